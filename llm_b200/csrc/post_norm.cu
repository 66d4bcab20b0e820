// Row-wise kernels of a layer whose parts are normed on both sides ("sandwich" norms), and the two
// element-wise steps its parts need.
//
// norm_add: the norm BEHIND a part, the residual sum and the norm in front of the next part in one
// launch, one block per token. y holds `terms` result rows per token (a part that leaves several
// partial results, e.g. one per chosen expert, has them added here in index order):
//     s = sum_k y[t * terms + k]         (32-bit, fixed order)
//     x[t] += s / sqrt(mean(s^2) + eps_post) * gain_post
//     h[t]  = x[t] / sqrt(mean(x[t]^2) + eps_next) * gain_next        (if gain_next; run dtype)
// Both sums of squares are reduced in one fixed order (thread order, lanes, warps), so a row's
// result does not depend on the batch.
//
// gelu: the tanh form, in place.  sigmoid_gate: out *= sigmoid(gate), rows with strides.
// fill: a constant into a 32-bit buffer.  add_terms: x[t] += the sum of a token's result rows.
#include "common.cuh"

using namespace llmb;

LLMB_DEFINE_LAST_ERROR(llmb_post_norm)

constexpr int THREADS = 256;

__device__ __forceinline__ float block_sum(float v, float* scratch) {
    v = warp_sum(v);
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) total += scratch[w];
    return total;
}

template <typename TOut>
__global__ void __launch_bounds__(THREADS)
norm_add_kernel(const float* __restrict__ y, int terms, const float* __restrict__ gain_post, float eps_post,
                float* __restrict__ x, const float* __restrict__ gain_next, float eps_next, TOut* __restrict__ h,
                int hidden) {
    extern __shared__ float row[];         // [hidden]
    __shared__ float scratch[THREADS / 32];
    griddep_launch();
    griddep_wait();
    size_t t = blockIdx.x;
    float sq = 0.f;
    for (int c = threadIdx.x; c < hidden; c += THREADS) {
        float s = 0.f;
        for (int k = 0; k < terms; ++k) s += y[(t * terms + k) * hidden + c];
        row[c] = s;
        sq = fmaf(s, s, sq);
    }
    float rstd = 1.0f / sqrtf(block_sum(sq, scratch) / (float)hidden + eps_post);
    sq = 0.f;
    for (int c = threadIdx.x; c < hidden; c += THREADS) {
        float v = x[t * hidden + c] + row[c] * rstd * gain_post[c];
        x[t * hidden + c] = v;
        row[c] = v;
        sq = fmaf(v, v, sq);
    }
    if (!gain_next) return;
    rstd = 1.0f / sqrtf(block_sum(sq, scratch) / (float)hidden + eps_next);
    for (int c = threadIdx.x; c < hidden; c += THREADS)
        h[t * hidden + c] = from_float<TOut>(row[c] * rstd * gain_next[c]);
}

// The same for rows of a multiple of four values up to 8,192, all arrays on 16-byte boundaries: NT threads (as many as the row
// has groups of four, up to 512) hold a row in registers, NV groups of four values each, and every load that does not wait
// for a sum is requested before the first one is needed (the gains even before the kernel in front has ended, where the
// caller says that they were complete before that one was launched: gains_bound). A row is one chain of load, sum, sum; the
// kernel above walks it element by element, with a chain of `terms` loads for each. Rows of 4,096, some of them with eight
// terms: 24 rows 14.7 -> 4.2 us, 2,077 rows 44.7 -> 37.0 us. Short rows, 4,096 of them with one term: of 64 values 8.3 us by the kernel above,
// 19.3 with 512 threads a row, 4.7 so; of 1,024 values 17.6, 20.6 and 9.3. The choice depends on the row's width and the
// addresses' alignment only, so that a row's sums have one order in every step.
constexpr int WIDE_THREADS = 512;      // most threads a row
template <typename TOut> __device__ __forceinline__ void store4(TOut* p, float4 v);
template <> __device__ __forceinline__ void store4<float>(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
template <> __device__ __forceinline__ void store4<__nv_bfloat16>(__nv_bfloat16* p, float4 v) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}
__device__ __forceinline__ float square4(float4 v, float sum) {
    return fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, fmaf(v.x, v.x, sum))));
}

template <typename TOut, int NV, int NT, bool BOUND>
__global__ void __launch_bounds__(NT)
norm_add_wide_kernel(const float* __restrict__ y, int terms, const float* __restrict__ gain_post, float eps_post,
                     float* __restrict__ x, const float* __restrict__ gain_next, float eps_next, TOut* __restrict__ h,
                     int hidden) {
    __shared__ float scratch[2][NT / 32];
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    griddep_launch();
    if constexpr (!BOUND) {
        griddep_wait();
        gain_post = behind_wait(gain_post);
        gain_next = behind_wait(gain_next);
    }
    float4 post[NV], next[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        int c = (threadIdx.x + i * NT) * 4;
        post[i] = next[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < hidden) {
            post[i] = *reinterpret_cast<const float4*>(gain_post + c);
            if (gain_next) next[i] = *reinterpret_cast<const float4*>(gain_next + c);
        }
    }
    if constexpr (BOUND) griddep_wait();
    y = behind_wait(y);
    size_t t = blockIdx.x;
    float* x_row = x + t * hidden;
    const float* y_rows = y + t * terms * hidden;
    float4 s[NV], v[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        int c = (threadIdx.x + i * NT) * 4;
        v[i] = s[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < hidden) {
            v[i] = *reinterpret_cast<const float4*>(x_row + c);
#pragma unroll 8
            for (int k = 0; k < terms; ++k) {
                float4 a = *reinterpret_cast<const float4*>(y_rows + (size_t)k * hidden + c);
                s[i].x += a.x; s[i].y += a.y; s[i].z += a.z; s[i].w += a.w;
            }
        }
    }
    auto total = [&](float sum, float* part) {
        sum = warp_sum(sum);
        if (lane == 0) part[warp] = sum;
        __syncthreads();
        float all = 0.f;
#pragma unroll
        for (int w = 0; w < NT / 32; ++w) all += part[w];
        return all;
    };
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) sq = square4(s[i], sq);
    float rstd = 1.0f / sqrtf(total(sq, scratch[0]) / (float)hidden + eps_post);
    sq = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        int c = (threadIdx.x + i * NT) * 4;
        v[i].x += s[i].x * rstd * post[i].x;
        v[i].y += s[i].y * rstd * post[i].y;
        v[i].z += s[i].z * rstd * post[i].z;
        v[i].w += s[i].w * rstd * post[i].w;
        if (c < hidden) *reinterpret_cast<float4*>(x_row + c) = v[i];
        sq = square4(v[i], sq);
    }
    if (!gain_next) return;
    rstd = 1.0f / sqrtf(total(sq, scratch[1]) / (float)hidden + eps_next);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        int c = (threadIdx.x + i * NT) * 4;
        if (c < hidden)
            store4(h + t * hidden + c, make_float4(v[i].x * rstd * next[i].x, v[i].y * rstd * next[i].y,
                                                   v[i].z * rstd * next[i].z, v[i].w * rstd * next[i].w));
    }
}

// The instance for a row: as many threads as it has groups of four, up to 512.
template <typename T, bool BOUND>
static auto norm_add_wide(int hidden, int* threads) {
    *threads = hidden <= 128 ? 32 : hidden <= 256 ? 64 : hidden <= 512 ? 128 : hidden <= 1024 ? 256 : WIDE_THREADS;
    return hidden <= 128    ? norm_add_wide_kernel<T, 1, 32, BOUND>
           : hidden <= 256  ? norm_add_wide_kernel<T, 1, 64, BOUND>
           : hidden <= 512  ? norm_add_wide_kernel<T, 1, 128, BOUND>
           : hidden <= 1024 ? norm_add_wide_kernel<T, 1, 256, BOUND>
           : hidden <= 2048 ? norm_add_wide_kernel<T, 1, 512, BOUND>
           : hidden <= 4096 ? norm_add_wide_kernel<T, 2, 512, BOUND>
                            : norm_add_wide_kernel<T, 4, 512, BOUND>;
}

// gains_bound: the gains were complete before the kernel in front of this call was launched.
LLMB_EXPORT int llmb_norm_add(const float* y, int terms, const float* gain_post, float eps_post, float* x,
                              const float* gain_next, float eps_next, void* h, int h_dtype, int n_rows, int hidden,
                              int gains_bound, cudaStream_t stream) {
    if (n_rows == 0) return LLMB_OK;
    LLMB_REQUIRE(hidden > 0 && terms > 0 && y && x && gain_post, "norm_add: bad sizes or a missing array");
    LLMB_REQUIRE(!gain_next || h, "norm_add: the next norm has no output");
    size_t smem = sizeof(float) * (size_t)hidden;
    LLMB_REQUIRE(smem <= 200 * 1024, "norm_add: a row of %d values does not fit in shared memory", hidden);
    size_t addresses = (size_t)y | (size_t)gain_post | (size_t)x | (size_t)gain_next | (size_t)h;
    bool wide = hidden % 4 == 0 && hidden <= 16 * WIDE_THREADS && addresses % 16 == 0;
#define LLMB_NORM_ADD(T)                                                                                           \
    do {                                                                                                           \
        if (wide) {                                                                                                \
            int threads = 0;                                                                                       \
            auto kernel = gains_bound ? norm_add_wide<T, true>(hidden, &threads) : norm_add_wide<T, false>(hidden, &threads); \
            LLMB_CUDA(llmb::launch(kernel, dim3(n_rows), dim3(threads), 0, stream, true, y, terms, gain_post,      \
                                   eps_post, x, gain_next, eps_next, (T*)h, hidden));                              \
            break;                                                                                                 \
        }                                                                                                          \
        if (smem > 48 * 1024)                                                                                      \
            LLMB_CUDA(cudaFuncSetAttribute(norm_add_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
        LLMB_CUDA(llmb::launch(norm_add_kernel<T>, dim3(n_rows), dim3(THREADS), smem, stream, true, y, terms,      \
                               gain_post, eps_post, x, gain_next, eps_next, (T*)h, hidden));                       \
    } while (0)
    if (h_dtype == LLMB_DTYPE_F32) LLMB_NORM_ADD(float);
    else if (h_dtype == LLMB_DTYPE_BF16) LLMB_NORM_ADD(__nv_bfloat16);
    else return fail(LLMB_ERR_ARGUMENT, "norm_add: unknown dtype %d", h_dtype);
#undef LLMB_NORM_ADD
    return check_launch("norm_add");
}
LLMB_PACKED(llmb_norm_add)

__device__ __forceinline__ float gelu_tanh(float z) {
    return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}

// 16 bytes a thread where the address allows it (`vectors`), the last elements one by one
template <typename T>
__global__ void gelu_kernel(T* __restrict__ a, long long n, int vectors) {
    griddep_launch();
    griddep_wait();
    constexpr int VEC = 16 / sizeof(T);
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (vectors) {
        long long first = i * VEC;
        if (first + VEC <= n) {
            uint4 raw = reinterpret_cast<const uint4*>(a)[i];
            T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
            for (int j = 0; j < VEC; ++j) e[j] = from_float<T>(gelu_tanh(to_float(e[j])));
            reinterpret_cast<uint4*>(a)[i] = raw;
        } else {
            for (long long k = first; k < n; ++k) a[k] = from_float<T>(gelu_tanh(to_float(a[k])));
        }
        return;
    }
    if (i < n) a[i] = from_float<T>(gelu_tanh(to_float(a[i])));
}

LLMB_EXPORT int llmb_gelu(void* a, int dtype, long long n, cudaStream_t stream) {
    if (n == 0) return LLMB_OK;
    LLMB_REQUIRE(n > 0 && a, "gelu: bad size");
    int vectors = ((size_t)a % 16) == 0;
    long long per_thread = vectors ? (dtype == LLMB_DTYPE_F32 ? 4 : 8) : 1;
    long long threads = (n + per_thread - 1) / per_thread;
    unsigned blocks = (unsigned)((threads + 255) / 256);
    if (dtype == LLMB_DTYPE_F32)
        LLMB_CUDA(llmb::launch(gelu_kernel<float>, dim3(blocks), dim3(256), 0, stream, true, (float*)a, n, vectors));
    else if (dtype == LLMB_DTYPE_BF16)
        LLMB_CUDA(llmb::launch(gelu_kernel<__nv_bfloat16>, dim3(blocks), dim3(256), 0, stream, true, (__nv_bfloat16*)a, n, vectors));
    else return fail(LLMB_ERR_ARGUMENT, "gelu: unknown dtype %d", dtype);
    return check_launch("gelu");
}
LLMB_PACKED(llmb_gelu)

// `vectors`: 16 bytes a thread (width, both strides and both addresses allow it)
template <typename T>
__global__ void sigmoid_gate_kernel(T* __restrict__ out, int out_stride, const T* __restrict__ gate, int gate_stride,
                                    int width, long long total, int vectors) {
    griddep_launch();
    griddep_wait();
    constexpr int VEC = 16 / sizeof(T);
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (vectors) {
        int per_row = width / VEC;
        if (i >= total / VEC) return;
        long long t = i / per_row;
        int c = (int)(i % per_row) * VEC;
        uint4 g_raw = *reinterpret_cast<const uint4*>(gate + t * gate_stride + c);
        uint4* dst = reinterpret_cast<uint4*>(out + t * out_stride + c);
        uint4 v_raw = *dst;
        const T* g = reinterpret_cast<const T*>(&g_raw);
        T* v = reinterpret_cast<T*>(&v_raw);
#pragma unroll
        for (int j = 0; j < VEC; ++j) v[j] = from_float<T>(to_float(v[j]) / (1.0f + expf(-to_float(g[j]))));
        *dst = v_raw;
        return;
    }
    if (i >= total) return;
    long long t = i / width;
    int c = (int)(i % width);
    float g = to_float(gate[t * gate_stride + c]);
    float v = to_float(out[t * out_stride + c]);
    out[t * out_stride + c] = from_float<T>(v / (1.0f + expf(-g)));
}

LLMB_EXPORT int llmb_sigmoid_gate(void* out, int out_stride, const void* gate, int gate_stride, int dtype, int n_rows,
                                  int width, cudaStream_t stream) {
    if (n_rows == 0) return LLMB_OK;
    LLMB_REQUIRE(width > 0 && out_stride >= width && gate_stride >= width, "sigmoid_gate: bad widths");
    long long total = (long long)n_rows * width;
    int vec = dtype == LLMB_DTYPE_F32 ? 4 : 8;
    int vectors = width % vec == 0 && out_stride % vec == 0 && gate_stride % vec == 0 && ((size_t)out % 16) == 0 &&
                  ((size_t)gate % 16) == 0;
    long long threads = vectors ? total / vec : total;
    unsigned blocks = (unsigned)((threads + 255) / 256);
    if (dtype == LLMB_DTYPE_F32)
        LLMB_CUDA(llmb::launch(sigmoid_gate_kernel<float>, dim3(blocks), dim3(256), 0, stream, true, (float*)out, out_stride,
                               (const float*)gate, gate_stride, width, total, vectors));
    else if (dtype == LLMB_DTYPE_BF16)
        LLMB_CUDA(llmb::launch(sigmoid_gate_kernel<__nv_bfloat16>, dim3(blocks), dim3(256), 0, stream, true,
                               (__nv_bfloat16*)out, out_stride, (const __nv_bfloat16*)gate, gate_stride, width, total, vectors));
    else return fail(LLMB_ERR_ARGUMENT, "sigmoid_gate: unknown dtype %d", dtype);
    return check_launch("sigmoid_gate");
}
LLMB_PACKED(llmb_sigmoid_gate)

__global__ void add_terms_kernel(float* __restrict__ x, const float* __restrict__ y, int terms, int hidden, long long total) {
    griddep_launch();
    griddep_wait();
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    long long t = i / hidden;
    int c = (int)(i % hidden);
    float s = 0.f;
    for (int k = 0; k < terms; ++k) s += y[(t * terms + k) * hidden + c];
    x[i] += s;
}

// x[t] += sum_k y[t * terms + k] (the terms in index order)
LLMB_EXPORT int llmb_add_terms(float* x, const float* y, int terms, int n_rows, int hidden, cudaStream_t stream) {
    if (n_rows == 0) return LLMB_OK;
    LLMB_REQUIRE(terms > 0 && hidden > 0 && x && y, "add_terms: bad sizes");
    long long total = (long long)n_rows * hidden;
    LLMB_CUDA(llmb::launch(add_terms_kernel, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, stream, true, x, y, terms,
                           hidden, total));
    return check_launch("add_terms");
}
LLMB_PACKED(llmb_add_terms)

__global__ void fill_kernel(float* __restrict__ x, long long n, float value) {
    griddep_launch();
    griddep_wait();
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = value;
}

LLMB_EXPORT int llmb_fill(float* x, long long n, float value, cudaStream_t stream) {
    if (n == 0) return LLMB_OK;
    LLMB_REQUIRE(n > 0 && x, "fill: bad size");
    LLMB_CUDA(llmb::launch(fill_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, true, x, n, value));
    return check_launch("fill");
}
LLMB_PACKED(llmb_fill)

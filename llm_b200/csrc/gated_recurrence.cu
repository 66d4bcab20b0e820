// A real-gated linear recurrence behind a short causal convolution (the recurrent block of De et al.,
// "Griffin"), on C channels cut into `blocks` equal parts of P = C / blocks:
//
//     u[t, c]  = conv_b[c] + sum_j conv_w[c, j] * x[t - (taps - 1) + j, c]       (x = 0 before a sequence's start)
//     r[t, c]  = sigmoid(gate_a_bias[c] + sum_i gate_a[b, c - bP, i] * u[t, bP + i])     b = c / P
//     i[t, c]  = sigmoid(gate_i_bias[c] + sum_i gate_i[b, c - bP, i] * u[t, bP + i])
//     a        = exp(rate[c] * r)                                                  (rate = -decay * softplus(lam) < 0)
//     S[t, c]  = a * S[t - 1, c] + sqrt(1 - a^2) * i * u                           (S = 0 before the start)
//     out[t, c] = out_scale * S[t, c] * gelu(y[t, c])                              (tanh form of gelu)
//
// x and y are the two branches' projections (with their biases) in the run's dtype. Everything between
// reading them and rounding `out` is 32-bit: the convolution's sum, both gates' matrix products (fixed order of
// summation per output; where the matrices are bfloat16 numbers on the tensor cores, of exact products), the decay, the
// recurrence and S.
//
// Per sequence the cache holds state[slot] = [taps, C] float32: rows 0 .. taps - 2 are the last taps - 1
// inputs x (oldest first), the last row is S. A slot's state is zeroed when the slot is taken, which is
// the convolution's zero padding and S = 0 for a sequence's first token: nothing treats it specially.
//
// Three kernels. conv: u of every token and channel, once, from x and the state (a value is `taps`
// multiply-adds; neighbouring threads take neighbouring channels). gates: tiles of 128 (long steps) or
// 32 tokens x 64 channels of one part over u; a thread owns 8 (or 2) tokens x 4 channels of both gates, so
// that 16 multiply-adds ride on every 16-byte read of shared memory; every output sums its inputs in
// rising order, whatever the tile; it writes a and the driving term sqrt(1 - a^2) i u of every token.
// scan: one thread per (sequence, channel) walks the sequence's tokens of this step in order, 16 at a
// time with the next 16 tokens' values already requested (the chain S <- a S + b is the only thing
// that has to wait), then brings the state up to date (S, and the last taps - 1 inputs). The first
// kernel only reads the state, the last writes it.
//
// Long steps (more than SCAN_SERIAL tokens) scan in three passes over chunks of 64 packed tokens, so that
// the tokens of a long prompt are not walked one after the other by a single thread: `scan_local` forms
// every chunk's product of a and its end value from a zero start (a sequence's first token of the step
// takes its S from the state there and stops the carry: a = 0), `scan_carry` walks the chunks in order
// (S at a chunk's start), `scan_apply` walks each chunk again from that start and writes the results, the
// new S of sequences that end in it and their convolution rows. The sums are the same up to rounding
// (a chunk's start value is formed from the chunk before it as a whole); short steps, and so every decode
// step, keep the token order exactly.
#include "tc.cuh"

using namespace llmb;
using namespace llmb::tc;

LLMB_DEFINE_LAST_ERROR(llmb_gated_recurrence)

constexpr int MAX_TAPS = 16;
constexpr int TN = 64;        // output channels of a tile
constexpr int KC = 16;        // input channels staged at a time
constexpr int SCAN_THREADS = 64;
constexpr int SCAN_AHEAD = 16;
constexpr int SCAN_SERIAL = 256;   // steps of up to this many tokens are scanned by one thread a (sequence, channel)
constexpr int SCAN_CHUNK = 64;
constexpr int SCAN_GROUP = 16;     // tokens whose values a thread of the chunked scan has in flight

// Where the convolution finds its inputs: the tokens of the same sequence in this step, and before the
// step's first token the rows of the state.
template <typename T>
struct ConvSource {
    const T* x;
    int x_stride;
    const float* state;       // [slots, taps, C]
    const float* conv_w;      // [C, taps]
    const float* conv_b;
    int taps, channels;

    __device__ __forceinline__ float value(int t, int seq_start, int slot, int c) const {
        float sum = conv_b[c];
        for (int j = 0; j < taps; ++j) {
            int src = t - (taps - 1) + j;
            float in = src >= seq_start ? to_float(x[(size_t)src * x_stride + c])
                                        : state[((size_t)slot * taps + (taps - 1 + src - seq_start)) * channels + c];
            sum = fmaf(conv_w[(size_t)c * taps + j], in, sum);
        }
        return sum;
    }
};

template <typename T>
__global__ void __launch_bounds__(256)
conv_kernel(ConvSource<T> source, const int* __restrict__ tok_seq, const int* __restrict__ cu_seqlens,
            const int* __restrict__ slot_ids, float* __restrict__ u) {
    griddep_launch();
    griddep_wait();
    int t = blockIdx.x;
    int c = blockIdx.y * 256 + threadIdx.x;
    if (c >= source.channels) return;
    int seq = tok_seq[t];
    u[(size_t)t * source.channels + c] = source.value(t, cu_seqlens[seq], slot_ids[seq], c);
}

// The same for four taps where four neighbouring channels lie on a boundary: a thread takes them for TOK tokens that follow
// each other, so that a row of x is read once for the TOK tokens, 8 or 16 bytes at a time, and the taps once. Every value is
// the sum of the kernel above in its order. Bound by memory: 2,500 tokens of 4,096 channels (61 MB) 68 -> 19 us.
// Shorter steps than four tokens an SM keep the kernel above: with one token a thread, 64 sequences took 9 us longer.
template <typename T> struct alignas(4 * sizeof(T)) Four { T v[4]; };
template <typename T, int TOK>
__global__ void __launch_bounds__(256)
conv_fours_kernel(ConvSource<T> source, const int* __restrict__ tok_seq, const int* __restrict__ cu_seqlens,
                  const int* __restrict__ slot_ids, float* __restrict__ u, int n_tokens) {
    griddep_launch();
    int c = (blockIdx.y * 256 + threadIdx.x) * 4;
    if (c >= source.channels) return;
    griddep_wait();
    const float* conv_w = behind_wait(source.conv_w);
    const float* conv_b = behind_wait(source.conv_b);
    float taps[4][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        float4 w = *reinterpret_cast<const float4*>(conv_w + (size_t)(c + e) * 4);
        taps[e][0] = w.x; taps[e][1] = w.y; taps[e][2] = w.z; taps[e][3] = w.w;
    }
    float4 bias4 = *reinterpret_cast<const float4*>(conv_b + c);
    const float bias[4] = {bias4.x, bias4.y, bias4.z, bias4.w};
    const T* x = behind_wait(source.x) + c;
    int t0 = blockIdx.x * TOK, count = min(TOK, n_tokens - t0);
    int seq0 = tok_seq[t0];
    bool plain = count == TOK && tok_seq[t0 + count - 1] == seq0 && t0 - cu_seqlens[seq0] >= 3;     // seven rows of one sequence
    if (!plain) {
        for (int k = 0; k < count; ++k) {
            int seq = tok_seq[t0 + k];
            float4 out;
            float* o = &out.x;
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = source.value(t0 + k, cu_seqlens[seq], slot_ids[seq], c + e);
            *reinterpret_cast<float4*>(u + (size_t)(t0 + k) * source.channels + c) = out;
        }
        return;
    }
    Four<T> in[TOK + 3];
#pragma unroll
    for (int r = 0; r < TOK + 3; ++r) in[r] = *reinterpret_cast<const Four<T>*>(x + (size_t)(t0 + r - 3) * source.x_stride);
#pragma unroll
    for (int k = 0; k < TOK; ++k) {
        float o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float sum = bias[e];
#pragma unroll
            for (int j = 0; j < 4; ++j) sum = fmaf(taps[e][j], to_float(in[k + j].v[e]), sum);
            o[e] = sum;
        }
        *reinterpret_cast<float4*>(u + (size_t)(t0 + k) * source.channels + c) = make_float4(o[0], o[1], o[2], o[3]);
    }
}

// TT: tokens a thread owns; a tile has 16 * TT tokens.
template <int TT>
__global__ void __launch_bounds__(256)
gates_kernel(const float* __restrict__ u, int channels, const float* __restrict__ gate_a, const float* __restrict__ gate_a_bias,
                  const float* __restrict__ gate_i, const float* __restrict__ gate_i_bias, int part,
                  const float* __restrict__ rate, float* __restrict__ decay, float* __restrict__ drive, int n_tokens) {
    constexpr int TM = 16 * TT;
    // rows padded by four floats: a thread's 16-byte reads stay aligned, and the stores (16 neighbouring threads
    // write one column) spread over the banks
    __shared__ __align__(16) float u_tile[KC][TM + 4];      // [input channel][token]
    __shared__ __align__(16) float a_tile[KC][TN + 4];      // [input channel][output channel]
    __shared__ __align__(16) float i_tile[KC][TN + 4];
    griddep_launch();
    griddep_wait();
    int tiles_per_part = (part + TN - 1) / TN;
    int b = blockIdx.y / tiles_per_part;                 // which part of the channels
    int o0 = (blockIdx.y % tiles_per_part) * TN;         // first output of the tile, inside the part
    int t0 = blockIdx.x * TM;
    // thread (ty, tx) owns tokens ty * TT .. + TT - 1 and outputs tx * 4 .. + 3
    int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float acc_a[TT][4], acc_i[TT][4];
#pragma unroll
    for (int m = 0; m < TT; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n) acc_a[m][n] = acc_i[m][n] = 0.f;
    const float* wa = gate_a + (size_t)b * part * part;
    const float* wi = gate_i + (size_t)b * part * part;
    // the next chunk's values are requested into registers before this chunk's products run
    constexpr int U_PER = TM * KC / 256, W_PER = TN * KC / 256;
    float u_next[U_PER], a_next[W_PER], i_next[W_PER];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int j = 0; j < U_PER; ++j) {
            int e = threadIdx.x + j * 256;
            int m = e / KC, k = e % KC;                 // neighbouring threads: neighbouring channels of one token
            int t = t0 + m;
            u_next[j] = (t < n_tokens && k0 + k < part) ? u[(size_t)t * channels + b * part + k0 + k] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < W_PER; ++j) {
            int e = threadIdx.x + j * 256;
            int n = e / KC, k = e % KC;                 // neighbouring threads: neighbouring inputs of one output row
            bool live = o0 + n < part && k0 + k < part;
            size_t at = (size_t)(o0 + n) * part + k0 + k;
            a_next[j] = live ? wa[at] : 0.f;
            i_next[j] = live ? wi[at] : 0.f;
        }
    };
    fetch(0);
    for (int k0 = 0; k0 < part; k0 += KC) {
#pragma unroll
        for (int j = 0; j < U_PER; ++j) {
            int e = threadIdx.x + j * 256;
            u_tile[e % KC][e / KC] = u_next[j];
        }
#pragma unroll
        for (int j = 0; j < W_PER; ++j) {
            int e = threadIdx.x + j * 256;
            a_tile[e % KC][e / KC] = a_next[j];
            i_tile[e % KC][e / KC] = i_next[j];
        }
        __syncthreads();
        if (k0 + KC < part) fetch(k0 + KC);
#pragma unroll
        for (int k = 0; k < KC; ++k) {
            float un[TT];
            if (TT % 4 == 0) {
#pragma unroll
                for (int m = 0; m < TT; m += 4) {
                    float4 v = *reinterpret_cast<const float4*>(&u_tile[k][ty * TT + m]);
                    un[m] = v.x; un[m + 1] = v.y; un[m + 2] = v.z; un[m + 3] = v.w;
                }
            } else {
#pragma unroll
                for (int m = 0; m < TT; ++m) un[m] = u_tile[k][ty * TT + m];
            }
            float4 av = *reinterpret_cast<const float4*>(&a_tile[k][tx * 4]);
            float4 iv = *reinterpret_cast<const float4*>(&i_tile[k][tx * 4]);
            float an[4] = {av.x, av.y, av.z, av.w}, in[4] = {iv.x, iv.y, iv.z, iv.w};
#pragma unroll
            for (int m = 0; m < TT; ++m)
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    acc_a[m][n] = fmaf(an[n], un[m], acc_a[m][n]);
                    acc_i[m][n] = fmaf(in[n], un[m], acc_i[m][n]);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int m = 0; m < TT; ++m) {
        int t = t0 + ty * TT + m;
        if (t >= n_tokens) continue;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            int o = o0 + tx * 4 + n;
            if (o >= part) continue;
            int c = b * part + o;
            float uc = u[(size_t)t * channels + c];
            float r = 1.0f / (1.0f + expf(-(acc_a[m][n] + gate_a_bias[c])));
            float g = 1.0f / (1.0f + expf(-(acc_i[m][n] + gate_i_bias[c])));
            float a = expf(rate[c] * r);
            decay[(size_t)t * channels + c] = a;
            drive[(size_t)t * channels + c] = sqrtf(1.0f - a * a) * g * uc;
        }
    }
}

// ------------------------------------------------------------------------- both gates on the tensor cores
// For matrices whose values are bfloat16 (a checkpoint in bfloat16, held in 32 bits): the 32-bit inputs u are taken apart
// instead of rounded. u = hi + mid + lo with bfloat16 parts of 8 bits each is exact (each part is cut off, not rounded),
// every product of a part with a weight is exact in 32 bits, and the tensor core adds them in 32 bits, hi's products in one
// accumulator and those of mid and lo, which are 2^-8 of them, in another, so that hi's chain stays short. One block an SM
// takes units of 128 tokens x 64 channels of one part, both gates of a channel side by side (128 columns):
//
// * warps 0-7: epilogue. A warp reads 32 tokens of 32 channels from tensor memory, forms the gates, a and the driving term.
// * warps 8-11: take u apart, a k-block of 64 at a time, into three swizzled tiles of 128 x 64.
// * warp 12: TMA loads of the weights' tile (128 rows x 64). Warp 13: the products. One elected lane of either issues.
//
// Bound by the epilogue's exponentials, divisions and roots (8 warps an SM) and the taking apart of u, which every group of 64
// channels of a part does again. 4,096 channels in 16 parts, the gates_kernel of the CUDA cores -> here, whole calls: 2,500 tokens
// 411 -> 202 us, 600 151 -> 76, 129 70 -> 41, 64 sequences of one token 27 -> 23, one token 22 -> 18; a is 5.0e-8 away from 64
// bits (5.3e-8 there), the driving term 9.3e-8 (9.9e-8).
//
// gate_rows: bfloat16 [2 C, P]: per group of 64 channels of a part, its 64 rows of gate_a, then its 64 rows of gate_i.
constexpr int TC_TOKENS = 128, TC_CHANNELS = 64, TC_K = 64, TC_STAGES = 3;
constexpr int TC_EPILOGUE_WARPS = 8, TC_SPLIT_WARPS = 4, TC_THREADS = (TC_EPILOGUE_WARPS + TC_SPLIT_WARPS + 2) * 32;
constexpr int TC_TILE = 128 * TC_K * 2;                           // bytes of a tile of bfloat16, of u's parts or of weights
constexpr int TC_STAGE = 4 * TC_TILE;                             // hi | mid | lo | weights
constexpr int TC_COLS = 2 * TC_CHANNELS;                          // columns of an accumulator: both gates

__device__ __forceinline__ uint32_t high_halves(float a, float b) {      // the top 16 bits of both, a's in the low half
    return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}
// v minus its top 16 bits: exact. An infinity has no rest.
__device__ __forceinline__ float below_high(float v) {
    float rest = v - __uint_as_float(__float_as_uint(v) & 0xffff0000u);
    return fabsf(v) == INFINITY ? 0.f : rest;
}

__global__ void __launch_bounds__(TC_THREADS, 1)
gates_tc_kernel(const __grid_constant__ CUtensorMap map_rows, const float* __restrict__ u, int channels,
                const float* __restrict__ gate_a_bias, const float* __restrict__ gate_i_bias, int part,
                const float* __restrict__ rate, float* __restrict__ decay, float* __restrict__ drive, int n_tokens,
                int n_units, int* status) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full_bar[TC_STAGES], empty_bar[TC_STAGES], acc_full_bar[2], acc_empty_bar[2];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;
    const int warp = warp_index(), lane = threadIdx.x & 31;
    griddep_launch();
    if (threadIdx.x == 0) {
        for (int s = 0; s < TC_STAGES; ++s) {
            mbar_init(smem_u32(&full_bar[s]), TC_SPLIT_WARPS + 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&acc_full_bar[b]), 1);
            mbar_init(smem_u32(&acc_empty_bar[b]), TC_EPILOGUE_WARPS);
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_shared();
    }
    if (warp == 13) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = tmem_slot;
    griddep_wait();
    u = behind_wait(u);
    gate_a_bias = behind_wait(gate_a_bias);
    gate_i_bias = behind_wait(gate_i_bias);
    rate = behind_wait(rate);

    // units: the groups of 64 channels run fastest, so that the blocks at work share the tokens' rows in L2
    const int groups = channels / TC_CHANNELS, kblocks = part / TC_K;
    if (warp < TC_EPILOGUE_WARPS) {
        const int quarter = warp & 3, half = warp >> 2;
        uint32_t n_done = 0;
        for (int unit = blockIdx.x; unit < n_units; unit += gridDim.x, ++n_done) {
            uint32_t buffer = n_done & 1, use = n_done >> 1;
            int t = unit / groups * TC_TOKENS + quarter * 32 + lane, c0 = unit % groups * TC_CHANNELS + half * 32;
            if (!mbar_wait_warp(smem_u32(&acc_full_bar[buffer]), use & 1, &abort_flag, status, 3)) break;
            tcgen05_fence_after();
            uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + buffer * (2 * TC_COLS) + half * 32;
#pragma unroll 1
            for (int c = 0; c < 32; c += 16) {
                uint32_t a_hi[16], a_low[16], i_hi[16], i_low[16];
                tmem_ld16(at + c, a_hi);
                tmem_ld16(at + TC_CHANNELS + c, i_hi);
                tmem_ld16(at + TC_COLS + c, a_low);
                tmem_ld16(at + TC_COLS + TC_CHANNELS + c, i_low);
                if (t < n_tokens) {
                    size_t place = (size_t)t * channels + c0 + c;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        float4 uc = *reinterpret_cast<const float4*>(u + place + 4 * q);
                        float4 ba = *reinterpret_cast<const float4*>(gate_a_bias + c0 + c + 4 * q);
                        float4 bi = *reinterpret_cast<const float4*>(gate_i_bias + c0 + c + 4 * q);
                        float4 r4 = *reinterpret_cast<const float4*>(rate + c0 + c + 4 * q);
                        const float us[4] = {uc.x, uc.y, uc.z, uc.w}, bas[4] = {ba.x, ba.y, ba.z, ba.w};
                        const float bis[4] = {bi.x, bi.y, bi.z, bi.w}, rates[4] = {r4.x, r4.y, r4.z, r4.w};
                        float as[4], ds[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            float sa = __uint_as_float(a_hi[4 * q + e]) + __uint_as_float(a_low[4 * q + e]);
                            float si = __uint_as_float(i_hi[4 * q + e]) + __uint_as_float(i_low[4 * q + e]);
                            float r = 1.0f / (1.0f + expf(-(sa + bas[e])));
                            float g = 1.0f / (1.0f + expf(-(si + bis[e])));
                            as[e] = expf(rates[e] * r);
                            ds[e] = sqrtf(1.0f - as[e] * as[e]) * g * us[e];
                        }
                        *reinterpret_cast<float4*>(decay + place + 4 * q) = make_float4(as[0], as[1], as[2], as[3]);
                        *reinterpret_cast<float4*>(drive + place + 4 * q) = make_float4(ds[0], ds[1], ds[2], ds[3]);
                    }
                }
                __syncwarp();
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty_bar[buffer]));
        }
    } else if (warp < TC_EPILOGUE_WARPS + TC_SPLIT_WARPS) {
        // a thread takes 8 neighbouring values of 8 tokens (16 apart) a k-block, requested before the stage is free
        const int thread = (int)threadIdx.x - TC_EPILOGUE_WARPS * 32, piece = thread & 7, row0 = thread >> 3;
        int s = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
            int t0 = unit / groups * TC_TOKENS, first = unit % groups * TC_CHANNELS / part * part;
            for (int kb = 0; kb < kblocks; ++kb) {
                float4 v[8][2];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    int t = t0 + row0 + 16 * i;
                    const float4* from = reinterpret_cast<const float4*>(u + (size_t)t * channels + first + kb * TC_K + piece * 8);
                    v[i][0] = t < n_tokens ? from[0] : make_float4(0.f, 0.f, 0.f, 0.f);
                    v[i][1] = t < n_tokens ? from[1] : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                ok = mbar_wait_warp(smem_u32(&empty_bar[s]), phase ^ 1, &abort_flag, status, 1);
                if (!ok) break;
                unsigned char* to = tiles + s * TC_STAGE;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    int row = row0 + 16 * i;
                    float x[8] = {v[i][0].x, v[i][0].y, v[i][0].z, v[i][0].w, v[i][1].x, v[i][1].y, v[i][1].z, v[i][1].w};
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        uint4 packed = make_uint4(high_halves(x[0], x[1]), high_halves(x[2], x[3]),
                                                  high_halves(x[4], x[5]), high_halves(x[6], x[7]));
                        // rows of 128 bytes, the 16-byte piece at place piece ^ (row % 8): the 128-byte swizzle
                        *reinterpret_cast<uint4*>(to + p * TC_TILE + row * 128 + ((piece ^ (row & 7)) << 4)) = packed;
                        if (p < 2) {
#pragma unroll
                            for (int e = 0; e < 8; ++e) x[e] = below_high(x[e]);
                        }
                    }
                }
                fence_async_shared();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&full_bar[s]));
                if (++s == TC_STAGES) { s = 0; phase ^= 1; }
            }
        }
    } else if (warp == 12) {
        int s = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
            int row = unit % groups * TC_COLS;
            for (int kb = 0; kb < kblocks; ++kb) {
                ok = mbar_wait_warp(smem_u32(&empty_bar[s]), phase ^ 1, &abort_flag, status, 1);
                if (!ok) break;
                if (elect_one()) {
                    mbar_expect_tx(smem_u32(&full_bar[s]), TC_TILE);
                    tma_load_2d(smem_u32(tiles + s * TC_STAGE + 3 * TC_TILE), &map_rows, smem_u32(&full_bar[s]), kb * TC_K, row);
                }
                __syncwarp();
                if (++s == TC_STAGES) { s = 0; phase ^= 1; }
            }
        }
    } else {
        // D 32-bit, A and B bfloat16, both K-major, M = 128, N = 128
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TC_COLS >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint64_t x0 = smem_desc(smem_u32(tiles));
        int s = 0;
        uint32_t phase = 0, n_done = 0;
        bool ok = true;
        for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x, ++n_done) {
            uint32_t buffer = n_done & 1, use = n_done >> 1, hi = tmem + buffer * (2 * TC_COLS), low = hi + TC_COLS;
            ok = mbar_wait_warp(smem_u32(&acc_empty_bar[buffer]), (use & 1) ^ 1, &abort_flag, status, 4);
            if (!ok) break;
            tcgen05_fence_after();
            for (int kb = 0; kb < kblocks; ++kb) {
                ok = mbar_wait_warp(smem_u32(&full_bar[s]), phase, &abort_flag, status, 2);
                if (!ok) break;
                tcgen05_fence_after();
                uint64_t x = x0 + (uint64_t)(s * (TC_STAGE >> 4)), w = x + (uint64_t)(3 * (TC_TILE >> 4));
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < TC_K / 16; ++k) {
                        tcgen05_mma(low, x + (uint64_t)(2 * (TC_TILE >> 4)) + 2 * k, w + 2 * k, idesc, kb > 0 || k > 0);
                        tcgen05_mma(low, x + (uint64_t)(TC_TILE >> 4) + 2 * k, w + 2 * k, idesc, 1u);
                        tcgen05_mma(hi, x + 2 * k, w + 2 * k, idesc, kb > 0 || k > 0);
                    }
                    tcgen05_commit(smem_u32(&empty_bar[s]));
                    if (kb + 1 == kblocks) tcgen05_commit(smem_u32(&acc_full_bar[buffer]));
                }
                __syncwarp();
                if (++s == TC_STAGES) { s = 0; phase ^= 1; }
            }
        }
    }
    __syncwarp();
    tcgen05_fence_before();
    __syncthreads();
    if (abort_flag) {
        // let copies that are still in flight land before shared memory is given up
        for (int i = 0; i < 100; ++i) __nanosleep(10000);
        __syncthreads();
    }
    if (warp == 13) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

template <typename T>
__device__ __forceinline__ void update_conv_rows(float* rows, int taps, int channels, const T* x, int x_stride,
                                                 int first, int count, int c);

__device__ __forceinline__ float gelu_tanh(float z) {
    return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}

template <typename T>
__global__ void __launch_bounds__(SCAN_THREADS)
scan_kernel(const T* __restrict__ y, int y_stride, const T* __restrict__ x, int x_stride,
            const float* __restrict__ decay, const float* __restrict__ drive, float* __restrict__ state, int taps,
            int channels, const int* __restrict__ cu_seqlens, const int* __restrict__ slot_ids, T* __restrict__ out,
            int out_stride, float out_scale) {
    griddep_launch();
    griddep_wait();
    int c = blockIdx.x * SCAN_THREADS + threadIdx.x;
    if (c >= channels) return;
    int seq = blockIdx.y;
    int first = cu_seqlens[seq], last = cu_seqlens[seq + 1];
    if (first >= last) return;
    float* rows = state + (size_t)slot_ids[seq] * taps * channels + c;      // row r at rows[r * channels]
    float s = rows[(size_t)(taps - 1) * channels];
    // the values of SCAN_AHEAD tokens are held while those of the next SCAN_AHEAD are on their way
    float a_now[SCAN_AHEAD], b_now[SCAN_AHEAD], y_now[SCAN_AHEAD], a_next[SCAN_AHEAD], b_next[SCAN_AHEAD], y_next[SCAN_AHEAD];
    auto fetch = [&](int t0, float (&a)[SCAN_AHEAD], float (&b)[SCAN_AHEAD], float (&g)[SCAN_AHEAD]) {
#pragma unroll
        for (int i = 0; i < SCAN_AHEAD; ++i) {
            int t = t0 + i;
            bool live = t < last;
            a[i] = live ? decay[(size_t)t * channels + c] : 0.f;
            b[i] = live ? drive[(size_t)t * channels + c] : 0.f;
            g[i] = live ? to_float(y[(size_t)t * y_stride + c]) : 0.f;
        }
    };
    fetch(first, a_now, b_now, y_now);
    for (int t0 = first; t0 < last; t0 += SCAN_AHEAD) {
        fetch(t0 + SCAN_AHEAD, a_next, b_next, y_next);
#pragma unroll
        for (int i = 0; i < SCAN_AHEAD; ++i) {
            int t = t0 + i;
            if (t < last) {
                s = fmaf(a_now[i], s, b_now[i]);
                out[(size_t)t * out_stride + c] = from_float<T>(s * gelu_tanh(y_now[i]) * out_scale);
            }
        }
#pragma unroll
        for (int i = 0; i < SCAN_AHEAD; ++i) { a_now[i] = a_next[i]; b_now[i] = b_next[i]; y_now[i] = y_next[i]; }
    }
    rows[(size_t)(taps - 1) * channels] = s;
    update_conv_rows(rows, taps, channels, x, x_stride, first, last - first, c);
}

// The last taps - 1 inputs of a sequence after a step of `count` tokens that began at packed token `first`: row r
// of the new state is input (count - (taps - 1) + r) of this step, or, where that lies before the step, row
// (r + count) of the old state. rows: the sequence's state at this channel, row r at rows[r * channels].
template <typename T>
__device__ __forceinline__ void update_conv_rows(float* rows, int taps, int channels, const T* x, int x_stride,
                                                 int first, int count, int c) {
    float old[MAX_TAPS];
#pragma unroll
    for (int r = 0; r < MAX_TAPS; ++r) old[r] = (r < taps - 1) ? rows[(size_t)r * channels] : 0.f;
#pragma unroll
    for (int r = 0; r < MAX_TAPS; ++r) {
        if (r >= taps - 1) break;
        int src = count - (taps - 1) + r;
        float v;
        if (src >= 0) {
            v = to_float(x[(size_t)(first + src) * x_stride + c]);
        } else {
            v = 0.f;
#pragma unroll
            for (int q = 0; q < MAX_TAPS; ++q) if (q == r + count) v = old[q];
        }
        rows[(size_t)r * channels] = v;
    }
}

// A step in which every sequence brings one token: token b is sequence b's, nothing is walked.
template <typename T>
__global__ void __launch_bounds__(256)
scan_single_kernel(const T* __restrict__ y, int y_stride, const T* __restrict__ x, int x_stride,
                   const float* __restrict__ decay, const float* __restrict__ drive, float* __restrict__ state, int taps,
                   int channels, const int* __restrict__ slot_ids, T* __restrict__ out, int out_stride, float out_scale) {
    griddep_launch();
    griddep_wait();
    int c = blockIdx.x * 256 + threadIdx.x;
    if (c >= channels) return;
    int t = blockIdx.y;
    float* rows = state + (size_t)slot_ids[t] * taps * channels + c;
    float s = fmaf(decay[(size_t)t * channels + c], rows[(size_t)(taps - 1) * channels], drive[(size_t)t * channels + c]);
    out[(size_t)t * out_stride + c] = from_float<T>(s * gelu_tanh(to_float(y[(size_t)t * y_stride + c])) * out_scale);
    rows[(size_t)(taps - 1) * channels] = s;
    for (int r = 0; r + 1 < taps - 1; ++r) rows[(size_t)r * channels] = rows[(size_t)(r + 1) * channels];
    if (taps > 1) rows[(size_t)(taps - 2) * channels] = to_float(x[(size_t)t * x_stride + c]);
}

// Which tokens of a chunk are a sequence's first ones (`edge` 0) or last ones (1): bit i for token t0 + i. Thread i looks at
// token i, so that no thread's walk waits for the look-up of a token's sequence. All threads of the block call it.
static_assert(SCAN_THREADS == SCAN_CHUNK && SCAN_CHUNK == 64, "a thread a token, two warps");
__device__ __forceinline__ unsigned long long chunk_edges(const int* tok_seq, const int* cu_seqlens, int t0, int t1, int edge) {
    __shared__ unsigned words[2];
    int t = t0 + threadIdx.x;
    bool hit = false;
    if (t < t1) {
        int seq = tok_seq[t];
        hit = edge ? t + 1 == cu_seqlens[seq + 1] : t == cu_seqlens[seq];
    }
    unsigned word = __ballot_sync(0xffffffffu, hit);
    if ((threadIdx.x & 31) == 0) words[threadIdx.x >> 5] = word;
    __syncthreads();
    return words[0] | ((unsigned long long)words[1] << 32);
}

// Pass 1 of the chunked scan. A sequence's first token of the step becomes a token without a carry: its
// driving term takes a * S(state) in, its a becomes 0 (both rewritten in place).
__global__ void __launch_bounds__(SCAN_THREADS)
scan_local_kernel(float* __restrict__ decay, float* __restrict__ drive, const float* __restrict__ state, int taps,
                  int channels, const int* __restrict__ tok_seq, const int* __restrict__ cu_seqlens,
                  const int* __restrict__ slot_ids, float* __restrict__ products, float* __restrict__ ends, int n_tokens) {
    griddep_launch();
    griddep_wait();
    int c = blockIdx.x * SCAN_THREADS + threadIdx.x;
    int chunk = blockIdx.y, t0 = chunk * SCAN_CHUNK, t1 = min(t0 + SCAN_CHUNK, n_tokens);
    unsigned long long firsts = chunk_edges(tok_seq, cu_seqlens, t0, t1, 0);
    if (c >= channels) return;
    float product = 1.f, s = 0.f;
    for (int g = t0; g < t1; g += SCAN_GROUP) {            // a group's values are requested before the first is used
        float a[SCAN_GROUP], b[SCAN_GROUP];
#pragma unroll
        for (int i = 0; i < SCAN_GROUP; ++i) {
            bool live = g + i < t1;
            a[i] = live ? decay[(size_t)(g + i) * channels + c] : 1.f;
            b[i] = live ? drive[(size_t)(g + i) * channels + c] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < SCAN_GROUP; ++i) {
            int t = g + i;
            if (t >= t1) break;
            if (firsts >> (t - t0) & 1) {
                b[i] = fmaf(a[i], state[((size_t)slot_ids[tok_seq[t]] * taps + taps - 1) * channels + c], b[i]);
                a[i] = 0.f;
                decay[(size_t)t * channels + c] = a[i];
                drive[(size_t)t * channels + c] = b[i];
            }
            product *= a[i];
            s = fmaf(a[i], s, b[i]);
        }
    }
    products[(size_t)chunk * channels + c] = product;
    ends[(size_t)chunk * channels + c] = s;
}

// Pass 2: ends[k] becomes S at the START of chunk k.
__global__ void __launch_bounds__(SCAN_THREADS)
scan_carry_kernel(const float* __restrict__ products, float* __restrict__ ends, int channels, int n_chunks) {
    griddep_launch();
    griddep_wait();
    int c = blockIdx.x * SCAN_THREADS + threadIdx.x;
    if (c >= channels) return;
    float s = 0.f;
    for (int k = 0; k < n_chunks; ++k) {
        float p = products[(size_t)k * channels + c], e = ends[(size_t)k * channels + c];
        ends[(size_t)k * channels + c] = s;
        s = fmaf(p, s, e);
    }
}

// Pass 3: each chunk again from its start value; results, and the state of the sequences that end here.
template <typename T>
__global__ void __launch_bounds__(SCAN_THREADS)
scan_apply_kernel(const T* __restrict__ y, int y_stride, const T* __restrict__ x, int x_stride,
                  const float* __restrict__ decay, const float* __restrict__ drive, const float* __restrict__ starts,
                  float* __restrict__ state, int taps, int channels, const int* __restrict__ tok_seq,
                  const int* __restrict__ cu_seqlens, const int* __restrict__ slot_ids, T* __restrict__ out,
                  int out_stride, float out_scale, int n_tokens) {
    griddep_launch();
    griddep_wait();
    int c = blockIdx.x * SCAN_THREADS + threadIdx.x;
    int chunk = blockIdx.y, t0 = chunk * SCAN_CHUNK, t1 = min(t0 + SCAN_CHUNK, n_tokens);
    unsigned long long lasts = chunk_edges(tok_seq, cu_seqlens, t0, t1, 1);
    if (c >= channels) return;
    float s = starts[(size_t)chunk * channels + c];
    for (int g = t0; g < t1; g += SCAN_GROUP) {
        float a[SCAN_GROUP], b[SCAN_GROUP];
        T z[SCAN_GROUP];
#pragma unroll
        for (int i = 0; i < SCAN_GROUP; ++i) {
            int t = min(g + i, t1 - 1);
            a[i] = decay[(size_t)t * channels + c];
            b[i] = drive[(size_t)t * channels + c];
            z[i] = y[(size_t)t * y_stride + c];
        }
#pragma unroll
        for (int i = 0; i < SCAN_GROUP; ++i) {
            int t = g + i;
            if (t >= t1) break;
            s = fmaf(a[i], s, b[i]);
            out[(size_t)t * out_stride + c] = from_float<T>(s * gelu_tanh(to_float(z[i])) * out_scale);
            if (lasts >> (t - t0) & 1) {                   // the sequence's last token of the step
                int seq = tok_seq[t], first = cu_seqlens[seq];
                float* rows = state + (size_t)slot_ids[seq] * taps * channels + c;
                rows[(size_t)(taps - 1) * channels] = s;
                update_conv_rows(rows, taps, channels, x, x_stride, first, t + 1 - first, c);
            }
        }
    }
}

// 0 if nothing went wrong since the last call of this function; else the code of the wait that ran out (1 operands, 2 products,
// 3 epilogue, 4 accumulator). Call after a synchronisation.
LLMB_EXPORT int llmb_gated_recurrence_status() {
    int* s = status_word();
    if (!s) return -1;
    int v = *s;
    *s = 0;
    return v;
}

// work [3, T, C] float32: u, a, the driving term. gate_rows: both gates' rows in bfloat16 as gates_tc_kernel reads them, or nullptr.
LLMB_EXPORT int llmb_gated_recurrence(const void* y, int y_stride, const void* x, int x_stride, int dtype,
                                      const float* conv_w, const float* conv_b, int taps, const float* gate_a,
                                      const float* gate_a_bias, const float* gate_i, const float* gate_i_bias,
                                      int blocks, const float* rate, float* state, const int* tok_seq,
                                      const int* cu_seqlens, const int* slot_ids, void* out, int out_stride,
                                      float out_scale, float* work, int n_tokens, int channels, int n_seqs,
                                      int single_tokens, const void* gate_rows, cudaStream_t stream) {
    if (n_tokens == 0) return LLMB_OK;
    LLMB_REQUIRE(taps >= 1 && taps <= MAX_TAPS, "gated_recurrence: %d taps (1 to %d are built)", taps, MAX_TAPS);
    LLMB_REQUIRE(channels > 0 && blocks > 0 && channels % blocks == 0 && n_seqs > 0,
                 "gated_recurrence: %d channels in %d parts", channels, blocks);
    int part = channels / blocks;
    bool long_step = n_tokens > 64;                 // the result is the same either way
    dim3 grid_gates(ceil_div(n_tokens, long_step ? 128 : 32), blocks * ceil_div(part, TN));
    dim3 grid_scan(ceil_div(channels, SCAN_THREADS), n_seqs);
    LLMB_REQUIRE(grid_gates.y <= 65535 && grid_scan.y <= 65535, "gated_recurrence: too many tiles or sequences");
    float* u = work;
    float* decay = work + (size_t)n_tokens * channels;
    float* drive = decay + (size_t)n_tokens * channels;
    auto gates = long_step ? gates_kernel<8> : gates_kernel<2>;
    // Up to 64 tokens a part of 64 or 128 channels is over on the CUDA cores before the tensor cores are set up: one token of 1,024
    // channels in 16 parts 10.1 us, 14.2 there, 64 tokens of 4,096 in 64 parts 14.8, 18.7; in 32 parts 18.7, 19.8. From 65
    // tokens (96 in 64 parts 28.7, 21.0) or parts of 192 channels (one token of 1,152 in 6 parts 17.7, 16.1) on it is not.
    bool on_tensor_cores = gate_rows && part % TC_CHANNELS == 0 && (long_step || part > 128) &&
                           (((size_t)gate_rows | (size_t)work | (size_t)gate_a_bias | (size_t)gate_i_bias | (size_t)rate) % 16) == 0;
    const size_t tc_smem = 1024 + (size_t)TC_STAGES * TC_STAGE;
    int n_units = ceil_div(n_tokens, TC_TOKENS) * (channels / TC_CHANNELS);
    static int n_sms = 0;
    CUtensorMap map_rows;
    int* status_dev = nullptr;
    if (on_tensor_cores) {
        if (n_sms == 0) {
            int device = 0, count = 0;
            LLMB_CUDA(cudaGetDevice(&device));
            LLMB_CUDA(cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device));
            LLMB_CUDA(cudaFuncSetAttribute(gates_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc_smem));
            n_sms = count;
        }
        int code = make_map_2d(&map_rows, gate_rows, 2LL * channels, part, part, TC_K, 128);
        if (code) return code;
        if (int* word = status_word()) cudaHostGetDevicePointer((void**)&status_dev, word, 0);
    }
#define LLMB_RECURRENCE(T)                                                                                          \
    do {                                                                                                            \
        ConvSource<T> source{(const T*)x, x_stride, state, conv_w, conv_b, taps, channels};                         \
        if (n_tokens >= 4 * 148 && taps == 4 && channels % 4 == 0 && x_stride % 4 == 0 &&                           \
            ((size_t)x % (4 * sizeof(T))) == 0 && (((size_t)conv_w | (size_t)conv_b | (size_t)work) % 16) == 0) {   \
            LLMB_CUDA(llmb::launch(conv_fours_kernel<T, 4>, dim3(ceil_div(n_tokens, 4), ceil_div(channels, 1024)),  \
                                   dim3(256), 0, stream, true, source, tok_seq, cu_seqlens, slot_ids, u, n_tokens)); \
        } else                                                                                                      \
            LLMB_CUDA(llmb::launch(conv_kernel<T>, dim3(n_tokens, ceil_div(channels, 256)), dim3(256), 0, stream,   \
                                   true, source, tok_seq, cu_seqlens, slot_ids, u));                                \
        if (on_tensor_cores)                                                                                        \
            LLMB_CUDA(llmb::launch(gates_tc_kernel, dim3(n_units < n_sms ? n_units : n_sms), dim3(TC_THREADS), tc_smem, stream, \
                                   true, map_rows, (const float*)u, channels, gate_a_bias, gate_i_bias, part, rate, \
                                   decay, drive, n_tokens, n_units, status_dev));                                   \
        else                                                                                                        \
        /* launched plainly, so that its blocks find the SMs empty: put down while the convolution drains, several of them \
           share an SM (64 sequences of one token, 4,096 channels: 49 us in all dependent, 26 plainly) */          \
        LLMB_CUDA(llmb::launch(gates, grid_gates, dim3(256), 0, stream, false, (const float*)u, channels, gate_a,    \
                               gate_a_bias, gate_i, gate_i_bias, part, rate, decay, drive, n_tokens));              \
        if (n_tokens == n_seqs && single_tokens) {                                                                  \
            LLMB_CUDA(llmb::launch(scan_single_kernel<T>, dim3(ceil_div(channels, 256), n_seqs), dim3(256), 0, stream, \
                                   true, (const T*)y, y_stride, (const T*)x, x_stride, (const float*)decay,         \
                                   (const float*)drive, state, taps, channels, slot_ids, (T*)out, out_stride,       \
                                   out_scale));                                                                     \
        } else if (n_tokens <= SCAN_SERIAL) {                                                                       \
            LLMB_CUDA(llmb::launch(scan_kernel<T>, grid_scan, dim3(SCAN_THREADS), 0, stream, true, (const T*)y,     \
                                   y_stride, (const T*)x, x_stride, (const float*)decay, (const float*)drive,       \
                                   state, taps, channels, cu_seqlens, slot_ids, (T*)out, out_stride, out_scale));   \
        } else {                                                                                                    \
            /* u is no longer needed: the chunks' products and end values take its place */                         \
            int n_chunks = ceil_div(n_tokens, SCAN_CHUNK);                                                          \
            float* products = u;                                                                                    \
            float* ends = u + (size_t)n_chunks * channels;                                                          \
            dim3 grid_chunks(ceil_div(channels, SCAN_THREADS), n_chunks);                                           \
            LLMB_REQUIRE(n_chunks <= 65535, "gated_recurrence: too many tokens in one call");                       \
            LLMB_CUDA(llmb::launch(scan_local_kernel, grid_chunks, dim3(SCAN_THREADS), 0, stream, true, decay,      \
                                   drive, (const float*)state, taps, channels, tok_seq, cu_seqlens, slot_ids,       \
                                   products, ends, n_tokens));                                                      \
            LLMB_CUDA(llmb::launch(scan_carry_kernel, dim3(ceil_div(channels, SCAN_THREADS)), dim3(SCAN_THREADS), 0, \
                                   stream, true, (const float*)products, ends, channels, n_chunks));                \
            LLMB_CUDA(llmb::launch(scan_apply_kernel<T>, grid_chunks, dim3(SCAN_THREADS), 0, stream, true,          \
                                   (const T*)y, y_stride, (const T*)x, x_stride, (const float*)decay,               \
                                   (const float*)drive, (const float*)ends, state, taps, channels, tok_seq,         \
                                   cu_seqlens, slot_ids, (T*)out, out_stride, out_scale, n_tokens));                \
        }                                                                                                           \
    } while (0)
    if (dtype == LLMB_DTYPE_F32) LLMB_RECURRENCE(float);
    else if (dtype == LLMB_DTYPE_BF16) LLMB_RECURRENCE(__nv_bfloat16);
    else return fail(LLMB_ERR_ARGUMENT, "gated_recurrence: unknown dtype %d", dtype);
#undef LLMB_RECURRENCE
    return check_launch("gated_recurrence");
}

LLMB_PACKED(llmb_gated_recurrence)

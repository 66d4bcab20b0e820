// Prefill of the differential attention (diff_attention.cu says what it computes) on the fifth-generation
// tensor cores.
//
// One block serves 128 queries of one head, both maps, and walks the visible keys page by page (64 keys). A map
// is a softmax attention of its own over its half of the key rows and the same values, so a block holds two
// pipelines that share the keys' and values' tiles:
//
// * warp 8: TMA for the queries (once) and the key pages; warp 10: TMA for the value pages; one elected lane of each
//   issues. 64 x 64 boxes, STAGES pages of each in flight.
// * warp 9, one elected lane: issues the products. Per map S[128, 64 keys] = Q K^T into one of two score buffers, and
//   O[128, DV] += P V with P read from tensor memory (over the buffer's first 32 columns) and V an MN-major
//   operand. The scores of page n + 2 of a map are issued right behind P V of page n, as in attention_prefill_tc.
// * warps 0-3 are the softmax of map 1, warps 4-7 that of map 2; a thread owns a query row. While one map's
//   products run, the other map's exponentials do: what two blocks an SM do for attention_prefill_tc. O is
//   rescaled in place by a warp one of whose rows has a new maximum.
// * tensor memory, all 512 columns: 2 maps x 2 score buffers x 64, 2 x DV for O. The two warps that own the same
//   lanes halve the columns of O1 and O2 at the end: o = a1 - lambda a2, the head's norm, the scale.
//
// Bound by the exponentials (2 x 64 a query and page at 16 a cycle and SM), with 4 + 4 products a map and page
// beside them. 3,001 tokens, 32 heads of 2 x 64 over 8, values of 128, on a B200: 440 us by tiles of 64 queries on
// mma.sync, 222 us here (1.2 us a page and block; 1,024 cycles of exponentials are 0.55), the same error.
// Which call comes here: every prefill of the map and value sizes below; the other sizes of LLMB_DIFF_SHAPES have
// rows that no 128-byte swizzle covers (48) or values narrower than one (32), and stay on mma.sync.
//
// All waits are bounded by a clock limit and report through the status word of this library.
#include "tc.cuh"
#include "page_walk.cuh"

using namespace llmb;
using namespace llmb::tc;

LLMB_DEFINE_LAST_ERROR(llmb_diff_attention_tc)

#define LLMB_DIFF_TC_SHAPES(X) X(32, 64) X(64, 64) X(64, 128) X(128, 128)

namespace {

constexpr int BQ = 128;                           // queries a block = lanes of tensor memory
constexpr int SOFTMAX_THREADS = 256;
constexpr int THREADS = SOFTMAX_THREADS + 96;
constexpr int Q_PIECE = BQ * 64 * 2;              // 128 query rows, 64 columns of the head's two maps
constexpr int KV_PIECE = LLMB_PAGE * 64 * 2;      // one page, 64 columns
constexpr uint32_t O_COL = 256, TMEM_COLS = 512;  // scores: (map * 2 + buffer) * 64

__device__ __forceinline__ void softmax_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(SOFTMAX_THREADS) : "memory"); }

template <int DK, int DV>
struct Tiles {
    static constexpr int K_PIECES = 2 * DK / 64, V_PIECES = DV / 64;
    static constexpr int Q_BYTES = K_PIECES * Q_PIECE, K_BYTES = K_PIECES * KV_PIECE, V_BYTES = V_PIECES * KV_PIECE;
    static constexpr int STAGES = DK > 64 ? 2 : 4;
    static constexpr int BARS = 1 + 4 * STAGES + 4 + 4 + 2;
    static constexpr size_t SMEM = 1024 + (size_t)Q_BYTES + (size_t)STAGES * (K_BYTES + V_BYTES) + BARS * 8 + 16 + 4 * BQ * 4;
};

template <int DK, int DV>
__global__ void __launch_bounds__(THREADS, 1)
diff_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, const int* __restrict__ block_table, int table_stride,
                         int ring_pages, const int* __restrict__ cu_seqlens, const int* __restrict__ seq_lens,
                         const int* __restrict__ seq_order, __nv_bfloat16* __restrict__ out, int out_stride, int n_heads,
                         int n_kv_heads, float scale_log2, int window, int keep_first, float lambda, float eps,
                         float out_scale, int head_norm, int* status) {
    using T = Tiles<DK, DV>;
    constexpr int STAGES = T::STAGES;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* q_tile = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* k_tile = q_tile + T::Q_BYTES;
    unsigned char* v_tile = k_tile + STAGES * T::K_BYTES;
    uint64_t* q_full = reinterpret_cast<uint64_t*>(v_tile + STAGES * T::V_BYTES);
    uint64_t* k_full = q_full + 1;
    uint64_t* k_empty = k_full + STAGES;
    uint64_t* v_full = k_empty + STAGES;
    uint64_t* v_empty = v_full + STAGES;
    uint64_t* s_full = v_empty + STAGES;          // [map * 2 + buffer] the scores are complete
    uint64_t* p_full = s_full + 4;                // [map * 2 + buffer] the probabilities are written and O has been rescaled
    uint64_t* o_full = p_full + 4;                // [map] a page's P V has been added to O
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* exchange = reinterpret_cast<float*>(tmem_slot + 4);        // [2][BQ] reciprocal sums, then [2][BQ] squares

    griddep_wait();
    int seq = seq_order ? seq_order[blockIdx.z] : (int)blockIdx.z, head = blockIdx.x;
    int first_token = cu_seqlens[seq];
    int n_new = cu_seqlens[seq + 1] - first_token;
    int n_tiles = (n_new + BQ - 1) / BQ;
    if ((int)blockIdx.y >= n_tiles) return;                  // uniform for the block: nothing is allocated yet
    int tile = n_tiles - 1 - blockIdx.y;                     // the heaviest tile of every head first
    int start = seq_lens[seq] - n_new;
    int kv_head = head / (n_heads / n_kv_heads);
    const int warp = warp_index(), lane = threadIdx.x & 31;
    PageWalk walk = page_walk(start + tile * BQ, start + min(tile * BQ + BQ - 1, n_new - 1), window, keep_first);
    const int* pages = block_table + (size_t)seq * table_stride;

    if (threadIdx.x == 0) {
        for (int i = 0; i < T::BARS; ++i) mbar_init(smem_u32(&q_full[i]), (&q_full[i] >= p_full && &q_full[i] < o_full) ? BQ : 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    uint32_t tmem_base = *tmem_slot;
    griddep_launch();            // behind the allocation: no block of the next kernel can hold this one's tensor memory

    if (warp == 8 || warp == 10) {
        const bool keys = warp == 8;
        if (keys && elect_one()) {
            uint32_t bar = smem_u32(q_full);
            mbar_expect_tx(bar, T::Q_BYTES);
            for (int h = 0; h < T::K_PIECES; ++h)
                tma_load_2d(smem_u32(q_tile + h * Q_PIECE), &map_q, bar, head * 2 * DK + h * 64, first_token + tile * BQ);
        }
        __syncwarp();
        const CUtensorMap* map = keys ? &map_k : &map_v;
        unsigned char* tiles = keys ? k_tile : v_tile;
        uint64_t* full = keys ? k_full : v_full;
        uint64_t* empty = keys ? k_empty : v_empty;
        const int bytes = keys ? T::K_BYTES : T::V_BYTES, pieces = keys ? T::K_PIECES : T::V_PIECES;
        for (int n = 0; n < walk.count; ++n) {
            int stage = n % STAGES, turn = n / STAGES;
            int row = (pages[walk.logical(n) % ring_pages] * n_kv_heads + kv_head) * LLMB_PAGE;
            if (turn > 0 && !mbar_wait_warp(smem_u32(&empty[stage]), (turn - 1) & 1, abort_flag, status, keys ? 1 : 2)) break;
            if (elect_one()) {
                uint32_t bar = smem_u32(&full[stage]);
                mbar_expect_tx(bar, bytes);
                for (int h = 0; h < pieces; ++h)
                    tma_load_2d(smem_u32(tiles + stage * bytes + h * KV_PIECE), map, bar, h * 64, row);
            }
            __syncwarp();
        }
    } else if (warp == 9) {
        // D 32-bit, A and B bfloat16, M = 128; S has N = 64 keys, O has N = DV with B MN-major
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BQ >> 4) << 24);
        constexpr uint32_t idesc_s = idesc | ((uint32_t)(LLMB_PAGE >> 3) << 17);
        constexpr uint32_t idesc_o = idesc | (1u << 16) | ((uint32_t)(DV >> 3) << 17);
        const uint64_t q_desc = smem_desc(smem_u32(q_tile)), k_desc = smem_desc(smem_u32(k_tile));
        const uint64_t v_desc = smem_desc_mn(smem_u32(v_tile), KV_PIECE);
        // scores of page n, map m (map 2's columns follow map 1's in a row of the tiles); a page's keys are free behind map 2
        auto issue_scores = [&](int n, int m) -> bool {
            int stage = n % STAGES;
            if (m == 0) {
                if (!mbar_wait_warp(smem_u32(&k_full[stage]), (n / STAGES) & 1, abort_flag, status, 3)) return false;
                tcgen05_fence_after();
            }
            uint64_t k_at = k_desc + (uint64_t)((stage * T::K_BYTES) >> 4);
            if (elect_one()) {
#pragma unroll
                for (int j = 0; j < DK / 16; ++j) {
                    int c = m * DK + j * 16;
                    tcgen05_mma(tmem_base + (m * 2 + (n & 1)) * LLMB_PAGE, q_desc + (uint64_t)(((c >> 6) * Q_PIECE + (c & 63) * 2) >> 4),
                                k_at + (uint64_t)(((c >> 6) * KV_PIECE + (c & 63) * 2) >> 4), idesc_s, j > 0 ? 1u : 0u);
                }
                tcgen05_commit(smem_u32(&s_full[m * 2 + (n & 1)]));
                if (m == 1) tcgen05_commit(smem_u32(&k_empty[stage]));
            }
            __syncwarp();
            return true;
        };
        bool ok = mbar_wait_warp(smem_u32(q_full), 0, abort_flag, status, 4);
        for (int n = 0; n < 2 && n < walk.count && ok; ++n) ok = issue_scores(n, 0) && issue_scores(n, 1);
        for (int n = 0; n < walk.count && ok; ++n) {
            int stage = n % STAGES;
            uint64_t v_at = v_desc + (uint64_t)((stage * T::V_BYTES) >> 4);
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                ok = mbar_wait_warp(smem_u32(&p_full[m * 2 + (n & 1)]), (n >> 1) & 1, abort_flag, status, 5);
                if (ok && m == 0) ok = mbar_wait_warp(smem_u32(&v_full[stage]), (n / STAGES) & 1, abort_flag, status, 6);
                if (!ok) break;
                tcgen05_fence_after();
                if (elect_one()) {
#pragma unroll
                    for (int j = 0; j < LLMB_PAGE / 16; ++j)      // 16 keys: 8 columns of P, 2048 bytes of value rows
                        tcgen05_mma_ts(tmem_base + O_COL + m * DV, tmem_base + (m * 2 + (n & 1)) * LLMB_PAGE + j * 8,
                                       v_at + (uint64_t)((j * 2048) >> 4), idesc_o, (n > 0 || j > 0) ? 1u : 0u);
                    tcgen05_commit(smem_u32(&o_full[m]));
                    if (m == 1) tcgen05_commit(smem_u32(&v_empty[stage]));
                }
                __syncwarp();
                if (n + 2 < walk.count) ok = issue_scores(n + 2, m);
                if (!ok) break;
            }
        }
    } else {
        int map = warp >> 2, quarter = warp & 3;
        int row = quarter * 32 + lane;                       // query row of the tile = lane of tensor memory
        int q_index = tile * BQ + row;                       // among the sequence's new tokens
        int pos = start + q_index;
        int warp_pos = start + tile * BQ + quarter * 32;     // the warp's first position
        uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
        uint32_t o_addr = lane_addr + O_COL + map * DV;
        float reference = -INFINITY, run_sum = 0.f;
        bool ok = true;
        for (int n = 0; n < walk.count && ok; ++n) {
            int b = map * 2 + (n & 1);
            ok = mbar_wait(smem_u32(&s_full[b]), (n >> 1) & 1, abort_flag, status, 7);
            if (!ok) break;
            __syncwarp();
            tcgen05_fence_after();
            int key0 = walk.logical(n) * LLMB_PAGE;
            uint32_t s_addr = lane_addr + b * LLMB_PAGE;
            uint32_t ra[32], rb[32];
            tmem_ld32_start(s_addr, ra);
            tmem_ld32_start(s_addr + 32, rb);
            tmem_ld32_wait(ra);
            tmem_ld32_wait(rb);
            // some key of the page may be hidden from some row of the warp: above the diagonal, or outside a window
            bool masked = key0 + LLMB_PAGE - 1 > warp_pos || (window > 0 && key0 < warp_pos + 31 - window + 1);
            if (masked) {
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    if (!key_visible(key0 + j, pos, window, keep_first)) ra[j] = __float_as_uint(-INFINITY);
                    if (!key_visible(key0 + 32 + j, pos, window, keep_first)) rb[j] = __float_as_uint(-INFINITY);
                }
            }
            float top = -INFINITY;
#pragma unroll
            for (int j = 0; j < 32; ++j) top = max3(top, __uint_as_float(ra[j]), __uint_as_float(rb[j]));
            // The exponent's reference is the row's maximum itself, as in the mma.sync kernel: the largest weights then lie just
            // below 1, where bfloat16 is finest. (A reference that lags by up to 2^8 saves most of the rescaling, 198 us
            // for 222, and is 4 % further from 64 bits.) A row that has seen no key yet keeps -inf: weights 0.
            float raised = fmaxf(reference, top * scale_log2);
            float alpha = raised > reference ? fast_exp2(reference - raised) : 1.f;
            float shift = raised == -INFINITY ? 0.f : raised;
            reference = raised;
            float add = 0.f;
            uint32_t packed[16];
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                float p0 = fast_exp2(fmaf(__uint_as_float(ra[j]), scale_log2, -shift));
                float p1 = fast_exp2(fmaf(__uint_as_float(ra[j + 1]), scale_log2, -shift));
                add += p0 + p1;
                packed[j >> 1] = pack2(p0, p1);
            }
            tmem_st16(s_addr, packed);
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                float p0 = fast_exp2(fmaf(__uint_as_float(rb[j]), scale_log2, -shift));
                float p1 = fast_exp2(fmaf(__uint_as_float(rb[j + 1]), scale_log2, -shift));
                add += p0 + p1;
                packed[j >> 1] = pack2(p0, p1);
            }
            tmem_st16(s_addr + 16, packed);
            run_sum = run_sum * alpha + add;
            if (n > 0) {                                     // the product before this one is complete: O may be rescaled
                ok = mbar_wait(smem_u32(&o_full[map]), (n - 1) & 1, abort_flag, status, 8);
                if (!ok) break;
                __syncwarp();
                tcgen05_fence_after();
                if (__any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll 1
                    for (int c = 0; c < DV; c += 16) {
                        uint32_t r[16];
                        tmem_ld16(o_addr + c, r);
#pragma unroll
                        for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * alpha);
                        tmem_st16(o_addr + c, r);
                    }
                }
            }
            tmem_st_wait();
            tcgen05_fence_before();
            mbar_arrive(smem_u32(&p_full[b]));
        }
        exchange[map * BQ + row] = 1.0f / run_sum;            // every stored row sees at least its own key
        for (int m = 0; m < 2 && ok; ++m) ok = mbar_wait(smem_u32(&o_full[m]), (walk.count - 1) & 1, abort_flag, status, 9);
        softmax_barrier();                                   // (reached on every path: a failed wait does not leave the other warps here)
        __syncwarp();
        tcgen05_fence_after();
        // the two warps of these lanes take half of the columns each
        constexpr int HALF = DV / 2;
        float inv1 = exchange[row], inv2 = exchange[BQ + row], square = 0.f;
        float o[HALF];
#pragma unroll
        for (int c = 0; c < HALF; c += 32) {
            uint32_t r1[32], r2[32];
            tmem_ld32_start(lane_addr + O_COL + map * HALF + c, r1);
            tmem_ld32_start(lane_addr + O_COL + DV + map * HALF + c, r2);
            tmem_ld32_wait(r1);
            tmem_ld32_wait(r2);
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                float v = __uint_as_float(r1[j]) * inv1 - lambda * (__uint_as_float(r2[j]) * inv2);
                square = fmaf(v, v, square);
                o[c + j] = v;
            }
        }
        float factor = out_scale;
        if (head_norm) {
            exchange[(2 + map) * BQ + row] = square;
            softmax_barrier();
            factor *= 1.0f / sqrtf((exchange[2 * BQ + row] + exchange[3 * BQ + row]) / (float)DV + eps);
        }
        if (ok && q_index < n_new) {
            __nv_bfloat16* to = out + (size_t)(first_token + q_index) * out_stride + (size_t)head * DV + map * HALF;
#pragma unroll
            for (int d = 0; d < HALF; d += 8) {
                uint4 line;
                line.x = pack2(o[d] * factor, o[d + 1] * factor);
                line.y = pack2(o[d + 2] * factor, o[d + 3] * factor);
                line.z = pack2(o[d + 4] * factor, o[d + 5] * factor);
                line.w = pack2(o[d + 6] * factor, o[d + 7] * factor);
                *reinterpret_cast<uint4*>(to + d) = line;
            }
        }
    }

    tcgen05_fence_before();
    __syncthreads();
    if (*abort_flag) {                                       // copies in flight land before the block's memory is given back
        for (int i = 0; i < 100; ++i) __nanosleep(10000);
        __syncthreads();
    }
    if (warp == 9) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

template <int DK, int DV>
int launch_tc(const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v, dim3 grid, const int* block_table,
              int table_stride, int ring_pages, const int* cu_seqlens, const int* seq_lens, const int* seq_order, void* out,
              int out_stride, int n_heads, int n_kv_heads, float scale, int window, int keep_first, float lambda, float eps,
              float out_scale, int head_norm, cudaStream_t stream) {
    constexpr size_t smem = Tiles<DK, DV>::SMEM;
    static bool configured = false;
    if (!configured) {
        LLMB_CUDA(cudaFuncSetAttribute(diff_attention_tc_kernel<DK, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured = true;
    }
    int* status = status_word();
    int* status_dev = nullptr;
    if (status) cudaHostGetDevicePointer((void**)&status_dev, status, 0);
    LLMB_CUDA(llmb::launch(diff_attention_tc_kernel<DK, DV>, grid, dim3(THREADS), smem, stream, true, map_q, map_k, map_v, block_table,
                           table_stride, ring_pages, cu_seqlens, seq_lens, seq_order, (__nv_bfloat16*)out, out_stride, n_heads,
                           n_kv_heads, scale * 1.4426950408889634f, window, keep_first, lambda, eps, out_scale, head_norm, status_dev));
    return check_launch("diff_attention_tc");
}

}  // namespace

LLMB_EXPORT int llmb_diff_attention_tc_status() {
    int* s = status_word();
    if (!s) return -1;
    int v = *s;
    *s = 0;
    return v;
}

// As llmb_diff_attention_prefill, with the number of token rows of q and of pages of the cache (the tensor maps' bounds) and
// the order in which sequences start (or null). A positive scale.
LLMB_EXPORT int llmb_diff_attention_tc(const void* q, int q_stride, int n_tokens, const void* k_cache, const void* v_cache,
                                       int n_cache_pages, const int* block_table, int table_stride, int ring_pages,
                                       const int* cu_seqlens, const int* seq_lens, const int* seq_order, void* out, int out_stride,
                                       int n_seqs, int max_new, int n_heads, int n_kv_heads, int dim, int vdim, float scale,
                                       int window, int keep_first, float lambda, float eps, float out_scale, int head_norm,
                                       cudaStream_t stream) {
    if (n_seqs == 0 || max_new == 0 || n_tokens == 0) return LLMB_OK;
    LLMB_REQUIRE(n_heads > 0 && n_kv_heads > 0 && n_heads % n_kv_heads == 0, "diff_attention_tc: %d heads are no multiple of %d kv heads",
                 n_heads, n_kv_heads);
    LLMB_REQUIRE(n_seqs <= 65535 && max_new / BQ < 65535 && ring_pages > 0 && n_cache_pages > 0 && window >= 0 && keep_first >= 0 &&
                 scale > 0.f, "diff_attention_tc: bad sizes");
    LLMB_REQUIRE(q_stride % 8 == 0 && out_stride % 8 == 0 && (reinterpret_cast<uintptr_t>(q) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(out) & 15) == 0 && (reinterpret_cast<uintptr_t>(k_cache) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(v_cache) & 15) == 0,
                 "diff_attention_tc: operands must be 16-byte aligned with row strides that are multiples of 8");
    long long cache_rows = (long long)n_cache_pages * n_kv_heads * LLMB_PAGE;
    LLMB_REQUIRE(cache_rows < (1LL << 31), "diff_attention_tc: too many cache rows");
    int code;
    CUtensorMap map_q, map_k, map_v;
    if ((code = make_map_2d(&map_q, q, n_tokens, (long long)n_heads * 2 * dim, q_stride, 64, BQ))) return code;
    if ((code = make_map_2d(&map_k, k_cache, cache_rows, 2 * dim, 2 * dim, 64, LLMB_PAGE))) return code;
    if ((code = make_map_2d(&map_v, v_cache, cache_rows, vdim, vdim, 64, LLMB_PAGE))) return code;
    dim3 grid(n_heads, (max_new + BQ - 1) / BQ, n_seqs);
#define X(DK, DVAL)                                                                                                          \
    if (dim == DK && vdim == DVAL)                                                                                           \
        return launch_tc<DK, DVAL>(map_q, map_k, map_v, grid, block_table, table_stride, ring_pages, cu_seqlens, seq_lens,   \
                                   seq_order, out, out_stride, n_heads, n_kv_heads, scale, window, keep_first, lambda, eps,  \
                                   out_scale, head_norm, stream);
    LLMB_DIFF_TC_SHAPES(X)
#undef X
    return fail(LLMB_ERR_ARGUMENT, "diff_attention_tc: map size %d with value size %d is not built", dim, vdim);
}

LLMB_PACKED(llmb_diff_attention_tc)

// Prefill of the sigmoid attention with mixed heads (sigmoid_attention.cu says what it computes) on the
// fifth-generation tensor cores. The mix of the heads' scores is linear in the queries, so it is done on
// them: with G key/value heads, the mixed score of head a is one product of a "mixed query" of G * D
// elements with the keys of all G heads at a position. That makes the scores a contraction of length
// G * D (1,024 in the 8b shape), eight to nine tenths of the work, and it runs as a matrix product does:
//
// * mix_queries writes the mixed queries [head, token, G * D] of some heads once (32-bit sums over a
//   group's heads in index order, rounded to bfloat16 as any query is). A thread holds its eight columns
//   of the group's queries in registers and walks the heads, so it is bound by its stores.
// * the main kernel serves 128 queries of one head a block and walks the keys in steps of up to 256 (four
//   cache pages). S[128, 256] = mixed Q . K^T over G * D / 64 k-blocks (TMA, four stages of 48 KB: 16 KB of
//   queries, 8 KB of every page's keys), then O[128, DV] += W V with the weights W read from tensor memory.
//   The 128 mixed queries are 256 KB, more than an SM's shared memory: they stream with the keys, and 256
//   keys a step is what makes a k-block's 48 KB worth 4.2 MFLOP.
// * tensor memory: S 256 columns, W 128 (bfloat16 pairs), O 128. Eight warps take S into registers (128
//   columns a thread) and release it at once; while they form the weights sigmoid(scale S + bias), the
//   scores of the next step are being multiplied. The product of step n's weights is issued behind the
//   scores of step n + 1, so the tensor pipe has work while the threads read S.
// * nothing is normalised: no maximum, no rescaling. Keys after a query's position and before its window
//   get the weight 0; pages that no query of the tile sees are not loaded.
//
// Which call comes here, and why: every prefill of bfloat16 with a mixing matrix, head and value sizes of
// 64 or 128 and groups of 1, 2, 4 or 8 heads. 2,500 tokens, window 2,048, 32 heads over 8 of 128 on a B200:
// 2,147 us by the tiles on mma.sync (104 TFLOP/s of visible work), 290 + 35 us here (main kernel, 770 TFLOP/s, and
// mix_queries, 164 MB of stores). Without a matrix the contraction is one head long and the kernel of
// sigmoid_attention.cu stays. What bounds it now: 48 KB a k-block and SM through the L2, where a pair of blocks with
// one instruction for both would need 32 KB.
//
// All waits are bounded by a clock limit and report through the status word of this library.
#include "tc.cuh"

using namespace llmb;
using namespace llmb::tc;

LLMB_DEFINE_LAST_ERROR(llmb_sigmoid_attention_tc)

namespace {

constexpr int BQ = 128;                      // queries a block = lanes of tensor memory
constexpr int STEP_PAGES = 4;                // cache pages a step
constexpr int STEP_KEYS = STEP_PAGES * LLMB_PAGE;
constexpr int EPILOGUE_WARPS = 8;            // two a quarter of the lanes, half of a step's keys each
constexpr int EPILOGUE_THREADS = EPILOGUE_WARPS * 32;
constexpr int THREADS = EPILOGUE_THREADS + 64;
constexpr int STAGES = 4;
constexpr int A_BYTES = BQ * 64 * 2;                      // 64 columns of the mixed queries
constexpr int PAGE_PIECE = LLMB_PAGE * 64 * 2;            // 64 columns of a page's keys or values
constexpr int STAGE_BYTES = A_BYTES + STEP_PAGES * PAGE_PIECE;
constexpr int VALUE_PAGES = 2;               // pages whose values a stage takes
constexpr uint32_t S_COL = 0, W_COL = 256, O_COL = 384, TMEM_COLS = 512;


// mixed[h][t][g * D + d] = sum over the heads b of group g of talk[first_head + h, b] * q[t][b][d]
constexpr int MIX_THREADS = 256;
template <int GROUP>
__global__ void __launch_bounds__(MIX_THREADS)
mix_queries_kernel(const __nv_bfloat16* __restrict__ q, int q_stride, const float* __restrict__ talk,
                   __nv_bfloat16* __restrict__ mixed, int n_tokens, int n_heads, int n_kv_heads, int dim,
                   int first_head, int heads) {
    extern __shared__ float talk_rows[];                 // [heads][n_heads]
    griddep_launch();
    griddep_wait();
    q = behind_wait(q);
    for (int i = threadIdx.x; i < heads * n_heads; i += MIX_THREADS) talk_rows[i] = talk[(size_t)first_head * n_heads + i];
    __syncthreads();
    int width = n_kv_heads * dim, pieces = width / 8;    // 8 columns a thread
    long long items = (long long)n_tokens * pieces;
    for (long long item = (long long)blockIdx.x * MIX_THREADS + threadIdx.x; item < items; item += (long long)gridDim.x * MIX_THREADS) {
        int t = (int)(item / pieces), c = (int)(item % pieces) * 8;
        int g = c / dim, d = c % dim;
        float held[GROUP][8];
#pragma unroll
        for (int b = 0; b < GROUP; ++b) {
            const __nv_bfloat162* from = reinterpret_cast<const __nv_bfloat162*>(q + (size_t)t * q_stride + (size_t)(g * GROUP + b) * dim + d);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float2 pair = __bfloat1622float2(from[e]);
                held[b][2 * e] = pair.x;
                held[b][2 * e + 1] = pair.y;
            }
        }
        __nv_bfloat16* to = mixed + (size_t)t * width + c;
        for (int h = 0; h < heads; ++h) {
            const float* row = talk_rows + h * n_heads + g * GROUP;
            float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int b = 0; b < GROUP; ++b) {
                float w = row[b];
#pragma unroll
                for (int e = 0; e < 8; ++e) sum[e] = fmaf(w, held[b][e], sum[e]);
            }
            uint4 out;
            out.x = pack2(sum[0], sum[1]);
            out.y = pack2(sum[2], sum[3]);
            out.z = pack2(sum[4], sum[5]);
            out.w = pack2(sum[6], sum[7]);
            *reinterpret_cast<uint4*>(to + (size_t)h * n_tokens * width) = out;
        }
    }
}

template <int D, int DV>
__global__ void __launch_bounds__(THREADS, 1)
sigmoid_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                            const __grid_constant__ CUtensorMap map_v, const int* __restrict__ block_table,
                            int table_stride, int ring_pages, const int* __restrict__ cu_seqlens,
                            const int* __restrict__ seq_lens, const int* __restrict__ seq_order,
                            __nv_bfloat16* __restrict__ out, int out_stride, int n_tokens, int n_heads, int n_kv_heads,
                            int first_head, float scale, int window, const float* __restrict__ head_bias,
                            float out_scale, int* status) {
    constexpr int PIECES = D / 64, V_PIECES = DV / 64;
    constexpr int V_PAGE = V_PIECES * PAGE_PIECE;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(ring + STAGES * STAGE_BYTES);
    uint64_t* full = bars;                       // [STAGES]
    uint64_t* empty = bars + STAGES;             // [STAGES]
    uint64_t* s_full = bars + 2 * STAGES;        // a step's scores are complete
    uint64_t* s_empty = s_full + 1;              // they are in registers
    uint64_t* w_full = s_full + 2;               // its weights are in tensor memory
    uint64_t* o_full = s_full + 3;               // their product has been added to O
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_full + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    griddep_wait();
    int seq = seq_order ? seq_order[blockIdx.z] : (int)blockIdx.z, head = first_head + blockIdx.x;
    int first_token = cu_seqlens[seq];
    int n_new = cu_seqlens[seq + 1] - first_token;
    int n_tiles = (n_new + BQ - 1) / BQ;
    if ((int)blockIdx.y >= n_tiles) return;                  // uniform for the block: nothing is allocated yet
    int tile = n_tiles - 1 - blockIdx.y;                     // the heaviest tile of every head first
    int start = seq_lens[seq] - n_new;
    int kv_head = head / (n_heads / n_kv_heads);
    const int warp = warp_index(), lane = threadIdx.x & 31;
    int tile_last_pos = start + min(tile * BQ + BQ - 1, n_new - 1);
    int n_pages = tile_last_pos / LLMB_PAGE + 1;
    int first_page = window > 0 ? max(start + tile * BQ - window + 1, 0) / LLMB_PAGE : 0;
    int n_steps = (n_pages - first_page + STEP_PAGES - 1) / STEP_PAGES;
    int n_kblocks = n_kv_heads * PIECES;
    const int* pages = block_table + (size_t)seq * table_stride;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2 * STAGES + 4; ++i) mbar_init(smem_u32(&bars[i]), (&bars[i] == s_empty || &bars[i] == w_full) ? EPILOGUE_THREADS : 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == EPILOGUE_WARPS + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    uint32_t tmem_base = *tmem_slot;
    griddep_launch();            // behind the allocation: no block of the next kernel can hold this one's tensor memory

    if (warp == EPILOGUE_WARPS) {
        // the ring's order is the products' order: the k-blocks of step n, then the values of step n - 1
        int unit = 0;
        bool ok = true;
        auto next = [&](uint32_t bytes, uint32_t& bar, unsigned char*& to) {
            int stage = unit % STAGES, turn = unit / STAGES;
            if (turn > 0 && !mbar_wait_warp(smem_u32(&empty[stage]), (turn - 1) & 1, abort_flag, status, 1)) return false;
            bar = smem_u32(&full[stage]);
            to = ring + stage * STAGE_BYTES;
            if (elect_one()) mbar_expect_tx(bar, bytes);
            __syncwarp();
            ++unit;
            return true;
        };
        int q_row = (head - first_head) * n_tokens + first_token + tile * BQ;
        for (int n = 0; n <= n_steps && ok; ++n) {
            if (n < n_steps) {
                int p0 = first_page + n * STEP_PAGES, count = min(STEP_PAGES, n_pages - p0);
                int row[STEP_PAGES];
#pragma unroll
                for (int p = 0; p < STEP_PAGES; ++p)
                    row[p] = p < count ? pages[(p0 + p) % ring_pages] * n_kv_heads * LLMB_PAGE : 0;
                for (int j = 0; j < n_kblocks && ok; ++j) {
                    uint32_t bar;
                    unsigned char* to;
                    ok = next(A_BYTES + count * PAGE_PIECE, bar, to);
                    if (!ok) break;
                    int g = j / PIECES, x = (j % PIECES) * 64;
                    if (elect_one()) {
                        tma_load_2d(smem_u32(to), &map_q, bar, j * 64, q_row);
#pragma unroll
                        for (int p = 0; p < STEP_PAGES; ++p)
                            if (p < count) tma_load_2d(smem_u32(to + A_BYTES + p * PAGE_PIECE), &map_k, bar, x, row[p] + g * LLMB_PAGE);
                    }
                    __syncwarp();
                }
            }
            if (n > 0) {
                int p0 = first_page + (n - 1) * STEP_PAGES, count = min(STEP_PAGES, n_pages - p0);
                for (int v = 0; v < count && ok; v += VALUE_PAGES) {
                    uint32_t bar;
                    unsigned char* to;
                    int here = min(VALUE_PAGES, count - v);
                    ok = next(here * V_PAGE, bar, to);
                    if (!ok) break;
                    for (int p = 0; p < here; ++p) {
                        int row = (pages[(p0 + v + p) % ring_pages] * n_kv_heads + kv_head) * LLMB_PAGE;
                        if (elect_one()) {
                            for (int h = 0; h < V_PIECES; ++h)
                                tma_load_2d(smem_u32(to + p * V_PAGE + h * PAGE_PIECE), &map_v, bar, h * 64, row);
                        }
                        __syncwarp();
                    }
                }
            }
        }
    } else if (warp == EPILOGUE_WARPS + 1) {
        // D 32-bit, A and B bfloat16, M = 128; S has N = the step's keys, O has N = DV with B MN-major
        constexpr uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BQ >> 4) << 24);
        constexpr uint32_t idesc_o = idesc_s | (1u << 16) | ((uint32_t)(DV >> 3) << 17);
        const uint64_t a_desc = smem_desc(smem_u32(ring)), b_desc = smem_desc(smem_u32(ring + A_BYTES));
        const uint64_t v_desc = smem_desc_mn(smem_u32(ring), PAGE_PIECE);
        constexpr uint64_t STAGE = (uint64_t)(STAGE_BYTES >> 4);
        int stage = 0, phase = 0;
        auto advance = [&]() { if (++stage == STAGES) { stage = 0; phase ^= 1; } };
        bool ok = true;
        for (int n = 0; n <= n_steps && ok; ++n) {
            if (n < n_steps) {
                int count = min(STEP_PAGES, n_pages - (first_page + n * STEP_PAGES));
                uint32_t idesc = idesc_s | ((uint32_t)((count * LLMB_PAGE) >> 3) << 17);
                if (n > 0) ok = mbar_wait_warp(smem_u32(s_empty), (n - 1) & 1, abort_flag, status, 2);
                if (!ok) break;
                tcgen05_fence_after();
                for (int j = 0; j < n_kblocks && ok; ++j) {
                    ok = mbar_wait_warp(smem_u32(&full[stage]), phase, abort_flag, status, 3);
                    if (!ok) break;
                    tcgen05_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            tcgen05_mma(tmem_base + S_COL, a_desc + stage * STAGE + k * 2, b_desc + stage * STAGE + k * 2, idesc,
                                        (j > 0 || k > 0) ? 1u : 0u);
                        tcgen05_commit(smem_u32(&empty[stage]));
                        if (j + 1 == n_kblocks) tcgen05_commit(smem_u32(s_full));
                    }
                    __syncwarp();
                    advance();
                }
                if (!ok) break;
            }
            if (n > 0) {
                int count = min(STEP_PAGES, n_pages - (first_page + (n - 1) * STEP_PAGES));
                ok = mbar_wait_warp(smem_u32(w_full), (n - 1) & 1, abort_flag, status, 4);
                if (!ok) break;
                tcgen05_fence_after();
                for (int v = 0; v < count && ok; v += VALUE_PAGES) {
                    ok = mbar_wait_warp(smem_u32(&full[stage]), phase, abort_flag, status, 5);
                    if (!ok) break;
                    tcgen05_fence_after();
                    int here = min(VALUE_PAGES, count - v);
                    if (elect_one()) {
                        for (int p = 0; p < here; ++p)
#pragma unroll
                            for (int k = 0; k < LLMB_PAGE / 16; ++k)      // 16 keys: 8 columns of W, 2048 bytes of value rows
                                tcgen05_mma_ts(tmem_base + O_COL, tmem_base + W_COL + (v + p) * (LLMB_PAGE / 2) + k * 8,
                                               v_desc + stage * STAGE + (uint64_t)((p * V_PAGE + k * 2048) >> 4), idesc_o,
                                               (n > 1 || v + p > 0 || k > 0) ? 1u : 0u);
                        tcgen05_commit(smem_u32(&empty[stage]));
                        if (v + VALUE_PAGES >= count) tcgen05_commit(smem_u32(o_full));
                    }
                    __syncwarp();
                    advance();
                }
                if (!ok) break;
            }
        }
    } else {
        int quarter = warp & 3, half = warp >> 2;
        int q_index = tile * BQ + quarter * 32 + lane;       // among the sequence's new tokens; lane of tensor memory
        int pos = start + q_index;
        int warp_pos = start + tile * BQ + quarter * 32;     // the warp's first position
        int low = window > 0 ? pos - window + 1 : 0;
        uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
        float bias = head_bias ? head_bias[head] : 0.f;
        // sigmoid(z) = 1 / (1 + 2^(-z log2 e)), z = scale * s + bias
        float slope = -scale * 1.4426950408889634f, offset = -bias * 1.4426950408889634f;
        bool ok = true;
        for (int n = 0; n < n_steps && ok; ++n) {
            int p0 = first_page + n * STEP_PAGES;
            int mine = min(STEP_PAGES, n_pages - p0) * LLMB_PAGE - half * (STEP_KEYS / 2);      // columns of this half that exist
            ok = mbar_wait(smem_u32(s_full), n & 1, abort_flag, status, 6);
            if (!ok) break;
            __syncwarp();
            tcgen05_fence_after();
            uint32_t r[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (c * 32 < mine) tmem_ld32_start(lane_addr + S_COL + half * (STEP_KEYS / 2) + c * 32, r[c]);
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (c * 32 < mine) tmem_ld32_wait(r[c]);
            tcgen05_fence_before();
            mbar_arrive(smem_u32(s_empty));
            int key0 = p0 * LLMB_PAGE + half * (STEP_KEYS / 2);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (c * 32 >= mine) continue;
                int k0 = key0 + c * 32;
                bool edge = k0 + 31 > warp_pos || (window > 0 && k0 < warp_pos + 31 - window + 1);
#pragma unroll
                for (int j = 0; j < 32; j += 2) {
                    float w0 = __frcp_rn(1.0f + fast_exp2(fmaf(__uint_as_float(r[c][j]), slope, offset)));
                    float w1 = __frcp_rn(1.0f + fast_exp2(fmaf(__uint_as_float(r[c][j + 1]), slope, offset)));
                    if (edge) {
                        if (k0 + j > pos || k0 + j < low) w0 = 0.f;
                        if (k0 + j + 1 > pos || k0 + j + 1 < low) w1 = 0.f;
                    }
                    r[c][j >> 1] = pack2(w0, w1);
                }
            }
            if (n > 0) {                                     // the weights before these have been multiplied
                ok = mbar_wait(smem_u32(o_full), (n - 1) & 1, abort_flag, status, 7);
                if (!ok) break;
                __syncwarp();
                tcgen05_fence_after();
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (c * 32 >= mine) continue;
                uint32_t packed[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) packed[j] = r[c][j];
                tmem_st16(lane_addr + W_COL + half * (STEP_KEYS / 4) + c * 16, packed);
            }
            tmem_st_wait();
            tcgen05_fence_before();
            mbar_arrive(smem_u32(w_full));
        }
        if (ok) ok = mbar_wait(smem_u32(o_full), (n_steps - 1) & 1, abort_flag, status, 8);
        if (ok) {
            __syncwarp();
            tcgen05_fence_after();
            __nv_bfloat16* o = out + (size_t)(first_token + q_index) * out_stride + (size_t)head * DV + half * (DV / 2);
#pragma unroll
            for (int c = 0; c < DV / 2; c += 32) {
                uint32_t r[32];
                tmem_ld32(lane_addr + O_COL + half * (DV / 2) + c, r);
                if (q_index < n_new) {
#pragma unroll
                    for (int d = 0; d < 32; d += 8) {
                        uint4 packed;
                        packed.x = pack2(__uint_as_float(r[d]) * out_scale, __uint_as_float(r[d + 1]) * out_scale);
                        packed.y = pack2(__uint_as_float(r[d + 2]) * out_scale, __uint_as_float(r[d + 3]) * out_scale);
                        packed.z = pack2(__uint_as_float(r[d + 4]) * out_scale, __uint_as_float(r[d + 5]) * out_scale);
                        packed.w = pack2(__uint_as_float(r[d + 6]) * out_scale, __uint_as_float(r[d + 7]) * out_scale);
                        *reinterpret_cast<uint4*>(o + c + d) = packed;
                    }
                }
            }
        }
    }

    tcgen05_fence_before();
    __syncthreads();
    if (*abort_flag) {                                       // copies in flight land before the block's memory is given back
        for (int i = 0; i < 100; ++i) __nanosleep(10000);
        __syncthreads();
    }
    if (warp == EPILOGUE_WARPS + 1) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

}  // namespace

LLMB_EXPORT int llmb_sigmoid_attention_tc_status() {
    int* s = status_word();
    if (!s) return -1;
    int v = *s;
    *s = 0;
    return v;
}

LLMB_EXPORT int llmb_sigmoid_attention_tc_supports(int n_heads, int n_kv_heads, int dim, int vdim) {
    LLMB_REQUIRE(n_heads > 0 && n_kv_heads > 0 && n_heads % n_kv_heads == 0,
                 "sigmoid_attention_tc: %d heads are no multiple of %d kv heads", n_heads, n_kv_heads);
    int group = n_heads / n_kv_heads;
    LLMB_REQUIRE(group == 1 || group == 2 || group == 4 || group == 8, "sigmoid_attention_tc: groups of %d heads are not built", group);
    LLMB_REQUIRE(n_heads <= 128, "sigmoid_attention_tc: %d heads (up to 128)", n_heads);
    LLMB_REQUIRE((dim == 64 || dim == 128) && (vdim == 64 || vdim == 128),
                 "sigmoid_attention_tc: head size %d with value size %d is not built", dim, vdim);
    return LLMB_OK;
}

namespace {
template <int D, int DV>
int launch_tc(const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v, dim3 grid, const int* block_table,
              int table_stride, int ring_pages, const int* cu_seqlens, const int* seq_lens, const int* seq_order, void* out,
              int out_stride, int n_tokens, int n_heads, int n_kv_heads, int first_head, float scale, int window,
              const float* head_bias, float out_scale, cudaStream_t stream) {
    constexpr size_t smem = 1024 + (size_t)STAGES * STAGE_BYTES + (2 * STAGES + 4) * 8 + 16;
    static bool configured = false;
    if (!configured) {
        LLMB_CUDA(cudaFuncSetAttribute(sigmoid_attention_tc_kernel<D, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured = true;
    }
    int* status = status_word();
    int* status_dev = nullptr;
    if (status) cudaHostGetDevicePointer((void**)&status_dev, status, 0);
    LLMB_CUDA(llmb::launch(sigmoid_attention_tc_kernel<D, DV>, grid, dim3(THREADS), smem, stream, true, map_q, map_k, map_v,
                           block_table, table_stride, ring_pages, cu_seqlens, seq_lens, seq_order, (__nv_bfloat16*)out,
                           out_stride, n_tokens, n_heads, n_kv_heads, first_head, scale, window, head_bias, out_scale, status_dev));
    return check_launch("sigmoid_attention_tc");
}
}  // namespace

// q: the new tokens' queries [n_tokens, q_stride], packed sequence after sequence; the rest as in
// llmb_sigmoid_attention_tiles, with talk [n_heads, n_heads] float32 given. mixed: room for the mixed queries of
// `heads_at_once` heads (bfloat16 [heads_at_once, n_tokens, n_kv_heads * dim]); the heads run in groups of that
// many, two launches a group.
LLMB_EXPORT int llmb_sigmoid_attention_tc(const void* q, int q_stride, int n_tokens, const void* k_cache, const void* v_cache,
                                          int n_cache_pages, const int* block_table, int table_stride, int ring_pages,
                                          const int* cu_seqlens, const int* seq_lens, const int* seq_order, void* out,
                                          int out_stride, void* mixed, int heads_at_once, int n_seqs, int max_new,
                                          int n_heads, int n_kv_heads, int dim, int vdim, float scale, int window,
                                          const float* talk, const float* head_bias, float out_scale, cudaStream_t stream) {
    if (n_seqs == 0 || max_new == 0 || n_tokens == 0) return LLMB_OK;
    int code = llmb_sigmoid_attention_tc_supports(n_heads, n_kv_heads, dim, vdim);
    if (code) return code;
    LLMB_REQUIRE(n_seqs <= 65535 && max_new / BQ < 65535 && ring_pages > 0 && n_cache_pages > 0 && window >= 0 && talk && mixed,
                 "sigmoid_attention_tc: bad sizes");
    LLMB_REQUIRE(heads_at_once > 0 && (long long)heads_at_once * n_tokens < (1LL << 31), "sigmoid_attention_tc: %d heads at once", heads_at_once);
    LLMB_REQUIRE(q_stride % 2 == 0 && (reinterpret_cast<uintptr_t>(q) & 3) == 0 && out_stride % 8 == 0 &&
                 (reinterpret_cast<uintptr_t>(out) & 15) == 0 && (reinterpret_cast<uintptr_t>(mixed) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(k_cache) & 15) == 0 && (reinterpret_cast<uintptr_t>(v_cache) & 15) == 0,
                 "sigmoid_attention_tc: out, mixed and the cache must be 16-byte aligned, out's row stride a multiple of 8, "
                 "q 4-byte aligned with an even row stride");
    int width = n_kv_heads * dim;
    long long cache_rows = (long long)n_cache_pages * n_kv_heads * LLMB_PAGE;
    LLMB_REQUIRE(cache_rows < (1LL << 31), "sigmoid_attention_tc: too many cache rows");
    CUtensorMap map_q, map_k, map_v;
    if ((code = make_map_2d(&map_k, k_cache, cache_rows, dim, dim, 64, LLMB_PAGE))) return code;
    if ((code = make_map_2d(&map_v, v_cache, cache_rows, vdim, vdim, 64, LLMB_PAGE))) return code;
    for (int first = 0; first < n_heads; first += heads_at_once) {
        int heads = n_heads - first < heads_at_once ? n_heads - first : heads_at_once;
        if ((code = make_map_2d(&map_q, mixed, (long long)heads * n_tokens, width, width, 64, BQ))) return code;
        int group = n_heads / n_kv_heads;
        auto mix = group == 1 ? mix_queries_kernel<1> : group == 2 ? mix_queries_kernel<2> : group == 4 ? mix_queries_kernel<4>
                                                                                                     : mix_queries_kernel<8>;
        long long blocks = ceil_div((long long)n_tokens * (width / 8), (long long)MIX_THREADS);
        if (blocks > 148 * 8) blocks = 148 * 8;
        size_t smem = sizeof(float) * heads * n_heads;
        if (smem > 48 * 1024) LLMB_CUDA(cudaFuncSetAttribute(mix, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        LLMB_CUDA(llmb::launch(mix, dim3((unsigned)blocks), dim3(MIX_THREADS), smem, stream, true, (const __nv_bfloat16*)q, q_stride,
                               talk, (__nv_bfloat16*)mixed, n_tokens, n_heads, n_kv_heads, dim, first, heads));
        dim3 grid(heads, (max_new + BQ - 1) / BQ, n_seqs);
#define X(DK, DVAL)                                                                                                       \
        if (dim == DK && vdim == DVAL)                                                                                    \
            code = launch_tc<DK, DVAL>(map_q, map_k, map_v, grid, block_table, table_stride, ring_pages, cu_seqlens,      \
                                       seq_lens, seq_order, out, out_stride, n_tokens, n_heads, n_kv_heads, first, scale, \
                                       window, head_bias, out_scale, stream);
        X(64, 64) X(64, 128) X(128, 64) X(128, 128)
#undef X
        if (code) return code;
    }
    return LLMB_OK;
}

LLMB_PACKED(llmb_sigmoid_attention_tc)

// C = A . B^T on the fifth-generation tensor cores: tcgen05.mma with the
// accumulator in tensor memory, operands staged in shared memory by TMA.
//
// A is [rows_a, K] and B is [rows_b, K], both bfloat16 with K contiguous (the
// row-major [out, in] weights of MythEclipse/llm, apps/engine/src/tensor.rs:14,91,
// and activations [tokens, K]). One block computes a 128 x BN tile of
// D[a_row, b_row] = sum_k A[a_row, k] B[b_row, k]. It replaces the mma.sync prompt
// kernel q8_matmul_mma (apps/engine/kernels/gpu.cu:907-1212): the tile loop,
// the token tile running fastest over the grid so that a weight tile is reused
// from L2 (gpu.cu:942-966) and the bias/residual epilogue (gpu.cu:1194-1209)
// are kept, the machinery is Blackwell's:
//
// * warp 0: TMA producer (one elected lane issues). Per k-block of 64 it waits for a free
//   stage, arms the stage's mbarrier with the byte count and issues two
//   cp.async.bulk.tensor.2d loads (128-byte swizzle), A rows and B rows.
// * warp 1: allocates BN columns of tensor memory; one elected lane issues four
//   tcgen05.mma (M 128, N BN, K 16) per k-block from shared-memory descriptors,
//   then tcgen05.commit frees the stage; a last commit signals the epilogue.
// * warps 2-5: epilogue. Each reads its 32 lanes of the accumulator with
//   tcgen05.ld, adds the bias, and stores bfloat16 or 32-bit, or adds into the
//   32-bit residual stream.
//
// Two orientations share the kernel. `swap == 0` (prefill): A = activations,
// B = weights, D[token, out] is stored row by row. `swap == 1` (decode, few
// tokens): A = weights, B = activations, so that the 128-row side of the
// instruction is filled by weight rows and the tokens are the narrow N side
// (16 to 64); D[out, token] is stored transposed. For decode the k-blocks are
// split over `splits` blocks per tile so that a product with few output tiles
// still fills 148 SMs: each block writes its partial tile to scratch, and the
// block that arrives last at the tile's counter adds the partials in split
// order and runs the epilogue (the counter returns to zero).
//
// The kernel is persistent: at most as many blocks as the GPU holds at once, each taking
// work units (an output tile and one slice of its k-blocks) round robin. The operand ring
// and two accumulator buffers in tensor memory carry on from unit to unit, so the loads and
// products of the next unit run under the epilogue of the last.
//
// Every wait on an mbarrier is bounded by a clock limit. A wait that runs out
// sets a status word that the host can read, raises the block's abort flag so that
// the roles that load and multiply leave their loops (the epilogue runs through
// its own, see accumulator_wait), and the block still frees its tensor memory.
#include <cuda.h>

#include "common.cuh"
#include "fusion.h"
#include "tc.cuh"

using namespace llmb;
using namespace llmb::tc;      // mbarrier, TMA and tcgen05 wrappers, descriptors, the tensor-map encoder

LLMB_DEFINE_LAST_ERROR(llmb_gemm_tc)

namespace {

constexpr int BM = 128;             // rows of A per tile = lanes of tensor memory
constexpr int BK = 64;              // k-values per stage: one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int THREADS = 192;        // producer warp, mma warp, four epilogue warps

struct Epilogue {
    const float* bias;       // indexed by the output column n
    void* out;               // [tokens, ldo]
    float* residual;         // [tokens, ldo] 32-bit, added into
    int out_is_bf16;
    int ldo;
    int tokens, outs;        // valid tokens and output columns (rows of the weight matrix)
    int glu;                 // gated activation: the weight rows alternate 16 gate rows, 16 up rows;
                             // out is bfloat16 [tokens, ldo] with outs / 2 columns act(gate) * up
    llmb_gemm_fusion f;      // what else the epilogue does (fusion.h); all zero: nothing
    float act_linear, act_cubic;      // which act (see gated)
};

// 1 / sqrt(mean of squares + eps) of an input row from the partial sums its producer left. A whole warp
// computes it: lane i adds parts i and i + 32, then the lanes are summed as a butterfly, so every
// consumer of a row gets the same bits, and the loads of a row are in flight together.
__device__ __forceinline__ float warp_row_rstd(const llmb_gemm_fusion& f, int token) {
    int lane = threadIdx.x & 31;
    const float* p = f.norm_sumsq + (size_t)token * LLMB_SUMSQ_LD;
    float v = (lane < f.norm_parts ? __ldcg(p + lane) : 0.f) + (lane + 32 < f.norm_parts ? __ldcg(p + lane + 32) : 0.f);
    v = warp_sum(v);
    return 1.0f / sqrtf(v / f.norm_width + f.norm_eps);
}

// The same value, bit for bit, computed by ONE thread: v[i] = part i + part i + 32 as lane i has it, then
// the butterfly's levels as a tree (lane i's sum after the level of offset w is v[i] + v[i + w] for
// i < w; additions commute). A thread has all of its row's loads in flight at once, so the rows of a
// wide tile take one trip to L2 together instead of one trip each.
__device__ __forceinline__ float thread_row_rstd(const llmb_gemm_fusion& f, int token) {
    const float4* p = reinterpret_cast<const float4*>(f.norm_sumsq + (size_t)token * LLMB_SUMSQ_LD);
    int parts = f.norm_parts;
    float v[32];
#pragma unroll
    for (int g = 0; g < 8; ++g) {
        float4 lo = 4 * g < parts ? __ldcg(p + g) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 hi = 32 + 4 * g < parts ? __ldcg(p + 8 + g) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float l[4] = {lo.x, lo.y, lo.z, lo.w}, h[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            int i = 4 * g + j;
            v[i] = (i < parts ? l[j] : 0.f) + (i + 32 < parts ? h[j] : 0.f);
        }
    }
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
#pragma unroll
        for (int i = 0; i < w; ++i) v[i] += v[i + w];
    }
    return 1.0f / sqrtf(v[0] / f.norm_width + f.norm_eps);
}
static_assert(LLMB_SUMSQ_LD == 64, "thread_row_rstd and warp_row_rstd read a row of 64 partial sums");

// The scales of a tile's token rows into shared memory, by the four epilogue warps, before the tile's
// accumulator is awaited: up to 16 rows a warp a row (quarter = 0..3 takes every fourth), more rows a
// thread a row. The caller synchronises the epilogue warps afterwards.
__device__ __forceinline__ void tile_rstd(const Epilogue& ep, float* rstd, int quarter, int first_token, int n_tile_tokens) {
    int lane = threadIdx.x & 31;
    if (n_tile_tokens > 16) {
        for (int i = quarter * 32 + lane; i < n_tile_tokens; i += 128) {
            int token = first_token + i;
            rstd[i] = token < ep.tokens ? thread_row_rstd(ep.f, token) : 1.f;
        }
        return;
    }
#pragma unroll 4
    for (int i = quarter; i < n_tile_tokens; i += 4) {
        int token = first_token + i;
        float r = token < ep.tokens ? warp_row_rstd(ep.f, token) : 1.f;
        if (lane == 0) rstd[i] = r;
    }
}

static_assert(LLMB_GLU_BLOCK == 16, "the gated epilogue reads 16 gate and 16 up columns of tensor memory per pair");

// act(gate) * up. Both activations are z sigmoid(t): silu has t = z, and the tanh form of gelu, 0.5 z (1 + tanh(u)) with
// u = sqrt(2 / pi) (z + 0.044715 z^3), is z sigmoid(2 u); t = z (act_linear + act_cubic z^2) gives either.
__device__ __forceinline__ float gated(const Epilogue& ep, float gate, float up) {
    float t = gate * fmaf(ep.act_cubic * gate, gate, ep.act_linear);
    return gate / (1.0f + expf(-t)) * up;
}

// One work unit: output tile (tile_a, tile_b) and one slice of its k-blocks.
struct Unit {
    int tile_a, tile_b, split;
};
__device__ __forceinline__ Unit unit_of(int u, int tiles_a, int splits) {
    Unit w;
    w.split = u % splits;
    int t = u / splits;
    w.tile_a = t % tiles_a;            // the A tile runs fastest: neighbours share a B tile in L2
    w.tile_b = t / tiles_a;
    return w;
}

// Stores 16 consecutive accumulator columns (c .. c+15) of this thread's row.
// `preloaded` (swapped products with a residual only): the residual's values at these 16 places,
// read by the caller earlier so that their latency ran under other loads.
// `rstd` (shared memory, or nullptr): the scales of the tile's token rows (a folded norm).
template <int BN>
__device__ __forceinline__ void store_columns(const Epilogue& ep, int swap, int a_row, int tile_b,
                                              int c, float (&v)[16], const float* preloaded = nullptr,
                                              const float* rstd = nullptr, int tile_row = 0) {
    if (rstd) {
        if (swap) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] *= rstd[c + j];
        } else {
            float r = rstd[tile_row];
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] *= r;
        }
    }
    if (swap && ep.glu) {
        // lanes 0-15 of a warp hold 16 gate rows, lanes 16-31 the up rows of the same features
        int lane = threadIdx.x & 31;
        int feature = (a_row >> 5) * 16 + (a_row & 15);
        __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(ep.out);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            float up = __shfl_xor_sync(0xffffffffu, v[j], 16);
            int token = tile_b * BN + c + j;
            if (lane < 16 && a_row < ep.outs && token < ep.tokens)
                o[(size_t)token * ep.ldo + feature] = __float2bfloat16_rn(gated(ep, v[j], up));
        }
        return;
    }
    if (swap) {
        // D[out column a_row, token]: one token at a time, lanes along the output row
        if (a_row >= ep.outs) return;
        float b = ep.bias ? ep.bias[a_row] : 0.f;
        int first_token = tile_b * BN + c;
        if (ep.residual) {
            // all loads first, then all stores: a load placed after a store would have to
            // wait for it (the compiler cannot know that the addresses differ)
            float old[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (preloaded) old[j] = preloaded[j];
                else old[j] = first_token + j < ep.tokens ? ep.residual[(size_t)(first_token + j) * ep.ldo + a_row] : 0.f;
            }
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (first_token + j < ep.tokens)
                    ep.residual[(size_t)(first_token + j) * ep.ldo + a_row] = old[j] + (v[j] + b);
            return;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            int token = first_token + j;
            if (token >= ep.tokens) break;
            size_t at = (size_t)token * ep.ldo + a_row;
            float value = v[j] + b;
            if (ep.out_is_bf16) reinterpret_cast<__nv_bfloat16*>(ep.out)[at] = __float2bfloat16_rn(value);
            else reinterpret_cast<float*>(ep.out)[at] = value;
        }
        return;
    }
    if (a_row >= ep.tokens) return;
    // D[token a_row, out column]: 16 consecutive columns of this thread's row
    int n0 = tile_b * BN + c;
    if (n0 >= ep.outs) return;
    size_t at = (size_t)a_row * ep.ldo + n0;
    bool whole = n0 + 16 <= ep.outs;
    if (ep.bias) {
#pragma unroll
        for (int j = 0; j < 16; ++j) if (n0 + j < ep.outs) v[j] += ep.bias[n0 + j];
    }
    if (ep.residual) {
        if (whole && (ep.ldo & 3) == 0) {
            float4* p = reinterpret_cast<float4*>(ep.residual + at);
            float4 old[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) old[j] = p[j];              // loads first, then stores
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                old[j].x += v[4 * j]; old[j].y += v[4 * j + 1]; old[j].z += v[4 * j + 2]; old[j].w += v[4 * j + 3];
                p[j] = old[j];
            }
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) if (n0 + j < ep.outs) ep.residual[at + j] += v[j];
        }
    } else if (ep.out_is_bf16) {
        __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(ep.out) + at;
        if (whole && (ep.ldo & 7) == 0) {
            uint4 packed[2];
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(packed);
#pragma unroll
            for (int j = 0; j < 8; ++j) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
            reinterpret_cast<uint4*>(o)[0] = packed[0];
            reinterpret_cast<uint4*>(o)[1] = packed[1];
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) if (n0 + j < ep.outs) o[j] = __float2bfloat16_rn(v[j]);
        }
    } else {
        float* o = reinterpret_cast<float*>(ep.out) + at;
        if (whole && (ep.ldo & 3) == 0) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                reinterpret_cast<float4*>(o)[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) if (n0 + j < ep.outs) o[j] = v[j];
        }
    }
}

// ---- the fused epilogues of a decode tile (weights on the 128-row side, tiles of 16 tokens), run by the
// four epilogue warps of the block that arrived last at the tile; v[j] is the summed (and scaled) product
// for output column a_row and token first_token + j, j < valid.

// Adds into the residual and also leaves what the next norm needs: the updated rows as bfloat16 and,
// per token, the sum of their squares over this tile's 128 columns as partial `tile_a` of the row.
// The sum runs over lanes, then over the four warps in a fixed order. exch: 64 floats.
__device__ __forceinline__ void finish_emit(const Epilogue& ep, int a_row, int tile_a, int first_token, int valid,
                                            float (&v)[16], const float (&old)[16], float* exch) {
    int lane = threadIdx.x & 31, quarter = (threadIdx.x >> 5) & 3;
    bool live = a_row < ep.outs;
    float b = (ep.bias && live) ? ep.bias[a_row] : 0.f;
    __nv_bfloat16* rows = reinterpret_cast<__nv_bfloat16*>(ep.f.emit_rows);
    float sq[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        float updated = old[j] + (v[j] + b);
        bool here = live && j < valid;
        if (here) {
            size_t at = (size_t)(first_token + j) * ep.ldo + a_row;
            ep.residual[at] = updated;
            rows[at] = __float2bfloat16_rn(updated);
        }
        sq[j] = here ? updated * updated : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 16; ++j)
        if (j < valid) sq[j] = warp_sum(sq[j]);          // (valid is the same for the whole block)
    if (lane == 0) {
#pragma unroll
        for (int j = 0; j < 16; ++j) exch[quarter * 16 + j] = sq[j];
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
    int local = (int)threadIdx.x - 64;
    if (local < valid)
        ep.f.emit_sumsq[(size_t)(first_token + local) * LLMB_SUMSQ_LD + tile_a] =
            ((exch[local] + exch[16 + local]) + exch[32 + local]) + exch[48 + local];
    asm volatile("bar.sync 1, 128;" ::: "memory");
}

// The q/k/v product's epilogue: bias, rotation of the query and key heads, queries to `out`, keys and
// values into the paged cache (what llmb_rope_cache_write does in a kernel of its own). A head's values
// lie in one tile (128 % head_dim == 0); pairs (p, p + head_dim/2) are exchanged through shared memory
// (exch: 16 x 128 floats), interleaved pairs (2p, 2p+1) between neighbouring lanes.
//
// What the epilogue needs from global memory besides the products is fetched before the products are
// awaited (stage_rope, by every block of the tile, since any may be the last): each token's position, the
// page of its position and its row of angles wait in shared memory. Read in the epilogue itself, these
// small loads miss the L2 (a layer's weights have passed through it since their last use) and two of
// them in a chain cost the last block of a tile three microseconds.
struct RopeStage {
    float angles[16][BM];          // [token of the tile][head_dim values: cosines, then sines]
    int pos[16];
    int page[16];
};

__device__ __forceinline__ void stage_rope(const Epilogue& ep, RopeStage* stage, int first_token) {
    const llmb_gemm_fusion& f = ep.f;
    int local = (int)threadIdx.x - 64;
    int valid = min(16, ep.tokens - first_token);
    if (local < 16) {
        int pos = 0, page = 0;
        if (local < valid) {
            pos = f.tok_pos[first_token + local];
            page = f.block_table[(size_t)f.tok_seq[first_token + local] * f.table_stride + ((pos / LLMB_PAGE) % f.ring_pages)];
        }
        stage->pos[local] = pos;
        stage->page[local] = page;
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (f.rope_table) {
        int dim = f.head_dim;
        for (int i = local; i < valid * dim; i += 128) {
            int j = i / dim, e = i - j * dim;
            stage->angles[j][e] = f.rope_table[(size_t)stage->pos[j] * dim + e];
        }
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
}

__device__ __forceinline__ void finish_rope(const Epilogue& ep, int a_row, int tile_row, int first_token, int valid,
                                            float (&v)[16], float* exch, const RopeStage* stage) {
    const llmb_gemm_fusion& f = ep.f;
    int dim = f.head_dim, half = dim >> 1;
    int head = a_row / dim, r = a_row - head * dim;
    bool live = a_row < ep.outs;
    float b = (ep.bias && live) ? ep.bias[a_row] : 0.f;
    float partner[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] += b;
    if (f.interleaved) {
#pragma unroll
        for (int j = 0; j < 16; ++j) partner[j] = __shfl_xor_sync(0xffffffffu, v[j], 1);
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) exch[j * BM + tile_row] = v[j];
        asm volatile("bar.sync 1, 128;" ::: "memory");
        int other = r < half ? tile_row + half : tile_row - half;
#pragma unroll
        for (int j = 0; j < 16; ++j) partner[j] = exch[j * BM + other];
        asm volatile("bar.sync 1, 128;" ::: "memory");
    }
    bool is_q = head < f.n_heads, is_k = !is_q && head < f.n_heads + f.n_kv_heads;
    bool rotates = f.rope_table != nullptr && (is_q || is_k);
    bool low = f.interleaved ? (r & 1) == 0 : r < half;
    int pair = f.interleaved ? r >> 1 : (r < half ? r : r - half);
    __nv_bfloat16* q_out = reinterpret_cast<__nv_bfloat16*>(ep.out);
    __nv_bfloat16* cache = reinterpret_cast<__nv_bfloat16*>(is_k ? f.k_cache : f.v_cache);
    int kv_head = is_k ? head - f.n_heads : head - f.n_heads - f.n_kv_heads;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        if (j >= valid || !live) break;
        float value = v[j];
        if (rotates) {
            float c = stage->angles[j][pair], s = stage->angles[j][half + pair];
            value = low ? v[j] * c - partner[j] * s : partner[j] * s + v[j] * c;
        }
        if (is_q) {
            q_out[(size_t)(first_token + j) * ep.ldo + a_row] = __float2bfloat16_rn(value);
        } else if (f.write_cache) {
            int pos = stage->pos[j];
            cache[(((size_t)stage->page[j] * f.n_kv_heads + kv_head) * LLMB_PAGE + (pos % LLMB_PAGE)) * dim + r] =
                __float2bfloat16_rn(value);
        }
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");      // the staged values are free for the block's next unit
}

// The epilogue's wait for an accumulator. What follows has barriers of the four epilogue warps, and one warp's wait may run out where
// another's ended: a warp that left its loop here would leave the others waiting for good. So all go on, with sums that are
// not valid (the status word says so), through every barrier of their units; the waits that are left end as soon as they see
// the abort flag. (A wait of each thread for itself, its answer unused, made the gated epilogue 8 % slower: 801 x 26880 x 384 68.7 -> 74.4
// us; with a warp's wait 68.5, and tiles of the row side leave 3 % sooner than before, 317 x 12288 x 256 10.6 -> 10.25.)
__device__ __forceinline__ void accumulator_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status) {
    mbar_wait_warp(bar, parity, abort_flag, status, 3);
}

// Persistent: the grid has at most as many blocks as fit on the GPU at once, and block b
// takes the units b, b + gridDim.x, ... . The shared-memory ring and the two accumulator
// buffers in tensor memory run on across units, so the loads and products of the next unit
// overlap the epilogue of this one.
//
// Split K: every block leaves its partial tile in global memory. Either the block that arrives
// last at the tile's counter sums them in split order (one round of loads for up to 8 tokens), or,
// with sum_later (more than 16 tokens: the tile is wide and one block would sum for a long time),
// the blocks only write and splitk_sum_kernel, launched behind this kernel, sums with the whole
// GPU. The order of the sum is the same on both ways.
template <int BN>
__global__ void __launch_bounds__(THREADS, 2)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
               Epilogue ep, int swap, int n_kblocks, int kblocks_per_split, int splits, int tiles_a,
               int n_units, float* __restrict__ partials, unsigned* __restrict__ counters,
               int* status, int stages, int sum_later) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2;
    constexpr int TMEM_COLS = 2 * BN < 32 ? 32 : 2 * BN;       // two accumulator buffers
    // 1024-byte alignment of every tile is required by the 128-byte swizzle
    unsigned char* base = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* a_tiles = base;
    unsigned char* b_tiles = base + (size_t)stages * A_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(b_tiles + (size_t)stages * B_BYTES);
    uint64_t* full_bar = bars;                         // [stages] operands landed
    uint64_t* empty_bar = bars + stages;               // [stages] operands consumed
    uint64_t* acc_full_bar = bars + 2 * stages;        // [2] accumulator complete
    uint64_t* acc_empty_bar = bars + 2 * stages + 2;   // [2] accumulator drained
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * stages + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* last_flag = reinterpret_cast<volatile int*>(tmem_slot + 2);
    float* exch = reinterpret_cast<float*>(tmem_slot + 4);      // the fused epilogues' exchange (sized by the host)
    RopeStage* rope_stage = reinterpret_cast<RopeStage*>(exch + 16 * BM);   // only with a fused rotation
    __shared__ float rstd_s[2][BM];                             // scales of a tile's token rows (a folded norm)

    const int warp = warp_index(), lane = threadIdx.x & 31;
    LLMB_STAMP(0, 0);                                           // the block has started
    griddep_launch();                                           // the next kernel of the stream may set itself up
    uint32_t early = 0;                                         // k-blocks whose weight tile is on its way (known to the producer warp)
    if (warp == 0 && (int)blockIdx.x < n_units) {
        int first = unit_of(blockIdx.x, tiles_a, splits).split * kblocks_per_split;
        early = (uint32_t)min(stages, min(n_kblocks, first + kblocks_per_split) - first);
    }

    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
        for (int s = 0; s < stages; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&acc_full_bar[b]), 1);
            mbar_init(smem_u32(&acc_empty_bar[b]), 4);          // one arrival per epilogue warp
        }
        *abort_flag = 0;
        *last_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the barriers, as the copy engine sees them
        // Fetch this block's first weight tiles at once (no kernel writes weights): this thread made the
        // barriers and is the producer, so it need not wait for the block's set-up, and the kernel before
        // this one may still be running. The activations, the residual and the split-K scratch are
        // touched only after griddep_wait().
        if ((int)blockIdx.x < n_units) {
            Unit w = unit_of(blockIdx.x, tiles_a, splits);
            int kb_begin = w.split * kblocks_per_split;
            for (uint32_t i = 0; i < early; ++i) {
                uint32_t bar = smem_u32(&full_bar[i]);
                mbar_expect_tx(bar, A_BYTES + B_BYTES);
                if (swap) tma_load_2d(smem_u32(a_tiles + (size_t)i * A_BYTES), &map_a, bar, (kb_begin + i) * BK, w.tile_a * BM);
                else tma_load_2d(smem_u32(b_tiles + (size_t)i * B_BYTES), &map_b, bar, (kb_begin + i) * BK, w.tile_b * BN);
            }
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    uint32_t tmem_base = *tmem_slot;
    LLMB_STAMP(1, 0);                                           // barriers and tensor memory are set up
    griddep_wait();
    LLMB_STAMP(2, 0);                                           // the kernel before this one has completed

    if (warp == 0) {
        uint32_t it = 0;                                        // k-blocks issued so far, over all units
        int s = 0;                                              // the stage of k-block `it`, and how often
        uint32_t round = 0;                                     // the ring has been walked through (no division here)
        bool ok = true;
        for (int u = blockIdx.x; u < n_units && ok; u += gridDim.x) {
            Unit w = unit_of(u, tiles_a, splits);
            int kb_begin = w.split * kblocks_per_split;
            int kb_end = min(n_kblocks, kb_begin + kblocks_per_split);
            for (int kb = kb_begin; kb < kb_end; ++kb, ++it, s = (s + 1 == stages ? 0 : s + 1), round += (s == 0)) {
                uint32_t bar = smem_u32(&full_bar[s]);
                if (it < early) {                               // armed above, the weight tile is in flight
                    if (elect_one()) {
                        if (swap) tma_load_2d(smem_u32(b_tiles + (size_t)s * B_BYTES), &map_b, bar, kb * BK, w.tile_b * BN);
                        else tma_load_2d(smem_u32(a_tiles + (size_t)s * A_BYTES), &map_a, bar, kb * BK, w.tile_a * BM);
                    }
                    __syncwarp();
                    continue;
                }
                ok = mbar_wait_warp(smem_u32(&empty_bar[s]), (round & 1) ^ 1, abort_flag, status, 1);
                if (!ok) break;
                if (elect_one()) {
                    mbar_expect_tx(bar, A_BYTES + B_BYTES);
                    tma_load_2d(smem_u32(a_tiles + (size_t)s * A_BYTES), &map_a, bar, kb * BK, w.tile_a * BM);
                    tma_load_2d(smem_u32(b_tiles + (size_t)s * B_BYTES), &map_b, bar, kb * BK, w.tile_b * BN);
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        // instruction descriptor: D 32-bit, A and B bfloat16, both K-major, N = BN, M = 128
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) |
                                   ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
        // (this warp's instructions are the products' pace: the stage and its phase are counted, the
        // descriptors of stage 0 are made once, and the k-block that overwrites the accumulator is
        // peeled off: see gemm_tc_pair_kernel)
        uint32_t n_done = 0;
        int s = 0;
        uint32_t phase = 0;
        bool first = true;
        const uint64_t a_desc0 = smem_desc(smem_u32(a_tiles)), b_desc0 = smem_desc(smem_u32(b_tiles));
        const uint32_t full0 = smem_u32(&full_bar[0]), empty0 = smem_u32(&empty_bar[0]);
        bool ok = true;
        for (int u = blockIdx.x; u < n_units && ok; u += gridDim.x, ++n_done) {
            Unit w = unit_of(u, tiles_a, splits);
            int kb_begin = w.split * kblocks_per_split;
            int kb_end = min(n_kblocks, kb_begin + kblocks_per_split);
            uint32_t buffer = n_done & 1, use = n_done >> 1;
            // the epilogue must have drained this buffer (its previous use)
            ok = mbar_wait_warp(smem_u32(&acc_empty_bar[buffer]), (use & 1) ^ 1, abort_flag, status, 4);
            if (!ok) break;
            tcgen05_fence_after();
            uint32_t d_tmem = tmem_base + buffer * BN;
            for (int kb = kb_begin; kb < kb_end; ++kb) {
                ok = mbar_wait_warp(full0 + 8 * s, phase, abort_flag, status, 2);
                if (!ok) break;
                if (first) { LLMB_STAMP(3, 32); first = false; }        // the first operand tiles have landed
                tcgen05_fence_after();
                uint64_t a_desc = a_desc0 + (uint64_t)(s * (A_BYTES >> 4));
                uint64_t b_desc = b_desc0 + (uint64_t)(s * (B_BYTES >> 4));
                if (elect_one()) {
                    // 16 k-values = 32 bytes further inside the swizzled row: +2 in 16-byte units
                    if (kb == kb_begin) {
                        tcgen05_mma(d_tmem, a_desc, b_desc, idesc, 0u);
#pragma unroll
                        for (int k = 1; k < BK / UMMA_K; ++k) tcgen05_mma(d_tmem, a_desc + 2 * k, b_desc + 2 * k, idesc, 1u);
                    } else {
#pragma unroll
                        for (int k = 0; k < BK / UMMA_K; ++k) tcgen05_mma(d_tmem, a_desc + 2 * k, b_desc + 2 * k, idesc, 1u);
                    }
                    tcgen05_commit(empty0 + 8 * s);
                    if (kb + 1 == kb_end) tcgen05_commit(smem_u32(&acc_full_bar[buffer]));
                }
                __syncwarp();
                if (++s == stages) { s = 0; phase ^= 1; }
            }
            LLMB_STAMP(4, 32);                                  // the unit's last product is issued
        }
    } else {
        int quarter = warp & 3;                          // the 32 lanes of tensor memory this warp may read
        int row = quarter * 32 + lane;                   // row of the tile = row of A
        uint32_t n_done = 0;
        for (int u = blockIdx.x; u < n_units; u += gridDim.x, ++n_done) {
            Unit w = unit_of(u, tiles_a, splits);
            uint32_t buffer = n_done & 1, use = n_done >> 1;
            // a folded norm: the scales of this tile's token rows, computed while the products run
            // (two buffers in turn and one barrier a unit: a warp that runs ahead writes the other one)
            const float* rstd = nullptr;
            if (ep.f.norm_sumsq) {
                tile_rstd(ep, rstd_s[n_done & 1], quarter, swap ? w.tile_b * BN : w.tile_a * BM,
                          swap ? (BN < BM ? BN : BM) : BM);
                asm volatile("bar.sync 1, 128;" ::: "memory");
                rstd = rstd_s[n_done & 1];
            }
            // a fused rotation: positions, pages and angles of the tile's tokens into shared memory
            // (read again only after this unit's epilogue, which ends with a barrier of these warps)
            if (BN == 16 && swap && splits > 1 && ep.f.rope) stage_rope(ep, rope_stage, w.tile_b * BN);
            accumulator_wait(smem_u32(&acc_full_bar[buffer]), use & 1, abort_flag, status);
            tcgen05_fence_after();
            uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buffer * BN;
            int a_row = w.tile_a * BM + row;             // swap: output column; else: token
            size_t tile_id = (size_t)w.tile_b * tiles_a + w.tile_a;
            if (splits == 1 && ep.glu && !swap) {
                float r = rstd ? rstd[row] : 1.f;
                // columns alternate 16 gate, 16 up: this thread's row gets 16 activations per pair
                __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(ep.out);
#pragma unroll 1
                for (int c = 0; c + 32 <= BN; c += 32) {
                    uint32_t g[16], u[16];
                    tmem_ld16(taddr + c, g);
                    tmem_ld16(taddr + c + 16, u);
                    int n0 = w.tile_b * BN + c;                      // first weight row of the pair
                    if (a_row < ep.tokens && n0 + 32 <= ep.outs) {
                        uint4 packed[2];
                        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(packed);
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            h[j] = __floats2bfloat162_rn(
                                gated(ep, __uint_as_float(g[2 * j]) * r, __uint_as_float(u[2 * j]) * r),
                                gated(ep, __uint_as_float(g[2 * j + 1]) * r, __uint_as_float(u[2 * j + 1]) * r));
                        __nv_bfloat16* dst = o + (size_t)a_row * ep.ldo + n0 / 2;
                        if ((ep.ldo & 7) == 0) {
                            reinterpret_cast<uint4*>(dst)[0] = packed[0];
                            reinterpret_cast<uint4*>(dst)[1] = packed[1];
                        } else {
                            const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(packed);
#pragma unroll
                            for (int j = 0; j < 16; ++j) dst[j] = e[j];
                        }
                    }
                }
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&acc_empty_bar[buffer]));
                continue;
            }
            if (splits == 1) {
#pragma unroll 1
                for (int c = 0; c < BN; c += 16) {
                    uint32_t r[16];
                    float v[16];
                    tmem_ld16(taddr + c, r);
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
                    store_columns<BN>(ep, swap, a_row, w.tile_b, c, v, nullptr, rstd, row);
                }
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&acc_empty_bar[buffer]));
                continue;
            }
            // split K: park the partial tile [BN columns][128 rows], free the accumulator, and
            // let the block that arrives last add all partials in split order
            float* mine = partials + (tile_id * splits + w.split) * (size_t)(BN * BM);
            int cols = swap ? min(BN, ep.tokens - w.tile_b * BN) : BN;      // columns that hold tokens: the rest is padding that nobody reads
#pragma unroll 1
            for (int c = 0; c < BN; c += 16) {
                uint32_t r[16];
                tmem_ld16(taddr + c, r);
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (c + j < cols) __stcg(mine + (size_t)(c + j) * BM + row, __uint_as_float(r[j]));
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty_bar[buffer]));
            if (sum_later) {
                LLMB_STAMP(5, 64);
                continue;                                           // the kernel's end publishes the partials
            }
            __threadfence();
            LLMB_STAMP(5, 64);                                      // the partial tile is written and fenced
            asm volatile("bar.sync 1, 128;" ::: "memory");          // the four epilogue warps
            if (threadIdx.x == 64) {
                unsigned arrived = atomicAdd(&counters[tile_id], 1u);
                *last_flag = arrived == (unsigned)(splits - 1);
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
            bool last = *last_flag != 0;     // the flag is next written after the next unit's first barrier
            LLMB_STAMP(6, 64);                                      // the tile's counter has answered
            if (!last) continue;
            __threadfence();
            const float* first = partials + tile_id * splits * (size_t)(BN * BM) + row;
#pragma unroll 1
            for (int c = 0; c < BN; c += 16) {
                float v[16], old[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = 0.f;
                // columns that hold tokens (swapped products: the rest of the 16 is padding)
                int valid = swap ? min(16, ep.tokens - (w.tile_b * BN + c)) : 16;
                // the residual's values first: their latency runs under the partials' loads
                bool preload = swap && ep.residual && !ep.glu && a_row < ep.outs;
                if (preload) {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        old[j] = j < valid ? ep.residual[(size_t)(w.tile_b * BN + c + j) * ep.ldo + a_row] : 0.f;
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) old[j] = 0.f;
                }
                // Partials are added in split order. With at most 8 valid columns, 8 splits' loads
                // are in flight at once (a decode step of up to 8 sequences sums 9 splits in two
                // rounds of loads instead of three over all 16 columns); else 4 splits of 16 columns.
                if (valid <= 8) {
                    for (int s0 = 0; s0 < splits; s0 += 8) {
                        float t[8][8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            bool live = s0 + i < splits;
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                t[i][j] = (live && j < valid) ? __ldcg(first + (size_t)(s0 + i) * (BN * BM) + (size_t)(c + j) * BM) : 0.f;
                        }
#pragma unroll
                        for (int i = 0; i < 8; ++i)
#pragma unroll
                            for (int j = 0; j < 8; ++j) v[j] += t[i][j];
                    }
                } else {
                    for (int s0 = 0; s0 < splits; s0 += 4) {
                        float t[4][16];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            bool live = s0 + i < splits;
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                t[i][j] = (live && j < valid) ? __ldcg(first + (size_t)(s0 + i) * (BN * BM) + (size_t)(c + j) * BM) : 0.f;
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i)
#pragma unroll
                            for (int j = 0; j < 16; ++j) v[j] += t[i][j];
                    }
                }
                if (swap && (ep.f.rope || ep.f.emit_rows)) {
                    // the fused decode epilogues (tiles of 16 tokens: this loop runs once)
                    if (rstd) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] *= rstd[c + j];
                    }
                    if (ep.f.rope) finish_rope(ep, a_row, row, w.tile_b * BN + c, valid, v, exch, rope_stage);
                    else finish_emit(ep, a_row, w.tile_a, w.tile_b * BN + c, valid, v, old, exch);
                } else {
                    store_columns<BN>(ep, swap, a_row, w.tile_b, c, v, preload ? old : nullptr, rstd, row);
                }
            }
            if (threadIdx.x == 64) counters[tile_id] = 0u;
            LLMB_STAMP(7, 64);                                      // the last arriver has summed and stored
        }
    }

    // teardown: everyone meets, then the allocating warp frees the tensor memory
    tcgen05_fence_before();
    __syncthreads();
    if (*abort_flag) {
        // let copies that are still in flight land before shared memory is given up
        for (int i = 0; i < 100; ++i) __nanosleep(10000);
        __syncthreads();
    }
    if (warp == 1) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// Sums the partial tiles of a swapped split-K product: one thread per (token, output feature),
// the splits added in order, then scale / bias / residual / store as the product's epilogue would;
// with a residual it can also leave the next norm's input (bfloat16 rows and one partial sum of
// squares per block of 256 features).
// Partials: [tile_b][tile_a][split][BN columns = tokens][128 rows = features].
__device__ __forceinline__ float split_sum(const float* partials, int tiles_a, int splits, int bn, int token,
                                           int weight_row) {
    size_t tile_floats = (size_t)bn * BM;
    int tile_a = weight_row / BM, row = weight_row % BM, tile_b = token / bn, col = token % bn;
    const float* p = partials + ((size_t)tile_b * tiles_a + tile_a) * splits * tile_floats + (size_t)col * BM + row;
    float v = 0.f;
    for (int s0 = 0; s0 < splits; s0 += 8) {
        float t[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) t[i] = s0 + i < splits ? __ldcg(p + (size_t)(s0 + i) * tile_floats) : 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) v += t[i];
    }
    return v;
}

__global__ void __launch_bounds__(256)
splitk_sum_kernel(const float* __restrict__ partials, Epilogue ep, int tiles_a, int splits, int bn) {
    griddep_launch();
    griddep_wait();
    __shared__ float scale_s;
    __shared__ float squares[8];
    int token = blockIdx.y;
    int feature = blockIdx.x * 256 + threadIdx.x;                  // with glu: the activated column
    int n_features = ep.glu ? ep.outs / 2 : ep.outs;
    if (ep.f.norm_sumsq) {
        if (threadIdx.x < 32) {
            float r = warp_row_rstd(ep.f, token);
            if (threadIdx.x == 0) scale_s = r;
        }
        __syncthreads();
    }
    float scale = ep.f.norm_sumsq ? scale_s : 1.f;
    float updated = 0.f;
    if (feature < n_features) {
        if (ep.glu) {
            // weight rows alternate 16 gate rows, 16 up rows
            int gate_row = (feature / LLMB_GLU_BLOCK) * 2 * LLMB_GLU_BLOCK + feature % LLMB_GLU_BLOCK;
            float gate = split_sum(partials, tiles_a, splits, bn, token, gate_row) * scale;
            float up = split_sum(partials, tiles_a, splits, bn, token, gate_row + LLMB_GLU_BLOCK) * scale;
            reinterpret_cast<__nv_bfloat16*>(ep.out)[(size_t)token * ep.ldo + feature] = __float2bfloat16_rn(gated(ep, gate, up));
        } else {
            float v = split_sum(partials, tiles_a, splits, bn, token, feature) * scale + (ep.bias ? ep.bias[feature] : 0.f);
            size_t at = (size_t)token * ep.ldo + feature;
            if (ep.residual) {
                updated = ep.residual[at] + v;
                ep.residual[at] = updated;
                if (ep.f.emit_rows) reinterpret_cast<__nv_bfloat16*>(ep.f.emit_rows)[at] = __float2bfloat16_rn(updated);
            } else if (ep.out_is_bf16) {
                reinterpret_cast<__nv_bfloat16*>(ep.out)[at] = __float2bfloat16_rn(v);
            } else {
                reinterpret_cast<float*>(ep.out)[at] = v;
            }
        }
    }
    if (ep.f.emit_sumsq) {                                          // uniform over the block
        float sq = warp_sum(updated * updated);
        if ((threadIdx.x & 31) == 0) squares[threadIdx.x >> 5] = sq;
        __syncthreads();
        if (threadIdx.x == 0) {
            float total = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) total += squares[i];
            ep.f.emit_sumsq[(size_t)token * LLMB_SUMSQ_LD + blockIdx.x] = total;
        }
    }
}

// The same sum, four neighbouring features a thread and four tokens a block (rows and strides that
// allow 16-byte accesses): every thread has its shares' loads and its residual in flight together, and a
// quarter of the blocks pass through the GPU. With one value a thread the sum of a 512 x 4,096 product
// took 27 us for 34 MB, each of its 8,192 small blocks a chain of three trips to memory.
__device__ __forceinline__ float4 split_sum4(const float* partials, int tiles_a, int splits, int bn, int token,
                                             int weight_row) {
    size_t tile_floats = (size_t)bn * BM;
    int tile_a = weight_row / BM, row = weight_row % BM, tile_b = token / bn, col = token % bn;
    const float4* p = reinterpret_cast<const float4*>(
        partials + ((size_t)tile_b * tiles_a + tile_a) * splits * tile_floats + (size_t)col * BM + row);
    size_t stride = tile_floats / 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s0 = 0; s0 < splits; s0 += 8) {
        float4 t[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) t[i] = s0 + i < splits ? __ldcg(p + (size_t)(s0 + i) * stride) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            v.x += t[i].x;
            v.y += t[i].y;
            v.z += t[i].z;
            v.w += t[i].w;
        }
    }
    return v;
}

__device__ __forceinline__ uint2 pack4(float a, float b, float c, float d) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
    uint2 r;
    r.x = *reinterpret_cast<uint32_t*>(&lo);
    r.y = *reinterpret_cast<uint32_t*>(&hi);
    return r;
}

__global__ void __launch_bounds__(256)
splitk_sum4_kernel(const float* __restrict__ partials, Epilogue ep, int tiles_a, int splits, int bn) {
    griddep_launch();
    griddep_wait();
    __shared__ float scale_s[4];
    __shared__ float squares[4][2];
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int slot = threadIdx.x >> 6;                                   // which of the block's four tokens
    int token = blockIdx.y * 4 + slot;
    int feature = blockIdx.x * 256 + (threadIdx.x & 63) * 4;       // with glu: the activated column
    int n_features = ep.glu ? ep.outs / 2 : ep.outs;
    if (ep.f.norm_sumsq) {
        if (warp < 4) {
            int t = blockIdx.y * 4 + warp;
            float r = t < ep.tokens ? warp_row_rstd(ep.f, t) : 1.f;
            if (lane == 0) scale_s[warp] = r;
        }
        __syncthreads();
    }
    float scale = ep.f.norm_sumsq ? scale_s[slot] : 1.f;
    float sq = 0.f;
    if (token < ep.tokens && feature < n_features) {
        if (ep.glu) {
            // weight rows alternate 16 gate rows, 16 up rows; four neighbours stay inside a block of 16
            int gate_row = (feature / LLMB_GLU_BLOCK) * 2 * LLMB_GLU_BLOCK + feature % LLMB_GLU_BLOCK;
            float4 g = split_sum4(partials, tiles_a, splits, bn, token, gate_row);
            float4 u = split_sum4(partials, tiles_a, splits, bn, token, gate_row + LLMB_GLU_BLOCK);
            *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(ep.out) + (size_t)token * ep.ldo + feature) =
                pack4(gated(ep, g.x * scale, u.x * scale), gated(ep, g.y * scale, u.y * scale),
                      gated(ep, g.z * scale, u.z * scale), gated(ep, g.w * scale, u.w * scale));
        } else {
            float4 v = split_sum4(partials, tiles_a, splits, bn, token, feature);
            float4 b = ep.bias ? *reinterpret_cast<const float4*>(ep.bias + feature) : make_float4(0.f, 0.f, 0.f, 0.f);
            v.x = v.x * scale + b.x;
            v.y = v.y * scale + b.y;
            v.z = v.z * scale + b.z;
            v.w = v.w * scale + b.w;
            size_t at = (size_t)token * ep.ldo + feature;
            if (ep.residual) {
                float4 r = *reinterpret_cast<const float4*>(ep.residual + at);
                r.x += v.x;
                r.y += v.y;
                r.z += v.z;
                r.w += v.w;
                *reinterpret_cast<float4*>(ep.residual + at) = r;
                if (ep.f.emit_rows)
                    *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(ep.f.emit_rows) + at) = pack4(r.x, r.y, r.z, r.w);
                sq = fmaf(r.w, r.w, fmaf(r.z, r.z, fmaf(r.y, r.y, r.x * r.x)));
            } else if (ep.out_is_bf16) {
                *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(ep.out) + at) = pack4(v.x, v.y, v.z, v.w);
            } else {
                *reinterpret_cast<float4*>(reinterpret_cast<float*>(ep.out) + at) = v;
            }
        }
    }
    if (ep.f.emit_sumsq) {                                          // uniform over the block
        sq = warp_sum(sq);
        if (lane == 0) squares[slot][warp & 1] = sq;
        __syncthreads();
        if (threadIdx.x < 4 && blockIdx.y * 4 + threadIdx.x < ep.tokens)
            ep.f.emit_sumsq[(size_t)(blockIdx.y * 4 + threadIdx.x) * LLMB_SUMSQ_LD + blockIdx.x] =
                squares[threadIdx.x][0] + squares[threadIdx.x][1];
    }
}

// The same sum for the q/k/v product with the rotation and the cache write behind it (see finish_rope):
// one thread per (token, item); an item is a rotation pair of a query or key head, or one value of a v head.
__global__ void __launch_bounds__(256)
splitk_sum_rope_kernel(const float* __restrict__ partials, Epilogue ep, int tiles_a, int splits, int bn) {
    griddep_launch();
    griddep_wait();
    __shared__ float scale_s;
    const llmb_gemm_fusion& f = ep.f;
    int token = blockIdx.y;
    int dim = f.head_dim, half = dim >> 1;
    int n_pairs = (f.n_heads + f.n_kv_heads) * half;
    int n_items = n_pairs + f.n_kv_heads * dim;
    int item = blockIdx.x * 256 + threadIdx.x;
    if (f.norm_sumsq) {
        if (threadIdx.x < 32) {
            float r = warp_row_rstd(f, token);
            if (threadIdx.x == 0) scale_s = r;
        }
        __syncthreads();
    }
    float scale = f.norm_sumsq ? scale_s : 1.f;
    if (item >= n_items) return;
    int pos = f.tok_pos[token];
    size_t cache_row = 0;
    if (f.write_cache) {
        int page = f.block_table[(size_t)f.tok_seq[token] * f.table_stride + ((pos / LLMB_PAGE) % f.ring_pages)];
        cache_row = ((size_t)page * f.n_kv_heads) * LLMB_PAGE + (pos % LLMB_PAGE);      // + kv_head * 64, times dim
    }
    __nv_bfloat16* q_out = reinterpret_cast<__nv_bfloat16*>(ep.out) + (size_t)token * ep.ldo;
    if (item < n_pairs) {
        int head = item / half, pair = item - head * half;
        int e0 = f.interleaved ? 2 * pair : pair, e1 = f.interleaved ? 2 * pair + 1 : pair + half;
        int row0 = head * dim + e0, row1 = head * dim + e1;
        float lo = split_sum(partials, tiles_a, splits, bn, token, row0) * scale + (ep.bias ? ep.bias[row0] : 0.f);
        float hi = split_sum(partials, tiles_a, splits, bn, token, row1) * scale + (ep.bias ? ep.bias[row1] : 0.f);
        if (f.rope_table) {
            float c = f.rope_table[(size_t)pos * dim + pair], s = f.rope_table[(size_t)pos * dim + half + pair];
            float a = lo * c - hi * s, b = lo * s + hi * c;
            lo = a;
            hi = b;
        }
        if (head < f.n_heads) {
            q_out[row0] = __float2bfloat16_rn(lo);
            q_out[row1] = __float2bfloat16_rn(hi);
        } else if (f.write_cache) {
            __nv_bfloat16* k = reinterpret_cast<__nv_bfloat16*>(f.k_cache) +
                               (cache_row + (size_t)(head - f.n_heads) * LLMB_PAGE) * dim;
            k[e0] = __float2bfloat16_rn(lo);
            k[e1] = __float2bfloat16_rn(hi);
        }
    } else if (f.write_cache) {
        int rest = item - n_pairs;
        int kv_head = rest / dim, e = rest - kv_head * dim;
        int row = (f.n_heads + f.n_kv_heads + kv_head) * dim + e;
        float v = split_sum(partials, tiles_a, splits, bn, token, row) * scale + (ep.bias ? ep.bias[row] : 0.f);
        reinterpret_cast<__nv_bfloat16*>(f.v_cache)[(cache_row + (size_t)kv_head * LLMB_PAGE) * dim + e] = __float2bfloat16_rn(v);
    }
}

// The same with four neighbouring rotation pairs (or four values of a v head) a thread and four tokens a
// block, as splitk_sum4_kernel (head sizes that are multiples of 8, rows that allow 8-byte stores).
__global__ void __launch_bounds__(256)
splitk_sum_rope4_kernel(const float* __restrict__ partials, Epilogue ep, int tiles_a, int splits, int bn) {
    griddep_launch();
    griddep_wait();
    __shared__ float scale_s[4];
    const llmb_gemm_fusion& f = ep.f;
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int slot = threadIdx.x >> 6;
    int token = blockIdx.y * 4 + slot;
    int dim = f.head_dim, half = dim >> 1;
    int n_pair_quads = (f.n_heads + f.n_kv_heads) * half / 4;
    int n_quads = n_pair_quads + f.n_kv_heads * dim / 4;
    int quad = blockIdx.x * 64 + (threadIdx.x & 63);
    if (f.norm_sumsq) {
        if (warp < 4) {
            int t = blockIdx.y * 4 + warp;
            float r = t < ep.tokens ? warp_row_rstd(f, t) : 1.f;
            if (lane == 0) scale_s[warp] = r;
        }
        __syncthreads();
    }
    float scale = f.norm_sumsq ? scale_s[slot] : 1.f;
    if (token >= ep.tokens || quad >= n_quads) return;
    int pos = f.tok_pos[token];
    size_t cache_row = 0;
    if (f.write_cache) {
        int page = f.block_table[(size_t)f.tok_seq[token] * f.table_stride + ((pos / LLMB_PAGE) % f.ring_pages)];
        cache_row = ((size_t)page * f.n_kv_heads) * LLMB_PAGE + (pos % LLMB_PAGE);      // + kv_head * 64, times dim
    }
    auto biased = [&](float4 v, int row) {
        float4 b = ep.bias ? *reinterpret_cast<const float4*>(ep.bias + row) : make_float4(0.f, 0.f, 0.f, 0.f);
        return make_float4(v.x * scale + b.x, v.y * scale + b.y, v.z * scale + b.z, v.w * scale + b.w);
    };
    __nv_bfloat16* q_out = reinterpret_cast<__nv_bfloat16*>(ep.out) + (size_t)token * ep.ldo;
    if (quad < n_pair_quads) {
        int item = quad * 4;                                         // the first of four pairs of one head
        int head = item / half, pair = item - head * half;
        // rows of the four pairs: (pair .. pair + 3) and the same half a head on, or 2 pair .. 2 pair + 7
        int row0 = head * dim + (f.interleaved ? 2 * pair : pair);
        int row1 = f.interleaved ? row0 + 4 : row0 + half;
        float4 a = biased(split_sum4(partials, tiles_a, splits, bn, token, row0), row0);
        float4 b = biased(split_sum4(partials, tiles_a, splits, bn, token, row1), row1);
        float lo[4], hi[4];
        if (f.interleaved) {
            lo[0] = a.x; hi[0] = a.y; lo[1] = a.z; hi[1] = a.w;
            lo[2] = b.x; hi[2] = b.y; lo[3] = b.z; hi[3] = b.w;
        } else {
            lo[0] = a.x; lo[1] = a.y; lo[2] = a.z; lo[3] = a.w;
            hi[0] = b.x; hi[1] = b.y; hi[2] = b.z; hi[3] = b.w;
        }
        if (f.rope_table) {
            float4 c4 = *reinterpret_cast<const float4*>(f.rope_table + (size_t)pos * dim + pair);
            float4 s4 = *reinterpret_cast<const float4*>(f.rope_table + (size_t)pos * dim + half + pair);
            const float c[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float x = lo[i] * c[i] - hi[i] * sn[i], y = lo[i] * sn[i] + hi[i] * c[i];
                lo[i] = x;
                hi[i] = y;
            }
        }
        __nv_bfloat16* dst = nullptr;
        if (head < f.n_heads) dst = q_out + (size_t)head * dim;
        else if (f.write_cache)
            dst = reinterpret_cast<__nv_bfloat16*>(f.k_cache) + (cache_row + (size_t)(head - f.n_heads) * LLMB_PAGE) * dim;
        if (dst) {
            if (f.interleaved) {
                *reinterpret_cast<uint2*>(dst + 2 * pair) = pack4(lo[0], hi[0], lo[1], hi[1]);
                *reinterpret_cast<uint2*>(dst + 2 * pair + 4) = pack4(lo[2], hi[2], lo[3], hi[3]);
            } else {
                *reinterpret_cast<uint2*>(dst + pair) = pack4(lo[0], lo[1], lo[2], lo[3]);
                *reinterpret_cast<uint2*>(dst + half + pair) = pack4(hi[0], hi[1], hi[2], hi[3]);
            }
        }
    } else if (f.write_cache) {
        int rest = (quad - n_pair_quads) * 4;
        int kv_head = rest / dim, e = rest - kv_head * dim;
        int row = (f.n_heads + f.n_kv_heads + kv_head) * dim + e;
        float4 v = biased(split_sum4(partials, tiles_a, splits, bn, token, row), row);
        *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(f.v_cache) + (cache_row + (size_t)kv_head * LLMB_PAGE) * dim + e) =
            pack4(v.x, v.y, v.z, v.w);
    }
}

// ------------------------------------------------------------------------- two SMs on one tile
// For large token counts the 128 x 256 tile above is held back by shared-memory fill: per
// k-block it loads 48 KB for 524 tensor-core cycles. Two blocks of a cluster (a CTA pair on
// neighbouring SMs) computing one 256 x 256 tile with tcgen05.mma.cta_group::2 halve the
// weight traffic per SM: each block loads its own 128 token rows and only half (128 rows) of
// the weight tile, and the instruction reads both halves. Block 0 of the pair issues the
// instructions for both; each block keeps its 128 x 256 half of the accumulator in its own
// tensor memory and runs its own epilogue.
//
// Barriers: both producers' TMA loads report their bytes to block 0's `full` barrier (the
// .cta_group::2 form of the load allows a barrier in the partner block); tcgen05.commit with
// a multicast mask frees the stage in both blocks and announces the accumulator to both
// epilogues; all eight epilogue warps of the pair arrive on block 0's `acc_empty`.

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t cluster_bar,
                                                 int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(cluster_bar), "r"(x), "r"(y) : "memory");
}
// `mask`: the blocks of the cluster whose barrier at this place is signalled
__device__ __forceinline__ void tcgen05_commit_pair(uint32_t bar, uint16_t mask = 3) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
        ::"r"(bar), "h"(mask) : "memory");
}
__device__ __forceinline__ void tcgen05_mma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                                 uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8, %9, %10, %11, %12}, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate),
          "r"(0u), "r"(0u), "r"(0u), "r"(0u), "r"(0u), "r"(0u), "r"(0u), "r"(0u) : "memory");
}

constexpr int PAIRS = 74;           // of SMs
constexpr int PAIR_BN = 256;        // columns of the pair's tile; each block loads half of them

// The order in which the pairs take the tiles. The 74 tiles that run at the same time read their
// operands' k-blocks at about the same time, so an operand tile that several of them share comes from
// HBM once. With the token tile running fastest over all tiles (unit_of) a long prompt's 74 tiles
// share ONE weight tile and read 74 different token tiles: at 65,536 tokens and K = 2,048 that is
// 74 MB per 10 us, more than HBM delivers (products of a 263,000-token prefill ran at half their
// rate). So the token tiles are taken in panels of 8: inside a panel the token tile runs fastest,
// then the weight tile, then the next panel. A round of 74 tiles then reads 8 token tiles and about 9
// weight tiles.
constexpr int PANEL = 8;
__device__ __forceinline__ Unit pair_unit_of(int u, int tiles_a, int tiles_b) {
    Unit w;
    w.split = 0;
    int per_panel = PANEL * tiles_b;
    int panel = u / per_panel;
    int first = panel * PANEL;
    int width = min(PANEL, tiles_a - first);          // the last panel may be narrower
    int r = u - panel * per_panel;
    w.tile_b = r / width;
    w.tile_a = first + (r - w.tile_b * width);
    return w;
}

// What the pairs do. The first n_full tiles (a multiple of the pairs, or all of them) run whole, one a pair and round. The
// tail_tiles that are left would keep only some of the pairs busy for a whole tile's time, so their k-blocks, laid one
// tile behind the other, are cut into pieces of tail_len (at most a tile's own number), one a pair: a pair gets the end of
// one tile and the start of the next, or one part. Where a tile has several parts, each is left in scratch, and a kernel
// behind (pair_tail_sum_kernel) adds them in the order of k and does what the epilogue would. (The block that brought the
// last part doing that alone, 128 threads reading 128 KB a part, took some 30 us.)
struct PairWork {
    int n_kblocks, tiles_a, tiles_b, n_full, tail_tiles, tail_len;
};
struct PairPiece {
    int tile_a, tile_b, k0, k1;      // the tile and its k-blocks [k0, k1)
    int tail;                        // the tile's number among the tail's, or -1: the whole tile
};
// The i-th piece of pair `pair`; false: there is none.
__device__ __forceinline__ bool pair_piece(const PairWork& w, int pair, int n_pairs, int i, PairPiece& p) {
    int u = pair + i * n_pairs;
    p.k0 = 0;
    p.k1 = w.n_kblocks;
    p.tail = -1;
    if (u >= w.n_full) {
        int done = w.n_full / n_pairs;                  // whole tiles of this pair (n_full is a multiple, where there is a tail)
        int begin = pair * w.tail_len, end = min(begin + w.tail_len, w.tail_tiles * w.n_kblocks);
        if (w.tail_tiles == 0 || begin >= end) return false;
        int t = begin / w.n_kblocks + (i - done), at = t * w.n_kblocks;
        if (at >= end) return false;
        p.k0 = max(begin - at, 0);
        p.k1 = min(end - at, w.n_kblocks);
        if (p.k0 > 0 || p.k1 < w.n_kblocks) p.tail = t;
        u = w.n_full + t;
    }
    Unit unit = pair_unit_of(u, w.tiles_a, w.tiles_b);
    p.tile_a = unit.tile_a;
    p.tile_b = unit.tile_b;
    return true;
}
// A piece's place in scratch: two a pair, 256 x 256 values each, the halves of the pair's blocks one after the other, four
// columns of a row together and the rows side by side (what a warp stores or loads at once is 512 bytes on end).
constexpr int PIECE_FLOATS = 2 * BM * PAIR_BN;
__device__ __forceinline__ float* piece_of(float* partials, const PairWork& w, int pair, int tail, uint32_t rank) {
    int which = tail - pair * w.tail_len / w.n_kblocks;
    return partials + (size_t)(pair * 2 + which) * PIECE_FLOATS + rank * (BM * PAIR_BN);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const __grid_constant__ CUtensorMap map_residual, Epilogue ep, PairWork work, float* partials,
                    int* status, int stages, int residual_by_tma) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    constexpr int A_BYTES = BM * BK * 2, B_BYTES = (PAIR_BN / 2) * BK * 2;
    constexpr int TMEM_COLS = 2 * PAIR_BN;
    unsigned char* base = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* a_tiles = base;
    unsigned char* b_tiles = base + (size_t)stages * A_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(b_tiles + (size_t)stages * B_BYTES);
    uint64_t* full_bar = bars;
    uint64_t* empty_bar = bars + stages;
    uint64_t* acc_full_bar = bars + 2 * stages;
    uint64_t* acc_empty_bar = bars + 2 * stages + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * stages + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    __shared__ float rstd_s[2][BM];                   // scales of this block's 128 token rows (a folded norm)
    // Adding into the residual: accumulator pieces of 128 rows x 32 columns leave through two 16 KB
    // staging buffers behind the ring, and the copy engine adds them into the 32-bit matrix
    // (cp.reduce.async.bulk.tensor). Reading the old values into registers, 64 bytes a lane and one
    // chunk after the other, cost the last tile of every block some 16 us of load latency.
    float* staging = reinterpret_cast<float*>(base + (size_t)stages * (A_BYTES + B_BYTES) + 1024);

    const int warp = warp_index(), lane = threadIdx.x & 31;
    uint32_t rank = cluster_rank();
    int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&acc_full_bar[b]), 1);
            mbar_init(smem_u32(&acc_empty_bar[b]), 8);          // four epilogue warps in each block
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync();                                   // the partner's barriers exist from here on
    tcgen05_fence_after();
    uint32_t tmem_base = *tmem_slot;

    // As in gemm_tc_kernel: the first weight tiles (operand B here) are fetched while the kernel
    // before this one may still be running; the tokens only after griddep_wait().
    griddep_launch();
    uint32_t early = 0;
    PairPiece p;
    if (warp == 0 && pair_piece(work, pair, n_pairs, 0, p)) {
        early = (uint32_t)min(stages, p.k1 - p.k0);
        if (elect_one()) {
            for (uint32_t i = 0; i < early; ++i) {
                if (rank == 0) mbar_expect_tx(smem_u32(&full_bar[i]), 2 * (A_BYTES + B_BYTES));
                uint32_t bar = map_to_rank(smem_u32(&full_bar[i]), 0);
                tma_load_2d_pair(smem_u32(b_tiles + (size_t)i * B_BYTES), &map_b, bar, (p.k0 + (int)i) * BK,
                                 p.tile_b * PAIR_BN + (int)rank * (PAIR_BN / 2));
            }
        }
        __syncwarp();
    }
    griddep_wait();

    if (warp == 0) {
        const uint32_t full_of_0 = map_to_rank(smem_u32(&full_bar[0]), 0);      // both blocks' bytes are counted on block 0's barriers
        uint32_t it = 0;
        int s = 0;
        uint32_t round = 0;                                     // how often the ring has been walked through
        bool ok = true;
        for (int i = 0; ok && pair_piece(work, pair, n_pairs, i, p); ++i) {
            const int a_row = p.tile_a * 2 * BM + (int)rank * BM, b_row = p.tile_b * PAIR_BN + (int)rank * (PAIR_BN / 2);
            for (int kb = p.k0; kb < p.k1; ++kb, ++it, s = (s + 1 == stages ? 0 : s + 1), round += (s == 0)) {
                if (it < early) {                               // armed above, the weight tile is in flight
                    if (elect_one()) tma_load_2d_pair(smem_u32(a_tiles + (size_t)s * A_BYTES), &map_a, full_of_0 + 8 * s, kb * BK, a_row);
                    __syncwarp();
                    continue;
                }
                ok = mbar_wait_warp(smem_u32(&empty_bar[s]), (round & 1) ^ 1, abort_flag, status, 1);
                if (!ok) break;
                if (elect_one()) {
                    if (rank == 0) mbar_expect_tx(smem_u32(&full_bar[s]), 2 * (A_BYTES + B_BYTES));
                    tma_load_2d_pair(smem_u32(a_tiles + (size_t)s * A_BYTES), &map_a, full_of_0 + 8 * s, kb * BK, a_row);
                    tma_load_2d_pair(smem_u32(b_tiles + (size_t)s * B_BYTES), &map_b, full_of_0 + 8 * s, kb * BK, b_row);
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // D 32-bit, A and B bfloat16, both K-major, N = 256, M = 256 over the pair
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) |
                                       ((uint32_t)(PAIR_BN >> 3) << 17) | ((uint32_t)((2 * BM) >> 4) << 24);
            // This warp's instructions are the products' pace: per k-block it waits for a barrier and its elected lane
            // issues four instructions and a commit, 512 cycles of the tensor cores. Nothing in the loop divides, reads a
            // clock or builds a descriptor from scratch: the stage and its phase are counted, the descriptors of stage 0
            // are made once and a stage adds a constant, and the first k-block (which overwrites the accumulator) is
            // peeled off so that the others accumulate unconditionally. Cycles a k-block: 616 with the loop run by one lane
            // (67 wait, 277 for the four, 72 commit), 520 run by the warp.
            uint32_t n_done = 0;
            int s = 0;
            uint32_t phase = 0;
            const uint64_t a_desc0 = smem_desc(smem_u32(a_tiles)), b_desc0 = smem_desc(smem_u32(b_tiles));
            const uint32_t full0 = smem_u32(&full_bar[0]), empty0 = smem_u32(&empty_bar[0]);
            bool ok = true;
            for (; ok && pair_piece(work, pair, n_pairs, (int)n_done, p); ++n_done) {
                uint32_t buffer = n_done & 1, use = n_done >> 1;
                ok = mbar_wait_warp(smem_u32(&acc_empty_bar[buffer]), (use & 1) ^ 1, abort_flag, status, 4);
                if (!ok) break;
                tcgen05_fence_after();
                uint32_t d_tmem = tmem_base + buffer * PAIR_BN;
                for (int kb = p.k0; kb < p.k1; ++kb) {
                    ok = mbar_wait_warp(full0 + 8 * s, phase, abort_flag, status, 2);
                    if (!ok) break;
                    tcgen05_fence_after();
                    uint64_t a_desc = a_desc0 + (uint64_t)(s * (A_BYTES >> 4));
                    uint64_t b_desc = b_desc0 + (uint64_t)(s * (B_BYTES >> 4));
                    if (elect_one()) {
                        if (kb == p.k0) {
                            tcgen05_mma_pair(d_tmem, a_desc, b_desc, idesc, 0u);
#pragma unroll
                            for (int k = 1; k < BK / UMMA_K; ++k) tcgen05_mma_pair(d_tmem, a_desc + 2 * k, b_desc + 2 * k, idesc, 1u);
                        } else {
#pragma unroll
                            for (int k = 0; k < BK / UMMA_K; ++k) tcgen05_mma_pair(d_tmem, a_desc + 2 * k, b_desc + 2 * k, idesc, 1u);
                        }
                        tcgen05_commit_pair(empty0 + 8 * s);           // frees the stage in both blocks
                        if (kb + 1 == p.k1) tcgen05_commit_pair(smem_u32(&acc_full_bar[buffer]));
                    }
                    __syncwarp();
                    if (++s == stages) { s = 0; phase ^= 1; }
                }
            }
        }
    } else {
        int quarter = warp & 3;
        int row = quarter * 32 + lane;
        uint32_t n_done = 0;
        for (; pair_piece(work, pair, n_pairs, (int)n_done, p); ++n_done) {
            uint32_t buffer = n_done & 1, use = n_done >> 1;
            const float* rstd = nullptr;
            if (ep.f.norm_sumsq) {                    // as in gemm_tc_kernel: while the products run
                tile_rstd(ep, rstd_s[n_done & 1], quarter, p.tile_a * 2 * BM + (int)rank * BM, BM);
                asm volatile("bar.sync 1, 128;" ::: "memory");
                rstd = rstd_s[n_done & 1];
            }
            accumulator_wait(smem_u32(&acc_full_bar[buffer]), use & 1, abort_flag, status);
            tcgen05_fence_after();
            uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buffer * PAIR_BN;
            int a_row = p.tile_a * 2 * BM + (int)rank * BM + row;
            if (p.tail >= 0) {                            // a part of a tile: the sums as they are
                float* mine = piece_of(partials, work, pair, p.tail, rank) + row * 4;
#pragma unroll 1
                for (int c = 0; c < PAIR_BN; c += 32) {
                    uint32_t r[32];
                    tmem_ld32(taddr + c, r);
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        __stcg(reinterpret_cast<float4*>(mine + (size_t)(c + 4 * q) * BM),
                               make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                                           __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3])));
                }
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_remote(map_to_rank(smem_u32(&acc_empty_bar[buffer]), 0));
                continue;
            }
            if (ep.glu) {
                float r = rstd ? rstd[row] : 1.f;
                __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(ep.out);
#pragma unroll 1
                for (int c = 0; c < PAIR_BN; c += 32) {
                    uint32_t g[16], uu[16];
                    tmem_ld16(taddr + c, g);
                    tmem_ld16(taddr + c + 16, uu);
                    int n0 = p.tile_b * PAIR_BN + c;
                    if (a_row < ep.tokens && n0 + 32 <= ep.outs) {
                        uint4 packed[2];
                        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(packed);
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            h[j] = __floats2bfloat162_rn(
                                gated(ep, __uint_as_float(g[2 * j]) * r, __uint_as_float(uu[2 * j]) * r),
                                gated(ep, __uint_as_float(g[2 * j + 1]) * r, __uint_as_float(uu[2 * j + 1]) * r));
                        __nv_bfloat16* dst = o + (size_t)a_row * ep.ldo + n0 / 2;
                        if ((ep.ldo & 7) == 0) {
                            reinterpret_cast<uint4*>(dst)[0] = packed[0];
                            reinterpret_cast<uint4*>(dst)[1] = packed[1];
                        } else {
                            const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(packed);
#pragma unroll
                            for (int j = 0; j < 16; ++j) dst[j] = e[j];
                        }
                    }
                }
            } else if (residual_by_tma) {
                float scale = rstd ? rstd[row] : 1.f;
                int tile_row0 = p.tile_a * 2 * BM + (int)rank * BM;
#pragma unroll 1
                for (int c = 0; c < PAIR_BN; c += 32) {
                    uint32_t r[32];
                    tmem_ld32(taddr + c, r);
                    int n0 = p.tile_b * PAIR_BN + c;
                    float* buffer_s = staging + ((c >> 5) & 1) * (BM * 32);
                    // the copy that last read this buffer (two pieces ago) must be done with it
                    if (threadIdx.x == 64) bulk_wait_read<1>();
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (n0 < ep.outs) {
                        // row `row` of the piece: eight 16-byte chunks, chunk q at place q ^ (row % 8)
                        // (the 128-byte swizzle of the tensor map; also spreads the lanes over the banks)
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            float4 piece;
                            piece.x = __uint_as_float(r[4 * q]) * scale;
                            piece.y = __uint_as_float(r[4 * q + 1]) * scale;
                            piece.z = __uint_as_float(r[4 * q + 2]) * scale;
                            piece.w = __uint_as_float(r[4 * q + 3]) * scale;
                            if (ep.bias) {
                                int n = n0 + 4 * q;
                                piece.x += n < ep.outs ? ep.bias[n] : 0.f;
                                piece.y += n + 1 < ep.outs ? ep.bias[n + 1] : 0.f;
                                piece.z += n + 2 < ep.outs ? ep.bias[n + 2] : 0.f;
                                piece.w += n + 3 < ep.outs ? ep.bias[n + 3] : 0.f;
                            }
                            *reinterpret_cast<float4*>(buffer_s + row * 32 + ((q ^ (row & 7)) << 2)) = piece;
                        }
                    }
                    fence_async_shared();
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (threadIdx.x == 64) {
                        if (n0 < ep.outs && tile_row0 < ep.tokens)
                            tma_reduce_add_2d(&map_residual, smem_u32(buffer_s), n0, tile_row0);
                        bulk_commit();
                    }
                }
            } else {
#pragma unroll 1
                for (int c = 0; c < PAIR_BN; c += 16) {
                    uint32_t r[16];
                    float v[16];
                    tmem_ld16(taddr + c, r);
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
                    store_columns<PAIR_BN>(ep, 0, a_row, p.tile_b, c, v, nullptr, rstd, row);
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(map_to_rank(smem_u32(&acc_empty_bar[buffer]), 0));
        }
    }

    if (threadIdx.x == 64) bulk_wait<0>();            // the copy engine is done with the staging buffers
    tcgen05_fence_before();
    __syncthreads();
    if (*abort_flag) {
        for (int i = 0; i < 100; ++i) __nanosleep(10000);
        __syncthreads();
    }
    cluster_sync();                                   // nobody leaves while the partner may still signal it
    if (warp == 1) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// The tiles that the pairs left in parts. A block takes 64 rows and 64 columns of one tile; a warp 8 rows, a lane four
// columns of one row in each of four column groups of 16 (its loads fall together to 128 bytes, its stores to 32 or 64): the
// parts added in the order of k, then the row's scale, the bias, and the store, the sum or the gated activation.
__global__ void __launch_bounds__(256)
pair_tail_sum_kernel(float* partials, Epilogue ep, PairWork work) {
    __shared__ float rstd[64];
    griddep_launch();
    griddep_wait();
    int tail = blockIdx.x, first_part = tail * work.n_kblocks / work.tail_len;
    int parts = ((tail + 1) * work.n_kblocks - 1) / work.tail_len - first_part + 1;
    if (parts == 1) return;                                        // one pair ran the whole tile
    Unit unit = pair_unit_of(work.n_full + tail, work.tiles_a, work.tiles_b);
    int rows = (blockIdx.y >> 2) * 64, cols = (blockIdx.y & 3) * 64;
    int token0 = unit.tile_a * 2 * BM + rows, n0 = unit.tile_b * PAIR_BN + cols;
    if (token0 >= ep.tokens || n0 >= ep.outs) return;
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int row = warp * 8 + (lane >> 2), quad = (lane & 3) * 4;       // of the block's rows; of a group's columns
    int at = rows + row;
    float4 sum[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) sum[g] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
    for (int i = 0; i < parts; ++i) {
        const float* from = piece_of(partials, work, first_part + i, tail, at / BM) + (at % BM) * 4;
        float4 v[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) v[g] = __ldcg(reinterpret_cast<const float4*>(from + (size_t)(cols + g * 16 + quad) * BM));
#pragma unroll
        for (int g = 0; g < 4; ++g) { sum[g].x += v[g].x; sum[g].y += v[g].y; sum[g].z += v[g].z; sum[g].w += v[g].w; }
    }
    float scale = 1.f;
    if (ep.f.norm_sumsq) {
        if (threadIdx.x < 64) rstd[threadIdx.x] = token0 + (int)threadIdx.x < ep.tokens ? thread_row_rstd(ep.f, token0 + threadIdx.x) : 1.f;
        __syncthreads();
        scale = rstd[row];
    }
    int token = token0 + row;
    if (token >= ep.tokens) return;
    if (ep.glu) {
        __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(ep.out) + (size_t)token * ep.ldo + n0 / 2 + quad;
        bool wide = (ep.ldo & 3) == 0 && (reinterpret_cast<uintptr_t>(ep.out) & 7) == 0;
#pragma unroll
        for (int g = 0; g < 4; g += 2) {
            if (n0 + g * 16 + 32 > ep.outs) break;
            float a[4] = {gated(ep, sum[g].x * scale, sum[g + 1].x * scale), gated(ep, sum[g].y * scale, sum[g + 1].y * scale),
                          gated(ep, sum[g].z * scale, sum[g + 1].z * scale), gated(ep, sum[g].w * scale, sum[g + 1].w * scale)};
            if (wide) {
                __nv_bfloat162 lo = __floats2bfloat162_rn(a[0], a[1]), hi = __floats2bfloat162_rn(a[2], a[3]);
                *reinterpret_cast<uint2*>(o + g * 8) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
            } else {
                for (int j = 0; j < 4; ++j) o[g * 8 + j] = __float2bfloat16_rn(a[j]);
            }
        }
        return;
    }
    const void* target = ep.residual ? (const void*)ep.residual : ep.out;
    bool wide = (ep.ldo & 3) == 0 && (reinterpret_cast<uintptr_t>(target) & 15) == 0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        int n = n0 + g * 16 + quad;
        float v[4] = {sum[g].x * scale, sum[g].y * scale, sum[g].z * scale, sum[g].w * scale};
        if (ep.bias) {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] += n + j < ep.outs ? ep.bias[n + j] : 0.f;
        }
        size_t place = (size_t)token * ep.ldo + n;
        if (wide && n + 4 <= ep.outs) {
            if (ep.residual) {
                float4* r = reinterpret_cast<float4*>(ep.residual + place);
                float4 old = *r;
                *r = make_float4(old.x + v[0], old.y + v[1], old.z + v[2], old.w + v[3]);
            } else if (ep.out_is_bf16) {
                __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
                *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(ep.out) + place) =
                    make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
            } else {
                *reinterpret_cast<float4*>(reinterpret_cast<float*>(ep.out) + place) = make_float4(v[0], v[1], v[2], v[3]);
            }
            continue;
        }
        for (int j = 0; j < 4 && n + j < ep.outs; ++j) {
            if (ep.residual) ep.residual[place + j] += v[j];
            else if (ep.out_is_bf16) reinterpret_cast<__nv_bfloat16*>(ep.out)[place + j] = __float2bfloat16_rn(v[j]);
            else reinterpret_cast<float*>(ep.out)[place + j] = v[j];
        }
    }
}

// ------------------------------------------------------------------------- weights on the pair's row side
// From some tokens to some thousand, 256 x 256 tiles with the tokens as rows are too coarse: 350 tokens fill 512 rows, a
// 4,096-wide output has 32 tiles for 74 pairs, and a tile takes its 18 us (64 k-blocks) whatever the other pairs do. Here the
// weights are the 256 rows of a pair's tile and the tokens its N side, whose width (64 to 256, a multiple of 32) is chosen
// so that the tokens fill it; and where the tiles are too few, `splits` pairs of one cluster share a tile, each with a
// slice of its k-blocks. Their accumulators meet in shared memory: when every pair of the cluster is done, each block
// writes the columns that another one finishes into that block's (now empty) operand ring, and after one cluster barrier
// every block adds its share of the columns in the order of k and runs the epilogue on it. (Partial tiles through global
// memory and a second kernel cost some 12 us a product.)
//
// The epilogue turns the tile around: a thread holds one output column (weight row) of 16 tokens at a time and writes
// them to a staging buffer [16 tokens][128 outputs], from which the copy engine stores (or adds, 32-bit residual) whole rows;
// tokens and outputs beyond the matrix are dropped by its bounds. Targets that a tensor map cannot describe are stored directly.
struct WideWork {
    int n_kblocks, tiles_t, tiles_w, bn, splits;      // token tiles of bn, weight tiles of 256
};

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];"
                 ::"l"(map), "r"(src), "r"(x), "r"(y) : "memory");
}

__global__ void __launch_bounds__(THREADS, 1)
gemm_tc_wide_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                    const __grid_constant__ CUtensorMap map_out, Epilogue ep, WideWork work, int* status, int stages,
                    int out_by_tma) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    constexpr int A_BYTES = BM * BK * 2;
    const int bn = work.bn, B_BYTES = (bn / 2) * BK * 2;
    unsigned char* base = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* a_tiles = base;
    unsigned char* b_tiles = base + (size_t)stages * A_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(b_tiles + (size_t)stages * B_BYTES);
    uint64_t* full_bar = bars;
    uint64_t* empty_bar = bars + stages;
    uint64_t* acc_full_bar = bars + 2 * stages;
    uint64_t* acc_empty_bar = bars + 2 * stages + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * stages + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    unsigned char* staging = base + (size_t)stages * (A_BYTES + B_BYTES) + 1024;       // two buffers of [16][128] values
    __shared__ float rstd_s[2][PAIR_BN];                // scales of a tile's tokens (a folded norm)

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const uint32_t cluster = cluster_rank(), rank = cluster & 1, lead = cluster & ~1u;
    const int split = (int)(cluster >> 1), splits = work.splits;
    const int n_units = work.tiles_t * work.tiles_w;
    const int n_teams = (int)gridDim.x / (2 * splits), team = (int)blockIdx.x / (2 * splits);
    const int k_begin = work.n_kblocks * split / splits, k_end = work.n_kblocks * (split + 1) / splits;
    int tmem_cols = 32;
    while (tmem_cols < (splits > 1 ? bn : 2 * bn)) tmem_cols *= 2;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&acc_full_bar[b]), 1);
            mbar_init(smem_u32(&acc_empty_bar[b]), 8);          // four epilogue warps in each block of the pair
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync();                                   // the partner's barriers exist from here on
    tcgen05_fence_after();
    uint32_t tmem_base = *tmem_slot;

    // As in gemm_tc_kernel: the first weight tiles (operand A here) are fetched while the kernel before this one may still be
    // running; the tokens only after griddep_wait().
    griddep_launch();
    uint32_t early = 0;
    if (warp == 0 && team < n_units) {
        Unit w = pair_unit_of(team, work.tiles_t, work.tiles_w);
        early = (uint32_t)min(stages, k_end - k_begin);
        if (elect_one()) {
            for (uint32_t i = 0; i < early; ++i) {
                if (rank == 0) mbar_expect_tx(smem_u32(&full_bar[i]), 2 * (A_BYTES + B_BYTES));
                tma_load_2d_pair(smem_u32(a_tiles + (size_t)i * A_BYTES), &map_w, map_to_rank(smem_u32(&full_bar[i]), lead),
                                 (k_begin + (int)i) * BK, w.tile_b * 2 * BM + (int)rank * BM);
            }
        }
        __syncwarp();
    }
    griddep_wait();

    if (warp == 0) {
        const uint32_t full_of_lead = map_to_rank(smem_u32(&full_bar[0]), lead);     // both blocks' bytes are counted there
        uint32_t it = 0;
        int s = 0;
        uint32_t round = 0;                                     // how often the ring has been walked through
        bool ok = true;
        for (int u = team; u < n_units && ok; u += n_teams) {
            Unit w = pair_unit_of(u, work.tiles_t, work.tiles_w);
            const int x_row = w.tile_a * bn + (int)rank * (bn / 2), w_row = w.tile_b * 2 * BM + (int)rank * BM;
            for (int kb = k_begin; kb < k_end; ++kb, ++it, s = (s + 1 == stages ? 0 : s + 1), round += (s == 0)) {
                const bool armed = it < early;                  // above, and the weight tile is in flight
                if (!armed) {
                    ok = mbar_wait_warp(smem_u32(&empty_bar[s]), (round & 1) ^ 1, abort_flag, status, 1);
                    if (!ok) break;
                }
                if (elect_one()) {
                    const uint32_t bar = full_of_lead + 8 * s;
                    if (!armed && rank == 0) mbar_expect_tx(smem_u32(&full_bar[s]), 2 * (A_BYTES + B_BYTES));
                    if (!armed) tma_load_2d_pair(smem_u32(a_tiles + (size_t)s * A_BYTES), &map_w, bar, kb * BK, w_row);
                    tma_load_2d_pair(smem_u32(b_tiles + (size_t)s * B_BYTES), &map_x, bar, kb * BK, x_row);
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // D 32-bit, A and B bfloat16, both K-major, N = bn, M = 256 over the pair (the loop as in gemm_tc_pair_kernel)
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) |
                                   ((uint32_t)(bn >> 3) << 17) | ((uint32_t)((2 * BM) >> 4) << 24);
            const uint16_t mask = (uint16_t)(3u << lead);
            uint32_t n_done = 0;
            int s = 0;
            uint32_t phase = 0;
            const uint64_t a_desc0 = smem_desc(smem_u32(a_tiles)), b_desc0 = smem_desc(smem_u32(b_tiles));
            const uint32_t full0 = smem_u32(&full_bar[0]), empty0 = smem_u32(&empty_bar[0]);
            const uint32_t b_step = (uint32_t)B_BYTES >> 4;
            bool ok = true;
            for (int u = team; u < n_units && ok; u += n_teams, ++n_done) {
                uint32_t buffer = n_done & 1, use = n_done >> 1;
                ok = mbar_wait_warp(smem_u32(&acc_empty_bar[buffer]), (use & 1) ^ 1, abort_flag, status, 4);
                if (!ok) break;
                tcgen05_fence_after();
                uint32_t d_tmem = tmem_base + buffer * bn;
                for (int kb = k_begin; kb < k_end; ++kb) {
                    ok = mbar_wait_warp(full0 + 8 * s, phase, abort_flag, status, 2);
                    if (!ok) break;
                    tcgen05_fence_after();
                    uint64_t a_desc = a_desc0 + (uint64_t)(s * (A_BYTES >> 4));
                    uint64_t b_desc = b_desc0 + (uint64_t)(s * b_step);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < BK / UMMA_K; ++k)
                            tcgen05_mma_pair(d_tmem, a_desc + 2 * k, b_desc + 2 * k, idesc, k > 0 || kb > k_begin);
                        tcgen05_commit_pair(empty0 + 8 * s, mask);     // frees the stage in both blocks
                        if (kb + 1 == k_end) tcgen05_commit_pair(smem_u32(&acc_full_bar[buffer]), mask);
                    }
                    __syncwarp();
                    if (++s == stages) { s = 0; phase ^= 1; }
                }
            }
        }
        __syncwarp();
    }

    const int quarter = warp & 3, row = quarter * 32 + lane, n_chunks = bn / 16;
    // Sixteen tokens of this thread's output column: scale, bias, then out. c: the first token's column in the tile.
    uint32_t turn = 0;                                  // which staging buffer is next
    auto finish = [&](const Unit& w, int c, float (&v)[16], const float* rstd) {
        int token0 = w.tile_a * bn + c, n0 = w.tile_b * 2 * BM + (int)rank * BM, n = n0 + row;
        if (rstd) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] *= rstd[c + j];
        }
        if (!out_by_tma) {
            store_columns<16>(ep, 1, n, 0, token0, v);
            return;
        }
        unsigned char* buffer = staging + (turn & 1) * (16 * BM * 4);
        ++turn;
        if (threadIdx.x == 64) bulk_wait_read<1>();     // the copy that last read this buffer is done with it
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (ep.glu) {
            // lanes 0-15 hold 16 gate rows, lanes 16-31 the up rows of the same features: the halves exchange so that a
            // gate lane gets the even tokens of its feature and an up lane the odd ones
            __nv_bfloat16* to = reinterpret_cast<__nv_bfloat16*>(buffer) + quarter * 16 + (lane & 15);
#pragma unroll
            for (int j = 0; j < 16; j += 2) {
                float other = __shfl_xor_sync(0xffffffffu, lane < 16 ? v[j + 1] : v[j], 16);
                float a = lane < 16 ? gated(ep, v[j], other) : gated(ep, other, v[j + 1]);
                to[(j + (lane >> 4)) * (BM / 2)] = __float2bfloat16_rn(a);
            }
        } else {
            float b = ep.bias && n < ep.outs ? ep.bias[n] : 0.f;
            if (ep.residual || !ep.out_is_bf16) {
                float* to = reinterpret_cast<float*>(buffer) + row;
#pragma unroll
                for (int j = 0; j < 16; ++j) to[j * BM] = v[j] + b;
            } else {
                __nv_bfloat16* to = reinterpret_cast<__nv_bfloat16*>(buffer) + row;
#pragma unroll
                for (int j = 0; j < 16; ++j) to[j * BM] = __float2bfloat16_rn(v[j] + b);
            }
        }
        fence_async_shared();
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (threadIdx.x == 64) {
            if (n0 < ep.outs && token0 < ep.tokens) {
                if (ep.residual) tma_reduce_add_2d(&map_out, smem_u32(buffer), n0, token0);
                else tma_store_2d(&map_out, smem_u32(buffer), ep.glu ? n0 / 2 : n0, token0);
            }
            bulk_commit();
        }
    };
    auto scales = [&](const Unit& w, uint32_t n_done) -> const float* {
        if (!ep.f.norm_sumsq) return nullptr;           // as in gemm_tc_kernel: while the products run
        tile_rstd(ep, rstd_s[n_done & 1], quarter, w.tile_a * bn, bn);
        asm volatile("bar.sync 1, 128;" ::: "memory");
        return rstd_s[n_done & 1];
    };

    if (splits == 1) {
        if (warp >= 2) {
            uint32_t n_done = 0;
            for (int u = team; u < n_units; u += n_teams, ++n_done) {
                Unit w = pair_unit_of(u, work.tiles_t, work.tiles_w);
                uint32_t buffer = n_done & 1, use = n_done >> 1;
                const float* rstd = scales(w, n_done);
                accumulator_wait(smem_u32(&acc_full_bar[buffer]), use & 1, abort_flag, status);
                tcgen05_fence_after();
                uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buffer * bn;
#pragma unroll 1
                for (int chunk = 0; chunk < n_chunks; ++chunk) {
                    uint32_t r[16];
                    float v[16];
                    tmem_ld16(taddr + chunk * 16, r);
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
                    finish(w, chunk * 16, v, rstd);
                }
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_remote(map_to_rank(smem_u32(&acc_empty_bar[buffer]), lead));
            }
        }
    } else {
        // one tile a cluster (n_units == n_teams). Block `split` of either half finishes the chunks [first, last).
        Unit w = pair_unit_of(team, work.tiles_t, work.tiles_w);
        const int first = n_chunks * split / splits, last = n_chunks * (split + 1) / splits;
        const float* rstd = nullptr;
        if (warp >= 2) {
            rstd = scales(w, 0);
            accumulator_wait(smem_u32(&acc_full_bar[0]), 0, abort_flag, status);
            tcgen05_fence_after();
        }
        __syncwarp();
        cluster_sync();                                 // every pair's products are done: the rings may be written over
        uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16);
        // a chunk's values from one pair: [4][128 rows] of four neighbouring columns
        const int slot = (n_chunks + splits - 1) / splits * 16 * BM;     // floats a pair sends to one block at most
        const uint32_t ring = smem_u32(base);
        if (warp >= 2) {
            for (int to = 0; to < splits; ++to) {
                if (to == split) continue;
                int its_first = n_chunks * to / splits, its_last = n_chunks * (to + 1) / splits;
                uint32_t there = map_to_rank(ring, (uint32_t)(2 * to) + rank) + (uint32_t)(split * slot + row * 4) * 4;
#pragma unroll 1
                for (int chunk = its_first; chunk < its_last; ++chunk) {
                    uint32_t r[16];
                    tmem_ld16(taddr + chunk * 16, r);
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};"
                                     ::"r"(there + (uint32_t)((((chunk - its_first) * 4 + q) * BM) * 16)),
                                       "r"(r[4 * q]), "r"(r[4 * q + 1]), "r"(r[4 * q + 2]), "r"(r[4 * q + 3]) : "memory");
                }
            }
        }
        __syncwarp();
        cluster_sync();
        if (warp >= 2) {
            const float4* mine = reinterpret_cast<const float4*>(base) + row;
#pragma unroll 1
            for (int chunk = first; chunk < last; ++chunk) {
                uint32_t r[16];
                float v[16];
                tmem_ld16(taddr + chunk * 16, r);
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = 0.f;
                for (int from = 0; from < splits; ++from) {              // in the order of k
                    if (from == split) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(r[j]);
                        continue;
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        float4 p = mine[from * (slot / 4) + ((chunk - first) * 4 + q) * BM];
                        v[4 * q] += p.x;
                        v[4 * q + 1] += p.y;
                        v[4 * q + 2] += p.z;
                        v[4 * q + 3] += p.w;
                    }
                }
                finish(w, chunk * 16, v, rstd);
            }
        }
        __syncwarp();
    }

    if (threadIdx.x == 64) bulk_wait<0>();            // the copy engine is done with the staging buffers
    tcgen05_fence_before();
    __syncthreads();
    if (*abort_flag) {
        for (int i = 0; i < 100; ++i) __nanosleep(10000);
        __syncthreads();
    }
    cluster_sync();                                   // nobody leaves while the partner may still signal it
    if (warp == 1) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
}

// ------------------------------------------------------------------------- host side

// rows x K bfloat16, K contiguous with `ld` elements between rows; box 64 x box_rows, 128-byte swizzle
int make_map(CUtensorMap* map, const void* ptr, long long rows, long long k, long long ld, int box_rows) {
    return make_map_2d(map, ptr, rows, k, ld, BK, box_rows);
}

// Whether a swapped split-K product leaves the sum to splitk_sum_kernel: from 17 tokens. Up to 16
// tokens both ways measured the same on a decode step (4.87 ms at batch 8), at 64 tokens the
// kernel of its own is far ahead (O projection 21.8 -> 12.0 us).
inline int sums_later(int swap, int splits, int bn) { return (swap && splits > 1 && bn >= 32) ? 1 : 0; }

template <int BN>
int launch(const CUtensorMap& map_a, const CUtensorMap& map_b, const Epilogue& ep, int swap,
           int tiles_a, int tiles_b, int n_kblocks, int per_split, int splits, float* partials,
           unsigned* counters, cudaStream_t stream) {
    constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2;
    int stages = (200 * 1024) / (A_BYTES + B_BYTES);
    if (stages > 8) stages = 8;
    int blocks_per_sm = 1;
    // the fused decode epilogues exchange values through shared memory behind the control words:
    // 64 floats for the sums of squares, 16 x 128 for rotation pairs that sit half a head apart
    size_t exchange = 256;
    if (swap && BN == 16 && splits > 1 && ep.f.rope) exchange = (size_t)16 * BM * 4 + sizeof(RopeStage);
    if (swap) {                                         // two blocks per SM for the decode stream
        stages = (int)((110 * 1024 - (exchange > 256 ? exchange : 0)) / (A_BYTES + B_BYTES));
        if (stages > 6) stages = 6;
        blocks_per_sm = 2;
    }
    size_t smem = 1024 + (size_t)stages * (A_BYTES + B_BYTES) + (2 * stages + 4) * 8 + 16 + exchange;
    static size_t configured = 0;
    if (smem > configured) {
        LLMB_CUDA(cudaFuncSetAttribute(gemm_tc_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured = smem;
    }
    static int n_sms = 0;
    if (n_sms == 0) {
        int device = 0;
        LLMB_CUDA(cudaGetDevice(&device));
        LLMB_CUDA(cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, device));
    }
    int* status = status_word();
    int* status_dev = nullptr;
    if (status) cudaHostGetDevicePointer((void**)&status_dev, status, 0);
    int n_units = tiles_a * tiles_b * splits;
    int grid = n_units < n_sms * blocks_per_sm ? n_units : n_sms * blocks_per_sm;
    int sum_later = sums_later(swap, splits, BN);
    llmb::launch(gemm_tc_kernel<BN>, grid, THREADS, smem, stream, true, map_a, map_b, ep, swap, n_kblocks, per_split,
                 splits, tiles_a, n_units, partials, counters, status_dev, stages, sum_later);
    int code = check_launch("gemm_tc");
    if (code || !sum_later) return code;
    auto aligned = [](const void* p, uintptr_t to) { return (reinterpret_cast<uintptr_t>(p) & (to - 1)) == 0; };
    if (ep.f.rope) {
        int n_items = (ep.f.n_heads + ep.f.n_kv_heads) * (ep.f.head_dim / 2) + ep.f.n_kv_heads * ep.f.head_dim;
        if (ep.f.head_dim % 8 == 0 && ep.ldo % 4 == 0 && aligned(ep.out, 8) && aligned(ep.bias, 16) &&
            aligned(ep.f.k_cache, 8) && aligned(ep.f.v_cache, 8) && aligned(ep.f.rope_table, 16)) {
            llmb::launch(splitk_sum_rope4_kernel, dim3((n_items / 4 + 63) / 64, (ep.tokens + 3) / 4), 256, 0, stream, true,
                         (const float*)partials, ep, tiles_a, splits, BN);
            return check_launch("gemm_tc (split-K sum with rotation, four pairs a thread)");
        }
        llmb::launch(splitk_sum_rope_kernel, dim3((n_items + 255) / 256, ep.tokens), 256, 0, stream, true,
                     (const float*)partials, ep, tiles_a, splits, BN);
        return check_launch("gemm_tc (split-K sum with rotation)");
    }
    int n_features = ep.glu ? ep.outs / 2 : ep.outs;
    bool by_fours = n_features % 4 == 0 && ep.ldo % 4 == 0 && aligned(ep.out, ep.out_is_bf16 ? 8 : 16) &&
                    aligned(ep.residual, 16) && aligned(ep.bias, 16) && aligned(ep.f.emit_rows, 8);
    if (by_fours) {
        llmb::launch(splitk_sum4_kernel, dim3((n_features + 255) / 256, (ep.tokens + 3) / 4), 256, 0, stream, true,
                     (const float*)partials, ep, tiles_a, splits, BN);
        return check_launch("gemm_tc (split-K sum, four features a thread)");
    }
    llmb::launch(splitk_sum_kernel, dim3((n_features + 255) / 256, ep.tokens), 256, 0, stream, true,
                 (const float*)partials, ep, tiles_a, splits, BN);
    return check_launch("gemm_tc (split-K sum)");
}

int launch_pair(const CUtensorMap& map_a, const CUtensorMap& map_b, const Epilogue& ep, const PairWork& work, int n_pairs,
                float* partials, cudaStream_t stream) {
    constexpr int STAGE_BYTES = BM * BK * 2 + (PAIR_BN / 2) * BK * 2;
    int stages = (192 * 1024) / STAGE_BYTES;
    if (stages > 8) stages = 8;
    // ring | 1 KB: barriers and control words | two staging buffers of 128 rows x 32 floats for the
    // residual epilogue (1024-byte aligned, as the swizzle wants)
    size_t smem = 1024 + (size_t)stages * STAGE_BYTES + 1024 + 2 * (size_t)BM * 32 * 4;
    static bool configured = false;
    if (!configured) {
        LLMB_CUDA(cudaFuncSetAttribute(gemm_tc_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured = true;
    }
    // the residual through the copy engine where a tensor map can describe it
    CUtensorMap map_residual = map_a;
    int residual_by_tma = 0;
    if (ep.residual && !ep.glu && ep.ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(ep.residual) & 15) == 0) {
        int code = make_map_2d_f32(&map_residual, ep.residual, ep.tokens, ep.outs, ep.ldo, BM);
        if (code) return code;
        residual_by_tma = 1;
    }
    int* status = status_word();
    int* status_dev = nullptr;
    if (status) cudaHostGetDevicePointer((void**)&status_dev, status, 0);
    llmb::launch(gemm_tc_pair_kernel, 2 * n_pairs, THREADS, smem, stream, true, map_a, map_b, map_residual, ep, work, partials,
                 status_dev, stages, residual_by_tma);
    int code = check_launch("gemm_tc_pair");
    if (code || work.tail_tiles == 0) return code;
    llmb::launch(pair_tail_sum_kernel, dim3(work.tail_tiles, 16), 256, 0, stream, true, partials, ep, work);
    return check_launch("gemm_tc_pair (the sums of the last round)");
}

int launch_wide(const void* x, int ldx, const void* w, const Epilogue& ep, const WideWork& work, int M, int N, int K,
                cudaStream_t stream) {
    CUtensorMap map_w, map_x, map_out;
    int code;
    if ((code = make_map(&map_w, w, N, K, K, BM))) return code;
    if ((code = make_map(&map_x, x, M, K, ldx, work.bn / 2))) return code;
    // ring | 1 KB: barriers and control words | two staging buffers of 16 tokens x 128 outputs
    const size_t stage_bytes = (size_t)BM * BK * 2 + (size_t)(work.bn / 2) * BK * 2, staging = 2 * 16 * BM * 4;
    int stages = (int)(204 * 1024 / stage_bytes);
    if (stages > 10) stages = 10;
    size_t smem = 1024 + stages * stage_bytes + 1024 + staging;
    static bool configured = false;
    if (!configured) {                                  // (every width's ring fits into what the widest takes and 227 KB hold)
        LLMB_CUDA(cudaFuncSetAttribute(gemm_tc_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 1024 + 204 * 1024 + 1024 + (int)staging));
        configured = true;
    }
    // the target as a tensor map, where one can describe it (boxes of one block's outputs x 16 tokens, no swizzle)
    map_out = map_w;
    bool wide = ep.residual || !ep.out_is_bf16;
    void* target = ep.residual ? (void*)ep.residual : ep.out;
    int columns = ep.glu ? N / 2 : N, out_by_tma = 0;
    if (ep.ldo % (wide ? 4 : 8) == 0 && (reinterpret_cast<uintptr_t>(target) & 15) == 0) {
        if ((code = make_map_plain(&map_out, target, wide, M, columns, ep.ldo, ep.glu ? BM / 2 : BM, 16))) return code;
        out_by_tma = 1;
    }
    int* status = status_word();
    int* status_dev = nullptr;
    if (status) cudaHostGetDevicePointer((void**)&status_dev, status, 0);
    int units = work.tiles_t * work.tiles_w, teams = work.splits > 1 || units < PAIRS ? units : PAIRS;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(teams * 2 * work.splits);
    config.blockDim = dim3(THREADS);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeClusterDimension;
    attributes[0].val.clusterDim.x = 2 * work.splits;
    attributes[0].val.clusterDim.y = attributes[0].val.clusterDim.z = 1;
    attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attributes;
    config.numAttrs = pdl_enabled() ? 2 : 1;
    LLMB_CUDA(cudaLaunchKernelEx(&config, gemm_tc_wide_kernel, map_w, map_x, map_out, ep, work, status_dev, stages, out_by_tma));
    return check_launch("gemm_tc_wide");
}

struct Plan {
    int swap, bn, tiles_a, tiles_b, n_kblocks, per_split, splits;
};

// The weights take the 128-row side of the tiles (tokens in tiles of up to 128 on the other) and K is split over blocks up to
// 128 tokens, and up to 1,024 tokens where 256 x 256 tiles are too few for the pairs of SMs even when cut along K. (With the
// tokens on the 128-row side a 128 x 4096 x 4096 product has 16 tiles and took 38 us; this way it takes 14. At 512 x 6144 x
// 4096 the 48 pair tiles are faster again: 27 against 32 us.)
constexpr int SWAP_TOKENS = 128, SWAP_TOKENS_MOST = 1024;

// How the pairs share the tiles (PairWork). A tile takes 0.35 us a k-block whatever the other pairs do, so a last round of R of
// 74 tiles wastes (74 - R) / 74 of it. Cut into pieces (multiples of four k-blocks, at least an eighth of a tile) it takes
// R / 74 of a tile's time, but leaving the parts and adding them in a kernel behind takes about 12 us, 34 k-blocks (30 when the line
// was drawn, at 0.4 us a k-block), and the pairs, each at another k, no longer share what they read, about a third of a piece. The cut
// is made where it saves more than 30 and that. Measured, whole tiles -> cut, with the norm's input behind a residual: 1300 x 4096 x
// 14336 (96 tiles) 178 -> 139 us, 2500 x 4096 x 14336 (160) 287 -> 231, 256 x 6144 x 4096 (24) 32.2 -> 29.4, 350 x 28672 x 4096 gated (224)
// 106 -> 99, and long gated ones about even at the power cap, 2048 x 28672 x 4096 (896) 351 -> 350, 3001 (1,344) 529 -> 535; not cut
// because slower: 512 x 4096 x 4096 (32) 29.4 -> 33.8, 2048 x 4096 x 14336 (128) 203 -> 205, 2048 x 6144 x 4096 (192) 81 -> 91.
PairWork plan_pairs(int M, int N, int K, int* n_pairs) {
    PairWork w;
    w.n_kblocks = (K + BK - 1) / BK;
    w.tiles_a = (M + 2 * BM - 1) / (2 * BM);
    w.tiles_b = (N + PAIR_BN - 1) / PAIR_BN;
    long long units = (long long)w.tiles_a * w.tiles_b;
    int rest = (int)(units % PAIRS);
    int length = (int)(((long long)rest * w.n_kblocks + PAIRS - 1) / PAIRS), least = (w.n_kblocks + 7) / 8;
    length = ((length > least ? length : least) + 3) / 4 * 4;
    if (rest > 0 && w.n_kblocks - length > 30 + (3 * length) / 10) {
        w.n_full = (int)(units - rest);
        w.tail_tiles = rest;
        w.tail_len = length;
        *n_pairs = w.n_full > 0 ? PAIRS : (rest * w.n_kblocks + length - 1) / length;
    } else {
        w.n_full = (int)units;
        w.tail_tiles = 0;
        w.tail_len = 1;
        *n_pairs = units < PAIRS ? (int)units : PAIRS;
    }
    return w;
}
bool on_pairs(const Plan& p, int M, int N) { return !p.swap && M > 128 && N >= 256; }

Plan make_plan(int M, int N, int K) {
    Plan p;
    p.n_kblocks = (K + BK - 1) / BK;
    long long pair_tiles = (long long)((M + 255) / 256) * ((N + 255) / 256);
    // (a pair's tile of 64 k-blocks takes 18 us alone, whatever fills the other pairs: with a short K the pairs win from some 24
    // tiles on, 512 x 6144 x 4096 in 27.3 against 31.8 us, 700 x 3072 x 2048 in 16.9 against 18.8; with a long K the split products
    // stay ahead until the pairs are well filled, 350 x 4096 x 14336 in 48 us against 59. What leaves the next norm's input in its
    // sum is ahead longer, 512 x 4096 x 4096 in 25.1 against 27.7 and 1000 x 2048 x 8192 in 38.6 against 43.3: the row side has most of those)
    bool few_tiles = p.n_kblocks <= 64 ? pair_tiles < 24 : pair_tiles * 5 < PAIRS * 3;
    p.swap = M <= SWAP_TOKENS || (M <= SWAP_TOKENS_MOST && few_tiles);
    if (p.swap) {
        p.bn = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
        p.tiles_a = (N + BM - 1) / BM;
        p.tiles_b = (M + p.bn - 1) / p.bn;
        // all blocks resident at once (two per SM): a second, partly filled wave would
        // double the time of a product this short
        int want = (2 * 148) / (p.tiles_a * p.tiles_b);
        int most = p.n_kblocks / 4 > 0 ? p.n_kblocks / 4 : 1; // at least four k-blocks a block
        if (want > most) want = most;
        if (want > 32) want = 32;
        if (want == 9 || want == 10) want = 8;      // the last block of a tile sums eight splits in one round of loads
        if (want < 1) want = 1;
        p.per_split = (p.n_kblocks + want - 1) / want;
        p.splits = (p.n_kblocks + p.per_split - 1) / p.per_split;
    } else {
        p.bn = N >= 256 ? 256 : N > 64 ? 128 : 64;
        p.tiles_a = (M + BM - 1) / BM;
        p.tiles_b = (N + p.bn - 1) / p.bn;
        p.per_split = p.n_kblocks;
        p.splits = 1;
    }
    return p;
}

// Where a product's results go: what an epilogue costs depends on it.
enum Target { TO_BF16, TO_F32, TO_RESIDUAL, TO_GATED };

// Whether a product runs with its weights on the pairs' row side, and how: the width of the token tiles and the pairs a tile, if any,
// whose estimate is below the other kernels' by 4 %, provided that it stays so when what leaves the tiles is counted. Estimates in us,
// from the measured times of 1,700 products of 129 to 2,100 tokens with 256 to 131,000 outputs and K from 64 to 16,384 (the layers'
// among them stand in profiles/gemm_tc__row_side_or_not.txt):
// * here, a round of 74 pairs takes 0.2 us a k-block up to 128 tokens a tile (the loads' pace) and 0.00151 us a token above, a call 4 us
//   more, or 8 where pairs share a tile; a gated tile's activations take 0.06 us a token, under the next round's products and
//   behind the last one's;
// * 256 x 256 tiles on pairs: 0.35 us a k-block and round, or, with the last round cut along K, 0.38 of the rounds' exact number (0.48
//   where there is no full one) and 12, and 6 for the last tiles' activations;
// * weights on one block's row side, tokens in tiles of 128: the weights at 6.5 TB/s, 1.4 ns a tile and k-block, 4.5 a call; it
//   leaves a norm's input or rotates in its sum, which takes a kernel of some 4 us behind this one;
// none faster than its weights at 5.5 TB/s. With a short K a round takes what its tiles need to leave: bfloat16 rows 1.8 us and 0.023 a
// token here and 5 there (9 the call), additions to the residual 1.25 and 0.022 (in a single round they are in its 4 us) and
// 5.5; 32-bit results are always faster here. Additions of more than 200 us stay there unless 12 % are in it, since at the power
// cap both ways end up together, and a gated round of more than 64 k-blocks against tiles on pairs took a third longer.
// Others -> here: 350 x 6144 x 4096 27.0 -> 19.3, 350 x 4096 x 4096 28.0 -> 18.4, 350 x 28672 x 4096 gated 101 -> 86, 350 x 4096 x 14336 47.5 ->
// 41.1, 600 x 4096 x 14336 85.9 -> 64.1, 1300 x 4096 x 4096 49.6 -> 39.1. Before what leaves was counted, short products of many
// outputs came here that are slower: 598 x 113152 x 128 107 -> 150, 855 x 24448 x 320 38 -> 51, 1365 x 16000 x 512 41 -> 51.
// Up to 128 tokens the sums' fused epilogues are worth more; a gated product, which has none, is faster here alone (64 x 16384 x
// 2048 18.5 -> 17.3), and a decode step of 64 sequences with it is not (2,558 -> 2,574 us): the kernel in front has its SMs longer.
bool plan_wide(int M, int N, int K, Target target, WideWork* best) {
    if (M <= SWAP_TOKENS || M > 2048 || N < 256) return false;
    Plan p = make_plan(M, N, K);
    const bool glu = target == TO_GATED;
    const int kblocks = p.n_kblocks, tiles_w = (N + 2 * BM - 1) / (2 * BM);
    const double weights = 2.0 * N * K * 1e-6, epilogue = glu ? 6.0 : 0.0, least = weights / 5.5 + 4.0 + epilogue;      // (bytes in MB, us)
    const double behind = p.swap && p.splits > 1 && !glu ? 4.0 : 0.0;
    // the other kernels, a round of whose 256 x 256 tiles takes `leave` at least
    auto others = [&](double leave) {
        double t;
        if (on_pairs(p, M, N)) {
            int n_pairs;
            PairWork w = plan_pairs(M, N, K, &n_pairs);
            const int units = w.tiles_a * w.tiles_b, rounds = (units + PAIRS - 1) / PAIRS;
            const double round = kblocks * 0.35;
            t = epilogue + (w.tail_tiles > 0 ? (double)units / PAIRS * kblocks * (units < PAIRS ? 0.48 : 0.38) + 12.0
                                             : rounds * (round > leave ? round : leave) + 4.0);
        } else {
            t = weights / 6.5 + 4.5 + epilogue + 0.0014 * p.tiles_a * p.tiles_b * kblocks;
        }
        return t > least ? t : least;
    };
    // this kernel, with tiles of bn tokens and `splits` pairs a tile
    auto here = [&](int bn, int splits, double leave, double slower) {
        const int units = (M + bn - 1) / bn * tiles_w, rounds = splits > 1 ? 1 : (units + PAIRS - 1) / PAIRS;
        const double last = glu ? 0.06 * bn : 0.0;
        double round = ((kblocks + splits - 1) / splits) * (bn <= 128 ? 0.2 : 0.00151 * bn) * slower;
        if (round < last) round = last;
        const double t = rounds * (round > leave ? round : leave) + (splits > 1 ? 8.0 : 4.0) + last;
        return (t > least ? t : least) + behind;
    };
    double lowest = others(0.0) / 1.04;
    bool found = false;
    for (int bn = 64; bn <= PAIR_BN; bn += 32) {
        const int tiles_t = (M + bn - 1) / bn, units = tiles_t * tiles_w;
        for (int splits = 1; splits <= 3; ++splits) {
            // (clusters of four blocks fit 34 times beside each other, of six 18 times; more would wait for a second wave)
            if (splits > 1 && (units > (splits == 2 ? 34 : 18) || kblocks < 8 * splits)) continue;
            const double t = here(bn, splits, 0.0, 1.0);
            if (t < lowest) {
                lowest = t;
                *best = WideWork{kblocks, tiles_t, tiles_w, bn, splits};
                found = true;
            }
        }
    }
    if (!found || target == TO_F32) return found;
    const bool one_round = best->splits > 1 || best->tiles_t * best->tiles_w <= PAIRS;
    const double leave = target == TO_BF16 ? 1.8 + 0.023 * best->bn : target == TO_RESIDUAL && !one_round ? 1.25 + 0.022 * best->bn : 0.0;
    double there = others(target == TO_BF16 ? 5.0 : target == TO_RESIDUAL ? 5.5 : 0.0);
    if (target == TO_BF16 && there < 9.0) there = 9.0;
    const double t = here(best->bn, best->splits, leave, glu && !p.swap && one_round && kblocks > 64 ? 1.3 : 1.0);
    return t * (target == TO_RESIDUAL && there > 200.0 ? 1.12 : 1.0) < there;
}

// Which kernel a product takes and what that kernel needs: the one answer that the launch and all questions about it share.
struct Choice {
    enum Kernel { BLOCKS, PAIRS_OF_SMS, ROW_SIDE } kernel;
    Plan plan;                          // BLOCKS
    PairWork pairs;                     // PAIRS_OF_SMS
    int n_pairs;
    WideWork wide;                      // ROW_SIDE
    long long scratch_floats;           // partial sums
    int counters, kernels;              // tile counters; kernels launched
    int emit_parts;                     // partial sums of squares a row (0: the kernels do not emit)
    bool can_rotate;                    // the q/k/v product's rotation, where its heads fit the tiles
};

Choice choose(int M, int N, int K, Target target, int allow_pair) {
    Choice c = {};
    c.kernels = 1;
    if (allow_pair && plan_wide(M, N, K, target, &c.wide)) {
        c.kernel = Choice::ROW_SIDE;
        return c;
    }
    const Plan p = c.plan = make_plan(M, N, K);
    if (allow_pair && on_pairs(p, M, N)) {
        c.kernel = Choice::PAIRS_OF_SMS;
        c.pairs = plan_pairs(M, N, K, &c.n_pairs);
        if (c.pairs.tail_tiles > 0) {
            c.scratch_floats = 2LL * c.n_pairs * PIECE_FLOATS;
            c.kernels = 2;
        }
        return c;
    }
    c.kernel = Choice::BLOCKS;
    if (p.splits > 1) {
        c.scratch_floats = (long long)p.tiles_a * p.tiles_b * p.splits * p.bn * BM;
        c.counters = p.tiles_a * p.tiles_b;
        c.kernels = 1 + sums_later(p.swap, p.splits, p.bn);
        if (p.swap) {
            const int parts = sums_later(p.swap, p.splits, p.bn) ? (N + 255) / 256 : p.tiles_a;
            c.emit_parts = parts <= LLMB_SUMSQ_LD ? parts : 0;
            c.can_rotate = true;
        }
    }
    return c;
}

}  // namespace

// 0 if nothing went wrong since the last call of this function; else the code of the
// wait that ran out (1 producer, 2 mma, 3 epilogue). Call after a synchronisation.
// The stamps of the last launches (a build with -DLLMB_TRACE): LLMB_TRACE_BLOCKS rows of
// LLMB_TRACE_SLOTS global-timer values, 0 where nothing was stamped. Returns 1 in a build without.
LLMB_EXPORT int llmb_gemm_tc_trace(unsigned long long* out, int clear) { return llmb_read_trace(out, clear); }

LLMB_EXPORT int llmb_gemm_tc_status() {
    int* s = status_word();
    if (!s) return -1;
    int v = *s;
    *s = 0;
    return v;
}

// What a call of these sizes does and needs, its results going to `target` (0 bfloat16, 1 float32, 2 the residual, 3 the gated
// activation in bfloat16): {kernel (0 blocks, 1 pairs, 2 row side), token or column width of its tiles, blocks
// or pairs that share a tile's K, tiles cut along K in the last round, floats of partial sums, tile counters, kernels launched,
// partial sums of squares a row that emit_rows / emit_sumsq leave (0: the caller runs llmb_cast_sumsq behind the product)}.
LLMB_EXPORT int llmb_gemm_tc_plan(int M, int N, int K, int target, int allow_pair, long long* out) {
    Choice c = choose(M, N, K, (Target)target, allow_pair);
    const bool blocks = c.kernel == Choice::BLOCKS, row_side = c.kernel == Choice::ROW_SIDE;
    const long long values[8] = {(long long)c.kernel, row_side ? c.wide.bn : blocks ? c.plan.bn : PAIR_BN,
                                 row_side ? c.wide.splits : blocks ? c.plan.splits : 1,
                                 c.kernel == Choice::PAIRS_OF_SMS ? c.pairs.tail_tiles : 0,
                                 c.scratch_floats, c.counters, c.kernels, c.emit_parts};
    for (int i = 0; i < 8; ++i) out[i] = values[i];
    return LLMB_OK;
}

// out[M, N] = x[M, K] . w[N, K]^T (+ bias[N]); or residual[M, N] += the same.
// allow_pair != 0: products with more than 128 rows run on pairs of SMs, as 256 x 256 tiles or with the weights on the row side.
// glu != 0: w holds gate and up rows alternating in blocks of 16 (N = 2 F rows, N % 32 == 0) and
// out is bfloat16 [M, ldo] with F columns act(gate) * up (1: silu, 2: the tanh form of gelu); no bias, no residual.
// fusion (optional): see fusion.h. *applied (optional) tells which parts ran inside the kernels:
// a folded norm always does; the rows and sums for the next norm and the rotation with the cache
// write only where the shape's kernels have them, else the caller runs them as kernels of their own.
LLMB_EXPORT int llmb_gemm_tc_ex(const void* x, int ldx, const void* w, const float* bias, void* out,
                                int out_dtype, float* residual, float* partials, long long partial_floats,
                                unsigned* counters, int n_counters, int M, int N, int K, int ldo, int glu,
                                int allow_pair, const llmb_gemm_fusion* fusion, int* applied,
                                cudaStream_t stream) {
    if (applied) *applied = 0;
    if (M == 0 || N == 0) return LLMB_OK;
    LLMB_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_tc: bad sizes");
    LLMB_REQUIRE(K % 8 == 0 && ldx % 8 == 0,
                 "gemm_tc: K %d and the row stride %d must be multiples of 8 (TMA strides of 16 bytes)", K, ldx);
    LLMB_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0,
                 "gemm_tc: operands must be 16-byte aligned");
    LLMB_REQUIRE((out != nullptr) != (residual != nullptr), "gemm_tc: give out or residual");
    LLMB_REQUIRE(residual || out_dtype == LLMB_DTYPE_BF16 || out_dtype == LLMB_DTYPE_F32,
                 "gemm_tc: unknown output dtype %d", out_dtype);
    LLMB_REQUIRE(glu >= 0 && glu <= 2, "gemm_tc: unknown gated activation %d", glu);
    if (glu) {
        LLMB_REQUIRE(N % 32 == 0 && !bias && !residual && out_dtype == LLMB_DTYPE_BF16 && ldo >= N / 2,
                     "gemm_tc: the gated epilogue needs N %% 32 == 0, a bfloat16 output and no bias");
    } else {
        LLMB_REQUIRE(ldo >= N, "gemm_tc: bad output stride");
    }
    const Target target = glu ? TO_GATED : residual ? TO_RESIDUAL : out_dtype == LLMB_DTYPE_BF16 ? TO_BF16 : TO_F32;
    const Choice choice = choose(M, N, K, target, allow_pair);
    const Plan& p = choice.plan;
    LLMB_REQUIRE((long long)p.tiles_a * p.tiles_b * p.splits < (1ll << 30), "gemm_tc: too many tiles");
    if (choice.counters > 0) {
        LLMB_REQUIRE(partials && counters && partial_floats >= choice.scratch_floats && n_counters >= choice.counters,
                     "gemm_tc: scratch is missing or too small");
    }
    Epilogue ep{bias, out, residual, out_dtype == LLMB_DTYPE_BF16, ldo, M, N, glu != 0, {},
                glu == 2 ? 1.5957691216057308f : 1.0f, glu == 2 ? 0.0713548162726009f : 0.0f};
    int did = 0;
    if (fusion) {
        llmb_gemm_fusion f = *fusion;
        if (f.norm_sumsq) {
            LLMB_REQUIRE(f.norm_parts >= 1 && f.norm_parts <= LLMB_SUMSQ_LD && f.norm_width > 0.f,
                         "gemm_tc: a folded norm needs 1 to %d partial sums a row", LLMB_SUMSQ_LD);
            did |= LLMB_FUSED_NORM;
        } else {
            f.norm_parts = 0;
        }
        if (f.emit_rows && f.emit_sumsq && residual && choice.emit_parts > 0) {
            did |= LLMB_FUSED_EMIT;
        } else {
            f.emit_rows = nullptr;
            f.emit_sumsq = nullptr;
        }
        if (f.rope) {
            LLMB_REQUIRE(out && out_dtype == LLMB_DTYPE_BF16 && !glu && !residual && f.tok_pos && f.tok_seq &&
                         f.block_table && f.k_cache && f.v_cache && f.ring_pages > 0,
                         "gemm_tc: the rotation needs a bfloat16 output, positions, a page table and the cache");
            if (choice.can_rotate && f.head_dim >= 2 && f.head_dim % 2 == 0 && BM % f.head_dim == 0 &&
                (long long)(f.n_heads + 2 * f.n_kv_heads) * f.head_dim == N) did |= LLMB_FUSED_ROPE;
            else f.rope = 0;
        }
        ep.f = f;
    }
    if (applied) *applied = did;
    if (choice.kernel == Choice::ROW_SIDE) return launch_wide(x, ldx, w, ep, choice.wide, M, N, K, stream);
    CUtensorMap map_a, map_b;
    int code;
    if (choice.kernel == Choice::PAIRS_OF_SMS) {
        // 256 x 256 tiles over pairs of SMs; each block's boxes are 128 rows
        int n_pairs = choice.n_pairs;
        PairWork work = choice.pairs;
        if (work.tail_tiles > 0 && (!partials || partial_floats < choice.scratch_floats)) {      // no room for parts: whole tiles only
            work.n_full = work.tiles_a * work.tiles_b;
            work.tail_tiles = 0;
            n_pairs = work.n_full < PAIRS ? work.n_full : PAIRS;
        }
        if ((code = make_map(&map_a, x, M, K, ldx, BM))) return code;
        if ((code = make_map(&map_b, w, N, K, K, PAIR_BN / 2))) return code;
        return launch_pair(map_a, map_b, ep, work, n_pairs, partials, stream);
    }
    if (p.swap) {
        if ((code = make_map(&map_a, w, N, K, K, BM))) return code;
        if ((code = make_map(&map_b, x, M, K, ldx, p.bn))) return code;
    } else {
        if ((code = make_map(&map_a, x, M, K, ldx, BM))) return code;
        if ((code = make_map(&map_b, w, N, K, K, p.bn))) return code;
    }
#define GO(BN) return launch<BN>(map_a, map_b, ep, p.swap, p.tiles_a, p.tiles_b, p.n_kblocks, \
                                 p.per_split, p.splits, partials, counters, stream)
    switch (p.bn) {
        case 16: GO(16);
        case 32: GO(32);
        case 64: GO(64);
        case 128: GO(128);
        default: GO(256);
    }
#undef GO
}

LLMB_EXPORT int llmb_gemm_tc(const void* x, int ldx, const void* w, const float* bias, void* out,
                             int out_dtype, float* residual, float* partials, long long partial_floats,
                             unsigned* counters, int n_counters, int M, int N, int K, int ldo, int glu,
                             int allow_pair, cudaStream_t stream) {
    return llmb_gemm_tc_ex(x, ldx, w, bias, out, out_dtype, residual, partials, partial_floats, counters,
                           n_counters, M, N, K, ldo, glu, allow_pair, nullptr, nullptr, stream);
}

// the packed doors of the launching entry points (common.cuh)
LLMB_PACKED(llmb_gemm_tc_ex)
LLMB_PACKED(llmb_gemm_tc)

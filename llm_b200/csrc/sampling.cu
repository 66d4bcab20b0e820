// Token sampling on the device, one block or a cluster of blocks per row of logits.
//
// The chain and its order are those of MythEclipse/llm's sampler
// (apps/engine/src/sampler.rs:54-96): repeat penalty over the recent window
// (sampler.rs:110-128, once per occurrence), greedy when temperature <= 0 with
// the first maximum winning (sampler.rs:167-175), else logits / temperature,
// top-k, softmax over the survivors in descending order, top-p, min-p, and an
// inverse-CDF walk in that order with a uniform number from xorshift64*
// (sampler.rs:98-107: state seed | 1, top 24 bits). Each row has its own
// parameters and its own generator state, so a row's draw does not depend on
// the batch it is in.
//
// top_k must lie in [1, MAX_TOP_K] for the ranked chain. top_k == 0 (no top-k)
// is served only with top_p >= 1: softmax over the whole row, min-p, and an
// inverse-CDF walk in index order (the same distribution; which token a given
// uniform number picks differs from a walk in descending order).
//
// What bounds it: half a megabyte a row through the few SMs that a batch of rows keeps busy. With one block a row
// (32 rows of 128,256: 32 of 148 SMs, the row read four times at some 100 GB/s an SM) a draw took 62 us. The blocks of a
// cluster (up to eight: blocks_a_row) each read their share of the row, tell each other how many elements they have from
// their own cut on, gather what can be among the row's top_k and hand it to the first block, which ranks it and draws. The
// row is read twice (the second time from L1), and two blocks an SM (64 registers a thread) keep the clusters of 32 rows in
// one wave: with one, 42 us. Copying 32 rows of 128,256 logits and drawing from them with the default parameters, call after
// call from the host: 76 us with one block a row, 44 with the row's histograms summed over the cluster digit by digit, 35 now, of
// which the copy takes 4.4, the penalty's four dependent reads 3.4, the cuts 4.4, the candidates 4.7, their sort 3.9 and the draw
// 2.2. (The figures below are of calls in a graph, where the launches' gaps are shorter: 38 and 31 us.) Rows of which all but some
// spread entries are -inf do the row's select behind the shares' cuts: 41 to 16,000 allowed ones 26 to 31 us, 36 to 38 before.
#include <cooperative_groups.h>

#include "common.cuh"

using namespace llmb;

LLMB_DEFINE_LAST_ERROR(llmb_sampling)

constexpr int THREADS = 512;
constexpr int MAX_TOP_K = 1024;
constexpr int CANDIDATES = 2048;   // room for ties at the top-k threshold
constexpr int RADIX_BINS = 2048;   // bins of the widest digit of the radix select
constexpr int WINDOW = 1024;       // recent tokens the penalty handles in parallel (longer windows: one thread)
constexpr int WINDOW_BINS = 32;    // bins from a share's cut on whose counts the blocks of a row exchange
constexpr int CLUSTER = 8;         // most blocks a row (the portable cluster size)

// The blocks of one row: a cluster, whose first block has the row's state and results in its shared memory, or one block.
template <bool CLUSTERED> struct Team {
    __device__ __forceinline__ int rank() const { return CLUSTERED ? (int)cooperative_groups::this_cluster().block_rank() : 0; }
    __device__ __forceinline__ int blocks() const { return CLUSTERED ? (int)cooperative_groups::this_cluster().num_blocks() : 1; }
    __device__ __forceinline__ void sync() const {
        if constexpr (CLUSTERED) cooperative_groups::this_cluster().sync();
        else __syncthreads();
    }
    template <typename T> __device__ __forceinline__ T* of(T* shared, int block) const {
        if constexpr (CLUSTERED) return cooperative_groups::this_cluster().map_shared_rank(shared, block);
        else return shared;
    }
};

// The part of a row of n entries that block `rank` of its cluster reads: [begin, end), begins on multiples of four entries.
struct Share {
    int begin, end;
};
__device__ __forceinline__ Share share_of(int n, int rank, int blocks) {
    int size = ((n + blocks - 1) / blocks + 3) / 4 * 4;
    int begin = min(rank * size, n);
    return {begin, min(begin + size, n)};
}

__device__ __forceinline__ unsigned ordered_key(float v) {
    unsigned u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);   // larger float -> larger key
}

struct ArgMax {
    float value;
    int index;
};
__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
    if (b.value > a.value || (b.value == a.value && b.index < a.index)) return b;
    return a;
}

// Calls visit(value, index) for every element of row[0..n) that falls to this thread, in rising
// index order. Rows that start on a 16-byte boundary are read four values a load and eight loads
// ahead: a thread's share of a 128,256-entry row is 8 rounds of loads instead of 250 dependent ones
// (one block has to keep enough bytes in flight to fetch half a megabyte quickly).
// `WHOLE`: the rounds that lie inside the row are read without looking at its end. That is the faster way where a block has
// several of them and little to do with a value (the maximum of 64 rows of 128,256 16.1 -> 13.5 us, of one row of 50,257 6.5 ->
// 5.2), and the slower one in a share of one round (the maximum of one row of 128,256 over eight blocks 4.9 -> 5.3).
template <bool WHOLE = false, typename Visit>
__device__ __forceinline__ void for_each_of_row(const float* row, int n, Visit visit) {
    int quads = (reinterpret_cast<uintptr_t>(row) & 15) == 0 ? n >> 2 : 0;
    const float4* row4 = reinterpret_cast<const float4*>(row);
    auto visit4 = [&](const float4& v, int q) {
        visit(v.x, 4 * q);
        visit(v.y, 4 * q + 1);
        visit(v.z, 4 * q + 2);
        visit(v.w, 4 * q + 3);
    };
    int q = threadIdx.x;
    if constexpr (WHOLE) {
        for (; q + 7 * THREADS < quads; q += 8 * THREADS) {
            float4 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = row4[q + u * THREADS];
#pragma unroll
            for (int u = 0; u < 8; ++u) visit4(v[u], q + u * THREADS);
        }
    }
    constexpr int ROUND = WHOLE ? 7 : 8;                                   // (behind whole rounds, fewer than eight are left)
    for (; q < quads; q += ROUND * THREADS) {
        float4 v[ROUND];
#pragma unroll
        for (int u = 0; u < ROUND; ++u)
            if (q + u * THREADS < quads) v[u] = row4[q + u * THREADS];     // all loads in flight, the last round's too
#pragma unroll
        for (int u = 0; u < ROUND; ++u)
            if (q + u * THREADS < quads) visit4(v[u], q + u * THREADS);
    }
    for (int i = 4 * quads + threadIdx.x; i < n; i += THREADS) visit(row[i], i);
}

// First maximum of scale * row[0..n); index INT_MAX where nothing is above -inf. NaN never wins (comparisons with NaN are
// false).
template <bool WHOLE>
__device__ ArgMax block_argmax_open(const float* row, int n, ArgMax* scratch, float scale = 1.0f) {
    ArgMax best{-INFINITY, 0x7fffffff};
    for_each_of_row<WHOLE>(row, n, [&](float v, int i) {
        v *= scale;
        if (v > best.value) best = ArgMax{v, i};
    });
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) {
        ArgMax other{__shfl_xor_sync(0xffffffffu, best.value, offset),
                     __shfl_xor_sync(0xffffffffu, best.index, offset)};
        best = better(best, other);
    }
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) scratch[warp] = best;
    __syncthreads();
    if (warp == 0) {
        int n_warps = blockDim.x >> 5;
        ArgMax v = lane < n_warps ? scratch[lane] : ArgMax{-INFINITY, 0x7fffffff};
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) {
            ArgMax other{__shfl_xor_sync(0xffffffffu, v.value, offset),
                         __shfl_xor_sync(0xffffffffu, v.index, offset)};
            v = better(v, other);
        }
        if (lane == 0) scratch[0] = v;
    }
    __syncthreads();
    ArgMax result = scratch[0];
    __syncthreads();
    return result;
}
__device__ ArgMax block_argmax(const float* row, int n, ArgMax* scratch, float scale = 1.0f) {
    ArgMax result = block_argmax_open<true>(row, n, scratch, scale);
    if (result.index == 0x7fffffff) result.index = 0;
    return result;
}

// The same over the blocks of a row: every block takes its share, block 0 has the result (the others' is their own share's).
template <bool CLUSTERED>
__device__ ArgMax team_argmax(const float* row, int n, ArgMax* scratch, ArgMax* gathered) {
    Team<CLUSTERED> team;
    if constexpr (!CLUSTERED) return block_argmax(row, n, scratch);
    const int rank = team.rank(), blocks = team.blocks();
    Share share = share_of(n, rank, blocks);
    ArgMax mine = block_argmax_open<false>(row + share.begin, share.end - share.begin, scratch);
    if (mine.index != 0x7fffffff) mine.index += share.begin;
    if (threadIdx.x == 0) team.of(gathered, 0)[rank] = mine;
    team.sync();
    ArgMax best = mine;
    if (rank == 0) {
        for (int r = 0; r < blocks; ++r) best = better(best, gathered[r]);
        if (best.index == 0x7fffffff) best.index = 0;
    }
    return best;
}

template <bool CLUSTERED>
__global__ void __launch_bounds__(THREADS, 2)
argmax_rows_kernel(const float* __restrict__ logits, int stride, int vocab, int* __restrict__ out) {
    __shared__ ArgMax scratch[32];
    __shared__ ArgMax gathered[CLUSTER];
    griddep_wait();
    logits = behind_wait(logits);
    Team<CLUSTERED> team;
    if constexpr (CLUSTERED) team.sync();                     // every block's shared memory exists from here on
    const int blocks = team.blocks();
    int row = blockIdx.x / blocks;
    ArgMax best = team_argmax<CLUSTERED>(logits + (size_t)row * stride, vocab, scratch, gathered);
    if (blockIdx.x % blocks == 0 && threadIdx.x == 0) out[row] = best.index;
}

// How many blocks share a row. A row of a large vocabulary is long enough for several, as long as they fill no more than the
// GPU. What a cluster costs a short row is its barriers. The default chain behind a copy of the logits, with the row's
// histograms summed over the cluster -> as it is now: 8 rows of 128,256 32 -> 25 us, 32 rows 38 -> 31, 64 rows 47 -> 39, 32 rows
// of 32,000 27 -> 21 (one block a row took 30 more at 8 rows of 128,256). Eight blocks where one is chosen, when that was
// decided: 256 rows of 128,256 147 -> 258, 148 rows of 32,000 36 -> 81, 1,024 rows of 4,096 82 -> 406.
static int blocks_a_row(int n_rows, int vocab) {
    if (vocab < 16384) return 1;
    if (n_rows <= 32) return 8;
    return n_rows <= 64 && vocab >= 65536 ? 2 : 1;
}

template <typename... Params, typename... Args>
static cudaError_t launch_rows(void (*kernel)(Params...), int blocks, int n_rows, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(n_rows * blocks);
    config.blockDim = dim3(THREADS);
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    int n = 0;
    if (pdl_enabled()) {
        attribute[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attribute[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (blocks > 1) {
        attribute[n].id = cudaLaunchAttributeClusterDimension;
        attribute[n].val.clusterDim.x = blocks;
        attribute[n].val.clusterDim.y = attribute[n].val.clusterDim.z = 1;
        ++n;
    }
    config.attrs = attribute;
    config.numAttrs = n;
    return cudaLaunchKernelEx(&config, kernel, Params(args)...);
}

LLMB_EXPORT int llmb_argmax_rows(const float* logits, int stride, int n_rows, int vocab, int* out,
                                 cudaStream_t stream) {
    if (n_rows == 0) return LLMB_OK;
    LLMB_REQUIRE(n_rows > 0 && vocab > 0 && stride >= vocab, "argmax: bad sizes");
    LLMB_REQUIRE(n_rows <= 0x7fffffff / CLUSTER, "argmax: too many rows");
    // (a maximum alone reads the row once: eight blocks pay from some 100,000 entries on, 16 rows of 128,256 6.0 -> 4.7 us,
    // 8 rows of 32,000 3.0 -> 3.6)
    int blocks = vocab >= 65536 && n_rows <= 32 ? blocks_a_row(n_rows, vocab) : 1;
    LLMB_CUDA(launch_rows(blocks > 1 ? argmax_rows_kernel<true> : argmax_rows_kernel<false>, blocks, n_rows, stream, logits, stride,
                          vocab, out));
    return check_launch("argmax_rows");
}

__device__ __forceinline__ float next_uniform(unsigned long long* state) {
    unsigned long long x = *state;
    x ^= x >> 12;
    x ^= x << 25;
    x ^= x >> 27;
    *state = x;
    unsigned long long value = x * 0x2545F4914F6CDD1DULL;
    return (float)(value >> 40) / 16777216.0f;
}

// Sum of `value` over the threads before this one (thread 0 first), for every thread of the block.
__device__ unsigned block_exclusive_sum(unsigned value, unsigned* warp_totals) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned inclusive = value;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
        unsigned below = __shfl_up_sync(0xffffffffu, inclusive, offset);
        if (lane >= offset) inclusive += below;
    }
    if (lane == 31) warp_totals[warp] = inclusive;
    __syncthreads();
    unsigned before = 0u;
    for (int w = 0; w < warp; ++w) before += warp_totals[w];
    __syncthreads();
    return before + inclusive - value;
}

// The candidates in order: descending by value, ascending by index among equals (a bitonic sort). Up to one a thread they are
// sorted in registers, and shared memory carries only the exchanges between warps (10 of the 45 steps of 512 candidates).
__device__ void sort_candidates(float* value, int* index, int count, int top_k) {
    const int tid = threadIdx.x;
    // whether the pair (a at the lower place, b) is in order
    auto in_order = [](float va, int ia, float vb, int ib) { return va > vb || (va == vb && ia < ib); };
    // The first of them is all that is asked for: one warp finds it (8 rows of 32,000 19.4 -> 16.1 us, 64 rows of 384 15.7 -> 13.4).
    if (top_k == 1) {
        if (tid < 32) {
            float v = value[min(tid, count - 1)];
            int i = index[min(tid, count - 1)];
            for (int at = tid + 32; at < count; at += 32)
                if (in_order(value[at], index[at], v, i)) { v = value[at]; i = index[at]; }
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                float pv = __shfl_xor_sync(0xffffffffu, v, step);
                int pi = __shfl_xor_sync(0xffffffffu, i, step);
                if (in_order(pv, pi, v, i)) { v = pv; i = pi; }
            }
            __syncwarp();
            if (tid == 0) { value[0] = v; index[0] = i; }
        }
        __syncthreads();
        return;
    }
    int padded = 1;
    while (padded < count) padded <<= 1;
    if (padded <= THREADS) {
        // the warps that have candidates; the others wait at the end
        const int threads = padded < 32 ? 32 : padded;
        if (tid < threads) {
            auto meet = [&]() { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); };
            float v = tid < count ? value[tid] : -INFINITY;
            int i = tid < count ? index[tid] : 0x7fffffff;
            for (int size = 2; size <= padded; size <<= 1) {
                for (int step = size >> 1; step > 0; step >>= 1) {
                    float pv;
                    int pi;
                    if (step < 32) {
                        pv = __shfl_xor_sync(0xffffffffu, v, step);
                        pi = __shfl_xor_sync(0xffffffffu, i, step);
                    } else {
                        meet();
                        value[tid] = v;
                        index[tid] = i;
                        meet();
                        pv = value[tid ^ step];
                        pi = index[tid ^ step];
                    }
                    bool lower = (tid & step) == 0, descending = (tid & size) == 0;
                    bool ordered = lower ? in_order(v, i, pv, pi) : in_order(pv, pi, v, i);
                    if (ordered != descending) { v = pv; i = pi; }
                }
            }
            meet();
            value[tid] = v;
            index[tid] = i;
        }
        __syncthreads();
        return;
    }
    for (int i = count + tid; i < padded; i += THREADS) { value[i] = -INFINITY; index[i] = 0x7fffffff; }
    __syncthreads();
    for (int size = 2; size <= padded; size <<= 1) {
        for (int step = size >> 1; step > 0; step >>= 1) {
            for (int i = tid; i < padded; i += THREADS) {
                int partner = i ^ step;
                if (partner > i) {
                    bool descending = (i & size) == 0;
                    float va = value[i], vb = value[partner];
                    int ia = index[i], ib = index[partner];
                    if (in_order(va, ia, vb, ib) != descending) {
                        value[i] = vb; value[partner] = va;
                        index[i] = ib; index[partner] = ia;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// The draw among the `kept` sorted candidates, by one warp: softmax, top-p, min-p and the walk. Every sum runs over the
// candidates one after the other, all lanes alike; the values come 32 at a time from the lanes, so that a step of a chain
// waits for an addition and not for shared memory. (Places past the end hold zero, which leaves a sum as it is.)
__device__ int draw(float* value, const int* index, int kept, float top_p, float min_p, unsigned long long* rng) {
    const int lane = threadIdx.x & 31;
    auto part = [&](int base, int n) { return base + lane < n ? value[base + lane] : 0.f; };
    auto sum_of = [&](int n) {
        float sum = 0.f;
        for (int base = 0; base < n; base += 32) {
            float v = part(base, n);
#pragma unroll
            for (int j = 0; j < 32; ++j) sum += __shfl_sync(0xffffffffu, v, j);
        }
        return sum;
    };
    unsigned long long state = *rng;                       // (requested before the sums)
    float top_value = value[0];
    __syncwarp();
    for (int i = lane; i < kept; i += 32) value[i] = expf(value[i] - top_value);
    __syncwarp();
    float sum = sum_of(kept);
    if (sum > 0.f)
        for (int i = lane; i < kept; i += 32) value[i] /= sum;
    __syncwarp();
    if (top_p >= 0.f && top_p < 1.f) {
        float cumulative = 0.f;
        int last = -1;
        for (int base = 0; base < kept && last < 0; base += 32) {
            float v = part(base, kept);
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                cumulative += __shfl_sync(0xffffffffu, v, j);
                if (last < 0 && cumulative > top_p) last = base + j;
            }
        }
        if (last >= 0) kept = min(kept, last + 1);
    }
    if (min_p > 0.f) {
        float cut = value[0] * min_p;
        int keep = kept;
        for (int base = 0; base < kept; base += 32) {
            unsigned below = __ballot_sync(0xffffffffu, base + lane < kept && !(value[base + lane] >= cut));
            if (below) { keep = base + __ffs(below) - 1; break; }
        }
        kept = keep;
    }
    float total = sum_of(kept);
    int pick = 0;
    if (total > 0.f) {
        float target = next_uniform(&state) * total;
        if (lane == 0) *rng = state;
        int found = -1;
        for (int base = 0; base < kept && found < 0; base += 32) {
            float v = part(base, kept);
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                target -= __shfl_sync(0xffffffffu, v, j);
                if (found < 0 && base + j < kept && target <= 0.f) found = base + j;
            }
        }
        if (found >= 0) pick = found;
    }
    return index[pick];
}

// params[row] = {temperature, top_p, min_p, repeat_penalty}; iparams[row] =
// {top_k, repeat_last_n}. recent[row, 0..recent_cap) holds the row's generated
// tokens as a ring: token number i (counted from 0) is at recent[row, i % cap],
// recent_len[row] counts all of them. `logits` is modified in place (the penalty
// on the recent tokens' entries). status[row] is set to 1 when the row was refused (its parameters, or
// more equal logits at the top-k cut than the kernel ranks) and token 0 stands in its place; the kernel
// never clears it, so a refusal in any step stays visible until the host has read and cleared it.
//
// Block 0 of a row's cluster owns the row's state and draws; the other blocks read their share of the row for the penalty,
// the histogram and the candidates. Where the chain walks the whole row in index order, one block does and the others leave.
template <bool CLUSTERED>
__global__ void __launch_bounds__(THREADS, 2)
sample_rows_kernel(float* __restrict__ logits, int stride, int vocab,
                   const float4* __restrict__ params, const int2* __restrict__ iparams,
                   int* __restrict__ recent, int* __restrict__ recent_len,
                   int recent_cap, unsigned long long* __restrict__ rng, int* __restrict__ out,
                   int* __restrict__ status, int record, const int* __restrict__ state_rows) {
    __shared__ ArgMax scratch[32];
    __shared__ unsigned histogram[RADIX_BINS];
    __shared__ unsigned block_sums_u[32];
    __shared__ float cand_value[CANDIDATES];
    __shared__ int cand_index[CANDIDATES];
    __shared__ unsigned shared_prefix, shared_need, shared_count, shared_gathered;
    __shared__ unsigned shared_counts[CLUSTER], window_counts[WINDOW_BINS], shared_windows[CLUSTER * WINDOW_BINS];
    __shared__ int shared_bins[CLUSTER];       // of the row's blocks: the bin of the first digit that holds a share's top_k-th largest
    __shared__ float block_sums[THREADS];
    __shared__ int window[WINDOW];
    __shared__ ArgMax gathered[CLUSTER];
    __shared__ int held_back;
    __shared__ float2 cuts;
    griddep_wait();
    params = behind_wait(params);
    iparams = behind_wait(iparams);
    state_rows = behind_wait(state_rows);
    Team<CLUSTERED> team;
    const int rank = team.rank(), blocks = team.blocks();

    // row of logits and of `out`; the sequence's parameters, window, generator and status are in
    // row state_rows[row] of their arrays (the same row if state_rows is null)
    int logits_row = blockIdx.x / blocks;
    int row_id = state_rows ? state_rows[logits_row] : logits_row;
    LLMB_STAMP(0, 0);
    float* row = logits + (size_t)logits_row * stride;
    float temperature = params[row_id].x, top_p = params[row_id].y, min_p = params[row_id].z;
    float penalty = params[row_id].w;
    int top_k = iparams[row_id].x, last_n = iparams[row_id].y;
    const int held = recent != nullptr && recent_len != nullptr ? recent_len[row_id] : 0;      // (requested together with the parameters)
    // what the draw at the end asks for waits in shared memory, not in every thread's registers (64 rows of 50,257, top_k 3: 40.7 -> 39.1 us)
    if (threadIdx.x == 0) { held_back = held; cuts = make_float2(top_p, min_p); }
    int tid = threadIdx.x;
    const Share share = share_of(vocab, rank, blocks);
    // the chains without a ranking (whole row, or refused) run in one block alone, each row in another: where the
    // clusters of several rows share SMs, their walking blocks do not (32 rows of 128,256: 67 us, and 88 in block 0 of each)
    const bool ranked = temperature > 0.f && (top_k > 0 || vocab <= MAX_TOP_K) && (top_k <= MAX_TOP_K || vocab <= MAX_TOP_K);
    const bool alone = temperature > 0.f && !ranked;
    if (alone && rank != logits_row % blocks) return;
    // the entries this block applies the penalty to: those that it reads
    const int own_begin = alone ? 0 : share.begin, own_end = alone ? vocab : share.end;
    // block 0's thread 0 calls this once: the token is the row's result and, with `record`, the newest entry
    // of the row's window (a ring over its generated tokens)
    auto finish = [&](int token) {
        out[logits_row] = token;
        if (record && recent != nullptr) {
            recent[(size_t)row_id * recent_cap + (held_back % recent_cap)] = token;
            recent_len[row_id] = held_back + 1;
        }
    };

    if (penalty != 1.0f && last_n > 0 && recent != nullptr) {
        // A token that occurs c times in the window is penalised c times, one after the other
        // (apps/engine/src/sampler.rs:115-127). One thread per window place; the first place of a
        // token applies all of its c steps, so the arithmetic is that of the serial loop.
        const int total = held;
        int span = min(min(total, last_n), recent_cap);
        if (span <= WINDOW) {
            for (int t = tid; t < span; t += THREADS)
                window[t] = recent[(size_t)row_id * recent_cap + ((total - span + t) % recent_cap)];
            __syncthreads();
            for (int t = tid; t < span; t += THREADS) {
                int id = window[t];
                if (id < own_begin || id >= own_end) continue;
                int count = 0;
                bool first = true;
                for (int u = 0; u < span; ++u) {
                    if (window[u] != id) continue;
                    if (u < t) { first = false; break; }
                    ++count;
                }
                if (!first) continue;
                float v = row[id];
                for (int c = 0; c < count; ++c) v = v > 0.f ? v / penalty : v * penalty;
                row[id] = v;
            }
        } else if (tid == 0) {
            for (int i = total - span; i < total; ++i) {
                int id = recent[(size_t)row_id * recent_cap + (i % recent_cap)];
                if (id < own_begin || id >= own_end) continue;
                float v = row[id];
                row[id] = v > 0.f ? v / penalty : v * penalty;
            }
        }
    }
    __syncthreads();

    if (tid == 0) shared_gathered = 0u;
    // every block's shared memory exists, and every block has read the row's state (block 0's finish() changes it)
    if (CLUSTERED && !alone) team.sync();

    if (!(temperature > 0.f)) {
        ArgMax best = team_argmax<CLUSTERED>(row, vocab, scratch, gathered);
        if (rank == 0 && tid == 0) finish(best.index);
        return;
    }
    // every later reading of the row takes its values times 1 / temperature (the same rounding each
    // time) instead of a pass that writes the scaled row back
    float inverse = 1.0f / temperature;
    LLMB_STAMP(1, 0);                                 // the penalty is applied

    if (top_k <= 0 || top_k >= vocab) {
        if (vocab <= MAX_TOP_K) {
            top_k = vocab;                      // a small row: rank all of it
        } else if (top_k > 0 || (top_p >= 0.f && top_p < 1.f)) {
            // the ranked chain is limited to MAX_TOP_K candidates
            if (tid == 0) { status[row_id] = 1; finish(0); }
            return;
        }
    } else if (top_k > MAX_TOP_K) {
        if (tid == 0) { status[row_id] = 1; finish(0); }
        return;
    }

    if (top_k <= 0) {
        // ---- whole row, index order: softmax, min-p, inverse CDF
        ArgMax best = block_argmax(row, vocab, scratch, inverse);
        float cut = min_p > 0.f ? min_p : 0.f;
        int per_thread = (vocab + THREADS - 1) / THREADS;
        int begin = min(tid * per_thread, vocab), end = min(begin + per_thread, vocab);
        float local = 0.f;
        for (int i = begin; i < end; ++i) {
            float p = expf(row[i] * inverse - best.value);
            if (p >= cut) local += p;
        }
        block_sums[tid] = local;
        __syncthreads();
        if (tid == 0) {
            // one thread's chains, each value fetched ahead of the addition that waits for the one before it: eight sums, four
            // entries at a time (8 rows of 32,000: 27 -> 20 us, 32 rows of 128,256: 71 -> 54)
            float total = 0.f;
            for (int base = 0; base < THREADS; base += 8) {
                float part[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) part[j] = block_sums[base + j];
#pragma unroll
                for (int j = 0; j < 8; ++j) total += part[j];
            }
            unsigned long long state = rng[row_id];
            float target = next_uniform(&state) * total;
            rng[row_id] = state;
            int owner = -1;
            float before = 0.f;
            for (int base = 0; base < THREADS && owner < 0; base += 8) {
                float part[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) part[j] = block_sums[base + j];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (owner < 0 && part[j] > 0.f && target - (before + part[j]) <= 0.f) owner = base + j;
                    if (owner < 0) before += part[j];
                }
            }
            int pick = best.index;
            if (owner >= 0) {
                float remaining = target - before;
                int b = min(owner * per_thread, vocab), e = min(b + per_thread, vocab);
                for (int i0 = b; i0 < e; i0 += 4) {
                    float p[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) p[j] = i0 + j < e ? row[i0 + j] : -INFINITY;
#pragma unroll
                    for (int j = 0; j < 4; ++j) p[j] = expf(p[j] * inverse - best.value);
                    bool found = false;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (found || i0 + j >= e || p[j] < cut) continue;
                        pick = i0 + j;
                        remaining -= p[j];
                        found = remaining <= 0.f;
                    }
                    if (found) break;
                }
            }
            finish(pick);
        }
        return;
    }

    // ---- ranked chain: radix select of the top_k-th largest key, three digits of 11, 11 and 10 bits.
    // The first digit is the sign, the exponent and two bits of the mantissa: wide enough to spread
    // a row of logits over some hundred bins, so that the threads' additions seldom meet. Every block counts its share,
    // block 0 has the sums and picks the bin. Once the elements that are not below the bin fit the candidate buffer, they
    // are gathered, and block 0 selects the digits that are left among them.
    auto bits = [](int digit) { return digit == 0 ? 21 : digit == 1 ? 10 : 0; };
    // block 0: the bin, counted from the top, in which the running count reaches what is still needed:
    // every thread sums four neighbouring bins, the block scans the threads from the top down
    auto pick_bin = [&](int digit) {
        const int n_bins = digit == 2 ? 1024 : 2048;
        unsigned need = shared_need, prefix = shared_prefix;
        int top_bin = n_bins - 1 - 4 * tid;                       // this thread's highest bin
        unsigned mine = 0u;
        if (top_bin >= 3)
            mine = histogram[top_bin] + histogram[top_bin - 1] + histogram[top_bin - 2] + histogram[top_bin - 3];
        unsigned before = block_exclusive_sum(mine, block_sums_u);  // of the threads with higher bins
        if (top_bin >= 3 && before < need && before + mine >= need) {
            unsigned left = need - before;
            int bin = top_bin;
            for (; bin > top_bin - 3; --bin) {
                if (histogram[bin] >= left) break;
                left -= histogram[bin];
            }
            shared_need = left;
            shared_prefix = prefix | ((unsigned)bin << bits(digit));
            // elements not below the bin: the ones above it are taken for certain
            shared_count = (unsigned)top_k - left + histogram[bin];
        }
        __syncthreads();
    };
    unsigned threshold = 0u;                   // keys of the gathered elements are not below it
    int digit = 0;                             // digits the threshold has
    bool gathered_all = false;
    if constexpr (CLUSTERED) {
        // Each block alone: the bin of the first digit down to which its own share has top_k elements, its cut. The row's cut is
        // no lower than any share's. Every block tells the others its cut and how many elements it has from there on and
        // from each of the bins above; all then know a bin down to which the row has top_k elements (counts past the window are
        // taken for zero, which lowers it at most), and everything down to it holds all that the row's select would keep,
        // ties included: some eighty elements of a row of logits. Three exchanges between the blocks instead of the six of
        // the row's select, which follows where they do not fit the buffer (rows that are mostly one value).
        for (int i = tid; i < RADIX_BINS; i += THREADS) histogram[i] = 0u;
        if (tid == 0) shared_prefix = 0u;
        __syncthreads();
        for_each_of_row(row + share.begin, share.end - share.begin, [&](float v, int) {
            atomicAdd(&histogram[ordered_key(v * inverse) >> 21], 1u);
        });
        __syncthreads();
        int top_bin = RADIX_BINS - 1 - 4 * tid;                   // as in pick_bin
        unsigned mine = histogram[top_bin] + histogram[top_bin - 1] + histogram[top_bin - 2] + histogram[top_bin - 3];
        unsigned before = block_exclusive_sum(mine, block_sums_u);
        if (before < (unsigned)top_k && before + mine >= (unsigned)top_k) {
            int bin = top_bin;
            for (unsigned have = before + histogram[bin]; have < (unsigned)top_k; have += histogram[bin]) --bin;
            shared_prefix = (unsigned)bin;
        }
        __syncthreads();
        // the number of elements from each bin of this thread's four on, into the window behind the cut
        const int cut = (int)shared_prefix;
        if (tid < WINDOW_BINS) window_counts[tid] = 0u;
        __syncthreads();
        if (top_bin >= cut) {
            unsigned from = before;
            for (int bin = top_bin; bin > top_bin - 4; --bin) {
                from += histogram[bin];
                if (bin >= cut && bin < cut + WINDOW_BINS) window_counts[bin - cut] = from;
            }
        }
        __syncthreads();
        if (tid < blocks * WINDOW_BINS) {
            const int to = tid / WINDOW_BINS, at = tid % WINDOW_BINS;
            team.of(shared_windows, to)[rank * WINDOW_BINS + at] = window_counts[at];
            if (at == 0) team.of(shared_bins, to)[rank] = cut;
        }
        team.sync();
        LLMB_STAMP(2, 0);                             // the shares have their cuts
        int bin = 0;
        for (int r = 0; r < blocks; ++r) bin = max(bin, shared_bins[r]);
        if ((tid & 31) < WINDOW_BINS) {               // a lane a bin from there on: the highest that has top_k elements
            unsigned have = 0u;
            for (int r = 0; r < blocks; ++r) {
                int at = bin + (tid & 31) - shared_bins[r];
                if (at < WINDOW_BINS) have += shared_windows[r * WINDOW_BINS + at];
            }
            unsigned enough = __ballot_sync(0xffffffffu, have >= (unsigned)top_k);
            if (enough) bin += 31 - __clz(enough);
        }
        threshold = (unsigned)bin << 21;
        // each block gathers its own, and the first block fetches what the others have (a counter and a buffer in the first
        // block's memory that all blocks write to took some 10 us for 450 candidates)
        for_each_of_row(row + share.begin, share.end - share.begin, [&](float v, int i) {
            v *= inverse;
            if (ordered_key(v) >= threshold) {
                unsigned at = atomicAdd(&shared_gathered, 1u);
                if (at < CANDIDATES) { cand_value[at] = v; cand_index[at] = share.begin + i; }
            }
        });
        __syncthreads();
        if (tid < blocks) team.of(shared_counts, tid)[rank] = shared_gathered;
        team.sync();
        unsigned total = 0u;
        for (int r = 0; r < blocks; ++r) total += shared_counts[r];
        gathered_all = total <= (unsigned)CANDIDATES;
        if (gathered_all) {
            if (rank == 0) {
                unsigned own = shared_counts[0];
                for (unsigned i = own + tid; i < total; i += THREADS) {
                    unsigned at = i - own;
                    int r = 1;
                    while (at >= shared_counts[r]) at -= shared_counts[r++];
                    cand_value[i] = team.of(cand_value, r)[at];
                    cand_index[i] = team.of(cand_index, r)[at];
                }
            }
            team.sync();                       // the others' memory has been read
            if (rank != 0) return;
            if (tid == 0) shared_gathered = total;
            __syncthreads();
        }
        threshold = 0u;
    }
    if (tid == 0) { shared_prefix = 0u; shared_need = (unsigned)top_k; shared_count = 0u; }
    if (!gathered_all) {
        for (; digit < 3;) {
            const int shift = bits(digit), n_bins = digit == 2 ? 1024 : 2048;
            for (int i = tid; i < RADIX_BINS; i += THREADS) histogram[i] = 0u;
            team.sync();                        // (block 0's bins are zero before the others add to them)
            unsigned mask = digit == 0 ? 0u : (0xffffffffu << bits(digit - 1));
            for_each_of_row(row + share.begin, share.end - share.begin, [&](float v, int) {
                unsigned key = ordered_key(v * inverse);
                if ((key & mask) == threshold) atomicAdd(&histogram[(key >> shift) & (unsigned)(n_bins - 1)], 1u);
            });
            __syncthreads();
            if (rank != 0) {
                unsigned* sums = team.of(histogram, 0);
                for (int i = tid; i < n_bins; i += THREADS)
                    if (histogram[i]) atomicAdd(&sums[i], histogram[i]);
            }
            team.sync();
            if (rank == 0) {
                pick_bin(digit);
                if (tid < blocks && tid > 0) {
                    *team.of(&shared_prefix, tid) = shared_prefix;
                    *team.of(&shared_count, tid) = shared_count;
                }
            }
            team.sync();
            threshold = shared_prefix;
            ++digit;
            if (shared_count <= (unsigned)CANDIDATES) break;
        }
        LLMB_STAMP(2, 0);                                 // the radix select has its threshold
        if (rank == 0 && tid == 0) shared_gathered = 0u;     // now the number of candidates
        team.sync();
        {
            unsigned* at_ = team.of(&shared_gathered, 0);
            float* values = team.of(cand_value, 0);
            int* indices = team.of(cand_index, 0);
            for_each_of_row(row + share.begin, share.end - share.begin, [&](float v, int i) {
                v *= inverse;
                if (ordered_key(v) >= threshold) {
                    unsigned at = atomicAdd(at_, 1u);
                    if (at < CANDIDATES) { values[at] = v; indices[at] = share.begin + i; }
                }
            });
        }
        team.sync();
        if (rank != 0) return;
    }
    LLMB_STAMP(3, 0);                                 // the candidates are gathered
    int count = (int)min(shared_gathered, (unsigned)CANDIDATES);
    if (shared_gathered > (unsigned)CANDIDATES) {
        // more ties at the threshold than the buffer holds
        if (tid == 0) { status[row_id] = 1; finish(0); }
        return;
    }
    if (digit < 3 && count > THREADS && top_k > 1) {
        // more than a sort in registers takes: the digits that are left, among the candidates; then those below the whole
        // threshold go
        for (; digit < 3; ++digit) {
            const int shift = bits(digit), n_bins = digit == 2 ? 1024 : 2048;
            for (int i = tid; i < RADIX_BINS; i += THREADS) histogram[i] = 0u;
            __syncthreads();
            unsigned prefix = shared_prefix, mask = digit == 0 ? 0u : (0xffffffffu << bits(digit - 1));
            for (int i = tid; i < count; i += THREADS) {
                unsigned key = ordered_key(cand_value[i]);
                if ((key & mask) == prefix) atomicAdd(&histogram[(key >> shift) & (unsigned)(n_bins - 1)], 1u);
            }
            __syncthreads();
            pick_bin(digit);
        }
        threshold = shared_prefix;
        float value[CANDIDATES / THREADS];
        int index[CANDIDATES / THREADS];
#pragma unroll
        for (int u = 0; u < CANDIDATES / THREADS; ++u) {
            int i = tid + u * THREADS;
            value[u] = i < count ? cand_value[i] : 0.f;
            index[u] = i < count && ordered_key(value[u]) >= threshold ? cand_index[i] : -1;
        }
        __syncthreads();
        if (tid == 0) shared_count = 0u;
        __syncthreads();
#pragma unroll
        for (int u = 0; u < CANDIDATES / THREADS; ++u) {
            if (index[u] < 0) continue;
            unsigned at = atomicAdd(&shared_count, 1u);
            cand_value[at] = value[u];
            cand_index[at] = index[u];
        }
        __syncthreads();
        count = (int)shared_count;
    }
    sort_candidates(cand_value, cand_index, count, top_k);
    LLMB_STAMP(4, 0);                                 // the candidates are sorted
    if (tid >= 32) return;
    int token = draw(cand_value, cand_index, min(count, top_k), cuts.x, cuts.y, rng + row_id);
    if (tid == 0) finish(token);
    LLMB_STAMP(5, 0);                                 // the token is drawn
}

// The stamps of the last sampling launch in a build with -DLLMB_TRACE (see common.cuh); 1 otherwise.
LLMB_EXPORT int llmb_sampling_trace(unsigned long long* out, int clear) { return llmb_read_trace(out, clear); }

LLMB_EXPORT int llmb_sample_rows(float* logits, int stride, int n_rows, int vocab,
                                 const float* params, const int* iparams, int* recent,
                                 int* recent_len, int recent_cap,
                                 unsigned long long* rng, int* out, int* status, int record,
                                 const int* state_rows, cudaStream_t stream) {
    if (n_rows == 0) return LLMB_OK;
    LLMB_REQUIRE(n_rows > 0 && vocab > 0 && stride >= vocab, "sample: bad sizes");
    LLMB_REQUIRE(recent == nullptr || recent_cap > 0, "sample: recent window without capacity");
    LLMB_REQUIRE(n_rows <= 0x7fffffff / CLUSTER, "sample: too many rows");
    int blocks = blocks_a_row(n_rows, vocab);
    LLMB_CUDA(launch_rows(blocks > 1 ? sample_rows_kernel<true> : sample_rows_kernel<false>, blocks, n_rows, stream, logits, stride,
                          vocab, (const float4*)params, (const int2*)iparams, recent, recent_len, recent_cap, rng, out, status,
                          record, state_rows));
    return check_launch("sample_rows");
}

// the packed doors of the launching entry points (common.cuh)
LLMB_PACKED(llmb_argmax_rows)
LLMB_PACKED(llmb_sample_rows)

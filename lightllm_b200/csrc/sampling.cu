// Token selection on the device: greedy argmax, and temperature sampling with the top-k,
// top-p and min-p filters, one block per row of logits.
//
// Order of operations as src/ops/sampling.cpp:22-335: temperature < 1e-5 is greedy (first
// index of the strictly largest logit, :36-59); else logits * 1/max(T, 1e-8) (:81-84); top-k
// keeps values >= the k-th largest, ties kept (:91-137); softmax with the maximum subtracted
// (:143-193); top-p keeps the most probable tokens until their mass reaches p and
// renormalises (:198-243); min-p drops probabilities below min_p * max and renormalises
// (:248-278); the draw is the first index whose cumulative mass reaches the uniform number,
// skipping entries without mass (:284-334).  The reference sorts on the CPU; here each filter
// is a threshold on the value, found over the float's ordered bit pattern (in short rows bit by
// bit, in long ones by bins of values), so a tie at the top-p boundary keeps all tied tokens where the
// reference's sort keeps an unspecified subset.  The uniform number comes from the caller
// (one per row), so the random stream belongs to the request, not to the kernel.
#include "common.cuh"

#include <cooperative_groups.h>
#include <math.h>

namespace cg = cooperative_groups;

namespace {

constexpr int THREADS = 1024;

// Order-preserving map from float to unsigned: a < b  <=>  key(a) < key(b).
__device__ __forceinline__ unsigned ordered_key(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float key_value(unsigned key) { return __uint_as_float((key & 0x80000000u) ? key ^ 0x80000000u : ~key); }

__device__ float block_sum(float v, float* sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    v = llb_warp_sum(v);
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    float t = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0f;
    if (w == 0) {
        t = llb_warp_sum(t);
        if (lane == 0) sh[32] = t;
    }
    __syncthreads();
    return sh[32];
}

__device__ float block_max(float v, float* sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    v = llb_warp_max(v);
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    float t = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : -INFINITY;
    if (w == 0) {
        t = llb_warp_max(t);
        if (lane == 0) sh[32] = t;
    }
    __syncthreads();
    return sh[32];
}

// First index of the largest value of a row.
// ``none`` is what a row without any value above -inf (or with NaNs only) gives.
__device__ int block_argmax(const float* x, int V, float* shf, int* shi, int none = 0) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
        const float v = x[i];
        if (v > best) { best = v; bi = i; }   // ascending i per thread keeps its first maximum
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) { shf[w] = best; shi[w] = bi; }
    __syncthreads();
    if (w == 0) {
        best = lane < (blockDim.x >> 5) ? shf[lane] : -INFINITY;
        bi = lane < (blockDim.x >> 5) ? shi[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        if (lane == 0) shi[32] = (bi == 0x7fffffff) ? none : bi;
    }
    __syncthreads();
    return shi[32];
}

__global__ void __launch_bounds__(THREADS) argmax_kernel(const float* __restrict__ logits, int V, long long stride,
                                                         int* __restrict__ out) {
    __shared__ float shf[33];
    __shared__ int shi[33];
    const int r = blockIdx.x;
    const int idx = block_argmax(logits + (size_t)r * stride, V, shf, shi);
    if (threadIdx.x == 0) out[r] = idx;
}

// The same over a long row, by many blocks: block (s, r) takes the s-th piece of row r and offers its first maximum to
// the row's slot as one 64-bit number (the value's ordered key above, 2^32 - 1 - index below: the larger value wins,
// among equal values the smaller index) with an atomic maximum.  The block that counts itself last on the row's
// counter writes the index and leaves slot and counter zero for the next launch.  A row without any value above
// -inf offers nothing and gets index 0, as in the one-block kernel.
constexpr int SPLIT_THREADS = 256;
constexpr int SPLIT_ELEMS = 4096;            // elements of a row per block

__global__ void __launch_bounds__(SPLIT_THREADS) argmax_split_kernel(const float* __restrict__ logits, int V, long long stride,
                                                                     unsigned long long* __restrict__ slots,
                                                                     int* __restrict__ counters, int* __restrict__ out) {
    __shared__ float shf[33];
    __shared__ int shi[33];
    const int r = blockIdx.y;
    const int begin = blockIdx.x * SPLIT_ELEMS;
    const int n = min(SPLIT_ELEMS, V - begin);
    const int idx = block_argmax(logits + (size_t)r * stride + begin, n, shf, shi, /*none=*/-1);
    if (threadIdx.x == 0) {
        if (idx >= 0) {
            const float v = logits[(size_t)r * stride + begin + idx] + 0.0f;        // -0 counts as +0
            const unsigned long long offer = ((unsigned long long)ordered_key(v) << 32) |
                                             (unsigned long long)(0xffffffffu - (unsigned)(begin + idx));
            atomicMax(slots + r, offer);
        }
        __threadfence();
        if (atomicAdd(counters + r, 1) == (int)gridDim.x - 1) {
            __threadfence();
            const unsigned long long best = atomicExch(slots + r, 0ull);
            out[r] = best == 0ull ? 0 : (int)(0xffffffffu - (unsigned)(best & 0xffffffffull));
            atomicExch(counters + r, 0);
        }
    }
}

// params per row: temperature, top_p, min_p, uniform; top_k per row as int.
__global__ void __launch_bounds__(THREADS) sample_kernel(const float* __restrict__ logits, int V, long long stride,
                                                         const float* __restrict__ temperature,
                                                         const int* __restrict__ top_k,
                                                         const float* __restrict__ top_p,
                                                         const float* __restrict__ min_p,
                                                         const float* __restrict__ uniform, int* __restrict__ out) {
    __shared__ float shf[33];
    __shared__ int shi[33];
    __shared__ float chunk_sum[THREADS];
    const int r = blockIdx.x;
    const float* x = logits + (size_t)r * stride;
    const float temp = temperature[r];
    if (temp < 1e-5f) {
        const int idx = block_argmax(x, V, shf, shi);
        if (threadIdx.x == 0) out[r] = idx;
        return;
    }
    const float inv_temp = 1.0f / fmaxf(temp, 1e-8f);
    const int k = top_k ? top_k[r] : 0;
    const float tp = top_p ? top_p[r] : 1.0f;
    const float mp = min_p ? min_p[r] : 0.0f;

    float mx = -INFINITY;
    for (int i = threadIdx.x; i < V; i += blockDim.x) mx = fmaxf(mx, x[i] * inv_temp);
    mx = block_max(mx, shf);
    if (mx == -INFINITY || !(mx == mx)) {  // every logit is -inf, or NaN: fall back to argmax
        const int idx = block_argmax(x, V, shf, shi);
        if (threadIdx.x == 0) out[r] = idx;
        return;
    }

    // top-k: key of the k-th largest scaled logit (largest K with count(key >= K) >= k).
    unsigned key_k = 0u;
    if (k > 0 && k < V) {
        for (int bit = 31; bit >= 0; --bit) {
            const unsigned cand = key_k | (1u << bit);
            float cnt = 0.0f;
            for (int i = threadIdx.x; i < V; i += blockDim.x) cnt += ordered_key(x[i] * inv_temp) >= cand ? 1.0f : 0.0f;
            cnt = block_sum(cnt, shf);
            if (cnt >= (float)k) key_k = cand;
        }
    }
    // e_i = exp(x_i/T - max) of the kept entries; everything below is in terms of e (max e = 1).
    auto e_of = [&](int i) -> float {
        const float s = x[i] * inv_temp;
        if (ordered_key(s) < key_k) return 0.0f;
        return expf(s - mx);
    };
    float z = 0.0f;
    for (int i = threadIdx.x; i < V; i += blockDim.x) z += e_of(i);
    z = block_sum(z, shf);

    // top-p: largest threshold on e whose kept mass still reaches p * z.
    unsigned key_p = 0u;
    if (tp < 1.0f) {
        const float need = tp * z;
        for (int bit = 31; bit >= 0; --bit) {
            const unsigned cand = key_p | (1u << bit);
            float mass = 0.0f;
            for (int i = threadIdx.x; i < V; i += blockDim.x) {
                const float e = e_of(i);
                if (e > 0.0f && ordered_key(e) >= cand) mass += e;
            }
            mass = block_sum(mass, shf);
            if (mass >= need) key_p = cand;
        }
    }
    // min-p: probabilities below min_p * max probability are dropped; max e is 1.
    const float e_min = mp > 0.0f ? mp : 0.0f;
    auto kept_of = [&](int i) -> float {
        const float e = e_of(i);
        if (e <= 0.0f || ordered_key(e) < key_p || e < e_min) return 0.0f;
        return e;
    };

    // Draw: first index whose running mass reaches u * total.  Threads own contiguous chunks.
    const int per = (V + blockDim.x - 1) / blockDim.x;
    const int begin = min(V, (int)threadIdx.x * per), end = min(V, begin + per);
    float mine = 0.0f;
    for (int i = begin; i < end; ++i) mine += kept_of(i);
    chunk_sum[threadIdx.x] = mine;
    const float total = block_sum(mine, shf);   // contains the barriers that publish chunk_sum
    if (threadIdx.x == 0) {
        int choice = -1;
        if (total > 0.0f) {
            const float target = uniform[r] * total;
            float run = 0.0f;
            int c = 0;
            for (; c < (int)blockDim.x; ++c) {
                if (chunk_sum[c] > 0.0f && run + chunk_sum[c] >= target) break;
                run += chunk_sum[c];
            }
            if (c < (int)blockDim.x) {
                const int b = min(V, c * per), e = min(V, b + per);
                int last_mass = -1;
                for (int i = b; i < e; ++i) {
                    const float m = kept_of(i);
                    if (m > 0.0f) {
                        last_mass = i;
                        run += m;
                        if (run >= target) { choice = i; break; }
                    }
                }
                if (choice < 0) choice = last_mass;
            }
            if (choice < 0) {  // rounding left the target above the total: last entry with mass
                for (int i = V - 1; i >= 0 && choice < 0; --i)
                    if (kept_of(i) > 0.0f) choice = i;
            }
        }
        shi[32] = choice;
    }
    __syncthreads();
    int choice = shi[32];
    if (choice < 0) choice = block_argmax(x, V, shf, shi);   // uniform over the block
    if (threadIdx.x == 0) out[r] = choice;
}

// ---------------------------------------------------------------------------------------------------------------
// The same selection for long rows (a vocabulary of 150,000), by a cluster of CL blocks per row.  The one-block
// kernel walks the whole row in memory for every counting pass (32 per filter, each with an exponential per
// element): 0.2 ms for temperature alone and 2 ms with all filters at this size.  Here block b of the cluster keeps
// its part of the row in shared memory (first the scaled logits, then their exponentials, then the kept masses), so a
// pass is a walk over shared memory, a reduction in the block and one exchange in the cluster: every block
// publishes its partial result in its own shared memory, the cluster meets on its barrier, and every block adds up
// all parts in rank order, so that all blocks hold the same bits and take the same branches.  The published
// values alternate between two places: a block writes the place of pass n+2 only after the barrier of pass n+1,
// which every block reaches only after it has read pass n.
constexpr int CL = 8;
constexpr int CL_THREADS = 512;

struct ClusterExchange {
    float f[2];
    int i[2];
    int turn;
};

__device__ __forceinline__ float cluster_max(cg::cluster_group& cl, ClusterExchange* xc, float block_value) {
    const int t = xc->turn;
    if (threadIdx.x == 0) xc->f[t] = block_value;
    cl.sync();
    float best = -INFINITY;
#pragma unroll
    for (int b = 0; b < CL; ++b) best = fmaxf(best, cl.map_shared_rank(xc, b)->f[t]);
    __syncthreads();
    if (threadIdx.x == 0) xc->turn = t ^ 1;
    __syncthreads();
    return best;
}

// The maxima of a and b over the cluster in one meeting.
__device__ __forceinline__ void cluster_max2(cg::cluster_group& cl, ClusterExchange* xc, float& a, float& b, float* sh) {
    static_assert(CL_THREADS == 512, "sixteen warps, two numbers each");
    const int t = xc->turn, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    a = llb_warp_max(a);
    b = llb_warp_max(b);
    if (lane == 0) {
        sh[w] = a;
        sh[16 + w] = b;
    }
    __syncthreads();
    if (w == 0) {
        float v = sh[lane];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) xc->f[t] = v;
        if (lane == 16) xc->i[t] = __float_as_int(v);
    }
    cl.sync();
    a = b = -INFINITY;
#pragma unroll
    for (int r = 0; r < CL; ++r) {
        const ClusterExchange* o = cl.map_shared_rank(xc, r);
        a = fmaxf(a, o->f[t]);
        b = fmaxf(b, __int_as_float(o->i[t]));
    }
    __syncthreads();
    if (threadIdx.x == 0) xc->turn = t ^ 1;
    __syncthreads();
}

// The threshold of a filter over a row that lies in its cluster's shared memory: the largest key for which the weight of all values
// with that key or a larger one reaches what is needed (a search bit by bit finds the same in 32 meetings of the cluster).  The weights
// are counted by bin, every block adds up all blocks' bins and finds the one in which the need is reached, and the values of
// that bin either go to a list of every block, where each is compared with all the others, or, where they are more than the list holds,
// are binned anew over the keys that they span: two meetings a level, one or two levels for most rows (ties end at once, their keys
// span one value).  A mass is added as a whole number of 2^-44 in three parts of 15 bits (32-bit atomics are the hardware's
// own, and the 56,000 values that a block holds at most leave them room), so no sum depends on the order of the atomics.
// What bounds it: the walks over shared memory (some 6 us a search at 151,936 values) and the meetings.  What falls into the last bin,
// where most of a wide row lies, is added up in registers.  (Adding up in the warp what shares a bin before the atomic helped rows
// of two values only, and cost all others a tenth.)  Three blocks fit a multiprocessor's registers at 40 a thread.
// 64 rows of 151,936, us, by bits -> this: top-k 40 256 -> 75, top-k 20 and top-p 0.95 435 -> 89, top-p 0.9 of normal logits of
// deviation 3 / 1 / 0.02: 221 / 228 / 229 -> 92 / 136 / 129, of equal ones 230 -> 126; one row 90 -> 28, 146 -> 33, 79 -> 40.
constexpr int BINS = 256;
constexpr int BIN_LIST = CL_THREADS / 4;      // four threads compare a member
struct ThresholdList {
    unsigned key[BIN_LIST];
    unsigned long long weight[BIN_LIST];
};
struct Threshold {
    unsigned hist[3][BINS];                   // counts or masses: bits 0-14, 15-29 and 30-44 of every value added up
    unsigned long long warp_total[BINS / 32];
    unsigned long long before, upto;          // what lies above the chosen bin, and with it
    int bin;
    unsigned value;                           // the threshold's key
    unsigned long long reached;               // the weight of the threshold's and all larger values
    float top, low;                           // of the whole row, kept here over the search by rank (registers are what limits blocks)
    // This block's values in the bin span these keys, and block 0's count of the list.  Two slots in turn for each search: a slot is set
    // anew two levels later, when everyone has met once more since its last reader; the second search's first one is set at the
    // kernel's start.  For the same reason each search has a list of its own: blocks write into one another's, and some are at the
    // second search while others still compare the first one's list.
    unsigned key_lo[4], key_hi[4];
    int listed[4];
    __device__ void start(int slot) {
        key_lo[slot] = 0xffffffffu;
        key_hi[slot] = 0u;
        listed[slot] = 0;
    }
    ThresholdList by_count;
    union {
        ThresholdList by_mass;
        float chunk_sum[CL_THREADS];          // of the draw
    };
};
__device__ __forceinline__ unsigned long long mass_of(float e) { return (unsigned long long)(e * 17592186044416.0f); }

__device__ __forceinline__ void add_mass(unsigned (*hist)[BINS], int b, unsigned long long w) {
    const unsigned lo = (unsigned)w & 0x7fffu, mid = (unsigned)(w >> 15) & 0x7fffu, hi = (unsigned)(w >> 30);
    if (lo) atomicAdd(&hist[0][b], lo);
    if (mid) atomicAdd(&hist[1][b], mid);
    if (hi) atomicAdd(&hist[2][b], hi);
}

// Of counts (MASS false): `share` is how many values; with `scale` > 0 the first bins are 1 / scale wide below `top` (rows of
// numbers), else they are steps of 2^24 keys.  Of masses: `share` of the whole mass; the values that are not zero take part,
// `top` is the smallest of them (or zero); with `few` they are known to fit in the list, which saves the bins.
template <bool MASS>
__device__ __forceinline__ unsigned cluster_threshold(Threshold* th, const float* mine, int n, float top, float scale, float share, bool few) {
    cg::cluster_group cl = cg::this_cluster();
    constexpr int UNROLL = 4, PARTS = MASS ? 3 : 1;
    const int tid = threadIdx.x, lane = tid & 31;
    bool linear = !MASS && scale > 0.0f;
    // the keys in play lie up to `reach` below `hi` (the largest mass is one), and the bins are made for a span of them: masses below
    // 2^-20 share the last bin (most values of a wide row are there, and few sums need them)
    unsigned hi = MASS ? ordered_key(1.0f) : 0xffffffffu, reach = MASS ? hi - (ordered_key(0.0f) + 1u) : hi;
    unsigned span = MASS ? hi - max(ordered_key(top), ordered_key(9.5367432e-7f)) : hi;
    unsigned long long before = 0ull, need = 0ull;
    Threshold* zero = cl.map_shared_rank(th, 0);
    for (int level = 0;; ++level) {
        const int slot = (MASS ? 2 : 0) + (level & 1);
        int first_rank = 0;          // (opaque, so that the eight blocks' addresses are made where they are used and not held in registers)
        asm volatile("" : "+r"(first_rank));
        // (span - 1) >> shift < BINS; all of a few in bin 0
        const int shift = MASS && few ? 31 : span <= (unsigned)BINS ? 0 : 24 - __clz(span - 1u);
        // the bins of UNROLL values from i0 on, higher values in lower bins; -1: not in play
        float x[UNROLL];
        int b[UNROLL];
        auto bins_from = [&](int i0) {
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                const int i = i0 + u * CL_THREADS + tid;
                x[u] = i < n ? mine[i] : 0.0f;
                b[u] = i < n ? 0 : -1;
            }
            if (linear) {
#pragma unroll
                for (int u = 0; u < UNROLL; ++u) b[u] |= (int)fminf((top - x[u]) * scale, (float)(BINS - 1));
            } else {
#pragma unroll
                for (int u = 0; u < UNROLL; ++u) {
                    const unsigned below = hi - (MASS ? __float_as_uint(x[u]) | 0x80000000u : ordered_key(x[u]));
                    b[u] |= below <= reach ? (int)min(below >> shift, (unsigned)(BINS - 1)) : -1;
                }
            }
        };
        int bin = 0;
        if (!(MASS && few)) {
            if (tid == 0 && (!MASS || level > 0)) th->start(slot);
            for (int i = tid; i < PARTS * BINS; i += CL_THREADS) (&th->hist[0][0])[i] = 0u;
            __syncthreads();
            unsigned long long least = 0ull;
#pragma unroll 1
            for (int i0 = 0; i0 < n; i0 += UNROLL * CL_THREADS) {
                bins_from(i0);
#pragma unroll
                for (int u = 0; u < UNROLL; ++u) {
                    if (b[u] < 0) continue;
                    const unsigned long long w = MASS ? mass_of(x[u]) : 1ull;
                    if (b[u] == BINS - 1) least += w;
                    else if (MASS) add_mass(th->hist, b[u], w);
                    else atomicAdd(&th->hist[0][b[u]], 1u);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) least += __shfl_xor_sync(0xffffffffu, least, o);
            if (lane == 0) {
                if (MASS) add_mass(th->hist, BINS - 1, least);
                else atomicAdd(&th->hist[0][BINS - 1], (unsigned)least);
            }
            cl.sync();
            // the bins of all blocks, as running sums
            unsigned long long own = 0ull, upto = 0ull;
            if (tid < BINS) {
#pragma unroll
                for (int r = 0; r < CL; ++r) {
                    const Threshold* o = cl.map_shared_rank(th, first_rank + r);
                    own += o->hist[0][tid];
                    if (MASS) own += ((unsigned long long)o->hist[1][tid] << 15) + ((unsigned long long)o->hist[2][tid] << 30);
                }
                upto = own;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned long long up = __shfl_up_sync(0xffffffffu, upto, o);
                    if (lane >= o) upto += up;
                }
                if (lane == 31) th->warp_total[tid >> 5] = upto;
            }
            __syncthreads();
            unsigned long long total = 0ull;
#pragma unroll
            for (int w = 0; w < BINS / 32; ++w) {
                if (w < (tid >> 5)) upto += th->warp_total[w];
                total += th->warp_total[w];
            }
            if (level == 0) need = max(MASS ? (unsigned long long)((double)share * (double)total) : (unsigned long long)share, 1ull);
            if (tid < BINS && before + upto - own < need && before + upto >= need) {          // one thread of the block
                th->bin = tid;
                th->before = before + upto - own;
                th->upto = before + upto;
            }
            __syncthreads();
            bin = th->bin;
            before = th->before;
        }
        // the bin's values: the keys that they span, and a list of them for every block as long as there is room
        unsigned key_lo = 0xffffffffu, key_hi = 0u;
        bool full = false;
#pragma unroll 1
        for (int i0 = 0; i0 < n; i0 += UNROLL * CL_THREADS) {
            bins_from(i0);
            bool any = false;
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) any |= b[u] == bin;
            if (!__any_sync(0xffffffffu, any)) continue;
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) {
                const bool member = b[u] == bin;
                const unsigned members = __ballot_sync(0xffffffffu, member);
                const unsigned key = ordered_key(x[u]);
                if (member) {
                    key_lo = min(key_lo, key);
                    key_hi = max(key_hi, key);
                }
                if (members == 0u || full) continue;
                const int first = __ffs(members) - 1;
                int at = 0;
                if (lane == first) at = atomicAdd(&zero->listed[slot], __popc(members));
                at = __shfl_sync(0xffffffffu, at, first);
                full = at >= BIN_LIST;
                at += __popc(members & ((1u << lane) - 1u));
                if (member && at < BIN_LIST) {
                    const unsigned long long w = MASS ? mass_of(x[u]) : 1ull;
#pragma unroll 1
                    for (int r = 0; r < CL; ++r) {
                        Threshold* o = cl.map_shared_rank(th, first_rank + r);
                        ThresholdList& list = MASS ? o->by_mass : o->by_count;
                        list.key[at] = key;
                        list.weight[at] = w;
                    }
                }
            }
        }
        key_lo = __reduce_min_sync(0xffffffffu, key_lo);
        key_hi = __reduce_max_sync(0xffffffffu, key_hi);
        if (lane == 0 && key_lo <= key_hi) {
            atomicMin(&th->key_lo[slot], key_lo);
            atomicMax(&th->key_hi[slot], key_hi);
        }
        cl.sync();
        const int m = zero->listed[slot];
        const Threshold* some = cl.map_shared_rank(th, lane % CL);
        hi = __reduce_max_sync(0xffffffffu, some->key_hi[slot]);
        reach = span = hi - __reduce_min_sync(0xffffffffu, some->key_lo[slot]);
        if (span == 0u) {
            if (tid == 0) th->reached = th->upto;
            return hi;
        }
        if (m <= BIN_LIST) {
            const ThresholdList& list = MASS ? th->by_mass : th->by_count;
            const int i = tid >> 2;
            const unsigned key = i < m ? list.key[i] : 0u;
            unsigned long long above = before, with = before;
            unsigned long long total = 0ull;
            if (i < m) {
                if (tid & 3) above = with = 0ull;
                for (int j = tid & 3; j < m; j += 4) {
                    const unsigned k = list.key[j];
                    const unsigned long long w = list.weight[j];
                    if (k > key) above += w;
                    if (k >= key) with += w;
                    if (MASS && few) total += w;
                }
            }
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                above += __shfl_xor_sync(0xffffffffu, above, o);
                with += __shfl_xor_sync(0xffffffffu, with, o);
                if (MASS && few) total += __shfl_xor_sync(0xffffffffu, total, o);
            }
            if (MASS && few) need = max((unsigned long long)((double)share * (double)total), 1ull);
            if (i < m && above < need && with >= need) {          // equal keys write the same
                th->value = key;
                th->reached = with;
            }
            __syncthreads();
            return th->value;
        }
        linear = false;
    }
}

// First index of the largest value of the whole row (0 if nothing lies above -inf), the same in every block.
__device__ int cluster_argmax(cg::cluster_group& cl, ClusterExchange* xc, const float* x, int begin, int n, float* shf,
                              int* shi) {
    const int local = n > 0 ? block_argmax(x + begin, n, shf, shi, -1) : -1;
    const int t = xc->turn;
    if (threadIdx.x == 0) {
        xc->f[t] = local >= 0 ? x[begin + local] : -INFINITY;
        xc->i[t] = local >= 0 ? begin + local : -1;
    }
    cl.sync();
    float best = -INFINITY;
    int at = -1;
#pragma unroll
    for (int b = 0; b < CL; ++b) {          // ascending ranks hold ascending indices: a later equal value does not win
        const ClusterExchange* o = cl.map_shared_rank(xc, b);
        const int oi = o->i[t];
        const float ov = o->f[t];
        if (oi >= 0 && (at < 0 || ov > best)) { best = ov; at = oi; }
    }
    __syncthreads();
    if (threadIdx.x == 0) xc->turn = t ^ 1;
    __syncthreads();
    return at < 0 ? 0 : at;
}

__global__ void __launch_bounds__(CL_THREADS, 3) sample_cluster_kernel(const float* __restrict__ logits, int V, long long stride,
                                                                    int part, const float* __restrict__ temperature,
                                                                    const int* __restrict__ top_k,
                                                                    const float* __restrict__ top_p,
                                                                    const float* __restrict__ min_p,
                                                                    const float* __restrict__ uniform,
                                                                    int* __restrict__ out) {
    extern __shared__ float mine[];            // this block's `part` elements of the row
    __shared__ Threshold th;
    __shared__ float shf[33];
    __shared__ int shi[33];
    __shared__ ClusterExchange xc;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const int r = blockIdx.y;
    const float* x = logits + (size_t)r * stride;
    const int begin = min(V, rank * part);
    const int n = min(part, V - begin);          // may be 0 for the last ranks of a short row
    if (threadIdx.x == 0) {
        xc.turn = 0;
        th.start(2);
    }
    __syncthreads();

    const float temp = temperature[r];
    if (temp < 1e-5f) {
        const int idx = cluster_argmax(cl, &xc, x, begin, n, shf, shi);
        if (rank == 0 && threadIdx.x == 0) out[r] = idx;
        cl.sync();                               // no block leaves while another may still read its shared memory
        return;
    }
    const float inv_temp = 1.0f / fmaxf(temp, 1e-8f);
    const int k = top_k ? top_k[r] : 0;
    const float tp = top_p ? top_p[r] : 1.0f;
    const float mp = min_p ? min_p[r] : 0.0f;

    const bool by_rank = k > 0 && k < V, by_mass = tp < 1.0f;
    float mx = -INFINITY, low = -INFINITY;          // low: minus the smallest finite value; +inf where a value is not a number
    if (by_rank || by_mass) {
        for (int i = threadIdx.x; i < n; i += CL_THREADS) {
            const float v = x[begin + i] * inv_temp;
            mine[i] = v;
            mx = fmaxf(mx, v);
            low = fmaxf(low, v == v ? (v > -INFINITY ? -v : -INFINITY) : INFINITY);
        }
        cluster_max2(cl, &xc, mx, low, shf);
    } else {
        for (int i = threadIdx.x; i < n; i += CL_THREADS) {
            const float v = x[begin + i] * inv_temp;
            mine[i] = v;
            mx = fmaxf(mx, v);
        }
        mx = cluster_max(cl, &xc, block_max(mx, shf));
    }
    if (mx == -INFINITY || !(mx == mx)) {        // every logit is -inf, or NaN: fall back to argmax
        const int idx = cluster_argmax(cl, &xc, x, begin, n, shf, shi);
        if (rank == 0 && threadIdx.x == 0) out[r] = idx;
        cl.sync();
        return;
    }

    // top-k: key of the k-th largest scaled logit (largest K with count(key >= K) >= k).  The first bins are 1/8 wide below the maximum,
    // and narrower where the whole row is narrower than they reach; a row with infinite values or NaN goes by keys alone.
    unsigned key_k = 0u;
    if (threadIdx.x == 0) {
        th.top = mx;
        th.low = low;
        th.reached = (unsigned long long)V;
    }
    __syncthreads();
    if (by_rank) {
        float scale = BINS / 32.0f;
        if (mx + low > 0.0f) scale = fmaxf(scale, fminf((float)(BINS - 1) / (mx + low), 1e30f));
        key_k = cluster_threshold<false>(&th, mine, n, mx, mx < INFINITY && low < INFINITY ? scale : 0.0f, (float)k, false);
        __syncthreads();
    }
    mx = th.top;
    // e_i = exp(x_i/T - max) of the kept entries; everything below is in terms of e (max e = 1).
    for (int i = threadIdx.x; i < n; i += CL_THREADS) {
        const float v = mine[i];
        mine[i] = ordered_key(v) < key_k ? 0.0f : expf(v - mx);
    }
    // top-p: largest threshold on e whose kept mass still reaches p of the whole.
    unsigned key_p = 0u;
    if (by_mass) {
        float least = expf(key_k ? key_value(key_k) - mx : -(mx + th.low));          // the smallest
        if (!(mx < INFINITY && th.low < INFINITY)) {          // where one is not a number, everything stays, and the draw falls back to the argmax
            least = -1.0f;
            for (int i = threadIdx.x; i < n; i += CL_THREADS) least = mine[i] == mine[i] ? least : INFINITY;
            least = cluster_max(cl, &xc, block_max(least, shf)) > 0.0f ? -1.0f : 0.0f;
        }
        if (least >= 0.0f) key_p = tp > 0.0f ? cluster_threshold<true>(&th, mine, n, least, 0.0f, tp, th.reached <= (unsigned long long)BIN_LIST) : 0xffffffffu;
    }
    // min-p: probabilities below min_p * max probability are dropped; max e is 1.  What is kept stays in `mine`.
    const float e_min = mp > 0.0f ? mp : 0.0f;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += CL_THREADS) {
        const float e = mine[i];
        if (e <= 0.0f || ordered_key(e) < key_p || e < e_min) mine[i] = 0.0f;
    }
    __syncthreads();

    // Draw: first index whose running mass reaches u * total.  Threads own contiguous chunks of their block's part,
    // blocks contiguous parts of the row.
    const int per = (part + CL_THREADS - 1) / CL_THREADS;
    const int cb = min(n, (int)threadIdx.x * per), ce = min(n, cb + per);
    float own = 0.0f;
    for (int i = cb; i < ce; ++i) own += mine[i];
    th.chunk_sum[threadIdx.x] = own;
    const float block_total = block_sum(own, shf);      // contains the barriers that publish chunk_sum
    // every block learns every block's total (the same exchange as cluster_max, but the parts are kept and added up in rank order)
    const int t = xc.turn;
    if (threadIdx.x == 0) xc.f[t] = block_total;
    cl.sync();
    float totals[CL];
    float total = 0.0f;
#pragma unroll
    for (int b = 0; b < CL; ++b) {
        totals[b] = cl.map_shared_rank(&xc, b)->f[t];
        total += totals[b];
    }
    __syncthreads();
    if (threadIdx.x == 0) xc.turn = t ^ 1;
    __syncthreads();
    if (!(total > 0.0f)) {                               // nothing kept (cannot happen with max e = 1, but stay safe)
        const int idx = cluster_argmax(cl, &xc, x, begin, n, shf, shi);
        if (rank == 0 && threadIdx.x == 0) out[r] = idx;
        cl.sync();
        return;
    }
    // the block in whose part the running mass reaches the target; if rounding leaves the target above the total,
    // the last block with mass, which then takes its last entry with mass
    const float target = uniform[r] * total;
    float run = 0.0f;
    int chosen = -1, last_with_mass = -1;
#pragma unroll
    for (int b = 0; b < CL; ++b) {
        if (chosen >= 0) continue;
        if (totals[b] > 0.0f) {
            last_with_mass = b;
            if (run + totals[b] >= target) { chosen = b; continue; }
        }
        run += totals[b];
    }
    const bool overshoot = chosen < 0;
    if (overshoot) chosen = last_with_mass;
    if (rank == chosen && threadIdx.x == 0) {
        int choice = -1;
        if (!overshoot) {
            int c = 0;
            for (; c < CL_THREADS; ++c) {
                if (th.chunk_sum[c] > 0.0f && run + th.chunk_sum[c] >= target) break;
                run += th.chunk_sum[c];
            }
            if (c < CL_THREADS) {
                const int b0 = min(n, c * per), e0 = min(n, b0 + per);
                int last_mass = -1;
                for (int i = b0; i < e0; ++i) {
                    const float m = mine[i];
                    if (m > 0.0f) {
                        last_mass = i;
                        run += m;
                        if (run >= target) { choice = i; break; }
                    }
                }
                if (choice < 0) choice = last_mass;
            }
        }
        if (choice < 0) {      // rounding left the target above the running mass: this block's last entry with mass
            for (int i = n - 1; i >= 0 && choice < 0; --i)
                if (mine[i] > 0.0f) choice = i;
        }
        out[r] = begin + choice;      // totals[chosen] > 0, so the block has an entry with mass
    }
    cl.sync();
}

}  // namespace

// logits [R, V] float with row stride `stride` elements; out [R] int32.  scratch (or null): 3 * scratch_rows ints,
// 8-byte aligned, zero on entry and left zero; with it, rows of 4 * 4096 elements or more are shared among blocks.
LLB_EXPORT int llb_argmax(const float* logits, int R, int V, long long stride, int* out, int* scratch, int scratch_rows,
                          cudaStream_t stream) {
    if (R == 0) return 0;
    LLB_REQUIRE(R > 0 && V > 0 && stride >= V, "argmax: bad sizes R=%d V=%d stride=%lld", R, V, stride);
    if (scratch && R <= scratch_rows && R <= 65535 && V >= 4 * SPLIT_ELEMS && (uintptr_t)scratch % 8 == 0) {
        unsigned long long* slots = (unsigned long long*)scratch;
        int* counters = scratch + 2 * (size_t)scratch_rows;
        argmax_split_kernel<<<dim3(llb_ceil_div(V, SPLIT_ELEMS), R), SPLIT_THREADS, 0, stream>>>(logits, V, stride, slots,
                                                                                               counters, out);
        return llb_check_launch("argmax");
    }
    argmax_kernel<<<R, THREADS, 0, stream>>>(logits, V, stride, out);
    return llb_check_launch("argmax");
}

// Per row: temperature [R]; top_k [R] int (0 = off) or null; top_p [R] (1 = off) or null;
// min_p [R] (0 = off) or null; uniform [R] in [0, 1).  out [R] int32.
LLB_EXPORT int llb_sample(const float* logits, int R, int V, long long stride, const float* temperature,
                          const int* top_k, const float* top_p, const float* min_p, const float* uniform, int* out,
                          cudaStream_t stream) {
    if (R == 0) return 0;
    LLB_REQUIRE(R > 0 && V > 0 && stride >= V, "sample: bad sizes R=%d V=%d stride=%lld", R, V, stride);
    LLB_REQUIRE(temperature && uniform && out, "sample: null argument");
    // long rows: a cluster of blocks per row, each with its part of the row in shared memory
    const int part = llb_ceil_div(V, CL);
    const size_t smem = (size_t)part * sizeof(float);
    if (V >= 8192 && smem <= 216 * 1024 && R <= 65535) {          // (beside it 7 KB of the kernel's own)
        static size_t configured = 0;
        if (smem > configured) {
            cudaError_t e = cudaFuncSetAttribute(sample_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return llb_fail("sample: cannot opt in to %zu bytes of shared memory: %s", smem,
                                                  cudaGetErrorString(e));
            configured = smem;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(CL, R);
        cfg.blockDim = dim3(CL_THREADS);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = CL;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        cudaError_t e = cudaLaunchKernelEx(&cfg, sample_cluster_kernel, logits, V, stride, part, temperature, top_k, top_p,
                                           min_p, uniform, out);
        if (e != cudaSuccess) return llb_fail("sample: launch failed: %s", cudaGetErrorString(e));
        return llb_check_launch("sample");
    }
    sample_kernel<<<R, THREADS, 0, stream>>>(logits, V, stride, temperature, top_k, top_p, min_p, uniform, out);
    return llb_check_launch("sample");
}

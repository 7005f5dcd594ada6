// The contraction of the decode step (at most 64 rows) on the tensor cores, fused with what stands
// before and after it so that a layer needs five launches instead of nine:
//
//   prologue NORM      the B operand is RMSNorm(residual) * weight, built by the block itself in shared
//                      memory (src/ops/norm.cu:19-55), instead of a separate norm kernel;
//   epilogue ROPE_KV   bias, rotary positions on q and k (src/ops/rope.cu:54-59, every pair), q to its
//                      buffer, k and v into their cache pages (src/kv_cache/paged_attention.cu:1150-1163);
//   epilogue SWIGLU    SiLU(gate) * up on interleaved weight rows (src/engine/engine_server.cpp:1875-1878);
//   epilogue RESIDUAL  adds into the float residual stream (engine_server.cpp:1870-1871);
//   epilogue STORE     bf16 output, optionally through a plain activation;
//   epilogue STORE_F32 float output (the head's logits).
//
// The weights take the MMA's 128-row A role and stream through a TMA ring; the few activation rows are
// the B operand (BN = 16, 32 or 64 columns of tensor memory).  Few tiles of features over a long K are cut along K among the
// blocks of a thread-block cluster: every block sends the sums it has of a token straight into the shared memory of the block
// that finishes that token (token t: block t mod C), the cluster meets once, and each block adds up and finishes its tokens in a
// fixed order.  A block alone does the same within its own shared memory.  So the epilogue reads its features side by side,
// whatever the tensor memory's layout, and is spread over eight warps of every block.  Measured (us that the launch adds to the chain
// of a step at the 0.5B sizes; four epilogue warps on the accumulators' layout and adds into memory -> now): 64 rows gate/up 16.3 ->
// 10.2, q/k/v 10.0 -> 8.0, o_proj 6.9 -> 6.4; 32 rows gate/up 11.5 -> 7.4, q/k/v 9.5 -> 5.6.  What bounds it: the launch before must have
// completed (1 us), then activations, products, the meeting and the outputs, each a trip to L2 or to another multiprocessor of
// half a microsecond to one; the weights' 17 MB of gate/up are 2.7 us of the copy rate.
//
// Every launch is a programmatic dependent
// launch: a block initialises its barriers, allocates tensor memory and already requests its first weight
// tiles while the kernel before it is still running, and only then waits for that kernel
// (griddepcontrol.wait) before it reads activations or writes anything.  Waits on mbarriers are bounded
// in time as in the other tensor-core kernels.
#include <atomic>
#include <utility>

#include "tcgen05_common.cuh"

namespace {

using namespace t5;

constexpr int TILE_M = 128;
constexpr int TILE_K = 64;
// Depth of the TMA ring: a block streams its weights at (bytes in flight) / latency.  Grids of a few blocks
// get a deep ring (8 stages, one block per SM; 6 where the received sums of 64 rows lie beside it); grids of many blocks (the
// head) a short one (4 stages), so that two blocks share an SM.
constexpr int DEEP = 8, MIDDLE = 6, SHALLOW = 4;
constexpr int WORKERS = 256;                // warps 2-9
constexpr int NUM_THREADS = 64 + WORKERS;
constexpr int MAX_CLUSTER = 8;
constexpr uint32_t A_BYTES = TILE_M * TILE_K * 2;

enum { DEPI_STORE_F32 = 1, DEPI_RESIDUAL = 2, DEPI_SWIGLU = 3, DEPI_ROPE_KV = 4, DEPI_STORE = 5 };

struct DecodeGemmParams {
    // NORM prologue
    const float* x;            // [*, K] float residual rows
    const int* x_rows;         // row r of the operand is x[x_rows[r]], or null for x[r]
    const void* norm_w;        // [K]
    int norm_w_bf16;
    float eps;
    // common
    const float* bias;         // [N] or null
    void* out;                 // SWIGLU: bf16 [M, N/2]; STORE_F32: float [M, N]
    float* residual;           // RESIDUAL: [M, N]
    int M, N, K, num_kb, kb_per_split;
    // ROPE_KV epilogue
    const int* slot_mapping;   // [M] cache row of each token, or null: nothing is written to the cache
    const float2* rope_table;  // [M, rotary_dim / 2] of (cos, sin) of pos * inv_freq
    int rotary_dim, interleaved, Hq, Hkv, hd;
    __nv_bfloat16* q_out;      // [M, Hq * hd]
    __nv_bfloat16* k_cache;    // [slots, Hkv, hd]
    __nv_bfloat16* v_cache;
    int cluster;               // blocks of a cluster: neighbouring pieces of K whose sums meet (1: a block alone)
    uint32_t recv_offset;      // where they meet, behind the operand tiles (over the weight ring when alone)
    int* error_flag;
    LlbGluArgs glu;            // the gated activation of the GLU epilogue, the plain one of STORE, the scale of the float ones
};

// How the rotary epilogue treats one output feature n (row `row` of the block's tile): whether it is rotated, with
// which row of the tile it pairs, which frequency it uses, and whether it is the pair's first member.
struct RopeRow {
    bool rotate, first;
    int partner, fi;
};
__device__ __forceinline__ RopeRow rope_row(const DecodeGemmParams& p, int n, int row) {
    RopeRow r;
    const int q_end = p.Hq * p.hd, k_end = q_end + p.Hkv * p.hd;
    const int head_row = n % p.hd;                    // q, k and v sections are multiples of hd
    const int half = p.rotary_dim / 2;
    r.rotate = n < p.N && n < k_end && head_row < p.rotary_dim;
    r.partner = row;
    r.fi = 0;
    r.first = true;
    if (r.rotate) {
        if (p.interleaved) { r.first = (head_row & 1) == 0; r.partner = r.first ? row + 1 : row - 1; r.fi = head_row >> 1; }
        else { r.first = head_row < half; r.partner = r.first ? row + half : row - half; r.fi = r.first ? head_row : head_row - half; }
    }
    return r;
}
// (cos, sin) and cache rows of four of the block's tokens (i0, i0 + 2, ..) for that feature; the loads do not depend on each other.
constexpr int ROPE_BATCH = 4;
__device__ __forceinline__ void rope_fetch(const DecodeGemmParams& p, const RopeRow& r, int n, int rank, int i0, int mine,
                                           float2 (&cs)[ROPE_BATCH], int (&slot)[ROPE_BATCH]) {
    const bool cached = n < p.N && n >= p.Hq * p.hd && p.slot_mapping != nullptr;
#pragma unroll
    for (int u = 0; u < ROPE_BATCH; ++u) {
        const int i = i0 + u * (WORKERS / TILE_M), m = rank + i * p.cluster;
        cs[u] = (r.rotate && i < mine) ? __ldg(p.rope_table + (size_t)m * (p.rotary_dim / 2) + r.fi) : make_float2(1.0f, 0.0f);
        slot[u] = (cached && i < mine) ? __ldg(p.slot_mapping + m) : -1;
    }
}
// The sum of what the blocks of the cluster sent of one token's features, in the order of K: slot i of every source, `slots` apart.
__device__ __forceinline__ float2 recv_pair(const float* recv, int cluster, int slots, int i, int f) {
    float2 v = *reinterpret_cast<const float2*>(recv + i * TILE_M + f);
    for (int src = 1; src < cluster; ++src) {
        const float2 u = *reinterpret_cast<const float2*>(recv + (src * slots + i) * TILE_M + f);
        v.x += u.x;
        v.y += u.y;
    }
    return v;
}
__device__ __forceinline__ float recv_one(const float* recv, int cluster, int slots, int i, int f) {
    float v = recv[i * TILE_M + f];
    for (int src = 1; src < cluster; ++src) v += recv[(src * slots + i) * TILE_M + f];
    return v;
}
// One token m and two neighbouring features n, n + 1 (n even).
template <int EPI>
__device__ __forceinline__ void finish_pair(const DecodeGemmParams& p, float2 v, float2 bias, int m, int n, bool alone) {
    const bool has1 = n + 1 < p.N;
    v.x += bias.x;
    v.y += bias.y;
    if (EPI == DEPI_SWIGLU) {
        if (has1)
            ((__nv_bfloat16*)p.out)[(size_t)m * (p.N / 2) + (n >> 1)] =
                __float2bfloat16_rn(llb_glu(v.x, v.y, p.glu.kind, p.glu.alpha, p.glu.limit, p.glu.up_shift));
        return;
    }
    const size_t at = (size_t)m * p.N + n;
    if (EPI == DEPI_STORE) {
        __nv_bfloat16* o = (__nv_bfloat16*)p.out + at;
        const __nv_bfloat162 h = __floats2bfloat162_rn(llb_act(v.x, p.glu.kind), llb_act(v.y, p.glu.kind));
        if (has1 && ((uintptr_t)o & 3) == 0) {
            *reinterpret_cast<__nv_bfloat162*>(o) = h;
        } else {
            o[0] = h.x;
            if (has1) o[1] = h.y;
        }
        return;
    }
    const float f = llb_out_scale(p.glu);
    v.x *= f;
    v.y *= f;
    float* o = (EPI == DEPI_STORE_F32 ? (float*)p.out : p.residual) + at;
    if (EPI == DEPI_RESIDUAL && !alone) {
        if (has1 && ((uintptr_t)o & 7) == 0) {
            asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(o), "f"(v.x), "f"(v.y) : "memory");
        } else {
            atomicAdd(o, v.x);
            if (has1) atomicAdd(o + 1, v.y);
        }
    } else if (has1 && ((uintptr_t)o & 7) == 0) {
        if (EPI == DEPI_RESIDUAL) {
            const float2 r = *reinterpret_cast<const float2*>(o);
            v.x += r.x;
            v.y += r.y;
        }
        *reinterpret_cast<float2*>(o) = v;
    } else {
        o[0] = EPI == DEPI_RESIDUAL ? o[0] + v.x : v.x;
        if (has1) o[1] = EPI == DEPI_RESIDUAL ? o[1] + v.y : v.y;
    }
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&r)[8]) {
    uint32_t* u = reinterpret_cast<uint32_t*>(r);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "r"(taddr)
                 : "memory");
    tmem_wait_ld();
}

// (Rings of up to five stages are for two blocks on a multiprocessor: ten warps lie three to a scheduler, so that both fit only from 80
// registers down; the bound for three blocks gives 64.)
template <int BN, int EPI, bool NORM, int STAGES>
__global__ void __launch_bounds__(NUM_THREADS, STAGES <= 5 ? 3 : 1)
gemm_decode_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                   const DecodeGemmParams p) {
    constexpr uint32_t B_BYTES = BN * TILE_K * 2;
    constexpr uint32_t TMEM_COLS = BN < 32 ? 32 : BN;
    __shared__ __align__(8) uint64_t full_bar[8];
    __shared__ __align__(8) uint64_t empty_bar[8];
    __shared__ __align__(8) uint64_t acc_bar, b_ready_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_s;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* a_tiles = smem;                             // STAGES weight tiles
    uint8_t* b_tiles = smem + STAGES * A_BYTES;          // NORM: num_kb resident tiles; else STAGES tiles
    float* recv = (float*)(smem + p.recv_offset);        // [cluster][slots][128]: this block's tokens' sums, from every block
    volatile int* abort_flag = &abort_s;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * TILE_M;                  // first weight row (output feature) of the block
    const int kb_begin = blockIdx.z * p.kb_per_split;
    const int kb_end = min(p.num_kb, kb_begin + p.kb_per_split);
    const int nkb = kb_end - kb_begin;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&acc_bar, 1);
        mbar_init(&b_ready_bar, 128);
        abort_s = 0;
        mbar_init_fence();
    }
    if (warp == 1) tmem_alloc(&tmem_slot, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;
    if (threadIdx.x == 0) griddep_launch_dependents();
    // the others of the cluster have begun: waited for before anything is sent to them
    __syncwarp();
    if (p.cluster > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    const int rank = (int)blockIdx.z % p.cluster, slots = (BN + p.cluster - 1) / p.cluster;
    bool ok = true;
    RopeRow rr;                     // the rotary epilogue's feature and first tokens
    float2 cs[ROPE_BATCH];
    int slot_of[ROPE_BATCH];

    {
        if (warp == 0) {
            if (lane == 0) {
                // Weights do not depend on the kernel before this one: request the first tiles at once.
                const int pre = min(STAGES, nkb);
                for (int i = 0; i < pre; ++i) {
                    mbar_expect_tx(&full_bar[i], A_BYTES + (NORM ? 0u : B_BYTES));
                    tma_load_2d(a_tiles + i * A_BYTES, &map_w, (kb_begin + i) * TILE_K, n0, &full_bar[i]);
                }
                griddep_wait();
                if (!NORM)
                    for (int i = 0; i < pre; ++i)
                        tma_load_2d(b_tiles + i * B_BYTES, &map_x, (kb_begin + i) * TILE_K, 0, &full_bar[i]);
                for (int i = pre; i < nkb; ++i) {
                    const int s = i % STAGES;
                    if (!mbar_wait(&empty_bar[s], ((i / STAGES) & 1) ^ 1, abort_flag)) break;
                    mbar_expect_tx(&full_bar[s], A_BYTES + (NORM ? 0u : B_BYTES));
                    tma_load_2d(a_tiles + s * A_BYTES, &map_w, (kb_begin + i) * TILE_K, n0, &full_bar[s]);
                    if (!NORM) tma_load_2d(b_tiles + s * B_BYTES, &map_x, (kb_begin + i) * TILE_K, 0, &full_bar[s]);
                }
            }
        } else if (warp == 1) {
            if (lane == 0) {
                constexpr uint32_t idesc = idesc_bf16(TILE_M, BN);
                if (NORM) ok = mbar_wait(&b_ready_bar, 0, abort_flag);
                for (int i = 0; i < nkb && ok; ++i) {
                    const int s = i % STAGES;
                    ok = mbar_wait(&full_bar[s], (i / STAGES) & 1, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(a_tiles + s * A_BYTES);
                    const uint32_t b_addr = smem_u32(b_tiles + (size_t)(NORM ? kb_begin + i : s) * B_BYTES);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_bf16(tmem_base, desc_kmajor(a_addr + k * 32), desc_kmajor(b_addr + k * 32), idesc,
                                  (i > 0 || k > 0) ? 1u : 0u);
                    umma_commit(&empty_bar[s]);
                }
                if (ok) umma_commit(&acc_bar);
            }
        } else {
            griddep_wait();
            if (NORM && warp < 6) {
                // B operand = RMSNorm(x) * w for all K, as bf16 in the swizzled K-major tiles.  One warp per row.
                if (p.K <= 1024 && p.M <= 8) {
                    // Few short rows: a warp asks for both of its rows at once and keeps them in registers (8 float4
                    // per lane and row), so the statistics and the scaled copy cost one trip to memory, not four.
                    const int ra = warp - 2, rb = warp + 2;
                    const bool has_a = ra < p.M, has_b = rb < p.M;
                    const float* xa = p.x + (size_t)(has_a ? (p.x_rows ? p.x_rows[ra] : ra) : 0) * p.K;
                    const float* xb = p.x + (size_t)(has_b ? (p.x_rows ? p.x_rows[rb] : rb) : 0) * p.K;
                    float4 va[8], vb[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int k = (i * 32 + lane) * 4;
                        const bool in_k = k < p.K;
                        va[i] = (has_a && in_k) ? *reinterpret_cast<const float4*>(xa + k) : make_float4(0.f, 0.f, 0.f, 0.f);
                        vb[i] = (has_b && in_k) ? *reinterpret_cast<const float4*>(xb + k) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                    float sa = 0.0f, sb = 0.0f;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        sa += va[i].x * va[i].x + va[i].y * va[i].y + va[i].z * va[i].z + va[i].w * va[i].w;
                        sb += vb[i].x * vb[i].x + vb[i].y * vb[i].y + vb[i].z * vb[i].z + vb[i].w * vb[i].w;
                    }
                    sa = llb_warp_sum(sa);
                    sb = llb_warp_sum(sb);
                    const float inva = 1.0f / sqrtf(sa / (float)p.K + p.eps), invb = 1.0f / sqrtf(sb / (float)p.K + p.eps);
                    // rows of the tile beyond M stay as they are: what the MMA makes of them is never read
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int k = (i * 32 + lane) * 4;       // 4 elements = half of a 16-byte chunk of the tile row
                        if ((k >> 6) < kb_begin || (k >> 6) >= kb_end) continue;
                        // columns from K to the end of the last tile are written as zeros: the weights there are the
                        // copy's zero fill, but zero times whatever the shared memory held before need not be zero
                        float nw[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                        if (k < p.K && p.norm_w_bf16) {
                            const uint2 u = *reinterpret_cast<const uint2*>((const __nv_bfloat16*)p.norm_w + k);
                            const float2 f0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
                            const float2 f1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
                            nw[0] = f0.x; nw[1] = f0.y; nw[2] = f1.x; nw[3] = f1.y;
                        } else if (k < p.K) {
                            const float4 c0 = *reinterpret_cast<const float4*>((const float*)p.norm_w + k);
                            nw[0] = c0.x; nw[1] = c0.y; nw[2] = c0.z; nw[3] = c0.w;
                        }
                        const int kb = k >> 6, q = (k & 63) >> 3, sub = (k & 7) * 2;       // tile, chunk, byte offset in it
                        if (has_a) {
                            const __nv_bfloat162 h0 = __floats2bfloat162_rn(va[i].x * inva * nw[0], va[i].y * inva * nw[1]);
                            const __nv_bfloat162 h1 = __floats2bfloat162_rn(va[i].z * inva * nw[2], va[i].w * inva * nw[3]);
                            uint8_t* dst = b_tiles + (size_t)kb * B_BYTES + (uint32_t)ra * 128 + ((q ^ (ra & 7)) * 16) + sub;
                            *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&h0),
                                                                        *reinterpret_cast<const uint32_t*>(&h1));
                        }
                        if (has_b) {
                            const __nv_bfloat162 h0 = __floats2bfloat162_rn(vb[i].x * invb * nw[0], vb[i].y * invb * nw[1]);
                            const __nv_bfloat162 h1 = __floats2bfloat162_rn(vb[i].z * invb * nw[2], vb[i].w * invb * nw[3]);
                            uint8_t* dst = b_tiles + (size_t)kb * B_BYTES + (uint32_t)rb * 128 + ((q ^ (rb & 7)) * 16) + sub;
                            *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&h0),
                                                                        *reinterpret_cast<const uint32_t*>(&h1));
                        }
                    }
                } else
                for (int r = warp - 2; r < BN; r += 4) {
                    const bool real = r < p.M;
                    const float* xr = p.x + (size_t)(real ? (p.x_rows ? p.x_rows[r] : r) : 0) * p.K;
                    float ss = 0.0f;
                    if (real)
                        for (int k = lane * 4; k < p.K; k += 128) {
                            const float4 v = *reinterpret_cast<const float4*>(xr + k);
                            ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
                        }
                    ss = llb_warp_sum(ss);
                    const float inv = 1.0f / sqrtf(ss / (float)p.K + p.eps);
                    // 16-byte chunks: chunk c of the row covers k = 8c .. 8c+7; tile kb = c / 8 (this split's tiles only)
                    for (int c = kb_begin * 8 + lane; c < kb_end * 8; c += 32) {
                        uint32_t w[4] = {0u, 0u, 0u, 0u};
                        const int k = c * 8;
                        if (real && k < p.K) {
                            const float4 a = *reinterpret_cast<const float4*>(xr + k);
                            const float4 b = *reinterpret_cast<const float4*>(xr + k + 4);
                            const float xv[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                            float nw[8];
                            if (p.norm_w_bf16) {
                                const uint4 u = *reinterpret_cast<const uint4*>((const __nv_bfloat16*)p.norm_w + k);
                                const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    const float2 f = __bfloat1622float2(h[i]);
                                    nw[2 * i] = f.x; nw[2 * i + 1] = f.y;
                                }
                            } else {
                                const float4 c0 = *reinterpret_cast<const float4*>((const float*)p.norm_w + k);
                                const float4 c1 = *reinterpret_cast<const float4*>((const float*)p.norm_w + k + 4);
                                nw[0] = c0.x; nw[1] = c0.y; nw[2] = c0.z; nw[3] = c0.w;
                                nw[4] = c1.x; nw[5] = c1.y; nw[6] = c1.z; nw[7] = c1.w;
                            }
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const __nv_bfloat162 h = __floats2bfloat162_rn(xv[2 * i] * inv * nw[2 * i],
                                                                               xv[2 * i + 1] * inv * nw[2 * i + 1]);
                                w[i] = *reinterpret_cast<const uint32_t*>(&h);
                            }
                        }
                        const int kb = c >> 3, q = c & 7;
                        uint8_t* dst = b_tiles + (size_t)kb * B_BYTES + (uint32_t)r * 128 + ((q ^ (r & 7)) * 16);
                        *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
                fence_async_smem();
                mbar_arrive(&b_ready_bar);
            }
            if (EPI == DEPI_ROPE_KV) {          // asked for while the tensor cores still work
                const int e = threadIdx.x - 64;
                rr = rope_row(p, n0 + (e & (TILE_M - 1)), e & (TILE_M - 1));
                rope_fetch(p, rr, n0 + (e & (TILE_M - 1)), rank, e >> 7, (p.M - rank + p.cluster - 1) / p.cluster, cs, slot_of);
            }
            ok = mbar_wait(&acc_bar, 0, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
        }
        __syncwarp();
        if (p.cluster > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (warp >= 2 && ok) {
            // eight warps: a quarter of the features and half of the tokens each; every token's sums go to the block that finishes it
            constexpr int COLS = BN / 2;
            const int row = (warp & 3) * 32 + lane, c0 = ((warp - 2) >> 2) * COLS;
            const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + c0;
            const uint32_t own = smem_u32(recv) + (uint32_t)((rank * slots) * TILE_M + row) * 4;
            int slot = c0 / p.cluster, dst = c0 - slot * p.cluster;          // of token c0 + c + j, counted on
#pragma unroll
            for (int c = 0; c < COLS; c += 8) {
                if (c0 + c >= p.M) break;          // (uniform)
                float v[8];
                tmem_ld8(taddr + c, v);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (c0 + c + j < p.M) {
                        const uint32_t at = own + (uint32_t)slot * (TILE_M * 4);
                        if (p.cluster > 1)
                            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(mapa_u32(at, (uint32_t)dst)), "f"(v[j]) : "memory");
                        else
                            recv[slot * TILE_M + row] = v[j];
                    }
                    if (++dst == p.cluster) { dst = 0; ++slot; }
                }
            }
        }
        tc_fence_before();
        __syncwarp();
        if (p.cluster > 1) {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else if (warp >= 2) {
            asm volatile("bar.sync 1, %0;" ::"n"(WORKERS) : "memory");
        }
        if (warp >= 2 && ok) {
            const int e = threadIdx.x - 64;
            const int mine = (p.M - rank + p.cluster - 1) / p.cluster;          // tokens rank, rank + cluster, ...
            const int piece = (int)blockIdx.z / p.cluster;                      // of K, when several clusters add into the residual
            if (EPI == DEPI_ROPE_KV) {
                // a feature a thread: rotate pairs of rows of one head and scatter to q and the cache pages
                const int row = e & (TILE_M - 1), n = n0 + row;
                const int q_end = p.Hq * p.hd, k_end = q_end + p.Hkv * p.hd;
                const float bias = (p.bias && n < p.N) ? p.bias[n] : 0.0f;
                const float other_bias = (p.bias && rr.rotate) ? p.bias[n0 + rr.partner] : 0.0f;
                for (int i0 = e >> 7; n < p.N && i0 < mine; i0 += ROPE_BATCH * (WORKERS / TILE_M)) {
                    if (i0 != e >> 7) rope_fetch(p, rr, n, rank, i0, mine, cs, slot_of);
#pragma unroll
                    for (int u = 0; u < ROPE_BATCH; ++u) {
                        const int i = i0 + u * (WORKERS / TILE_M), m = rank + i * p.cluster;
                        if (i >= mine) break;
                        float val = recv_one(recv, p.cluster, slots, i, row) + bias;
                        if (rr.rotate) {
                            const float other = recv_one(recv, p.cluster, slots, i, rr.partner) + other_bias;
                            val = rr.first ? val * cs[u].x - other * cs[u].y : val * cs[u].x + other * cs[u].y;
                        }
                        const __nv_bfloat16 h = __float2bfloat16_rn(val);
                        if (n < q_end) {
                            p.q_out[(size_t)m * q_end + n] = h;
                        } else if (slot_of[u] >= 0) {
                            if (n < k_end) p.k_cache[(size_t)slot_of[u] * (p.Hkv * p.hd) + (n - q_end)] = h;
                            else p.v_cache[(size_t)slot_of[u] * (p.Hkv * p.hd) + (n - k_end)] = h;
                        }
                    }
                }
            } else {
                const int f = (e & 63) * 2, n = n0 + f;
                float2 bias = make_float2(0.0f, 0.0f);
                if (p.bias && piece == 0) {
                    if (n < p.N) bias.x = p.bias[n];
                    if (n + 1 < p.N) bias.y = p.bias[n + 1];
                }
                const bool alone = (int)gridDim.z == p.cluster;
                if (n < p.N)
                    for (int i = e >> 6; i < mine; i += WORKERS / 64)
                        finish_pair<EPI>(p, recv_pair(recv, p.cluster, slots, i, f), bias, rank + i * p.cluster, n, alone);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (abort_s && threadIdx.x == 0 && p.error_flag) atomicExch(p.error_flag, 4);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

// Weight maps are cached by (pointer, shape); activations get a fresh map per launch.
struct MapKey {
    const void* ptr; long long rows, cols; int box;
    bool operator==(const MapKey& o) const { return ptr == o.ptr && rows == o.rows && cols == o.cols && box == o.box; }
};
struct MapKeyHash {
    size_t operator()(const MapKey& k) const {
        return std::hash<const void*>()(k.ptr) ^ ((size_t)k.rows * 1000003u) ^ ((size_t)k.cols << 20) ^ ((size_t)k.box << 44);
    }
};
int cached_map(const void* ptr, long long rows, long long cols, int box, CUtensorMap* out) {
    static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
    static std::mutex mu;
    MapKey key{ptr, rows, cols, box};
    {
        std::lock_guard<std::mutex> g(mu);
        auto it = cache.find(key);
        if (it != cache.end()) { *out = it->second; return 0; }
    }
    int rc = make_map_bf16(ptr, rows, cols, box, out);
    if (rc) return rc;
    std::lock_guard<std::mutex> g(mu);
    if (cache.size() > 4096) cache.clear();
    cache[key] = *out;
    return 0;
}

// Operand tiles, and behind them room for what a cluster's blocks send (a block alone uses the ring, which is idle by then).
size_t tile_bytes(int BN, int stages, int b_tiles) { return (size_t)stages * A_BYTES + (size_t)b_tiles * BN * TILE_K * 2; }
size_t recv_bytes(int BN, int cluster) { return cluster > 1 ? (size_t)cluster * llb_ceil_div(BN, cluster) * TILE_M * 4 : 0; }
// The most that any cluster takes: not always the largest (16 tokens: three slots in each of 7 blocks, two in each of 8).
size_t recv_bytes_most(int BN) {
    size_t most = 0;
    for (int c = 2; c <= MAX_CLUSTER; ++c) most = recv_bytes(BN, c) > most ? recv_bytes(BN, c) : most;
    return most;
}
constexpr size_t SMEM_LIMIT = 224 * 1024;

// How many clusters of `size` blocks of this kernel the device holds at once (asked once a kernel, size and device: a normed operand's
// shared memory grows with K, but with rings of six and eight stages a multiprocessor holds one block whatever K is).
template <int BN, int EPI, bool NORM, int STAGES>
int clusters_at_once(int size, size_t smem) {
    static std::atomic<int> known[64][MAX_CLUSTER + 1] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    const bool cached = dev >= 0 && dev < 64;
    if (cached && known[dev][size].load()) return known[dev][size].load() - 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, 1, size);
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = size;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_decode_kernel<BN, EPI, NORM, STAGES>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    if (cached) known[dev][size].store(n + 1);
    return n;
}

// The kernel's limit on shared memory, one figure whatever a launch takes: threads that come here at the same time set the same, and
// none lowers what another's launch needs.
template <int BN, int EPI, bool NORM, int STAGES>
int configure() {
    static std::atomic<bool> configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    const bool cached = dev >= 0 && dev < 64;
    if (cached && configured[dev].load()) return 0;
    const size_t room = tile_bytes(BN, STAGES, STAGES) + recv_bytes_most(BN) + 1024, most = NORM || room > SMEM_LIMIT ? SMEM_LIMIT : room;
    const cudaError_t e = cudaFuncSetAttribute(gemm_decode_kernel<BN, EPI, NORM, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e != cudaSuccess) return llb_fail("gemm_decode: cannot opt in to %zu bytes of shared memory: %s", most, cudaGetErrorString(e));
    if (cached) configured[dev].store(true);
    return 0;
}

template <int BN, int EPI, bool NORM, int STAGES>
int launch_stages(const CUtensorMap& mw, const CUtensorMap& mx, DecodeGemmParams p, int cluster, int pieces, cudaStream_t stream) {
    const int b_tiles = NORM ? p.num_kb : STAGES;
    const size_t tiles = tile_bytes(BN, STAGES, b_tiles), smem = tiles + recv_bytes(BN, cluster) + 1024;
    LLB_REQUIRE(smem <= SMEM_LIMIT, "gemm_decode: K=%d with %d rows needs %zu bytes of shared memory", p.K, BN, smem);
    int rc = configure<BN, EPI, NORM, STAGES>();
    if (rc) return rc;
    p.kb_per_split = llb_ceil_div(p.num_kb, cluster * pieces);
    p.cluster = cluster;
    p.recv_offset = cluster > 1 ? (uint32_t)tiles : 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(llb_ceil_div(p.N, TILE_M), 1, cluster * pieces);
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = 1;
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = cluster;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_decode_kernel<BN, EPI, NORM, STAGES>, mw, mx, p);
    if (e != cudaSuccess) return llb_fail("gemm_decode: launch failed: %s", cudaGetErrorString(e));
    return llb_check_launch("gemm_decode");
}

// K in `pieces` x `cluster` parts.  Asked for a number of parts: clusters of up to 8 of them.  Asked to choose (split_k = 0): the tiles
// of features alone leave most multiprocessors idle where there are few of them, and a block's part of K then is its time, so the
// largest clusters that all find a place at once; tiles that fill more than half of the multiprocessors get two blocks each with short
// rings, two blocks a multiprocessor (9,728 x 896, us with the norm before it: 8 rows 8.7 -> 7.4, 64 rows 12.6 -> 11.3; 17,920 x 1,536 at 27
// rows 15.0 -> 13.8).  Up to 32 rows the residual is cheap enough to add to from every block, with as many parts as multiprocessors
// and no meeting (896 x 896, 8 rows 4.2 us; in clusters 19 rows 5.5); 64 rows' additions are not (6.9 -> 6.4).
template <int BN, int EPI, bool NORM>
int launch(const CUtensorMap& mw, const CUtensorMap& mx, const DecodeGemmParams& p, int split_k, cudaStream_t stream) {
    constexpr int RING = BN == 64 ? MIDDLE : DEEP;          // beside the received sums
    const int tiles = llb_ceil_div(p.N, TILE_M), sms = llb_device_sms();
    const bool may_cut = EPI != DEPI_STORE_F32 && !(EPI == DEPI_SWIGLU && p.N % 2);
    int cluster = 1, pieces = 1;
    auto even = [&](int parts) { return llb_ceil_div(p.num_kb, llb_ceil_div(p.num_kb, parts)); };          // without empty parts
    if (may_cut && EPI == DEPI_RESIDUAL && BN <= 32) {
        pieces = even(split_k > 0 ? (split_k < p.num_kb ? split_k : p.num_kb) : tiles < sms ? (sms / tiles < p.num_kb ? sms / tiles : p.num_kb) : 1);
    } else if (may_cut) {
        const int most = split_k > 0 ? split_k : tiles < sms ? sms / tiles : 1;
        cluster = even(most < p.num_kb ? most : p.num_kb);
        if (cluster > MAX_CLUSTER) cluster = even(MAX_CLUSTER);
        const size_t room = tile_bytes(BN, RING, NORM ? p.num_kb : RING) + recv_bytes_most(BN) + 1024;
        if (cluster > 1 && room > SMEM_LIMIT) cluster = 1;          // (a normed operand that is resident over a long K)
        if (cluster > 1) {
            const int rc = configure<BN, EPI, NORM, RING>();
            if (rc) return rc;
            while (split_k == 0 && cluster > 1 && clusters_at_once<BN, EPI, NORM, RING>(cluster, room) < tiles) cluster = even(cluster - 1);
            // several clusters along K add into the residual
            if (EPI == DEPI_RESIDUAL && split_k == 0 && cluster == even(MAX_CLUSTER))
                while (llb_ceil_div(p.num_kb, cluster * pieces) > 6 && even(cluster * (pieces + 1)) == cluster * (pieces + 1) &&
                       clusters_at_once<BN, EPI, NORM, RING>(cluster, room) >= tiles * (pieces + 1))
                    ++pieces;
        }
    }
    if (cluster > 1) return launch_stages<BN, EPI, NORM, RING>(mw, mx, p, cluster, pieces, stream);
    if constexpr (!NORM && EPI != DEPI_STORE_F32) {
        // more tiles than half the multiprocessors: two blocks a tile, and two of them on a multiprocessor
        constexpr int PAIR = BN == 16 ? 5 : BN == 32 ? 4 : 3;
        if (split_k == 0 && may_cut && pieces == 1 && tiles <= sms && p.num_kb >= 4)
            return launch_stages<BN, EPI, NORM, PAIR>(mw, mx, p, 2, 1, stream);
    }
    // the float-store epilogue is the head's: a vocabulary's worth of blocks
    if constexpr (EPI == DEPI_STORE_F32 && !NORM)
        if (tiles >= 256) return launch_stages<BN, EPI, NORM, SHALLOW>(mw, mx, p, 1, pieces, stream);
    return launch_stages<BN, EPI, NORM, DEEP>(mw, mx, p, 1, pieces, stream);
}

template <int BN, bool NORM>
int dispatch_epi(int epi, const CUtensorMap& mw, const CUtensorMap& mx, const DecodeGemmParams& p, int split_k,
                 cudaStream_t s) {
    switch (epi) {
        case DEPI_STORE_F32: return launch<BN, DEPI_STORE_F32, NORM>(mw, mx, p, split_k, s);
        case DEPI_RESIDUAL: return launch<BN, DEPI_RESIDUAL, NORM>(mw, mx, p, split_k, s);
        case DEPI_SWIGLU: return launch<BN, DEPI_SWIGLU, NORM>(mw, mx, p, split_k, s);
        case DEPI_ROPE_KV: return launch<BN, DEPI_ROPE_KV, NORM>(mw, mx, p, split_k, s);
        case DEPI_STORE:
            if constexpr (!NORM) return launch<BN, DEPI_STORE, false>(mw, mx, p, split_k, s);
    }
    return llb_fail("gemm_decode: unknown epilogue %d", epi);
}

template <bool NORM>
int dispatch_bn(int epi, const CUtensorMap& mw, const CUtensorMap& mx, const DecodeGemmParams& p, int split_k,
                cudaStream_t s) {
    if (p.M <= 16) return dispatch_epi<16, NORM>(epi, mw, mx, p, split_k, s);
    if (p.M <= 32) return dispatch_epi<32, NORM>(epi, mw, mx, p, split_k, s);
    return dispatch_epi<64, NORM>(epi, mw, mx, p, split_k, s);
}

}  // namespace

// Whether the fused decode contraction takes this shape.
LLB_EXPORT int llb_gemm_decode_supports(int M, int N, int K, int norm, int epilogue, int hd) {
    if (M < 1 || M > 64 || K % 8 != 0 || N < 1) return 0;
    const int BN = M <= 16 ? 16 : M <= 32 ? 32 : 64;
    const int num_kb = llb_ceil_div(K, TILE_K);
    if (tile_bytes(BN, DEEP, norm ? num_kb : DEEP) + 1024 > SMEM_LIMIT) return 0;
    if (epilogue == DEPI_SWIGLU && N % 2) return 0;
    if (epilogue == DEPI_ROPE_KV && (hd < 2 || TILE_M % hd != 0)) return 0;
    if (epilogue == DEPI_STORE && norm) return 0;
    return 1;
}

// W [N, K] bf16 (K a multiple of 8).  Activations: with norm != 0 the float rows x[x_rows[r]] (or x[r])
// of width K, normalised with norm_w (float, or bf16 when norm_w_bf16) and eps inside the kernel; else
// a_bf16 [M, K].  Epilogues: 1 store float out[M, N]; 2 add into residual[M, N];
// 3 SwiGLU out[M, N/2] bf16; 4 rotary + q_out + cache write (N = (Hq + 2 Hkv) * hd; without
// slot_mapping only q is written and N = Hq * hd); rope_table [M, rotary_dim/2] holds (cos, sin) of each
// token's angle (llb_rope_table); 5 store bf16 out[M, N].  split_k: into how many parts K is cut (8 at most where the parts meet in a
// cluster), 0: as the sizes and the device suggest.
static int gemm_decode_impl(const void* W, const void* a_bf16, const float* x, const int* x_rows, const void* norm_w,
                            int norm_w_bf16, float eps, int norm, const float* bias, void* out, float* residual,
                            int epilogue, int M, int N, int K, int split_k,
                            const int* slot_mapping, const float* rope_table, int rotary_dim, int interleaved, int Hq,
                            int Hkv, int hd, void* q_out, void* k_cache, void* v_cache, int* error_flag, LlbGluArgs glu,
                            cudaStream_t stream) {
    if (M == 0) return 0;
    LLB_REQUIRE(llb_gemm_decode_supports(M, N, K, norm, epilogue, hd), "gemm_decode: unsupported shape M=%d N=%d K=%d", M, N, K);
    LLB_REQUIRE(((uintptr_t)W % 16 == 0), "gemm_decode: weights must be 16-byte aligned");
    LLB_REQUIRE(norm ? (x != nullptr && norm_w != nullptr && (uintptr_t)x % 16 == 0 && (uintptr_t)norm_w % 16 == 0)
                     : (a_bf16 != nullptr && (uintptr_t)a_bf16 % 16 == 0), "gemm_decode: bad activation operand");
    LLB_REQUIRE(split_k >= 0 && (epilogue != DEPI_STORE_F32 || split_k <= 1), "gemm_decode: the float-store epilogue takes no split_k");
    if (epilogue == DEPI_ROPE_KV) {
        const int hkv = slot_mapping ? Hkv : 0;
        LLB_REQUIRE(N == (Hq + 2 * hkv) * hd && rotary_dim % 2 == 0 && rotary_dim <= hd && q_out &&
                    (rotary_dim == 0 || rope_table), "gemm_decode: rotary epilogue arguments do not fit");
    }
    DecodeGemmParams p = {};
    p.x = x; p.x_rows = x_rows; p.norm_w = norm_w; p.norm_w_bf16 = norm_w_bf16; p.eps = eps;
    p.bias = bias; p.out = out; p.residual = residual; p.M = M; p.N = N; p.K = K;
    p.num_kb = llb_ceil_div(K, TILE_K);
    p.slot_mapping = slot_mapping; p.rope_table = (const float2*)rope_table; p.rotary_dim = rotary_dim;
    p.interleaved = interleaved; p.Hq = Hq; p.Hkv = slot_mapping ? Hkv : 0; p.hd = hd;
    p.q_out = (__nv_bfloat16*)q_out; p.k_cache = (__nv_bfloat16*)k_cache; p.v_cache = (__nv_bfloat16*)v_cache;
    p.error_flag = error_flag;
    p.glu = glu;
    CUtensorMap mw, mx;
    int rc = cached_map(W, N, K, TILE_M, &mw);
    if (rc) return rc;
    const int BN = M <= 16 ? 16 : M <= 32 ? 32 : 64;
    if (norm) {
        mx = mw;   // unused
        return dispatch_bn<true>(epilogue, mw, mx, p, split_k, stream);
    }
    if ((rc = make_map_bf16(a_bf16, M, K, BN, &mx))) return rc;
    return dispatch_bn<false>(epilogue, mw, mx, p, split_k, stream);
}

LLB_EXPORT int llb_gemm_decode(const void* W, const void* a_bf16, const float* x, const int* x_rows, const void* norm_w,
                               int norm_w_bf16, float eps, int norm, const float* bias, void* out, float* residual,
                               int epilogue, int M, int N, int K, int split_k,
                               const int* slot_mapping, const float* rope_table, int rotary_dim, int interleaved, int Hq,
                               int Hkv, int hd, void* q_out, void* k_cache, void* v_cache, int* error_flag, cudaStream_t stream) {
    return gemm_decode_impl(W, a_bf16, x, x_rows, norm_w, norm_w_bf16, eps, norm, bias, out, residual, epilogue, M, N, K,
                            split_k, slot_mapping, rope_table, rotary_dim, interleaved, Hq, Hkv, hd, q_out, k_cache, v_cache,
                            error_flag, llb_glu_silu(), stream);
}

// The GLU epilogue with another gated activation (LLB_GLU_*, see llb_glu), or the store epilogue with a plain one (a kind of LlbAct,
// else none); bf16 operand, no norm prologue.
LLB_EXPORT int llb_gemm_decode_glu(const void* W, const void* a_bf16, const float* bias, void* out, int epilogue, int M, int N, int K,
                                   int split_k, int* error_flag, int glu_kind, float glu_alpha, float glu_limit, float glu_up_shift,
                                   cudaStream_t stream) {
    LLB_REQUIRE(epilogue == DEPI_SWIGLU || epilogue == DEPI_STORE, "gemm_decode_glu: epilogue %d takes no activation", epilogue);
    return gemm_decode_impl(W, a_bf16, nullptr, nullptr, nullptr, 0, 0.0f, 0, bias, out, nullptr, epilogue, M, N, K,
                            split_k, nullptr, nullptr, 0, 0, 0, 0, 0, nullptr, nullptr, nullptr, error_flag,
                            LlbGluArgs{glu_kind, glu_alpha, glu_limit, glu_up_shift}, stream);
}

// The float-store and residual epilogues (bf16 operand, no norm prologue) with every output (bias included) times `scale`.
LLB_EXPORT int llb_gemm_decode_scaled(const void* W, const void* a_bf16, const float* bias, void* out, float* residual,
                                      int epilogue, int M, int N, int K, int split_k, float scale, int* error_flag,
                                      cudaStream_t stream) {
    LLB_REQUIRE(epilogue == DEPI_STORE_F32 || epilogue == DEPI_RESIDUAL, "gemm_decode_scaled: epilogue %d takes no scale", epilogue);
    return gemm_decode_impl(W, a_bf16, nullptr, nullptr, nullptr, 0, 0.0f, 0, bias, out, residual, epilogue, M, N, K,
                            split_k, nullptr, nullptr, 0, 0, 0, 0, 0, nullptr, nullptr, nullptr, error_flag,
                            LlbGluArgs{LLB_OUT_SCALE, scale, 0.0f, 0.0f}, stream);
}

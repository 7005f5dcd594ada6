// Contraction of 32-bit operands on the 5th-generation tensor cores (sm_100a) with 32-bit accuracy, for more rows than a few.
//
// C[M,N] = A[M,K] * W[N,K]^T, W stored [out, in] as in the checkpoint (src/engine/engine_server.cpp:1542-1544; the reference
// calls cublasSgemm, src/ops/gemm.cu:92-97).  The tensor cores multiply bf16 exactly but take no floats, and they cut off what
// does not fit a float after every instruction instead of rounding it.  So (the splitting is a published method: G. Henry, P. T. P. Tang
// and A. Heinecke, Leveraging the bfloat16 Artificial Intelligence Datatype For Higher-Precision Computations, 2019)
//   * every operand is the sum of three bf16 numbers, x = x1 + x2 + x3 (each rounded to nearest from what is left, which is
//     exact for a float's 24 bits, see UP).  The weights are split on the way into shared memory, so no copy of them is kept; the
//     tokens, which every tile of features reads, by a kernel before this one (split in every block they took most of its
//     instructions: 1,670 issue cycles a slice of 32 columns beside 900 of products);
//   * of the nine products the six that matter are computed: x1 w1 into an accumulator of its own, x1 w2, x2 w1, x2 w2,
//     x1 w3, x3 w1 into a second one (the other three are below 2^-25 of the product);
//   * the accumulator of x1 w1 is read, and begun anew, every 32 columns of K, and its values are added up in registers,
//     rounded to nearest.  Left in tensor memory over all of K the cut-off bits add up: 8.6e-7 off 64 bits (2-norm) at K = 896
//     where FFMA is 2.7e-7 off; the corrections are 2^-9 of the sum and may stay.
// What does not fit that form (an infinity, a NaN, operands beyond 2^104, sums beyond 2^80) shows as a sum that is no finite
// number; a block that sees one does its tile again with FFMA, so such inputs give what float arithmetic gives.
//
// A block makes a tile of 128 features (the MMA's 128 rows) x up to 160 tokens.  Sixteen warps fetch weights (two slices of 32
// columns ahead, in registers), split them into swizzled shared-memory tiles, and drain and add up the accumulators; one warp asks
// for the tokens (TMA) and one issues tcgen05.mma.  Few tiles over a long K are cut along K among the blocks of a cluster, whose sums
// meet in shared memory in the order of K.  Waits are bounded as in the other tensor-core kernels.
//
// Measured (us, FFMA tiles of csrc/gemm_simt.cu -> here, the split of the tokens included): 389 rows x 9,728 features x 896
// 228 -> 60 (113 TFLOP/s), 389 x 896 x 4,864 160 -> 42, 389 x 151,936 x 896 3,230 -> 730 (145), 160 x 9,728 x 896 119 -> 31.  2-norm error
// against 64 bits at 389 x 1,500 x K, FFMA -> here: K = 4 4.0e-8 -> 2.7e-8, 64 8.4e-8 -> 5.4e-8, 256 1.5e-7 -> 6.7e-8, 896 2.7e-7 -> 9.1e-8,
// 4,864 6.3e-7 -> 1.7e-7; 17 x 6,200 x 896 1.7e-7 -> 9.1e-8.  Sums of numbers of one sign, whose result's own rounding is 2.5e-8, are
// about even: K = 64 5.0e-8 -> 5.7e-8, 128 5.7e-8 -> 5.9e-8, 256 6.9e-8 -> 6.4e-8, 896 1.1e-7 -> 8.5e-8; 64 rows, K = 512 5.2e-8 -> 5.9e-8.
// What bounds it: a slice takes about 1,300 cycles at 32 tokens (each warp's chain of split, fence
// and drain) and 1,500 at 144, of which 12 products are 860 and their operands' reads from shared memory as many.
#include <cooperative_groups.h>

#include <atomic>

#include "tcgen05_common.cuh"
#include "warp_mma.cuh"

namespace {

using namespace t5;
using wm::pack_bf16;

constexpr int FEATURES = 128;              // of a tile: the MMA's rows
constexpr int MAX_TOKENS = 160;            // of a tile: the MMA's columns; three accumulators of that many fit tensor memory
constexpr int SLICE = 32;                  // columns of K per stage: rows of 64 bytes in bf16
constexpr int STAGES = 4;
constexpr int WORKERS = 512;               // 16 warps: a quarter of tensor memory's lanes x 40 tokens each
constexpr int WARP_TOKENS = 40;
constexpr int THREADS = WORKERS + 64;
constexpr int MMA_WARP = WORKERS / 32, LOAD_WARP = MMA_WARP + 1;
constexpr uint32_t W_PLANE = FEATURES * SLICE * 2, X_PLANE = MAX_TOKENS * SLICE * 2;
constexpr uint32_t STAGE_BYTES = 3 * W_PLANE + 3 * X_PLANE;
constexpr uint32_t SMEM_BYTES = STAGES * STAGE_BYTES + 1024;
constexpr uint32_t COL_CORR = 2 * MAX_TOKENS, TMEM_COLS = 512;
static_assert(3 * MAX_TOKENS <= 512 && MAX_TOKENS * FEATURES * 4 <= STAGES * STAGE_BYTES, "accumulators and the tile of sums fit");

struct F32Params {
    const float* A;
    const float* W;
    const float* bias;
    void* out;
    float* residual;
    int M, N, K;
    int tokens;            // of a tile, a multiple of 16
    uint32_t x_bytes;      // of a slice's tokens in shared memory, all three planes
    int k_part;            // columns of K of a block, a multiple of SLICE
    int* error_flag;
    LlbGluArgs glu;
};

// K-major operand tile with 64-byte rows and the 64-byte swizzle (layout type 4): groups of 8 rows 512 bytes apart.
__device__ __forceinline__ uint64_t desc_kmajor64(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)4 << 61);
}
// Operands are split at 2^24 times their size and the sums taken back: every float is a whole multiple of 2^-149, so that a part is zero or
// at least 2^-125, within what bf16 holds without losing bits (split as it is, a float below 2^-109 loses the third part, below 2^-117
// the second: 2.7e-4 off at 1e-37).  Powers of two leave all other roundings as they are.
constexpr float UP = 16777216.0f, DOWN = 1.0f / (UP * UP);
__device__ __forceinline__ float2 scaled_up2(float x, float y) {          // two products an instruction
    float2 r;
    asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmul.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a;\n\t}" : "=f"(r.x), "=f"(r.y) : "f"(x), "f"(y), "f"(UP));
    return r;
}
__device__ __forceinline__ float4 scaled_up(const float4& v) {
    const float2 a = scaled_up2(v.x, v.y), b = scaled_up2(v.z, v.w);
    return make_float4(a.x, a.y, b.x, b.y);
}
// Two floats as three pairs of bf16 that add up to them.
__device__ __forceinline__ void split2(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = pack_bf16(x, y);
    x -= __uint_as_float(h << 16);
    y -= __uint_as_float(h & 0xffff0000u);
    m = pack_bf16(x, y);
    x -= __uint_as_float(m << 16);
    y -= __uint_as_float(m & 0xffff0000u);
    l = pack_bf16(x, y);
}
// Eight columns of a row into the three planes of a tile.
__device__ __forceinline__ void store_split(uint8_t* at, const float4& a, const float4& b) {
    uint4 h, m, l;
    split2(a.x, a.y, h.x, m.x, l.x);
    split2(a.z, a.w, h.y, m.y, l.y);
    split2(b.x, b.y, h.z, m.z, l.z);
    split2(b.z, b.w, h.w, m.w, l.w);
    *reinterpret_cast<uint4*>(at) = h;
    *reinterpret_cast<uint4*>(at + W_PLANE) = m;
    *reinterpret_cast<uint4*>(at + 2 * W_PLANE) = l;
}

// The tokens as three planes [M, Kp] of bf16 (Kp: K rounded up to whole slices, zeros behind K), eight columns a thread.
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ A, __nv_bfloat16* __restrict__ planes, int M, int K,
                                                         int Kp) {
    // (in this order: the kernel after this one reads its weights before it waits, and whatever wrote them is complete then)
    griddep_wait();
    griddep_launch_dependents();
    const int per_row = Kp / 8;
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= (long long)M * per_row) return;
    const int m = (int)(i / per_row), k = (int)(i - (long long)m * per_row) * 8;
    const float* src = A + (size_t)m * K + k;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 a = scaled_up(k < K ? *reinterpret_cast<const float4*>(src) : zero);
    const float4 b = scaled_up(k + 4 < K ? *reinterpret_cast<const float4*>(src + 4) : zero);
    uint4 h, m4, l;
    split2(a.x, a.y, h.x, m4.x, l.x);
    split2(a.z, a.w, h.y, m4.y, l.y);
    split2(b.x, b.y, h.z, m4.z, l.z);
    split2(b.z, b.w, h.w, m4.w, l.w);
    __nv_bfloat16* dst = planes + (size_t)m * Kp + k;
    const size_t plane = (size_t)M * Kp;
    *reinterpret_cast<uint4*>(dst) = h;
    *reinterpret_cast<uint4*>(dst + plane) = m4;
    *reinterpret_cast<uint4*>(dst + 2 * plane) = l;
}

template <int EPI>
__device__ __forceinline__ void finish_pair(const F32Params& p, float2 v, int m, int n) {
    const bool has1 = n + 1 < p.N;
    if (p.bias) {
        v.x += p.bias[n];
        if (has1) v.y += p.bias[n + 1];
    }
    if (EPI == LLB_EPI_SWIGLU) {
        ((float*)p.out)[(size_t)m * (p.N / 2) + (n >> 1)] = llb_glu(v.x, v.y, p.glu.kind, p.glu.alpha, p.glu.limit, p.glu.up_shift);
        return;
    }
    float* o = (EPI == LLB_EPI_RESIDUAL ? p.residual : (float*)p.out) + (size_t)m * p.N + n;
    const bool vec = has1 && ((uintptr_t)o & 7) == 0;
    if (EPI == LLB_EPI_RESIDUAL) {
        const float f = llb_out_scale(p.glu);
        if (vec) {
            float2 r = *reinterpret_cast<float2*>(o);
            r.x = fmaf(v.x, f, r.x);
            r.y = fmaf(v.y, f, r.y);
            *reinterpret_cast<float2*>(o) = r;
            return;
        }
        o[0] = fmaf(v.x, f, o[0]);
        if (has1) o[1] = fmaf(v.y, f, o[1]);
        return;
    }
    if (EPI == LLB_EPI_STORE_F32) {
        const float f = llb_out_scale(p.glu);
        v.x *= f;
        v.y *= f;
    } else {
        v.x = llb_act(v.x, p.glu.kind);
        v.y = llb_act(v.y, p.glu.kind);
    }
    if (vec) {
        *reinterpret_cast<float2*>(o) = v;
    } else {
        o[0] = v.x;
        if (has1) o[1] = v.y;
    }
}

// Eight consecutive columns of this thread's lane of tensor memory; tcgen05.wait::ld must follow.
__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, float (&r)[8]) {
    uint32_t* u = reinterpret_cast<uint32_t*>(r);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "r"(taddr)
                 : "memory");
}

// A tile's sums in float arithmetic, by the worker warps: for a tile with a sum that is no finite number.  Slices of K go through shared
// memory (columns first, the next slice on its way in registers), and a thread adds 10 (few rows: 4) tokens x 4 features up in the
// order of K.  A call of its own, so that its registers are not the kernel's.  Measured, ms, every thread from memory by itself -> here
// (FFMA throughout): 389 x 9,728 x 896 with one NaN 14.7 -> 0.25, with one in every row 27.9 -> 0.43 (0.23); 389 x 151,936 x 896 114 -> 2.5
// and 284 -> 5.2 (3.2); 389 x 896 x 4,864 17.1 -> 0.30 (0.16); 24 x 9,728 x 896 1.49 -> 0.10 (0.035).
// Floats of a column: even, and four columns 8 banks on, so that the eight pieces of four rows that a warp stores meet two by two.
constexpr int REDO_X = MAX_TOKENS + 2, REDO_W = FEATURES + 2;
static_assert(REDO_X * 4 % 32 == 8 && REDO_W * 4 % 32 == 8, "see above");
constexpr int REDO_AT = MAX_TOKENS * FEATURES * 4;                     // behind the sums
static_assert(REDO_AT + SLICE * (REDO_X + REDO_W) * 4 <= STAGES * STAGE_BYTES, "a slice of floats beside the sums");
__device__ __forceinline__ void workers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(WORKERS) : "memory"); }
template <int RT>          // tokens of a thread; 16 times as many of the tile
__device__ __noinline__ void redo_tile(const float* __restrict__ A, const float* __restrict__ W, int K, int rows, int features, int k_lo,
                                       int k_hi, uint8_t* smem) {
    float* xs = reinterpret_cast<float*>(smem + REDO_AT);          // [SLICE][REDO_X]
    float* ws = xs + SLICE * REDO_X;                               // [SLICE][REDO_W]
    constexpr int RF = 4;                                          // a warp: 4 x RT tokens, 8 x 4 features
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int f0 = (warp & 3) * 32 + (lane & 7) * RF, t0 = ((warp >> 2) * 4 + (lane >> 3)) * RT;
    constexpr int PIECES = SLICE / 4;                              // of four columns of a row, neighbouring threads'
    constexpr int XN = (16 * RT * PIECES + WORKERS - 1) / WORKERS, WN = FEATURES * PIECES / WORKERS;
    const int row = tid / PIECES, c = tid % PIECES * 4;
    constexpr int STRIDE = WORKERS / PIECES;                       // rows on, the thread's next piece
    float4 x[XN], w[WN];
    auto fetch = [&](int k) {
#pragma unroll
        for (int u = 0; u < XN; ++u)
            x[u] = row + u * STRIDE < rows && k < k_hi ? __ldg(reinterpret_cast<const float4*>(A + (size_t)(row + u * STRIDE) * K + k))
                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < WN; ++u)
            w[u] = row + u * STRIDE < features && k < k_hi ? __ldg(reinterpret_cast<const float4*>(W + (size_t)(row + u * STRIDE) * K + k))
                                                          : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto store = [](float* at, int column, const float4& v) {
        at[0] = v.x; at[column] = v.y; at[2 * column] = v.z; at[3 * column] = v.w;
    };
    float acc[RT][RF];
#pragma unroll
    for (int j = 0; j < RT; ++j)
#pragma unroll
        for (int f = 0; f < RF; ++f) acc[j][f] = 0.0f;
    fetch(k_lo + c);
    for (int k0 = k_lo; k0 < k_hi; k0 += SLICE) {
        workers_sync();          // the slice before has been read
#pragma unroll
        for (int u = 0; u < XN; ++u)
            if (row + u * STRIDE < 16 * RT) store(xs + c * REDO_X + row + u * STRIDE, REDO_X, x[u]);
#pragma unroll
        for (int u = 0; u < WN; ++u) store(ws + c * REDO_W + row + u * STRIDE, REDO_W, w[u]);
        workers_sync();
        fetch(k0 + SLICE + c);       // (nothing beyond the last column)
        const int columns = (warp >> 2) * 4 * RT < rows ? min(SLICE, k_hi - k0) : 0;
#pragma unroll 4
        for (int k = 0; k < columns; ++k) {
            const float2 v0 = *reinterpret_cast<const float2*>(ws + k * REDO_W + f0), v1 = *reinterpret_cast<const float2*>(ws + k * REDO_W + f0 + 2);
#pragma unroll
            for (int j = 0; j < RT; j += 2) {
                const float2 t = *reinterpret_cast<const float2*>(xs + k * REDO_X + t0 + j);
                acc[j][0] = fmaf(t.x, v0.x, acc[j][0]);
                acc[j][1] = fmaf(t.x, v0.y, acc[j][1]);
                acc[j][2] = fmaf(t.x, v1.x, acc[j][2]);
                acc[j][3] = fmaf(t.x, v1.y, acc[j][3]);
                acc[j + 1][0] = fmaf(t.y, v0.x, acc[j + 1][0]);
                acc[j + 1][1] = fmaf(t.y, v0.y, acc[j + 1][1]);
                acc[j + 1][2] = fmaf(t.y, v1.x, acc[j + 1][2]);
                acc[j + 1][3] = fmaf(t.y, v1.y, acc[j + 1][3]);
            }
        }
    }
    float* sums = reinterpret_cast<float*>(smem);
#pragma unroll
    for (int j = 0; j < RT; ++j)
        if (t0 + j < rows) *reinterpret_cast<float4*>(sums + (t0 + j) * FEATURES + f0) = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
}

template <int EPI>
__global__ void __launch_bounds__(THREADS, 1) gemm_f32_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x, const F32Params p) {
    __shared__ __align__(8) uint64_t full[STAGES];      // the slice's operands are there (every worker warp, and the tokens' copies)
    __shared__ __align__(8) uint64_t done[STAGES];      // its products are computed
    __shared__ __align__(8) uint64_t drained[2];        // the accumulator of x1 w1 has been read (every worker warp)
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_s;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    volatile int* abort_flag = &abort_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * p.tokens, n0 = blockIdx.y * FEATURES;
    const int k_lo = blockIdx.z * p.k_part, k_hi = min(p.K, k_lo + p.k_part);
    const int slices = (k_hi - k_lo + SLICE - 1) / SLICE;
    const int rows = min(p.tokens, p.M - m0);           // tokens of this tile

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], WORKERS / 32 + 1);
            mbar_init(&done[s], 1);
        }
        mbar_init(&drained[0], WORKERS / 32);
        mbar_init(&drained[1], WORKERS / 32);
        abort_s = 0;
        mbar_init_fence();
    }
    if (warp == MMA_WARP) tmem_alloc(&tmem_slot, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;
    const int quarter = warp & 3, t0 = (warp >> 2) * WARP_TOKENS;          // a worker warp's lanes and first token of the tile
    const int feature = quarter * 32 + lane;
    float acc[WARP_TOKENS];
    bool ok = true, bad = false;

    if (warp == LOAD_WARP) {
        if (lane == 0) {
            griddep_wait();          // the tokens are split by the kernel before this one
            for (int i = 0; i < slices; ++i) {
                const int s = i % STAGES;
                if (i >= STAGES && !mbar_wait(&done[s], (i / STAGES - 1) & 1, abort_flag)) break;
                mbar_expect_tx(&full[s], p.x_bytes);
                uint8_t* x = smem + s * STAGE_BYTES + 3 * W_PLANE;
                // (rows behind the last token are the next plane's: they make columns that nobody reads)
                for (int c = 0; c < 3; ++c) tma_load_2d(x + c * X_PLANE, &map_x, k_lo + i * SLICE, c * p.M + m0, &full[s]);
            }
        }
        __syncwarp();
    } else if (warp == MMA_WARP) {
        if (lane == 0) {
            const uint32_t idesc = idesc_bf16(FEATURES, p.tokens);
            const uint64_t base = desc_kmajor64(smem_u32(smem));
            for (int i = 0; i < slices; ++i) {
                const int s = i % STAGES;
                ok = mbar_wait(&full[s], (i / STAGES) & 1, abort_flag);
                if (ok && i >= 2) ok = mbar_wait(&drained[i & 1], ((i >> 1) - 1) & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                // descriptors count 16 bytes, and the largest address stays below 2^18: no carry leaves the field
                const uint64_t w = base + (uint64_t)(s * (STAGE_BYTES >> 4)), x = w + (3 * W_PLANE >> 4);
                const uint32_t main = tmem_base + (i & 1) * MAX_TOKENS, corr = tmem_base + COL_CORR;
                umma_bf16_first(main, w, x, idesc);
                umma_bf16_acc(main, w + 2, x + 2, idesc);
                // (feature plane, token plane), the smallest products first
                constexpr int pw[5] = {2, 0, 1, 1, 0}, px[5] = {0, 2, 1, 0, 1};
#pragma unroll
                for (int c = 0; c < 10; ++c) {
                    const uint64_t wa = w + (pw[c >> 1] * (W_PLANE >> 4) + (c & 1) * 2), xa = x + (px[c >> 1] * (X_PLANE >> 4) + (c & 1) * 2);
                    if (c == 0) umma_bf16(corr, wa, xa, idesc, i > 0 ? 1u : 0u);
                    else umma_bf16_acc(corr, wa, xa, idesc);
                }
                umma_commit(&done[s]);
            }
        }
        __syncwarp();
    } else {
        const int row = tid >> 2, q = tid & 3;                     // eight columns of a feature
        const bool in_w = n0 + row < p.N;
        const float* wp = p.W + (size_t)(in_w ? n0 + row : 0) * p.K + k_lo + q * 8;
        const int k_left = in_w ? k_hi - k_lo - q * 8 : 0;         // columns from wp on
        // the 16-byte chunk c of row r lies at chunk c ^ ((r >> 1) & 3)
        uint8_t* at = smem + row * (SLICE * 2) + ((q ^ ((row >> 1) & 3)) * 16);
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        float4 w[2][2];
        auto fetch = [&](int i, int u) {
            w[u][0] = i * SLICE < k_left ? __ldg(reinterpret_cast<const float4*>(wp + i * SLICE)) : zero;
            w[u][1] = i * SLICE + 4 < k_left ? __ldg(reinterpret_cast<const float4*>(wp + i * SLICE + 4)) : zero;
        };
        const uint32_t t_at = tmem_base + ((uint32_t)(quarter * 32) << 16) + t0;
        auto add = [&](uint32_t col) {          // 40 tokens of this thread's feature
            float a[8], b[8];          // 16, 16 and 8: as many in flight as there are registers for
#pragma unroll
            for (int h = 0; h < WARP_TOKENS; h += 16) {
                tmem_ld8_nowait(t_at + col + h, a);
                if (h + 8 < WARP_TOKENS) tmem_ld8_nowait(t_at + col + h + 8, b);
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    acc[h + j] += a[j];
                    if (h + 8 < WARP_TOKENS) acc[(h + 8 + j) % WARP_TOKENS] += b[j];
                }
            }
        };
#pragma unroll
        for (int j = 0; j < WARP_TOKENS; ++j) acc[j] = 0.0f;
        const bool drains = t0 < p.tokens;
        fetch(0, 0);
        fetch(1, 1);
        for (int i0 = 0; i0 < slices + 2; i0 += 2) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int i = i0 + u;
                if (i < slices) {
                    // (the stage is free: this thread has waited for the products of slice i - 4)
                    if (ok) store_split(at + (i % STAGES) * STAGE_BYTES, scaled_up(w[u][0]), scaled_up(w[u][1]));
                    fetch(i + 2, u);
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&full[i % STAGES]);
                }
                if (i >= 2 && i < slices + 2) {
                    const int d = i - 2;
                    ok = ok && mbar_wait(&done[d % STAGES], (d / STAGES) & 1, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);          // tcgen05.ld is a warp's instruction
                    tc_fence_after();
                    if (ok && drains) add(u * MAX_TOKENS);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&drained[u]);
                }
            }
        }
        if (ok && drains) add(COL_CORR);
        tc_fence_before();
#pragma unroll
        for (int j = 0; j < WARP_TOKENS; ++j) bad = bad || (t0 + j < rows && !(fabsf(acc[j]) < INFINITY));
        bad = bad && n0 + feature < p.N && ok;
    }
    griddep_wait();
    bad = __syncthreads_or(bad);
    // the sums as [token][feature] over the stages: every product has been computed
    float* sums = reinterpret_cast<float*>(smem);
    if (warp < MMA_WARP) {
        if (bad) {
            if (rows > 64) redo_tile<10>(p.A + (size_t)m0 * p.K, p.W + (size_t)n0 * p.K, p.K, rows, p.N - n0, k_lo, k_hi, smem);
            else redo_tile<4>(p.A + (size_t)m0 * p.K, p.W + (size_t)n0 * p.K, p.K, rows, p.N - n0, k_lo, k_hi, smem);
        } else {
#pragma unroll
            for (int j = 0; j < WARP_TOKENS; ++j)
                if (t0 + j < rows) sums[(t0 + j) * FEATURES + feature] = acc[j] * DOWN;
        }
    }
    namespace cg = cooperative_groups;
    const int parts = gridDim.z;
    __syncthreads();
    if (parts > 1) cg::this_cluster().sync();
    // every block of the cluster finishes its share of the tile's tokens (pairs of features: the gated epilogue takes two)
    if (!*abort_flag) {
        const int r_lo = rows * (int)blockIdx.z / parts, r_hi = rows * ((int)blockIdx.z + 1) / parts;
        for (int i = tid; i < (r_hi - r_lo) * (FEATURES / 2); i += THREADS) {
            const int t = r_lo + i / (FEATURES / 2), c = (i % (FEATURES / 2)) * 2, n = n0 + c;
            if (n >= p.N) continue;
            float2 v = make_float2(0.0f, 0.0f);
            if (parts > 1) {
                for (int z = 0; z < parts; ++z) {
                    const float2 u = *reinterpret_cast<const float2*>(cg::this_cluster().map_shared_rank(sums, z) + t * FEATURES + c);
                    v.x += u.x;
                    v.y += u.y;
                }
            } else {
                v = *reinterpret_cast<const float2*>(sums + t * FEATURES + c);
            }
            finish_pair<EPI>(p, v, m0 + t, n);
        }
    }
    if (parts > 1) cg::this_cluster().sync();          // the others may still read this block's sums
    if (*abort_flag && tid == 0 && p.error_flag) atomicExch(p.error_flag, 5);
    if (warp == MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

// A map over the planes [rows, cols] of bf16 with boxes of box_rows x 32 and the 64-byte swizzle.
int make_planes_map(const void* ptr, long long rows, long long cols, int box_rows, CUtensorMap* out) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return llb_fail("cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    cuuint32_t box[2] = {(cuuint32_t)SLICE, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult rc = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) return llb_fail("cuTensorMapEncodeTiled failed with code %d", (int)rc);
    return 0;
}

template <int EPI>
int launch(const F32Params& p0, __nv_bfloat16* planes, cudaStream_t stream) {
    F32Params p = p0;
    static std::atomic<bool> configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev].load()) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tcgen05_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e != cudaSuccess) return llb_fail("gemm_f32: cannot opt in to %u bytes of shared memory: %s", SMEM_BYTES, cudaGetErrorString(e));
        if (dev >= 0 && dev < 64) configured[dev].store(true);
    }
    // Tiles of equal height, and K in as many pieces (powers of two, six slices at least) as leave every cluster a place at once: a
    // block takes a multiprocessor, and a GPC's multiprocessors hold whole clusters only (16 clusters of 8 take a second round: 2,048 x
    // 1,536, 128 tokens 26 us, in 32 clusters of 4 19 us).
    const int even = llb_ceil_div(p.M, llb_ceil_div(p.M, MAX_TOKENS));
    p.tokens = llb_ceil_div(even, 16) * 16;
    const int mt = llb_ceil_div(p.M, p.tokens), nt = llb_ceil_div(p.N, FEATURES), slices = llb_ceil_div(p.K, SLICE);
    int split = 1;
    while (split < 8 && (long long)mt * nt * split * 2 <= llb_device_sms() * (split < 4 ? 9 : 8) / 10 && slices >= split * 6) split *= 2;
    const int per = llb_ceil_div(slices, split);
    split = llb_ceil_div(slices, per);
    p.k_part = per * SLICE;
    p.x_bytes = (uint32_t)p.tokens * SLICE * 2 * 3;
    const int Kp = slices * SLICE;
    CUtensorMap map_x;
    int rc = make_planes_map(planes, 3ll * p.M, Kp, p.tokens, &map_x);
    if (rc) return rc;
    const long long groups = (long long)p.M * (Kp / 8);
    cudaError_t e0 = launch_pdl(split_rows_kernel, dim3((unsigned)((groups + 255) / 256)), dim3(256), 0, stream, p.A, planes, p.M, p.K, Kp);
    if (e0 != cudaSuccess) return llb_fail("gemm_f32: %s", cudaGetErrorString(e0));
    if ((rc = llb_check_launch("split_rows"))) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(mt, nt, split);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = 1;
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = split;
    cfg.attrs = at;
    cfg.numAttrs = split > 1 ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_f32_tcgen05_kernel<EPI>, map_x, p);
    if (e != cudaSuccess) return llb_fail("gemm_f32: %s", cudaGetErrorString(e));
    return llb_check_launch("gemm_f32");
}

}  // namespace

// Whether the kernel takes these operands: rows in 16-byte steps, tiles of features in the grid's second dimension, three planes
// of the tokens that a copy's row coordinate counts.
bool llb_gemm_f32_tcgen05_takes(const void* A, const void* W, int M, int N, int K) {
    return M > 0 && K % 4 == 0 && ((uintptr_t)A | (uintptr_t)W) % 16 == 0 && llb_ceil_div(N, FEATURES) <= 65535 && M <= (1 << 28);
}

// Bytes of scratch (16-byte aligned) that a contraction of M rows of K floats on the tensor cores needs: the split tokens.
LLB_EXPORT long long llb_gemm_f32_scratch_bytes(int M, int K) { return 6ll * M * (llb_ceil_div(K, SLICE) * SLICE); }

// A [M,K], W [N,K], bias [N] or null, all float; epilogues and glu as llb_gemm_simt_glu; scratch as llb_gemm_f32_scratch_bytes says.
LLB_EXPORT int llb_gemm_f32_tcgen05(const void* A, const void* W, const void* bias, void* out, float* residual, int epilogue, int M,
                                    int N, int K, int glu_kind, float glu_alpha, float glu_limit, float glu_up_shift, void* scratch,
                                    int* error_flag, cudaStream_t stream) {
    LLB_REQUIRE(llb_gemm_f32_tcgen05_takes(A, W, M, N, K), "gemm_f32: unsupported operands (M=%d N=%d K=%d)", M, N, K);
    LLB_REQUIRE(scratch && (uintptr_t)scratch % 16 == 0, "gemm_f32: no scratch, or not in 16-byte steps");
    F32Params p = {};
    p.A = (const float*)A;
    p.W = (const float*)W;
    p.bias = (const float*)bias;
    p.out = out;
    p.residual = residual;
    p.M = M;
    p.N = N;
    p.K = K;
    p.error_flag = error_flag;
    p.glu = LlbGluArgs{glu_kind, glu_alpha, glu_limit, glu_up_shift};
    __nv_bfloat16* planes = (__nv_bfloat16*)scratch;
    switch (epilogue) {
        case LLB_EPI_STORE: return launch<LLB_EPI_STORE>(p, planes, stream);
        case LLB_EPI_STORE_F32: return launch<LLB_EPI_STORE_F32>(p, planes, stream);
        case LLB_EPI_RESIDUAL: return launch<LLB_EPI_RESIDUAL>(p, planes, stream);
        case LLB_EPI_SWIGLU: return launch<LLB_EPI_SWIGLU>(p, planes, stream);
    }
    return llb_fail("gemm_f32: unknown epilogue %d", epilogue);
}

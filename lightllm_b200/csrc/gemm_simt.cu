// Dense contraction on CUDA cores with float accumulation: the 32-bit path of every linear layer with few rows or little
// work (floats with more of both go to csrc/gemm_f32_tcgen05.cu, at no larger error), and the path for shapes the bf16
// tensor-core kernel refuses.
//
// C[M,N] = A[M,K] * W[N,K]^T, W stored [out, in] as in the checkpoint
// (src/engine/engine_server.cpp:1542-1544; the reference calls cublasSgemm for it,
// src/ops/gemm.cu:92-97, and keeps tiled teaching kernels at :44-81).  Products and sums are
// float FFMA: no tensor cores, no TF32.  Epilogues add the bias (which the reference never
// loads, engine_server.cpp:436-450), add into the float residual stream
// (engine_server.cpp:1870-1871), or apply SiLU(gate)*up on interleaved rows
// (src/ops/elementwise.cu:27-33, engine_server.cpp:1875-1878).
//
// Three kernels: a row-streaming kernel for few rows (decode), where every weight row is read once by one warp with
// 16-byte loads; a tile kernel for float operands whose rows are 16-byte multiples;
// and a 64x64x16 tile kernel for everything else (odd inner sizes, 16-bit operands).
#include <cooperative_groups.h>

#include <atomic>

#include "common.cuh"

// csrc/gemm_f32_tcgen05.cu: the same of float operands on the tensor cores, split into bf16 numbers that add up to them.
bool llb_gemm_f32_tcgen05_takes(const void* A, const void* W, int M, int N, int K);
LLB_EXPORT long long llb_gemm_f32_scratch_bytes(int M, int K);
LLB_EXPORT int llb_gemm_f32_tcgen05(const void* A, const void* W, const void* bias, void* out, float* residual, int epilogue, int M,
                                    int N, int K, int glu_kind, float glu_alpha, float glu_limit, float glu_up_shift, void* scratch,
                                    int* error_flag, cudaStream_t stream);

namespace {

template <typename TO, int EPI>
struct Epilogue {
    // Called with two adjacent columns (n even) so that SwiGLU sees its gate/up pair.
    static __device__ __forceinline__ void pair(float a0, float a1, int m, int n, int N, void* out,
                                                float* residual, bool has1, const LlbGluArgs& glu) {
        if (EPI == LLB_EPI_STORE) {
            TO* o = (TO*)out + (size_t)m * N + n;
            o[0] = llb_from_float<TO>(llb_act(a0, glu.kind));
            if (has1) o[1] = llb_from_float<TO>(llb_act(a1, glu.kind));
        } else if (EPI == LLB_EPI_STORE_F32) {
            float* o = (float*)out + (size_t)m * N + n;
            const float f = llb_out_scale(glu);
            o[0] = a0 * f;
            if (has1) o[1] = a1 * f;
        } else if (EPI == LLB_EPI_RESIDUAL) {
            float* r = residual + (size_t)m * N + n;
            const float f = llb_out_scale(glu);
            r[0] = fmaf(a0, f, r[0]);
            if (has1) r[1] = fmaf(a1, f, r[1]);
        } else {  // SWIGLU: column pair (2j, 2j+1) -> output column j of N/2
            TO* o = (TO*)out + (size_t)m * (N / 2) + (n >> 1);
            o[0] = llb_from_float<TO>(llb_glu(a0, a1, glu.kind, glu.alpha, glu.limit, glu.up_shift));
        }
    }
};

constexpr int BM = 64, BN = 64, BK = 16;

template <typename TA, typename TW, typename TO, int EPI>
__global__ void __launch_bounds__(256) gemm_tile_kernel(const TA* __restrict__ A, const TW* __restrict__ W,
                                                        const float* __restrict__ bias, void* __restrict__ out,
                                                        float* __restrict__ residual, int M, int N, int K,
                                                        const LlbGluArgs glu) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int idx = tid + i * 256;  // 0..1023 over a 64x16 tile
            const int r = idx >> 4, kk = idx & 15;
            const int k = k0 + kk;
            const int am = m0 + r, wn = n0 + r;
            As[kk][r] = (am < M && k < K) ? llb_to_float(A[(size_t)am * K + k]) : 0.0f;
            Ws[kk][r] = (wn < N && k < K) ? llb_to_float(W[(size_t)wn * K + k]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            const bool has1 = n + 1 < N;
            float a0 = acc[i][j], a1 = acc[i][j + 1];
            if (bias) {
                a0 += bias[n];
                if (has1) a1 += bias[n + 1];
            }
            Epilogue<TO, EPI>::pair(a0, a1, m, n, N, out, residual, has1, glu);
        }
    }
}

// Few rows (M <= MAXM): one warp owns a pair of weight rows (n, n+1) and streams them once.
// Lane l reads elements k = (c*32 + l)*VEC .. +VEC-1 of each chunk c; sums are float.
template <typename TA, typename TW, typename TO, int EPI, int MAXM, int VEC>
__global__ void __launch_bounds__(256) gemm_rows_kernel(const TA* __restrict__ A, const TW* __restrict__ W,
                                                        const float* __restrict__ bias, void* __restrict__ out,
                                                        float* __restrict__ residual, int M, int N, int K,
                                                        const LlbGluArgs glu) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int n = warp * 2;
    if (n >= N) return;
    const bool has1 = n + 1 < N;
    const TW* w0 = W + (size_t)n * K;
    const TW* w1 = W + (size_t)(has1 ? n + 1 : n) * K;
    float acc0[MAXM], acc1[MAXM];
#pragma unroll
    for (int m = 0; m < MAXM; ++m) acc0[m] = acc1[m] = 0.0f;

    for (int k = lane * VEC; k < K; k += 32 * VEC) {
        float x0[VEC], x1[VEC];
        if (VEC == 8) {  // 16-byte loads of bf16 weights
            const uint4 p0 = *reinterpret_cast<const uint4*>(w0 + k);
            const uint4 p1 = *reinterpret_cast<const uint4*>(w1 + k);
            const __nv_bfloat162* h0 = reinterpret_cast<const __nv_bfloat162*>(&p0);
            const __nv_bfloat162* h1 = reinterpret_cast<const __nv_bfloat162*>(&p1);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 f0 = __bfloat1622float2(h0[i]);
                const float2 f1 = __bfloat1622float2(h1[i]);
                x0[2 * i] = f0.x; x0[2 * i + 1] = f0.y;
                x1[2 * i] = f1.x; x1[2 * i + 1] = f1.y;
            }
        } else if (VEC == 4) {  // 16-byte loads of float weights
            const float4 p0 = *reinterpret_cast<const float4*>(w0 + k);
            const float4 p1 = *reinterpret_cast<const float4*>(w1 + k);
            x0[0] = p0.x; x0[1] = p0.y; x0[2] = p0.z; x0[3] = p0.w;
            x1[0] = p1.x; x1[1] = p1.y; x1[2] = p1.z; x1[3] = p1.w;
        } else {
            x0[0] = llb_to_float(w0[k]);
            x1[0] = llb_to_float(w1[k]);
        }
#pragma unroll
        for (int m = 0; m < MAXM; ++m) {
            if (m < M) {
                const TA* a = A + (size_t)m * K + k;
#pragma unroll
                for (int i = 0; i < VEC; ++i) {
                    const float av = llb_to_float(a[i]);
                    acc0[m] = fmaf(av, x0[i], acc0[m]);
                    acc1[m] = fmaf(av, x1[i], acc1[m]);
                }
            }
        }
    }
#pragma unroll
    for (int m = 0; m < MAXM; ++m) {
        if (m < M) {  // M is uniform over the warp, so every lane takes part in the shuffles
            float a0 = llb_warp_sum(acc0[m]);
            float a1 = llb_warp_sum(acc1[m]);
            if (lane == 0) {
                if (bias) {
                    a0 += bias[n];
                    if (has1) a1 += bias[n + 1];
                }
                Epilogue<TO, EPI>::pair(a0, a1, m, n, N, out, residual, has1, glu);
            }
        }
    }
}

// ---- many rows of floats ----------------------------------------------------------------------------------------------
// A block makes a BM x 64 tile with four groups of 64 threads, each group over its own 8 columns of every 32-wide slice of
// K; a thread holds BM/8 x 8 sums.  What bounds it is the dispatch of FFMA (256 of them against 16 16-byte shared loads per thread
// and 4 columns; two thirds of the cycles issue, their pipe is busy for 47 %, and ready warps wait for the register file's ports),
// so the rest is arranged to keep two blocks of eight warps on every multiprocessor issuing them:
// operands by cp.async three slices deep, rows 36 floats apart (16-byte reads of 8 neighbouring rows meet no bank twice),
// and K cut among the blocks of a cluster where the tiles alone would leave multiprocessors idle.  The groups' and then
// the cluster's sums meet in shared memory in a fixed order.
// Measured (us, before -> after): 389 rows x 9,728 features x 896 (gate/up of the 0.5B sizes) 386 -> 232, 389 x 896 x 4,864
// 430 -> 160, 389 x 151,936 x 896 5,176 -> 3,110 (34 TFLOP/s of the 71 that FFMA alone reaches).  Slices of 64 columns and two
// products an instruction (fma.rn.f32x2, one block a multiprocessor) measured 3 to 15 % slower.
constexpr int F_BN = 64, F_BK = 32, F_STAGES = 3, F_PAD = F_BK + 4, F_RED = F_BN + 8, F_THREADS = 256;
constexpr int F_MAX_SPLIT = 8;
template <int BM> constexpr int f32_stage_floats() { return (BM + F_BN) * F_PAD; }
template <int BM> constexpr int f32_smem_bytes() {
    return 4 * (F_STAGES * f32_stage_floats<BM>() > 3 * BM * F_RED ? F_STAGES * f32_stage_floats<BM>() : 3 * BM * F_RED);
}

__device__ __forceinline__ void cp_async16_or_zero(float* dst, const float* src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

template <int EPI, int BM>
__global__ void __launch_bounds__(F_THREADS, 2) gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W,
                                                                const float* __restrict__ bias, void* __restrict__ out,
                                                                float* __restrict__ residual, int M, int N, int K,
                                                                int k_part, const LlbGluArgs glu) {
    extern __shared__ __align__(16) float fsm[];
    constexpr int RM = BM / 8;                       // rows of a thread
    constexpr int CH = F_BK / 4;                     // 16-byte pieces of a row of a slice
    const int tid = threadIdx.x;
    const int group = tid >> 6, tm = (tid & 63) >> 3, tn = tid & 7;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * F_BN;
    const int k_lo = blockIdx.z * k_part, k_hi = min(K, k_lo + k_part);
    const int slices = (k_hi - k_lo + F_BK - 1) / F_BK;

    auto request = [&](int slice) {
        float* stage = fsm + (slice % F_STAGES) * f32_stage_floats<BM>();
        const int k0 = k_lo + slice * F_BK;
#pragma unroll
        for (int i = 0; i < ((BM + F_BN) * CH + F_THREADS - 1) / F_THREADS; ++i) {
            const int c = tid + i * F_THREADS;
            if ((BM + F_BN) * CH % F_THREADS && c >= (BM + F_BN) * CH) break;
            const int row = c / CH, k = k0 + (c % CH) * 4;
            const bool is_a = row < BM;
            const int r = is_a ? m0 + row : n0 + row - BM;
            const bool valid = k < k_hi && r < (is_a ? M : N);
            const float* src = is_a ? A : W;
            cp_async16_or_zero(stage + row * F_PAD + (c % CH) * 4, valid ? src + (size_t)r * K + k : src, valid);
        }
    };
    float acc[RM][8];
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;

#pragma unroll
    for (int s = 0; s < F_STAGES - 1; ++s) {
        if (s < slices) request(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int s = 0; s < slices; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(F_STAGES - 2) : "memory");
        __syncthreads();          // slice s has landed for everyone, and slice s - 1 has been read by everyone
        if (s + F_STAGES - 1 < slices) request(s + F_STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* as = fsm + (s % F_STAGES) * f32_stage_floats<BM>() + group * (F_BK / 4);
        const float* ws = as + BM * F_PAD;
#pragma unroll
        for (int kk = 0; kk < F_BK / 4; kk += 4) {
            float4 a[RM];
#pragma unroll
            for (int i = 0; i < RM; ++i) a[i] = *reinterpret_cast<const float4*>(as + (tm + 8 * i) * F_PAD + kk);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 w = *reinterpret_cast<const float4*>(ws + (tn + 8 * j) * F_PAD + kk);
#pragma unroll
                for (int i = 0; i < RM; ++i) {
                    acc[i][j] = fmaf(a[i].x, w.x, acc[i][j]);
                    acc[i][j] = fmaf(a[i].y, w.y, acc[i][j]);
                    acc[i][j] = fmaf(a[i].z, w.z, acc[i][j]);
                    acc[i][j] = fmaf(a[i].w, w.w, acc[i][j]);
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (group > 0) {
        float* red = fsm + (group - 1) * BM * F_RED;
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) red[(tm + 8 * i) * F_RED + tn + 8 * j] = acc[i][j];
    }
    __syncthreads();
    if (group == 0) {
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int at = (tm + 8 * i) * F_RED + tn + 8 * j;
                fsm[at] = acc[i][j] + fsm[at] + fsm[BM * F_RED + at] + fsm[2 * BM * F_RED + at];
            }
    }
    namespace cg = cooperative_groups;
    const int parts = gridDim.z;
    if (parts > 1) cg::this_cluster().sync();
    else __syncthreads();
    // every block of the cluster finishes its share of the tile's rows (pairs of columns: the gated epilogue takes two)
    const int r_lo = BM * (int)blockIdx.z / parts, r_hi = BM * ((int)blockIdx.z + 1) / parts;
    for (int i = tid; i < (r_hi - r_lo) * (F_BN / 2); i += F_THREADS) {
        const int row = r_lo + i / (F_BN / 2), c = (i % (F_BN / 2)) * 2;
        const int m = m0 + row, n = n0 + c;
        if (m >= M || n >= N) continue;
        float2 v = make_float2(0.0f, 0.0f);
        if (parts > 1) {
            for (int z = 0; z < parts; ++z) {
                const float2 u = *reinterpret_cast<const float2*>(cg::this_cluster().map_shared_rank(fsm, z) + row * F_RED + c);
                v.x += u.x;
                v.y += u.y;
            }
        } else {
            v = *reinterpret_cast<const float2*>(fsm + row * F_RED + c);
        }
        const bool has1 = n + 1 < N;
        if (bias) {
            v.x += bias[n];
            if (has1) v.y += bias[n + 1];
        }
        Epilogue<float, EPI>::pair(v.x, v.y, m, n, N, out, residual, has1, glu);
    }
    if (parts > 1) cg::this_cluster().sync();          // the others may still read this block's sums
}

// Into how many pieces K is cut: two blocks are resident on a multiprocessor, and the tiles shall fill them once; no piece
// below four slices.  The order of a row's sum depends on it, and so its last bits depend on how many rows are beside it.
int f32_split(int tiles, int slices) {
    int split = 2 * llb_device_sms() / tiles;
    split = split > slices / 4 ? slices / 4 : split;
    return split < 1 ? 1 : split > F_MAX_SPLIT ? F_MAX_SPLIT : split;
}

// Whether M rows, five to eight of them, are for the streaming kernel (fewer always are, more never).  It reads the rows again for every
// pair of features; the tile kernel takes as long for five rows as for 16, and mostly less: 896 x 4,864 (features x K) 12 us, streaming
// 29 to 41 at five to eight rows, 3,584 x 3,584 21 / 29 to 39, 2,048 x 64 3.3 / 3.3 to 3.9, 13,824 x 896 24 / 27 to 38.  Streaming is
// ahead where a tile's chain of slices is the longer one: K of three to eight slices, which tiles hardly cut, under few features (896 x
// 256 5.0 us, streaming 3.9 to 5.0; 2,048 x 128 4.1 / 3.3 to 4.1; 4,096 x 256 at five rows 5.2 / 4.7), and a longer K that is not cut
// because every multiprocessor has a tile but few have two (9,728 x 896 23.6 / 17 to 21 at up to seven rows, 10,624 x 4,096 98 / 70 to 83).
bool f32_streamed(int M, int N, int K) {
    const int nt = llb_ceil_div(N, F_BN), slices = llb_ceil_div(K, F_BK), sms = llb_device_sms();
    if (M <= 4 || M > 8) return M <= 4;
    if (slices <= 8) return slices >= 3 && (long long)nt * M <= 320;
    return slices >= 16 && nt > sms && nt <= sms * 6 / 5 && nt * M <= 8 * sms;
}

// Whether floats go to the tensor cores (csrc/gemm_f32_tcgen05.cu).  That kernel and the one before it take 7 to 10 us whatever they are
// given, so the products (of the rows that the tiles here would pad to) have to be worth it; us there / here at features x K:
//   389 rows  64 x 896 13 / 10, 512 x 256 15 / 11, 256 x 896 14 / 15, 4,096 x 64 13 / 20, 9,728 x 896 58 / 227, 151,936 x 896 703 / 3,110
//   100 rows  4,096 x 128 12 / 11, 4,096 x 256 14 / 16, 896 x 896 13 / 15, 4,096 x 896 15 / 35
//   48 rows   2,048 x 512 11 / 10, 4,096 x 256 11 / 11, 4,096 x 512 11 / 15, 896 x 4,864 22 / 26
// At 17 to 32 rows the tiles here are as low as the rows, and only many features make up for the long chain of slices there
// (24 rows: 896 x 4,864 21 / 15, 4,096 x 896 13 / 13, 6,144 x 896 18 / 23, 9,728 x 896 26 / 31, 151,936 x 896 235 / 250).
bool f32_split_pays(int M, int N, int K) {
    if (M <= 16) return false;
    if (M <= 32) return N >= 6144 && K >= 512;
    return (long long)llb_ceil_div(M, 64) * 64 * N * K >= 80000000ll;
}

template <int EPI, int BM>
int launch_f32(const float* A, const float* W, const float* bias, void* out, float* residual, int M, int N, int K, LlbGluArgs glu,
               cudaStream_t stream) {
    constexpr int smem = f32_smem_bytes<BM>();
    static std::atomic<bool> configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev].load()) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_f32_kernel<EPI, BM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return llb_fail("gemm: cannot opt in to %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
        if (dev >= 0 && dev < 64) configured[dev].store(true);
    }
    const int mt = llb_ceil_div(M, BM), nt = llb_ceil_div(N, F_BN), slices = llb_ceil_div(K, F_BK);
    const int per = llb_ceil_div(slices, f32_split(mt * nt, slices));
    const int split = llb_ceil_div(slices, per);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(mt, nt, split);
    cfg.blockDim = dim3(F_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = split;
    cfg.attrs = at;
    cfg.numAttrs = split > 1 ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_f32_kernel<EPI, BM>, A, W, bias, out, residual, M, N, K, per * F_BK, glu);
    if (e != cudaSuccess) return llb_fail("gemm_f32: %s", cudaGetErrorString(e));
    return llb_check_launch("gemm_f32");
}

template <int EPI>
int dispatch_f32(const float* A, const float* W, const float* bias, void* out, float* residual, int M, int N, int K, LlbGluArgs glu,
                 cudaStream_t stream) {
    if (M <= 16) return launch_f32<EPI, 16>(A, W, bias, out, residual, M, N, K, glu, stream);
    if (M <= 32) return launch_f32<EPI, 32>(A, W, bias, out, residual, M, N, K, glu, stream);
    return launch_f32<EPI, 64>(A, W, bias, out, residual, M, N, K, glu, stream);
}

template <typename TA, typename TW, typename TO, int EPI>
int launch(const void* A, const void* W, const void* bias, void* out, float* residual, int M, int N, int K, LlbGluArgs glu,
           cudaStream_t stream) {
    const TA* a = (const TA*)A;
    const TW* w = (const TW*)W;
    const float* b = (const float*)bias;
    constexpr int MAXM = 8;
    if constexpr (sizeof(TA) == 4 && sizeof(TW) == 4) {
        // The tile kernel: rows in 16-byte steps for cp.async, 64-column tiles in the grid's y, not a call that the streaming kernel is
        // better at.  (More rows than the general kernel's grid counts are refused below, whatever their form.)
        if (!f32_streamed(M, N, K) && K % 4 == 0 && ((uintptr_t)A | (uintptr_t)W) % 16 == 0 && llb_ceil_div(N, F_BN) <= 65535 &&
            llb_ceil_div(M, BM) <= 65535)
            return dispatch_f32<EPI>((const float*)A, (const float*)W, b, out, residual, M, N, K, glu, stream);
    }
    if (M <= MAXM) {
        const int warps = (N + 1) / 2;
        const int threads = 128;
        const int blocks = llb_ceil_div(warps * 32, threads);
        constexpr int WVEC = sizeof(TW) == 2 ? 8 : 4;
        const bool aligned = (K % WVEC == 0) && ((uintptr_t)W % 16 == 0);
        if (aligned)
            gemm_rows_kernel<TA, TW, TO, EPI, MAXM, WVEC><<<blocks, threads, 0, stream>>>(a, w, b, out, residual, M, N, K, glu);
        else
            gemm_rows_kernel<TA, TW, TO, EPI, MAXM, 1><<<blocks, threads, 0, stream>>>(a, w, b, out, residual, M, N, K, glu);
        return llb_check_launch("gemm_rows");
    }
    dim3 grid(llb_ceil_div(N, BN), llb_ceil_div(M, BM));
    LLB_REQUIRE(grid.y <= 65535, "gemm: M=%d is too large for one launch", M);
    gemm_tile_kernel<TA, TW, TO, EPI><<<grid, 256, 0, stream>>>(a, w, b, out, residual, M, N, K, glu);
    return llb_check_launch("gemm_tile");
}

template <typename TA, typename TW>
int dispatch_epilogue(int epi, const void* A, const void* W, const void* bias, void* out, float* residual, int M,
                      int N, int K, LlbGluArgs glu, cudaStream_t s) {
    switch (epi) {
        case LLB_EPI_STORE: return launch<TA, TW, TA, LLB_EPI_STORE>(A, W, bias, out, residual, M, N, K, glu, s);
        case LLB_EPI_STORE_F32: return launch<TA, TW, float, LLB_EPI_STORE_F32>(A, W, bias, out, residual, M, N, K, glu, s);
        case LLB_EPI_RESIDUAL: return launch<TA, TW, float, LLB_EPI_RESIDUAL>(A, W, bias, out, residual, M, N, K, glu, s);
        case LLB_EPI_SWIGLU: return launch<TA, TW, TA, LLB_EPI_SWIGLU>(A, W, bias, out, residual, M, N, K, glu, s);
    }
    return llb_fail("gemm: unknown epilogue %d", epi);
}

}  // namespace

// Bytes of scratch with which a contraction of these sizes goes to the tensor cores (0: it stays on CUDA cores).
LLB_EXPORT long long llb_gemm_simt_scratch_bytes(int a_dtype, int w_dtype, int M, int N, int K) {
    if (a_dtype != LLB_F32 || w_dtype != LLB_F32 || M <= 0 || N <= 0 || K <= 0 || K % 4 != 0 || llb_ceil_div(M, BM) > 65535) return 0;
    return f32_split_pays(M, N, K) ? llb_gemm_f32_scratch_bytes(M, K) : 0;
}

// A [M,K] (a_dtype), W [N,K] (w_dtype), bias [N] float or null.  `out` is [M,N] of a_dtype
// (STORE), [M,N] float (STORE_F32) or [M,N/2] of a_dtype (SWIGLU, N even); `residual` is
// [M,N] float (RESIDUAL).  Supported: (float,float), (bf16,bf16), (bf16 activations, float weights).
// glu_kind .. glu_up_shift: the gated activation of the GLU epilogue (LLB_GLU_*, see llb_glu); under STORE a kind of LlbAct
// is a plain activation of every output.
// scratch (16-byte aligned): null, or as llb_gemm_simt_scratch_bytes says; error_flag: raised when a wait ran out of time.
LLB_EXPORT int llb_gemm_simt_glu(const void* A, int a_dtype, const void* W, const void* bias, int w_dtype, void* out,
                                 float* residual, int epilogue, int M, int N, int K, int glu_kind, float glu_alpha,
                                 float glu_limit, float glu_up_shift, void* scratch, long long scratch_bytes,
                                 int* error_flag, cudaStream_t stream) {
    const LlbGluArgs glu = LlbGluArgs{glu_kind, glu_alpha, glu_limit, glu_up_shift};
    if (M == 0) return 0;
    LLB_REQUIRE(M > 0 && N > 0 && K > 0, "gemm: bad sizes M=%d N=%d K=%d", M, N, K);
    LLB_REQUIRE(epilogue != LLB_EPI_SWIGLU || N % 2 == 0, "gemm: SwiGLU epilogue needs an even N, got %d", N);
    LLB_REQUIRE(epilogue != LLB_EPI_RESIDUAL || residual != nullptr, "gemm: residual epilogue without residual");
    LLB_REQUIRE(epilogue == LLB_EPI_RESIDUAL || out != nullptr, "gemm: output pointer is null");
    const long long need = llb_gemm_simt_scratch_bytes(a_dtype, w_dtype, M, N, K);
    if (need > 0 && scratch && scratch_bytes >= need && llb_gemm_f32_tcgen05_takes(A, W, M, N, K))
        return llb_gemm_f32_tcgen05(A, W, bias, out, residual, epilogue, M, N, K, glu_kind, glu_alpha, glu_limit, glu_up_shift,
                                    scratch, error_flag, stream);
    if (a_dtype == LLB_F32 && w_dtype == LLB_F32)
        return dispatch_epilogue<float, float>(epilogue, A, W, bias, out, residual, M, N, K, glu, stream);
    if (a_dtype == LLB_BF16 && w_dtype == LLB_BF16)
        return dispatch_epilogue<__nv_bfloat16, __nv_bfloat16>(epilogue, A, W, bias, out, residual, M, N, K, glu, stream);
    if (a_dtype == LLB_BF16 && w_dtype == LLB_F32)
        return dispatch_epilogue<__nv_bfloat16, float>(epilogue, A, W, bias, out, residual, M, N, K, glu, stream);
    return llb_fail("gemm: unsupported dtype pair activations=%d weights=%d", a_dtype, w_dtype);
}

// The same with SiLU as the GLU epilogue's activation.
LLB_EXPORT int llb_gemm_simt(const void* A, int a_dtype, const void* W, const void* bias, int w_dtype, void* out,
                             float* residual, int epilogue, int M, int N, int K, void* scratch, long long scratch_bytes,
                             int* error_flag, cudaStream_t stream) {
    return llb_gemm_simt_glu(A, a_dtype, W, bias, w_dtype, out, residual, epilogue, M, N, K, LLB_GLU_SILU, 1.0f, 0.0f, 0.0f,
                             scratch, scratch_bytes, error_flag, stream);
}

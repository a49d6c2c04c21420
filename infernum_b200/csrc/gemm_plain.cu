// Plain matrix product on the CUDA cores in true 32-bit:
//   C[M, N] = A[M, K] . W[N, K]^T      (W in checkpoint layout [out, in])
// Every output element is one chain of fused multiply-adds over k = 0..K-1 in
// ascending order, so a row of C does not depend on M, on the other rows, or
// on how the rows were batched.  Operands may be bf16 (widened exactly); the
// products and sums are 32-bit; no tensor-core or reduced-precision mode.
// It stands where the reference calls cuBLAS with 32-bit compute
// (infernum-cuda/src/inner/cuda/ops/matmul.rs:68-116) on its f32 path.
//
// Three kernels with one arithmetic, so that all of them give the same bits:
//   gemm_rows_kernel   float32, at most 64 rows, 32 where N x batch >= 8,192 (decode): the weights stream through shared
//                      memory once
//   gemm_tile_kernel   float32, more rows: register tiles, two tile sizes
//   gemm_plain_kernel  any operand types, strides and alignments
#include "common.cuh"

using namespace ib;

namespace {
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

// `bytes` (0 or 16) are copied, the rest of the sixteen is filled with zeros.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int bytes) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
}  // namespace

// Few rows.  A CTA takes 16 NC weight rows for all the rows of A; both operands come through a ring of stages of 128 k
// by cp.async, which four warps of their own issue.  A thread of the other warps owns NC columns, 16 apart, and MR
// rows, G apart (G * MR >= M), and fetches a few k of both from shared memory under the multiply-adds of those before.
// Rows of a stage are 132 floats apart: the eight weight rows of a quarter warp's 16-byte loads lie in different banks.
// Bound by the chain where the SMs hold a CTA or two (a stage of 128 k takes some 1,200 cycles, 536 of them dependent
// multiply-adds), by the loads from shared memory where they hold more.  Eight rows, the general kernel's time behind:
// 3072 x 2048 15.6 us (175), 16384 x 2048 36.7 us = 3.7 TB/s (225), 2048 x 8192 49.5 us = 1.4 TB/s (710).
constexpr int ROWS_BK = 128, ROWS_PITCH = ROWS_BK + 4;
template <int MR, int NC, int G>
struct RowsRing {
    static constexpr int ROWS = 16 * NC + G * MR;            // of W, then of A
    static constexpr int STAGE = ROWS * ROWS_PITCH;          // floats
    static constexpr int STAGES = ROWS <= 24 ? 5 : ROWS <= 48 ? 4 : 3;
    static constexpr int BYTES = STAGES * STAGE * (int)sizeof(float);
    static constexpr int COMPUTE = 16 * G, THREADS = COMPUTE + 128;
    static constexpr int KB = MR * NC <= 2 ? 16 : MR * NC <= 8 ? 8 : 4;  // k fetched together: 64 cycles of arithmetic
};

template <int MR, int NC, int G>
__global__ void __launch_bounds__(RowsRing<MR, NC, G>::THREADS)
gemm_rows_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, float* __restrict__ C,
                 int ldc, int M, int N, int K, long long a_bs, long long w_bs, long long c_bs) {
    using Ring = RowsRing<MR, NC, G>;
    pdl_trigger();
    pdl_wait();
    A += (size_t)blockIdx.z * a_bs;
    W += (size_t)blockIdx.z * w_bs;
    C += (size_t)blockIdx.z * c_bs;
    constexpr int BN = 16 * NC, ROWS = Ring::ROWS, STAGES = Ring::STAGES, STAGE = Ring::STAGE, KB = Ring::KB;
    constexpr int COMPUTE = Ring::COMPUTE;
    static_assert(G % 2 == 0, "whole warps compute");
    extern __shared__ __align__(16) float ring[];
    const int tid = threadIdx.x, n0 = blockIdx.x * BN;
    const int col = tid % 16, group = tid / 16;
    const int n_k = (K + ROWS_BK - 1) / ROWS_BK;

    auto fetch = [&](int t) {  // by the last four warps
        if (t < n_k) {
            float* dst = ring + (size_t)(t % STAGES) * STAGE + (tid % 32) * 4;
            const int k = t * ROWS_BK + (tid % 32) * 4;
            const int kept = k < K ? 16 : 0;  // (K is a multiple of four)
            const int ks = k < K ? k : 0;
#pragma unroll
            for (int row = 0; row < (ROWS + 3) / 4 * 4; row += 4) {
                const int r = row + (tid - COMPUTE) / 32;
                if (r < BN) {
                    const int n = n0 + r;
                    cp_async16(dst + r * ROWS_PITCH, W + (size_t)(n < N ? n : 0) * ldw + ks, n < N ? kept : 0);
                } else if (r < ROWS) {
                    const int m = r - BN;
                    cp_async16(dst + r * ROWS_PITCH, A + (size_t)(m < M ? m : 0) * lda + ks, m < M ? kept : 0);
                }
            }
        }
        cp_async_commit();
    };
    if (tid >= COMPUTE) {
#pragma unroll
        for (int t = 0; t < STAGES - 1; ++t) fetch(t);
    }
    float acc[MR][NC];
#pragma unroll
    for (int i = 0; i < MR; ++i)
#pragma unroll
        for (int j = 0; j < NC; ++j) acc[i][j] = 0.f;
    for (int t = 0; t < n_k; ++t) {
        if (tid >= COMPUTE) cp_async_wait<STAGES - 2>();
        __syncthreads();  // stage t has come, and stage t - 1 is read by all
        if (tid >= COMPUTE) {
            fetch(t + STAGES - 1);
        } else {
            const float* w = ring + (size_t)(t % STAGES) * STAGE + col * ROWS_PITCH;
            const float* a = ring + (size_t)(t % STAGES) * STAGE + (BN + group) * ROWS_PITCH;
            float4 wv[2][KB / 4][NC], av[2][KB / 4][MR];
            auto frag = [&](int k, int f) {
#pragma unroll
                for (int q = 0; q < KB / 4; ++q) {
#pragma unroll
                    for (int j = 0; j < NC; ++j)
                        wv[f][q][j] = *reinterpret_cast<const float4*>(w + j * 16 * ROWS_PITCH + k + 4 * q);
#pragma unroll
                    for (int i = 0; i < MR; ++i)
                        av[f][q][i] = *reinterpret_cast<const float4*>(a + i * G * ROWS_PITCH + k + 4 * q);
                }
            };
            auto mul = [&](int f) {
#pragma unroll
                for (int q = 0; q < KB / 4; ++q) {
#define IB_STEP(u)                                                                                             \
    _Pragma("unroll") for (int i = 0; i < MR; ++i)                                                             \
        _Pragma("unroll") for (int j = 0; j < NC; ++j) acc[i][j] = fmaf(av[f][q][i].u, wv[f][q][j].u, acc[i][j]);
                    IB_STEP(x) IB_STEP(y) IB_STEP(z) IB_STEP(w)
#undef IB_STEP
                }
            };
            frag(0, 0);
#pragma unroll 1
            for (int k = 0; k < ROWS_BK; k += 2 * KB) {
                frag(k + KB, 1);
                mul(0);
                if (k + 2 * KB < ROWS_BK) frag(k + 2 * KB, 0);
                mul(1);
            }
        }
    }
    if (tid < COMPUTE) {
#pragma unroll
        for (int i = 0; i < MR; ++i)
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                const int m = group + i * G, n = n0 + col + 16 * j;
                if (m < M && n < N) C[(size_t)m * ldc + n] = acc[i][j];
            }
    }
}

// Many rows: bound by the multiply-adds.  A thread owns FM x FN outputs; per k it loads FM + FN values as 16-byte
// pieces of rows of k (A and W are turned while they are stored), a k ahead of its arithmetic, and the next block of 16
// k is fetched into registers meanwhile.  Two neighbouring outputs are one packed multiply-add (fma.rn.f32x2: each half
// rounds as fmaf does).  A warp is 4 x 8 lanes, so its loads of either operand touch every bank once.
// 700 x 16384 x 2048: 1,055 us = 44 TFLOP/s (the general kernel 1,919 us; 8 x 8 outputs a thread 1,021 us, without
// the packed form 1,280); 700 x 2048 x 2048: 172 us (314; 8 x 8 outputs, whose tiles fill the SMs worse, 232).
// Launched in order, and its operands are read past the L1: as a programmatic dependent that read them through the
// read-only path it met lines that an SM had kept of what lay in the same memory before (outputs 4 % off).
__device__ __forceinline__ float2 fma2(float a, float2 b, float2 c) {
    const float2 aa = make_float2(a, a);
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<const unsigned long long&>(aa)), "l"(reinterpret_cast<const unsigned long long&>(b)),
          "l"(reinterpret_cast<const unsigned long long&>(c)));
    return d;
}

template <int TILE_M, int TILE_N, int FM, int FN>
__global__ void __launch_bounds__((TILE_M / (4 * FM)) * (TILE_N / (8 * FN)) * 32)
gemm_tile_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, float* __restrict__ C,
                 int ldc, int M, int N, int K, long long a_bs, long long w_bs, long long c_bs) {
    A += (size_t)blockIdx.z * a_bs;
    W += (size_t)blockIdx.z * w_bs;
    C += (size_t)blockIdx.z * c_bs;
    constexpr int WARPS_M = TILE_M / (4 * FM), WARPS_N = TILE_N / (8 * FN), THREADS = WARPS_M * WARPS_N * 32;
    constexpr int A_LOADS = TILE_M * 4 / THREADS, W_LOADS = TILE_N * 4 / THREADS;
    static_assert(A_LOADS * THREADS == TILE_M * 4 && W_LOADS * THREADS == TILE_N * 4, "tile and threads do not fit");
    __shared__ __align__(16) float As[2][BK][TILE_M + 4];
    __shared__ __align__(16) float Ws[2][BK][TILE_N + 4];
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const int ly = lane / 8, lx = lane % 8;
    const int wm = (warp / WARPS_N) * (4 * FM), wn = (warp % WARPS_N) * (8 * FN);
    const int m0 = blockIdx.y * TILE_M, n0 = blockIdx.x * TILE_N;
    const int lrow = tid / 4, lk = (tid % 4) * 4;

    float2 acc[FM][FN / 2];
#pragma unroll
    for (int i = 0; i < FM; ++i)
#pragma unroll
        for (int j = 0; j < FN / 2; ++j) acc[i][j] = make_float2(0.f, 0.f);

    float4 ra[A_LOADS], rw[W_LOADS];
    auto load = [&](int k0) {
        const bool in = k0 + lk < K;  // (K is a multiple of four)
#pragma unroll
        for (int r = 0; r < A_LOADS; ++r) {
            const int m = m0 + lrow + r * (THREADS / 4);
            ra[r] = in && m < M ? __ldcg(reinterpret_cast<const float4*>(A + (size_t)m * lda + k0 + lk))
                                : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int r = 0; r < W_LOADS; ++r) {
            const int n = n0 + lrow + r * (THREADS / 4);
            rw[r] = in && n < N ? __ldcg(reinterpret_cast<const float4*>(W + (size_t)n * ldw + k0 + lk))
                                : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int r = 0; r < A_LOADS; ++r) {
            const int m = lrow + r * (THREADS / 4);
            As[buf][lk][m] = ra[r].x;
            As[buf][lk + 1][m] = ra[r].y;
            As[buf][lk + 2][m] = ra[r].z;
            As[buf][lk + 3][m] = ra[r].w;
        }
#pragma unroll
        for (int r = 0; r < W_LOADS; ++r) {
            const int n = lrow + r * (THREADS / 4);
            Ws[buf][lk][n] = rw[r].x;
            Ws[buf][lk + 1][n] = rw[r].y;
            Ws[buf][lk + 2][n] = rw[r].z;
            Ws[buf][lk + 3][n] = rw[r].w;
        }
    };
    float4 fa[2][FM / 4], fw[2][FN / 4];
    auto frag = [&](int buf, int kk, int f) {
#pragma unroll
        for (int i = 0; i < FM / 4; ++i) fa[f][i] = *reinterpret_cast<const float4*>(&As[buf][kk][wm + i * 16 + ly * 4]);
#pragma unroll
        for (int j = 0; j < FN / 4; ++j) fw[f][j] = *reinterpret_cast<const float4*>(&Ws[buf][kk][wn + j * 32 + lx * 4]);
    };
    load(0);
    store(0);
    __syncthreads();
    frag(0, 0, 0);
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += BK, buf ^= 1) {
        const bool more = k0 + BK < K;
        if (more) load(k0 + BK);
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            if (kk < BK - 1) {
                frag(buf, kk + 1, (kk + 1) & 1);
            } else {
                if (more) store(buf ^ 1);  // (read by nobody since the barrier of the block before)
                __syncthreads();
                if (more) frag(buf ^ 1, 0, 0);
            }
            const float* a = reinterpret_cast<const float*>(fa[kk & 1]);
            const float2* w = reinterpret_cast<const float2*>(fw[kk & 1]);
#pragma unroll
            for (int i = 0; i < FM; ++i)
#pragma unroll
                for (int j = 0; j < FN / 2; ++j) acc[i][j] = fma2(a[i], w[j], acc[i][j]);
        }
    }
    const bool wide = N % 4 == 0 && ldc % 4 == 0 && ((uintptr_t)C & 15) == 0;
#pragma unroll
    for (int i = 0; i < FM; ++i) {
        const int m = m0 + wm + (i / 4) * 16 + ly * 4 + i % 4;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < FN; j += 4) {
            const int n = n0 + wn + j * 8 + lx * 4;
            float* dst = C + (size_t)m * ldc + n;
            const float2 lo = acc[i][j / 2], hi = acc[i][j / 2 + 1];
            if (wide) {
                if (n < N) *reinterpret_cast<float4*>(dst) = make_float4(lo.x, lo.y, hi.x, hi.y);
            } else {
                if (n < N) dst[0] = lo.x;
                if (n + 1 < N) dst[1] = lo.y;
                if (n + 2 < N) dst[2] = hi.x;
                if (n + 3 < N) dst[3] = hi.y;
            }
        }
    }
}

template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(256)
gemm_plain_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W, int ldw,
                  TC* __restrict__ C, int ldc, int M, int N, int K, long long a_bs, long long w_bs,
                  long long c_bs) {
    // blockIdx.z is the member of a batch: its operands lie a_bs, w_bs, c_bs elements apart
    A += (size_t)blockIdx.z * a_bs;
    W += (size_t)blockIdx.z * w_bs;
    C += (size_t)blockIdx.z * c_bs;
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int lrow = tid / 4, lk = (tid % 4) * 4;

    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        {
            const int gm = m0 + lrow;
            const TA* src = A + (size_t)gm * lda + k0 + lk;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                As[lk + u][lrow] = (gm < M && k0 + lk + u < K) ? to_f32(src[u]) : 0.f;
            const int gn = n0 + lrow;
            const TW* wsrc = W + (size_t)gn * ldw + k0 + lk;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                Ws[lk + u][lrow] = (gn < N && k0 + lk + u < K) ? to_f32(wsrc[u]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], w[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = Ws[kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * TM + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx * TN + j;
            if (gn < N) C[(size_t)gm * ldc + gn] = from_f32<TC>(acc[i][j]);
        }
    }
}

template <typename TA, typename TW, typename TC>
static int launch(const void* A, int lda, const void* W, int ldw, void* C, int ldc, int M, int N,
                  int K, cudaStream_t s, int batch = 1, long long a_bs = 0, long long w_bs = 0,
                  long long c_bs = 0) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batch);
    gemm_plain_kernel<TA, TW, TC><<<grid, 256, 0, s>>>((const TA*)A, lda, (const TW*)W, ldw,
                                                        (TC*)C, ldc, M, N, K, a_bs, w_bs, c_bs);
    IB_LAUNCH_CHECK();
    return IB_OK;
}

template <int MR, int NC, int G>
static int launch_rows(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K,
                       cudaStream_t s, int batch, long long a_bs, long long w_bs, long long c_bs) {
    static bool attr_done = false;
    if (!attr_done) {
        cudaError_t e = cudaFuncSetAttribute(gemm_rows_kernel<MR, NC, G>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             RowsRing<MR, NC, G>::BYTES);
        if (e != cudaSuccess) return (int)e;
        attr_done = true;
    }
    cudaError_t le = launch_kernel(gemm_rows_kernel<MR, NC, G>, dim3((N + 16 * NC - 1) / (16 * NC), 1, batch),
                                   dim3(RowsRing<MR, NC, G>::THREADS), (size_t)RowsRing<MR, NC, G>::BYTES, s, A, lda, W,
                                   ldw, C, ldc, M, N, K, a_bs, w_bs, c_bs);
    if (le != cudaSuccess) return (int)le;
    IB_LAUNCH_CHECK();
    return IB_OK;
}

template <int TILE_M, int TILE_N, int FM, int FN>
static int launch_tile(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K,
                       cudaStream_t s, int batch, long long a_bs, long long w_bs, long long c_bs) {
    cudaError_t le = launch_kernel_in_order(
        gemm_tile_kernel<TILE_M, TILE_N, FM, FN>, dim3((N + TILE_N - 1) / TILE_N, (M + TILE_M - 1) / TILE_M, batch),
        dim3((TILE_M / (4 * FM)) * (TILE_N / (8 * FN)) * 32), 0, s, A, lda, W, ldw, C, ldc, M, N, K, a_bs, w_bs, c_bs);
    if (le != cudaSuccess) return (int)le;
    IB_LAUNCH_CHECK();
    return IB_OK;
}

constexpr double SMALL_TILE_COST = 1.6;  // of an output in a tile of 32 x 32 against one of 64 x 64

// float32 throughout.  Sixteen-byte loads need 16-byte aligned rows of a multiple of four values; everything else
// goes to the general kernel.
static int launch_f32(const void* A, int lda, const void* W, int ldw, void* C, int ldc, int M, int N, int K,
                      cudaStream_t s, int batch = 1, long long a_bs = 0, long long w_bs = 0, long long c_bs = 0) {
    const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && a_bs % 4 == 0 && w_bs % 4 == 0 &&
                     !((uintptr_t)A & 15) && !((uintptr_t)W & 15);
    if (!vec) return launch<float, float, float>(A, lda, W, ldw, C, ldc, M, N, K, s, batch, a_bs, w_bs, c_bs);
#define IB_F32(F) F((const float*)A, lda, (const float*)W, ldw, (float*)C, ldc, M, N, K, s, batch, a_bs, w_bs, c_bs)
    // (more columns a thread from the width on that still gives every SM several warps)
    const bool many = (long long)N * batch >= 8192;
    if (M <= 2) return IB_F32((launch_rows<1, 1, 2>));
    if (M <= 4) return many ? IB_F32((launch_rows<2, 2, 2>)) : IB_F32((launch_rows<2, 1, 2>));
    if (M <= 8) return many ? IB_F32((launch_rows<2, 4, 4>)) : IB_F32((launch_rows<2, 1, 4>));
    if (M <= 16) return many ? IB_F32((launch_rows<4, 2, 4>)) : IB_F32((launch_rows<2, 1, 8>));
    if (M <= 32) return many ? IB_F32((launch_rows<8, 2, 4>)) : IB_F32((launch_rows<4, 1, 8>));
    if (M <= 64 && !many) return IB_F32((launch_rows<8, 1, 8>));
    // The time of a tile size is that of the SM with the most tiles: rounds of 148 times a tile's work, which costs
    // more per output the smaller the tile.
    auto rounds = [&](int t) {
        return (double)(((long long)((M + t - 1) / t) * ((N + t - 1) / t) * batch + 147) / 148);
    };
    // (the rows' tiles are on the grid's y; small ones are cheaper at any number of rows where N <= 32)
    return (M + 31) / 32 <= 65535 && rounds(32) * 0.25 * SMALL_TILE_COST < rounds(64) ? IB_F32((launch_tile<32, 32, 4, 4>))
                                                            : IB_F32((launch_tile<64, 64, 8, 4>));
#undef IB_F32
}

// dtypes: 0 = f32, 1 = bf16.  Leading dimensions are in elements.
IB_EXPORT int ib_gemm_plain(const void* A, int a_dtype, int lda, const void* W, int w_dtype,
                            int ldw, void* C, int c_dtype, int ldc, int M, int N, int K,
                            void* stream) {
    if (M <= 0 || N <= 0) return IB_OK;
    if (!A || !W || !C || K <= 0 || lda < K || ldw < K || ldc < N) return IB_ERR_BAD_ARG;
    if ((M + BM - 1) / BM > 65535) return IB_ERR_TOO_LARGE;
    cudaStream_t s = (cudaStream_t)stream;
    const int key = a_dtype * 100 + w_dtype * 10 + c_dtype;
    switch (key) {
        case 0: return launch_f32(A, lda, W, ldw, C, ldc, M, N, K, s);
        case 10: return launch<float, bf16, float>(A, lda, W, ldw, C, ldc, M, N, K, s);
        case 100: return launch<bf16, float, float>(A, lda, W, ldw, C, ldc, M, N, K, s);
        case 101: return launch<bf16, float, bf16>(A, lda, W, ldw, C, ldc, M, N, K, s);
        case 110: return launch<bf16, bf16, float>(A, lda, W, ldw, C, ldc, M, N, K, s);
        case 111: return launch<bf16, bf16, bf16>(A, lda, W, ldw, C, ldc, M, N, K, s);
        default: return IB_ERR_UNSUPPORTED;
    }
}

// A batch of such products, member b on A + b * a_bs, W + b * w_bs, C + b * c_bs
// (strides in elements): one product per head, say, with the heads side by side
// in the rows of A and C.  Same arithmetic, member by member.
IB_EXPORT int ib_gemm_plain_batched(const void* A, int a_dtype, int lda, long long a_bs, const void* W,
                                    int w_dtype, int ldw, long long w_bs, void* C, int c_dtype, int ldc,
                                    long long c_bs, int batch, int M, int N, int K, void* stream) {
    if (M <= 0 || N <= 0 || batch <= 0) return IB_OK;
    if (!A || !W || !C || K <= 0 || lda < K || ldw < K || ldc < N) return IB_ERR_BAD_ARG;
    if ((M + BM - 1) / BM > 65535 || batch > 65535) return IB_ERR_TOO_LARGE;
    cudaStream_t s = (cudaStream_t)stream;
    const int key = a_dtype * 100 + w_dtype * 10 + c_dtype;
    switch (key) {
        case 0: return launch_f32(A, lda, W, ldw, C, ldc, M, N, K, s, batch, a_bs, w_bs, c_bs);
        case 10: return launch<float, bf16, float>(A, lda, W, ldw, C, ldc, M, N, K, s, batch, a_bs, w_bs, c_bs);
        case 110: return launch<bf16, bf16, float>(A, lda, W, ldw, C, ldc, M, N, K, s, batch, a_bs, w_bs, c_bs);
        case 111: return launch<bf16, bf16, bf16>(A, lda, W, ldw, C, ldc, M, N, K, s, batch, a_bs, w_bs, c_bs);
        default: return IB_ERR_UNSUPPORTED;
    }
}

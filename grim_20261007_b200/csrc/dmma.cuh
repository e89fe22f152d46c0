// Complex128 GEMM C = (BETA ? C : 0) + (NEG ? -1 : 1) A B on the FP64 tensor cores
// (mma.sync m8n8k4 .f64, the only FP64 tensor-core instruction; tcgen05 has no FP64 kind).
//
// CTA tile 16 TM x 16 TN complex, 4 warps in 2 x 2, each warp TM x TN MMA tiles with separate
// real and imaginary FP64 accumulators (64 doubles per thread at 4 x 4).  One
// complex k-step of a tile is four real MMAs:
//   re += Ar Br,  re += (-Ai) Bi,  im += Ar Bi,  im += Ai Br.
// K in stages of 8 complex (two MMA k-steps), three to six of them in shared memory, filled
// with cp.async (16 bytes = one complex element, zero-filled outside the matrices).
// Fragments of m8n8k4 (PTX ISA): A 8 x 4 row-major, lane holds A[lane / 4][lane % 4];
// B 4 x 8 column-major, lane holds B[lane % 4][lane / 4]; C 8 x 8, lane holds
// C[lane / 4][2 (lane % 4) + {0, 1}].
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define DM_BM 64
#define DM_BN 64
#define DM_BK 8
#define DM_THREADS 128
// shared tiles padded by two complex elements per k (conflict-free fragment reads)
// Stages in flight by tile: the small ones run short K on few CTAs an SM and wait for L2 (six
// stages and C read before the main loop: rank-64 updates of N = 2048 11.0 -> 8.3 us, of N = 333
// 10.1 -> 7.3, 1024 x 361 x 1024 0.160 -> 0.148 ms); 64 x 64 holds two CTAs an SM with three.
__host__ __device__ constexpr int dm_stages(int tm, int tn) { return tm * tn <= 4 ? 6 : tm * tn <= 8 ? 4 : 3; }
__host__ __device__ constexpr int dm_smem(int tm, int tn) {
    return dm_stages(tm, tn) * DM_BK * (16 * tm + 16 * tn + 4) * 16;
}
#define DM_SMEM_BYTES dm_smem(4, 4)

__device__ __forceinline__ void dm_cp16(void *smem, const void *gmem, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem);
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(gmem), "r"(bytes) : "memory");
}

__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

template <bool NEG, bool BETA, int TM = 4, int TN = 4>
__device__ __forceinline__ void gemm_dmma_cta(int M, int N, int K, const double2 *__restrict__ A, int64_t lda,
                                              const double2 *__restrict__ B, int64_t ldb, double2 *__restrict__ C,
                                              int64_t ldc, int m0, int n0) {
    constexpr int STAGES = dm_stages(TM, TN);
    constexpr int BM = 16 * TM, BN = 16 * TN, LDA = BM + 2, LDB = BN + 2;
    extern __shared__ __align__(16) unsigned char dm_tiles[];
    double2 *As = reinterpret_cast<double2 *>(dm_tiles);              // [stage][k][LDA]
    double2 *Bs = As + STAGES * DM_BK * LDA;                     // [stage][k][LDB] (k-major rows of n)
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int g = lane >> 2, q = lane & 3;
    const int wm = (warp >> 1) * 8 * TM, wn = (warp & 1) * 8 * TN;
    const int nk = (K + DM_BK - 1) / DM_BK;

    auto load_stage = [&](int stage, int kt) {
        const int k0 = kt * DM_BK;
        double2 *as = As + stage * DM_BK * LDA;
        double2 *bs = Bs + stage * DM_BK * LDB;
#pragma unroll
        for (int i = 0; i < (BM * DM_BK) / DM_THREADS; ++i) {
            const int e = t + DM_THREADS * i;
            const int m = e % BM, k = e / BM;  // consecutive threads: consecutive rows of a column
            const int gm = m0 + m, gk = k0 + k;
            const bool ok = gm < M && gk < K;
            dm_cp16(as + k * LDA + m, ok ? (const void *)(A + (int64_t)gk * lda + gm) : (const void *)A, ok);
        }
#pragma unroll
        for (int i = 0; i < (BN * DM_BK) / DM_THREADS; ++i) {
            const int e = t + DM_THREADS * i;
            const int k = e % DM_BK, n = e / DM_BK;  // consecutive threads: consecutive k of a column of B
            const int gk = k0 + k, gn = n0 + n;
            const bool ok = gk < K && gn < N;
            dm_cp16(bs + k * LDB + n, ok ? (const void *)(B + (int64_t)gn * ldb + gk) : (const void *)B, ok);
        }
    };

    double re[TM][TN][2], im[TM][TN][2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;

    // small tiles (short K, latency-bound): C arrives under the main loop
    constexpr bool early = BETA && TM * TN <= 4;
    double2 old[early ? TM : 1][early ? TN : 1][2];
    if constexpr (early) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int gm = min(m0 + wm + 8 * i + g, M - 1), gn = min(n0 + wn + 8 * j + 2 * q + c, N - 1);
                    old[i][j][c] = C[(int64_t)gn * ldc + gm];
                }
    }
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < nk) load_stage(s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int kt = 0; kt < nk; ++kt) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();
        // prefetch stage kt + STAGES - 1 into the buffer freed by stage kt - 1
        if (kt + STAGES - 1 < nk) load_stage((kt + STAGES - 1) % STAGES, kt + STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const double2 *as = As + (kt % STAGES) * DM_BK * LDA;
        const double2 *bs = Bs + (kt % STAGES) * DM_BK * LDB;
#pragma unroll
        for (int ks = 0; ks < DM_BK; ks += 4) {
            double ar[TM], ai[TM], nai[TM], br[TN], bi[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const double2 a = as[(ks + q) * LDA + wm + 8 * i + g];
                ar[i] = a.x;
                ai[i] = a.y;
                nai[i] = -a.y;
            }
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const double2 b = bs[(ks + q) * LDB + wn + 8 * j + g];
                br[j] = b.x;
                bi[j] = b.y;
            }
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    dmma(re[i][j][0], re[i][j][1], ar[i], br[j]);
                    dmma(re[i][j][0], re[i][j][1], nai[i], bi[j]);
                    dmma(im[i][j][0], im[i][j][1], ar[i], bi[j]);
                    dmma(im[i][j][0], im[i][j][1], ai[i], br[j]);
                }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // epilogue: lane holds rows wm + 8 i + g, columns wn + 8 j + 2 q + {0, 1}
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + wm + 8 * i + g;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int gn = n0 + wn + 8 * j + 2 * q + c;
                if (gn >= N) continue;
                double vr = re[i][j][c], vi = im[i][j][c];
                if (NEG) {
                    vr = -vr;
                    vi = -vi;
                }
                double2 *p = C + (int64_t)gn * ldc + gm;
                if (BETA) {
                    double2 o;
                    if constexpr (early) o = old[i][j][c];
                    else o = *p;
                    vr += o.x;
                    vi += o.y;
                }
                *p = make_double2(vr, vi);
            }
        }
    }
}

// grid = (ceil(M / 16 TM), ceil(N / 16 TN)).
template <bool NEG, bool BETA, int TM, int TN>
__global__ void __launch_bounds__(DM_THREADS)
k_gemm_dmma(int M, int N, int K, const double2 *__restrict__ A, int64_t lda, const double2 *__restrict__ B,
            int64_t ldb, double2 *__restrict__ C, int64_t ldc) {
    gemm_dmma_cta<NEG, BETA, TM, TN>(M, N, K, A, lda, B, ldb, C, ldc, blockIdx.x * 16 * TM, blockIdx.y * 16 * TN);
}

// Triangular solves of complex128 getrs, one launch per triangle.
//
// The right-hand-side columns are independent, so a CTA takes a strip of eight of them (the
// width of an FP64 tensor-core tile) through the whole substitution: no launch, no barrier
// between CTAs per 64-row block.  (64-row blocks solved by one launch and applied by a
// rank-64 GEMM by another spend 12 us and 25-50 us a block on launches, prologues and
// partly filled waves: N = 2048, 720 columns 2.1 ms a triangle.)
// Per 64-row block i, with X the solved rows of the strip:
//   1. W = B_i - T_i X over every solved row (mma.sync m8n8k4 .f64): sixteen warps, each eight
//      rows by every other group of four k-steps (eight warps left half the tensor pipe idle:
//      two a scheduler do not cover the instructions between the MMAs).  Fragments come
//      straight from L2 -- eight consecutive rows of a column are one 128-byte line, read once
//      per strip by one warp -- two groups ahead; the solved rows, each read by the eight warps
//      of its half of the groups, from L1; meanwhile the diagonal block arrives in shared memory
//      with cp.async;
//   2. the 64-row substitution, one warp per column, two rows per lane;
//   3. X_i to global memory, where step 1 of the next block reads it.
// Bound by the FP64 tensor pipe of the SMs that have a strip (8 n^2 x 8 / 2 flops a strip and
// triangle; 51 % of it over the whole chip at 90 strips) and the substitution chain (about 4 us a
// block).  getrs, both triangles with the
// interchanges, blocked launches before -> strips: N = 400, 722 columns 0.53 -> 0.18 ms;
// N = 1024, 361 1.30 -> 0.61 ms; N = 2048, 720 3.40 -> 1.99 ms; N = 4096, 720 9.5 -> 7.2 ms.
#pragma once
#include "dmma.cuh"
#include "lu.cuh"
#include "pivot.cuh"

#define TRS_COLS 8
#define TRS_THREADS 512
#define TRS_GROUP 4   // k-steps (of four columns of T) per prefetched group
#define TRS_DEPTH 1   // groups in flight ahead of the one multiplied (odd: two B buffers alternate)
#define TRS_LDT (NB + 1)
#define TRS_SMEM ((size_t)(NB * TRS_LDT + 2 * TRS_COLS * TRS_LDT + NB) * sizeof(double2))

// A read-once element of the factor: not kept in L1 (the solved rows, read by eight warps, are).
__device__ __forceinline__ double2 trs_stream(const double2 *p) {
    double2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}

// Unit lower 64-row substitution of one column by a warp: x0, x1 rows lane, lane + 32.  Rows
// take only what is above them, so an Inf or NaN stays in its column and the rows below it.
__device__ __forceinline__ void trs_lower(const double2 *T, int lane, double2 &x0, double2 &x1) {
#pragma unroll 8
    for (int k = 0; k < 32; ++k) {
        const double2 xk = shfl_c(x0, k);
        if (lane > k) cfms(x0, T[k * TRS_LDT + lane], xk);
        cfms(x1, T[k * TRS_LDT + lane + 32], xk);
    }
#pragma unroll 8
    for (int k = 32; k < NB; ++k) {
        const double2 xk = shfl_c(x1, k - 32);
        if (lane > k - 32) cfms(x1, T[k * TRS_LDT + lane + 32], xk);
    }
}

template <bool UPPER>
__global__ void __launch_bounds__(TRS_THREADS, 1)
k_trsolve_strip(int n, int nrhs, const double2 *__restrict__ LU, int64_t lda, double2 *B, int64_t ldb) {
    extern __shared__ __align__(16) unsigned char trs_smem[];
    double2 *T = reinterpret_cast<double2 *>(trs_smem);  // [column][TRS_LDT] diagonal block
    double2 *W = T + NB * TRS_LDT;                        // [strip column][TRS_LDT], and the odd groups' sums
    double2 *rd = W + 2 * TRS_COLS * TRS_LDT;                 // reciprocals of the diagonal
    const int t = threadIdx.x, warp = (t >> 5) & 7, odd = t >> 8, lane = t & 31, g = lane >> 2, q = lane & 3;
    const int c0 = blockIdx.x * TRS_COLS, nblk = (n + NB - 1) / NB;
    const double2 *bcol = B + (int64_t)min(c0 + g, nrhs - 1) * ldb;
    for (int s = 0; s < nblk; ++s) {
        const int i = UPPER ? nblk - 1 - s : s, j = i * NB, nbj = min(NB, n - j);
        for (int e = t; e < NB * NB; e += TRS_THREADS) {
            const int r = e % NB, c = e / NB;
            const bool ok = r < nbj && c < nbj && (UPPER ? r <= c : r > c);
            dm_cp16(T + c * TRS_LDT + r, ok ? (const void *)(LU + (int64_t)(j + c) * lda + j + r) : (const void *)LU, ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        // solved rows [k0, k1), oldest first: forward from row 0, backward from row n - 1 (a
        // last partial group there, its missing rows skipped; every other group is whole)
        const int k0 = UPPER ? j + nbj : 0, k1 = UPPER ? n : j;
        const int row = j + 8 * warp + g;
        const bool row_ok = row < n;
        // rows past n and columns past nrhs repeat the last one: their sums are not stored
        const double2 *ap = LU + (row_ok ? row : n - 1) + (int64_t)(k0 + q) * lda, *bp = bcol + k0 + q;
        const int ngrp = (k1 - k0 + 4 * TRS_GROUP - 1) / (4 * TRS_GROUP), mine = (ngrp + 1 - odd) / 2;
        double re[TRS_GROUP][2] = {}, im[TRS_GROUP][2] = {};
        double2 a[TRS_DEPTH + 1][TRS_GROUP], b[2][TRS_GROUP];
        auto load_a = [&](double2(&v)[TRS_GROUP], int grp) {
            if (grp >= mine) return;
            const int off = 4 * TRS_GROUP * (UPPER ? ngrp - 1 - 2 * grp - odd : 2 * grp + odd);
            const double2 *p = ap + (int64_t)off * lda;
            const bool whole = k0 + off + 4 * TRS_GROUP <= k1;
#pragma unroll
            for (int u = 0; u < TRS_GROUP; ++u) {
                if (whole || k0 + off + q + 4 * u < k1) v[u] = trs_stream(p + (int64_t)(4 * u) * lda);
                else v[u] = czero<double2>();
            }
        };
        auto load_b = [&](double2(&v)[TRS_GROUP], int grp) {
            if (grp >= mine) return;
            const int off = 4 * TRS_GROUP * (UPPER ? ngrp - 1 - 2 * grp - odd : 2 * grp + odd);
            const bool whole = k0 + off + 4 * TRS_GROUP <= k1;
#pragma unroll
            for (int u = 0; u < TRS_GROUP; ++u) {
                if (whole || k0 + off + q + 4 * u < k1) v[u] = bp[off + 4 * u];
                else v[u] = czero<double2>();
            }
        };
        // the group's k-steps side by side, each its own accumulators
        auto mma = [&](const double2(&x)[TRS_GROUP], const double2(&y)[TRS_GROUP]) {
#pragma unroll
            for (int u = 0; u < TRS_GROUP; ++u) {
                dmma(re[u][0], re[u][1], x[u].x, y[u].x);
                dmma(im[u][0], im[u][1], x[u].x, y[u].y);
            }
#pragma unroll
            for (int u = 0; u < TRS_GROUP; ++u) {
                dmma(re[u][0], re[u][1], -x[u].y, y[u].y);
                dmma(im[u][0], im[u][1], x[u].y, y[u].x);
            }
        };
#pragma unroll
        for (int v = 0; v < TRS_DEPTH; ++v) load_a(a[v], v);
        load_b(b[0], 0);
        for (int grp = 0; grp < mine; grp += TRS_DEPTH + 1) {
#pragma unroll
            for (int v = 0; v < TRS_DEPTH + 1; ++v) {
                if (grp + v >= mine) break;
                load_a(a[(v + TRS_DEPTH) % (TRS_DEPTH + 1)], grp + v + TRS_DEPTH);
                load_b(b[(v + 1) % 2], grp + v + 1);
                mma(a[v], b[v % 2]);
            }
        }
#pragma unroll
        for (int u = 1; u < TRS_GROUP; ++u)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                re[0][e] += re[u][e];
                im[0][e] += im[u][e];
            }
        // lane holds row 8 warp + g, strip columns 2 q, 2 q + 1
        if (odd) {
#pragma unroll
            for (int e = 0; e < 2; ++e)
                W[(TRS_COLS + 2 * q + e) * TRS_LDT + 8 * warp + g] = make_double2(re[0][e], im[0][e]);
        }
        __syncthreads();
        if (!odd) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int c = 2 * q + e;
                double2 v = czero<double2>();
                if (row_ok && c0 + c < nrhs) v = B[(int64_t)(c0 + c) * ldb + row];
                const double2 w = W[(TRS_COLS + c) * TRS_LDT + 8 * warp + g];
                W[c * TRS_LDT + 8 * warp + g] = make_double2(v.x - (re[0][e] + w.x), v.y - (im[0][e] + w.y));
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (UPPER && t < NB) rd[t] = t < nbj ? crecip(T[t * TRS_LDT + t]) : czero<double2>();
        if (UPPER) __syncthreads();
        // one column per warp (the first eight); rows at and past nbj hold zeros and are left alone
        if (!odd) {
            double2 x0 = W[warp * TRS_LDT + lane], x1 = W[warp * TRS_LDT + lane + 32];
            if (!UPPER) {
                trs_lower(T, lane, x0, x1);
            } else {
#pragma unroll 8
                for (int k = NB - 1; k >= 32; --k) {
                    if (lane == k - 32) x1 = cmul(x1, rd[k]);
                    const double2 xk = shfl_c(x1, k - 32);
                    if (lane < k - 32) cfms(x1, T[k * TRS_LDT + lane + 32], xk);
                    cfms(x0, T[k * TRS_LDT + lane], xk);
                }
#pragma unroll 8
                for (int k = 31; k >= 0; --k) {
                    if (lane == k) x0 = cmul(x0, rd[k]);
                    const double2 xk = shfl_c(x0, k);
                    if (lane < k) cfms(x0, T[k * TRS_LDT + lane], xk);
                }
            }
            if (c0 + warp < nrhs) {
                double2 *out = B + (int64_t)(c0 + warp) * ldb + j;
                if (lane < nbj) out[lane] = x0;
                if (lane + 32 < nbj) out[lane + 32] = x1;
            }
        }
        __syncthreads();  // X_i in place, T and W free
    }
}

// Forward elimination of the right-hand sides by panels [p0, p1) of a running partial-pivoting
// factorization (LU: the panels' columns as factored, later panels' interchanges not yet
// applied; moves_all: each panel's row moves).  A strip of eight columns per CTA as above, but
// right-looking, because the rows of L still move: per panel the row moves, the substitution,
// and W -= L X on all rows below, a warp eight rows of all 64 columns at a time.
//
// The panel chain of the factorization leaves most SMs idle; this runs in its shadow, so that of
// the forward substitution (N = 2048, 720 columns 0.98 ms, N = 1024, 361 0.28 ms) only the last
// launch is waited for.  A launch takes the panels of about TRS_FWD_ROWS rows of updates (at
// 90 strips 80 us, within the 115 us of the panel that starts with it: strips still running
// keep the next panel's 16-CTA cluster waiting, 200 us with four panels of 1900 rows a launch),
// at most TRS_FWD_PANELS.  256 threads and half the registers of an SM: the chain's short
// kernels fit beside it.  Whole solves: N = 333, 19 columns 1.16 -> 1.08 ms, N = 2048, 720
// columns 9.49 -> 8.58 ms (four panels a launch from the start: 9.05).
#define TRS_FWD_THREADS 256
#define TRS_FWD_PANELS 4
#define TRS_FWD_ROWS 1536
#define TRS_FWD_LDX (NB + 4)  // eight columns' 16-byte elements in different banks
#define TRS_FWD_SMEM ((size_t)(NB * TRS_LDT + TRS_COLS * TRS_FWD_LDX) * sizeof(double2))
__global__ void __launch_bounds__(TRS_FWD_THREADS, 2)
k_forward_strip(int n, int nrhs, const double2 *__restrict__ LU, int64_t lda, double2 *B, int64_t ldb, int p0, int p1,
                const int *__restrict__ moves_all) {
    extern __shared__ __align__(16) unsigned char trs_smem[];
    double2 *T = reinterpret_cast<double2 *>(trs_smem);
    double2 *X = T + NB * TRS_LDT;  // [strip column][TRS_FWD_LDX]
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, q = lane & 3;
    const int c0 = blockIdx.x * TRS_COLS;
    for (int p = p0; p < p1; ++p) {
        const int j = p * NB, nbj = min(NB, n - j);
        for (int e = t; e < NB * NB; e += TRS_FWD_THREADS) {
            const int r = e % NB, c = e / NB;
            const bool ok = r < nbj && c < r;
            dm_cp16(T + c * TRS_LDT + r, ok ? (const void *)(LU + (int64_t)(j + c) * lda + j + r) : (const void *)LU, ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        // row moves: every source before any destination
        const int *mv = moves_all + (size_t)p * GEPP_MOVES_STRIDE;
        const int cnt = min(mv[0], GEPP_MAX_MOVES), mc = t % TRS_COLS, mi = t / TRS_COLS;
        constexpr int per = TRS_FWD_THREADS / TRS_COLS, rounds = GEPP_MAX_MOVES / per;
        double2 *mcol = B + (int64_t)(c0 + mc) * ldb;
        double2 tmp[rounds];
#pragma unroll
        for (int u = 0; u < rounds; ++u)
            if (mi + per * u < cnt && c0 + mc < nrhs) tmp[u] = mcol[mv[1 + GEPP_MAX_MOVES + mi + per * u]];
        __syncthreads();
#pragma unroll
        for (int u = 0; u < rounds; ++u)
            if (mi + per * u < cnt && c0 + mc < nrhs) mcol[mv[1 + mi + per * u]] = tmp[u];
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        {
            double2 x0 = czero<double2>(), x1 = x0;
            double2 *col = B + (int64_t)(c0 + warp) * ldb + j;
            const bool ok = c0 + warp < nrhs;
            if (ok && lane < nbj) x0 = col[lane];
            if (ok && lane + 32 < nbj) x1 = col[lane + 32];
            trs_lower(T, lane, x0, x1);
            if (ok && lane < nbj) col[lane] = x0;
            if (ok && lane + 32 < nbj) col[lane + 32] = x1;
            X[warp * TRS_FWD_LDX + lane] = x0;
            X[warp * TRS_FWD_LDX + lane + 32] = x1;
        }
        __syncthreads();
        const int j1 = j + NB, groups = (n - j1 + 7) / 8;  // none after the last panel
        const double2 *xf = X + g * TRS_FWD_LDX + q;
        for (int rg = warp; rg < groups; rg += TRS_FWD_THREADS / 32) {
            // rows past n repeat the last one: their sums are not stored
            const int row = j1 + 8 * rg + g, rowc = min(row, n - 1);
            const double2 *ap = LU + rowc + (int64_t)(j + q) * lda;
            double2 a[2][TRS_GROUP], w[2];
            double re[TRS_GROUP][2] = {}, im[TRS_GROUP][2] = {};
#pragma unroll
            for (int u = 0; u < TRS_GROUP; ++u) a[0][u] = trs_stream(ap + (int64_t)(4 * u) * lda);
#pragma unroll
            for (int e = 0; e < 2; ++e) w[e] = B[(int64_t)min(c0 + 2 * q + e, nrhs - 1) * ldb + rowc];
#pragma unroll
            for (int v = 0; v < NB / (4 * TRS_GROUP); ++v) {
                if (v + 1 < NB / (4 * TRS_GROUP)) {
#pragma unroll
                    for (int u = 0; u < TRS_GROUP; ++u)
                        a[(v + 1) & 1][u] = trs_stream(ap + (int64_t)(4 * (TRS_GROUP * (v + 1) + u)) * lda);
                }
#pragma unroll
                for (int u = 0; u < TRS_GROUP; ++u) {
                    const double2 l = a[v & 1][u], x = xf[4 * (TRS_GROUP * v + u)];
                    dmma(re[u][0], re[u][1], l.x, x.x);
                    dmma(im[u][0], im[u][1], l.x, x.y);
                    dmma(re[u][0], re[u][1], -l.y, x.y);
                    dmma(im[u][0], im[u][1], l.y, x.x);
                }
            }
#pragma unroll
            for (int u = 1; u < TRS_GROUP; ++u)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    re[0][e] += re[u][e];
                    im[0][e] += im[u][e];
                }
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (row < n && c0 + 2 * q + e < nrhs)
                    B[(int64_t)(c0 + 2 * q + e) * ldb + row] = make_double2(w[e].x - re[0][e], w[e].y - im[0][e]);
        }
        __syncthreads();  // every row updated, T and X free
    }
}

// Partial-pivoting panel factorization on a thread-block cluster (LAPACK getf2 order, the
// reference's scipy lu_factor pivots: |re| + |im|, first row on ties).
//
// The 64-column panel rows j..n-1 are spread over the CS CTAs of one cluster, CTA c holding
// panel rows [c rpc, (c+1) rpc) in shared memory (rows past its capacity in a global
// scratch, which stays in L2).  Column step k:
//   1. every CTA reduces its best candidate for column k among its rows >= k, pushes its
//      (value, row) into every CTA's shared memory and publishes the candidate's whole row
//      (and row k, if it owns it) in a double-buffered slot, with step k - 1's rank-1
//      update (still pending on columns > k) applied on the fly;
//   2. it arrives at the cluster barrier, finishes that pending update on its own rows
//      while the other CTAs arrive, and waits;
//   3. one warp finds the winner among the pushed candidates, then reads its row and row
//      k through distributed shared memory; the owners of rows k and p swap them;
//   4. one thread per row forms l = a_rk / a_kk, updates column k + 1 at once and finds
//      the candidates of step k + 1.
// One cluster barrier per column: a slot (pushed or published) is rewritten two steps
// later, after every CTA has passed the barrier that follows its reads.  Every CTA runs the same steps, barriers
// included, whatever its rows.
//
// The panel's interchanges reach the other columns in two ways: the trailing columns take
// them before U12 is formed (k_panel_u_moves, from a list of at most 128 row moves that
// CTA 0 derives from the 64 interchanges), the factored columns on the left at the end of
// the factorization (k_laswp_left, from ipiv).
#pragma once
#include <cooperative_groups.h>

#include "lu.cuh"

namespace cg = cooperative_groups;

#define GEPP_THREADS 256
#define GEPP_LDR (NB + 1)   // padded row stride of the panel rows in shared memory
#define GEPP_MAX_MOVES (2 * NB)

template <typename C>
struct GeppPub {
    C row[NB];    // the CTA's best candidate row of this step
    C krow[NB];   // panel row k, from the CTA that owns it
    double val;   // |re| + |im| of the candidate in column k (-1: no row >= k)
    int idx;      // its panel row
    int pad;
};

// Fixed shared memory of the panel kernel (the rows follow it).
template <typename C>
__host__ __device__ constexpr size_t gepp_fixed_smem() {
    return (2 * sizeof(GeppPub<C>) + 2 * NB * sizeof(C) /* prow */ + (size_t)GEPP_THREADS / 32 * 16 /* reduce */ +
            4 * NB * sizeof(int) /* ipiv, first, slot, content */ + 2 * NB * sizeof(int) /* extras */ + 64 + 15) /
           16 * 16;
}

// Better candidate: larger |re| + |im|, then the smaller row.
__device__ __forceinline__ bool gepp_better(double v, int i, double bv, int bi) {
    return v > bv || (v == bv && i < bi);
}

// Row moves of one panel's interchanges (one warp): ipiv_s[k] is the panel row that step k
// swapped with row k (k < nbj).  Simulating the swaps on the touched rows -- the panel's
// first nbj rows and the targets below them -- gives, for each touched row, the row whose
// content ends there: moves[0] = count, then count destination rows and, GEPP_MAX_MOVES
// entries on, count source rows (absolute: + j).  Scratch (shared): first, slot (NB ints),
// content (2 NB), extra (NB).  Returns the count (every lane).
__device__ __forceinline__ int panel_moves(const int *ipiv_s, int nbj, int j, int *moves, int *first, int *slot,
                                           int *content, int *extra) {
    const int lane = threadIdx.x & 31;
    // first[k]: the first interchange with the same target row; extra targets (rows >= nbj)
    // get slots nbj, nbj + 1, ... in order of first appearance
    for (int k = lane; k < nbj; k += 32) {
        int f = k;
        for (int q = 0; q < k; ++q)
            if (ipiv_s[q] == ipiv_s[k]) { f = q; break; }
        first[k] = f;
    }
    __syncwarp();
    int base = 0;
    for (int k0 = 0; k0 < nbj; k0 += 32) {
        const int k = k0 + lane;
        const bool is_new = k < nbj && ipiv_s[k] >= nbj && first[k] == k;
        const unsigned bal = __ballot_sync(0xffffffffu, is_new);
        if (is_new) {
            const int at = base + __popc(bal & ((1u << lane) - 1u));
            slot[k] = nbj + at;
            extra[at] = ipiv_s[k];
        }
        base += __popc(bal);
    }
    __syncwarp();
    int cnt = 0;
    if (lane == 0) {
        for (int s = 0; s < nbj + base; ++s) content[s] = s < nbj ? s : extra[s - nbj];
        for (int k = 0; k < nbj; ++k) {
            const int pk_ = ipiv_s[k];
            if (pk_ == k) continue;
            const int sp = pk_ < nbj ? pk_ : slot[first[k]];
            const int t = content[k];
            content[k] = content[sp];
            content[sp] = t;
        }
        for (int s = 0; s < nbj + base; ++s) {
            const int pos = s < nbj ? s : extra[s - nbj];
            if (content[s] != pos) {
                moves[1 + cnt] = j + pos;                        // destination row
                moves[1 + GEPP_MAX_MOVES + cnt] = j + content[s];  // source row
                ++cnt;
            }
        }
        moves[0] = cnt;
    }
    return __shfl_sync(0xffffffffu, cnt, 0);
}

// Row moves of every panel of a factorization, from its ipiv (1-based, absolute): one warp
// per panel, moves of panel p at moves_all + p * GEPP_MOVES_STRIDE.
#define GEPP_MOVES_STRIDE (1 + 2 * GEPP_MAX_MOVES)
__global__ void __launch_bounds__(128) k_ipiv_moves(int n, const int *__restrict__ ipiv, int *__restrict__ moves_all) {
    __shared__ int sc[4][NB * 6];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p = blockIdx.x * 4 + warp;
    const int npan = (n + NB - 1) / NB;
    if (p >= npan) return;
    const int j = p * NB, nbj = min(NB, n - j);
    int *ip = sc[warp], *first = ip + NB, *slot = first + NB, *content = slot + NB, *extra = content + 2 * NB;
    for (int k = lane; k < nbj; k += 32) ip[k] = ipiv[j + k] - 1 - j;
    __syncwarp();
    panel_moves(ip, nbj, j, moves_all + (size_t)p * GEPP_MOVES_STRIDE, first, slot, content, extra);
}

// Applies the row moves of panels first.. npan-1 to columns of B (one CTA per column, the
// rows it can change staged in shared memory): the interchanges of getrs' right-hand
// sides (left = 0: every panel, every row) and of the factored columns left of later
// panels (left = 1: column c of panel c / NB takes the panels after it, rows from the next
// panel on).  ident (may be NULL): nothing to do when *ident is set.  Dynamic smem: n
// elements (n * sizeof(C) <= GEPP_MOVES_SMEM_MAX).
#define GEPP_MOVES_SMEM_MAX (200 * 1024)
template <typename C>
__global__ void __launch_bounds__(256)
k_apply_moves(int n, C *__restrict__ B, int64_t ldb, int col0, int left, const int *__restrict__ moves_all,
              const int *__restrict__ ident) {
    extern __shared__ __align__(16) unsigned char mv_smem[];
    C *col = reinterpret_cast<C *>(mv_smem);
    const int c = col0 + blockIdx.x;
    const int npan = (n + NB - 1) / NB;
    const int first = left ? c / NB + 1 : 0;
    if (first >= npan || (ident && *ident)) return;
    const int row0 = first * NB;
    C *b = B + (int64_t)c * ldb;
    for (int r = row0 + threadIdx.x; r < n; r += blockDim.x) col[r - row0] = b[r];
    __syncthreads();
    for (int p = first; p < npan; ++p) {
        const int *mv = moves_all + (size_t)p * GEPP_MOVES_STRIDE;
        const int cnt = min(mv[0], GEPP_MAX_MOVES);
        C v = czero<C>();
        const bool act = threadIdx.x < cnt;
        if (act) v = col[mv[1 + GEPP_MAX_MOVES + threadIdx.x] - row0];
        __syncthreads();
        if (act) col[mv[1 + threadIdx.x] - row0] = v;
        __syncthreads();
    }
    for (int r = row0 + threadIdx.x; r < n; r += blockDim.x) b[r] = col[r - row0];
}

// A CTA's candidate of one step, pushed into every CTA of the cluster.
struct GeppCand {
    double val;
    int idx;
    int pad;
};

// Cluster barrier halves: the arrive of threads whose writes other CTAs read carries release
// semantics, the others' is relaxed; the wait acquires.
__device__ __forceinline__ void gepp_arrive(bool release) {
    if (release) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    else asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void gepp_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

template <typename C>
__global__ void __launch_bounds__(GEPP_THREADS)
k_panel_gepp(int n, C *__restrict__ A, int64_t lda, int j, int nbj, int rpc, int rows_smem, C *__restrict__ gscratch,
             int *__restrict__ ipiv, int *__restrict__ info, int *__restrict__ swapped, int *__restrict__ moves,
             PanelPack pk) {
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int cs = (int)cluster.num_blocks();
    extern __shared__ __align__(16) unsigned char gepp_smem[];
    GeppPub<C> *pub = reinterpret_cast<GeppPub<C> *>(gepp_smem);
    C *prow = reinterpret_cast<C *>(pub + 2);  // [2][NB]: the pivot rows of the last two steps
    double *red_v = reinterpret_cast<double *>(prow + 2 * NB);
    int *red_i = reinterpret_cast<int *>(red_v + GEPP_THREADS / 32);
    int *ipiv_s = red_i + GEPP_THREADS / 32;
    int *first = ipiv_s + NB, *slot = first + NB, *content = slot + NB, *extra = content + 2 * NB;
    C *rows = reinterpret_cast<C *>(gepp_smem + gepp_fixed_smem<C>());
    __shared__ GeppCand cand[2][16];  // [parity][rank]: every CTA's candidate, pushed here
    __shared__ int s_p, s_zero;
    __shared__ C s_rp;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m = n - j;
    const int r0 = rank * rpc;
    const int nr = max(0, min(m - r0, rpc));
    C *gs = gscratch + (size_t)rank * (size_t)max(0, rpc - rows_smem) * NB;
    auto rowp = [&](int r) -> C * { return r < rows_smem ? rows + (size_t)r * GEPP_LDR : gs + (size_t)(r - rows_smem) * NB; };

    // load the CTA's rows (coalesced along each column)
    for (int e = tid; e < nr * NB; e += GEPP_THREADS) {
        const int c = e / nr, r = e - c * nr;
        rowp(r)[c] = c < nbj ? A[(int64_t)(j + c) * lda + j + r0 + r] : czero<C>();
    }
    __syncthreads();

    // Step k starts with column k up to date on every row g >= k and the rank-1 update of
    // step k - 1 still pending on columns > k (multipliers in column k - 1, pivot row in
    // prow[(k - 1) & 1]); it finishes it while the cluster barrier completes.
    double bv = -1.0;
    int bi = 0x7fffffff;
    for (int r = tid; r < nr; r += GEPP_THREADS) {
        const double v = (double)cabs1(rowp(r)[0]);
        if (gepp_better(v, r0 + r, bv, bi)) { bv = v; bi = r0 + r; }
    }
    for (int k = 0; k < nbj; ++k) {
        const int par = k & 1;
        const C *uprev = prow + (par ^ 1) * NB;
        // 1. the CTA's candidate for column k: warp maxima, then every thread takes the
        //    largest of the 8 (first row on ties)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_down_sync(0xffffffffu, bv, o);
            const int oi = __shfl_down_sync(0xffffffffu, bi, o);
            if (gepp_better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
        }
        if (lane == 0) { red_v[warp] = bv; red_i[warp] = bi; }
        __syncthreads();
        bv = red_v[0];
        bi = red_i[0];
#pragma unroll
        for (int w = 1; w < GEPP_THREADS / 32; ++w)
            if (gepp_better(red_v[w], red_i[w], bv, bi)) { bv = red_v[w]; bi = red_i[w]; }
        //    published with the pending update applied: its row (threads 0-63), row k if this
        //    CTA owns it (64-127); its (value, row) pushed into every CTA (warp 4)
        if (tid < 2 * NB) {
            const int c = tid & (NB - 1);
            const int src = tid < NB ? bi : k;
            const bool want = tid < NB ? bi != 0x7fffffff : (k >= r0 && k < r0 + nr);
            if (want) {
                const C *a = rowp(src - r0);
                C x = a[c];
                if (k > 0 && c > k) cfms(x, a[k - 1], uprev[c]);
                if (tid < NB) pub[par].row[c] = x;
                else pub[par].krow[c] = x;
            }
        } else if (warp == 4 && lane < cs) {
            GeppCand *dst = cluster.map_shared_rank(&cand[par][rank], lane);
            dst->val = bv;
            dst->idx = bi;
        }
        // the published rows are read before any warp applies the pending update to them
        __syncthreads();
        gepp_arrive(warp <= 4);
        // 2. the pending update of step k - 1 on the CTA's rows >= k, columns > k: two
        //    threads per row, alternate columns
        if (k > 0) {
            const int half = tid & 1;
            for (int r = tid >> 1; r < nr; r += GEPP_THREADS / 2) {
                if (r0 + r >= k) {
                    C *a = rowp(r);
                    const C l = a[k - 1];
#pragma unroll 4
                    for (int c = k + 1 + half; c < NB; c += 2) cfms(a[c], l, uprev[c]);
                }
            }
        }
        gepp_wait();
        __syncthreads();
        // 3. warp 0: the winner from the pushed candidates (local), then its row and row k
        //    through distributed shared memory; the owners of rows k and p swap them
        if (warp == 0) {
            double v = -1.0;
            int i = 0x7fffffff;
            for (int w = 0; w < cs; ++w) {
                const GeppCand cw = cand[par][w];
                if (gepp_better(cw.val, cw.idx, v, i)) { v = cw.val; i = cw.idx; }
            }
            const bool zero = !(v > 0.0);
            const int ck = k / rpc, cw = i == 0x7fffffff ? 0 : i / rpc;
            const GeppPub<C> *wp = cluster.map_shared_rank(&pub[par], cw);
            const GeppPub<C> *kp = cluster.map_shared_rank(&pub[par], ck);
            const C x0 = wp->row[lane], x1 = wp->row[lane + 32];
            const C k0 = kp->krow[lane], k1 = kp->krow[lane + 32];
            prow[par * NB + lane] = x0;
            prow[par * NB + lane + 32] = x1;
            if (lane == (k & 31)) s_rp = zero ? one_c<C>() : crecip(k < 32 ? x0 : x1);
            if (i != k && !zero) {
                if (rank == ck) {
                    C *a = rowp(k - r0);
                    a[lane] = x0;
                    a[lane + 32] = x1;
                }
                if (rank == cw) {
                    C *a = rowp(i - r0);
                    a[lane] = k0;
                    a[lane + 32] = k1;
                }
            }
            if (lane == 0) {
                s_p = i;
                s_zero = zero;
                if (rank == 0) ipiv_s[k] = zero ? k : i;
            }
        }
        __syncthreads();
        const bool zero = s_zero;
        if (zero && rank == 0 && tid == 0) atomicCAS(info, 0, j + k + 1);
        // 4. multipliers of the CTA's rows below k (LAPACK leaves a zero pivot column
        //    unscaled), column k + 1 updated at once, and the candidates of step k + 1
        const C *u = prow + par * NB;
        const C rp = s_rp;
        bv = -1.0;
        bi = 0x7fffffff;
        for (int r = tid; r < nr; r += GEPP_THREADS) {
            const int g = r0 + r;
            if (g > k) {
                C *a = rowp(r);
                const C l = zero ? a[k] : cmul(a[k], rp);
                a[k] = l;
                if (k + 1 < NB) {
                    cfms(a[k + 1], l, u[k + 1]);
                    const double v = (double)cabs1(a[k + 1]);
                    if (gepp_better(v, g, bv, bi)) { bv = v; bi = g; }
                }
            }
        }
    }
    // every CTA has finished reading every other CTA's slots before any CTA exits
    cluster.sync();

    // write the factored rows back; complex64: the trailing update's packed A operand (L21)
    for (int e = tid; e < nr * NB; e += GEPP_THREADS) {
        const int cc = e / nr, r = e - cc * nr;
        if (cc < nbj) A[(int64_t)(j + cc) * lda + j + r0 + r] = rowp(r)[cc];
    }
    if constexpr (sizeof(C) == sizeof(float2)) {
        if (pk.a_hi) {
            // L21 rows are panel rows >= nbj (= NB here); padding rows up to a_rows / 2 are zero
            const int rest = m - nbj;
            const int pad_rows = pk.a_rows / 2;
            for (int e = tid; e < rpc * NB; e += GEPP_THREADS) {
                const int cc = e / rpc, r = e - cc * rpc;
                const int mrow = r0 + r - nbj;
                if (mrow < 0 || mrow >= pad_rows) continue;
                float xr = 0.f, xi = 0.f;
                if (mrow < rest && r < nr) {
                    const float2 x = *reinterpret_cast<const float2 *>(&rowp(r)[cc]);
                    xr = x.x;
                    xi = x.y;
                }
                pack_pair(pk.a_hi, pk.a_lo, tc_tile_offset(2 * mrow, 2 * cc, pk.a_rows), xr, -xi);
                pack_pair(pk.a_hi, pk.a_lo, tc_tile_offset(2 * mrow + 1, 2 * cc, pk.a_rows), xi, xr);
            }
            // rows past the rows of every CTA (rpc * CS may not reach pad_rows): zero
            const int covered = (int)cluster.num_blocks() * rpc - nbj;
            if (rank == 0)
                for (int e = tid; e < (pad_rows - covered) * NB; e += GEPP_THREADS) {
                    const int mrow = covered + e / NB, cc = e % NB;
                    if (mrow < 0) continue;
                    pack_pair(pk.a_hi, pk.a_lo, tc_tile_offset(2 * mrow, 2 * cc, pk.a_rows), 0.f, 0.f);
                    pack_pair(pk.a_hi, pk.a_lo, tc_tile_offset(2 * mrow + 1, 2 * cc, pk.a_rows), 0.f, 0.f);
                }
        }
    }

    // CTA 0: ipiv, the swapped flag and the row moves of the panel's interchanges
    if (rank != 0) return;
    if (tid < nbj) ipiv[j + tid] = j + ipiv_s[tid] + 1;
    if (warp == 0) {
        const int cnt = panel_moves(ipiv_s, nbj, j, moves, first, slot, content, extra);
        if (lane == 0) *swapped = cnt > 0;
    }
}

// Candidate keys: the bits of |re| + |im| (a non-negative double) plus one order like the
// values; 0 marks "no candidate" (and NaN, which LAPACK's search never picks either).
__device__ __forceinline__ unsigned long long gepp_key(double v) {
    return v == v ? (unsigned long long)__double_as_longlong(v) + 1ull : 0ull;
}

// Warp maximum of the keys (every lane) and the lowest lane that holds it (-1: all zero).
__device__ __forceinline__ int gepp_warp_argmax(unsigned long long key, unsigned long long &kmax) {
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
    const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
    kmax = ((unsigned long long)mhi << 32) | mlo;
    const unsigned bal = __ballot_sync(0xffffffffu, kmax != 0ull && key == kmax);
    return bal ? __ffs(bal) - 1 : -1;
}

// L x = a (L unit lower in T, zero elsewhere) for one 64-long column vector shared by 8 lanes
// (v[i] = row 8 i + s), right-looking: an entry, once final, is broadcast to its lanes and
// subtracted from the later ones; after each block of eight the pending entries shift down a
// register (the loop body stays in the instruction cache).  Blocks [b0, b0 + 4), 8 - b0 live.
template <typename C, int B0>
__device__ __forceinline__ void umoves_blocks(C (&v)[8], C (&x)[8], const C *T, int s) {
    const int base = (int)(threadIdx.x & 31u) & ~7;
#pragma unroll 1
    for (int b = B0; b < B0 + 4; ++b) {
#pragma unroll
        for (int cc = 0; cc < 8; ++cc) {
            const C xr = shfl_c(v[0], base | cc);
            const C *col = T + (8 * b + cc) * NBP + 8 * b + s;
            if (s > cc) cfms(v[0], xr, col[0]);
#pragma unroll
            for (int i = 1; i < 8 - B0; ++i)
                if (b + i < 8) cfms(v[i], xr, col[8 * i]);
        }
#pragma unroll
        for (int i = 0; i < 7; ++i) x[i] = x[i + 1];
        x[7] = v[0];
#pragma unroll
        for (int i = 0; i + 1 < 8 - B0; ++i) v[i] = v[i + 1];
    }
}

// U12 = inv(L11) A12 of the trailing columns after the panel's row moves: 16 columns per CTA, 8
// threads a column (a panel's substitution chains on as many SMs as there are 16-column
// blocks; with 4 threads a column and 32 columns an SM the FP64 issue, not the chain, set the
// time).  Between a panel and the next on the critical chain, and all latency, so the loads
// wait on one another as little as they can: L11 comes with cp.async under the move list (one
// read, whatever its count), and the panel's rows are read straight from where the moves take
// them, together with the rows that leave for below it (each column gathers every source
// before any write).  N = 2048: complex128 13.8 -> 11.3 us a panel (11.8 with 4 threads a column),
// complex64 11.4 -> 8.9.  complex64: also writes the trailing update's packed B operand.
// Dynamic smem: NB * NBP elements (L11).
#define UMOVES_THREADS 128
#define UMOVES_COLS (UMOVES_THREADS / 8)
template <typename C>
__global__ void __launch_bounds__(UMOVES_THREADS)
k_panel_u_moves(int n, C *__restrict__ A, int64_t lda, int j, int nbj, const int *__restrict__ moves, PanelPack pk) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *T = reinterpret_cast<C *>(smem_raw);
    __shared__ int s_from[NB];                 // the source of each panel row
    __shared__ int s_dst[NB], s_src[NB];       // rows that end below the panel (at most NB)
    __shared__ int s_below;
    const int t = threadIdx.x, s = t & 7, lane_vec = t >> 3;
    for (int e = t; e < NB * NB; e += UMOVES_THREADS) {
        const int r = e % NB, c = e / NB;
        cp_async_elem(T + c * NBP + r, A + (int64_t)(j + min(c, nbj - 1)) * lda + j + min(r, nbj - 1), c < r && r < nbj);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    static_assert(UMOVES_THREADS == GEPP_MAX_MOVES, "one move a thread");
    const int cnt = min(moves[0], GEPP_MAX_MOVES), dst = moves[1 + t], src = moves[1 + GEPP_MAX_MOVES + t];
    if (t < NB) s_from[t] = j + t;
    if (t == 0) s_below = 0;
    __syncthreads();
    if (t < cnt) {
        if (dst < j + nbj) s_from[dst - j] = src;
        else {
            const int at = atomicAdd(&s_below, 1);
            if (at < NB) {
                s_dst[at] = dst;
                s_src[at] = src;
            }
        }
    }
    __syncthreads();
    const int below = min(s_below, NB);
    const int col = j + nbj + UMOVES_COLS * blockIdx.x + lane_vec;
    const bool ok = col < n;
    C *a = A + (int64_t)col * lda;
    C v[8], x[8], tmp[NB / 8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = 8 * i + s;
        v[i] = (ok && r < nbj) ? a[s_from[r]] : czero<C>();
    }
#pragma unroll
    for (int q = 0; q < NB / 8; ++q)
        if (ok && 8 * q + s < below) tmp[q] = a[s_src[8 * q + s]];
    // a column's 8 threads (one warp) have read all they need; the warp barrier stays outside
    // the per-column condition, which differs between the lanes of a warp at the matrix edge
    __syncwarp();
#pragma unroll
    for (int q = 0; q < NB / 8; ++q)
        if (ok && 8 * q + s < below) a[s_dst[8 * q + s]] = tmp[q];
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = czero<C>();
    umoves_blocks<C, 0>(v, x, T, s);
    umoves_blocks<C, 4>(v, x, T, s);
    if (ok) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = 8 * i + s;
            if (r < nbj) A[(int64_t)col * lda + j + r] = x[i];
        }
    }
    if constexpr (sizeof(C) == sizeof(float2)) {
        if (pk.b_hi) {
            const int nb_row = UMOVES_COLS * blockIdx.x + lane_vec;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = 8 * i + s;
                pack_pair(pk.b_hi, pk.b_lo, tc_tile_offset(nb_row, 2 * r, pk.b_rows), ok ? (float)x[i].x : 0.f,
                          ok ? (float)x[i].y : 0.f);
            }
        }
    }
}

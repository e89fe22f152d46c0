// Partial-pivoting panel factorization on a thread-block cluster, rows in registers.
//
// LAPACK getf2's pivots (|re| + |im|, first position on ties), one exchange between the
// CTAs per column.  The work is small (0.3 TFLOP/s); what bounds it is the chain of one
// column: the best row of the warp, of the CTA and of the cluster, the reciprocal, the next
// column.  On this GPU a cluster barrier takes 410-445 cycles, a distributed shared-memory
// load 275, a CTA barrier 27, a warp reduction 23 and an FP64 operation 8, so the chain
// holds one cluster barrier and no remote load:
//   * rows never move: each row stays in the registers of its two threads (thread half h
//     holding columns h, h + 2, ...) with its current position, so an interchange is two
//     position updates; the rows are written to their final places at the end, and the
//     panel's row moves are the rows whose position changed;
//   * a CTA's candidate is pushed with its elements in columns K (the pivot) and K + 1,
//     which is all the other rows need to form their multipliers and column K + 1, the next
//     step's candidates;
//   * the rest of the pivot row is fetched through distributed shared memory by a helper
//     warp that holds no rows; it is first used in the shadow of the next step's barrier,
//     where step K - 1's rank-1 update of the columns > K runs;
//   * the reciprocals of all candidates are formed beside the search for the winner, one
//     per lane;
//   * complex64 keys are one word; complex128 keys are compared by their high words, and
//     only where those tie by the low words and positions.
// After each pair of columns the row registers shift down one, so register q holds column
// 2 (q + t) + h at pair t and every register index is a compile-time constant; finished
// columns retire to shared memory.  The loop runs in four phases of eight pairs keeping 32,
// 24, 16 and 8 registers, from the instruction cache.
// Column step K (owner half H = K & 1, its value in register 0, up to date; columns > K
// lack step K - 1's update):
//   1. the warp's and the CTA's best alive row, published as it stands; its header pushed
//      into every CTA of the cluster;
//   2. the cluster barrier; meanwhile, with the helper's pivot row of step K - 1 in place,
//      that step's update of the columns > K;
//   3. every warp: the winner among the headers (its column K + 1 completed); positions,
//      multipliers, column K retired, column K + 1 updated.  Helper: the winner's row.
// Double-buffered slots are rewritten two steps later, after every CTA has passed the
// cluster barrier that follows their last reads.
#pragma once
#include "pivot.cuh"

// Threads of the row warps: two per row.  Complex128 rows fill the register file at 128 rows
// a CTA; complex64 rows allow 256 (panels above 16 x 128 rows).
#define GEPPL_THREADS 256
#define GEPPL_THREADS_WIDE 512
#define GEPPL_HELPER 32

// Ordered keys of |re| + |im|: the value's bits plus one, 0 for none (and NaN, which LAPACK's
// search never picks either).
template <typename C>
struct GeppLKey;
template <>
struct GeppLKey<float2> {
    using type = unsigned;
    __device__ static type of(float2 a) {
        const float v = cabs1(a);
        return v == v ? __float_as_uint(v) + 1u : 0u;
    }
};
template <>
struct GeppLKey<double2> {
    using type = unsigned long long;
    __device__ static type of(double2 a) { return gepp_key(cabs1(a)); }
};

template <typename C>
struct __align__(16) GeppLHead {
    C piv;                   // the candidate's element in the step's column
    C next;                  // and in the next one, the previous step's update pending
    C lp;                    // its multiplier of the previous step
    unsigned long long key;  // 0: no candidate, 1: the value 0
    int pos;                 // its current position in the panel
    int pad;
};

template <typename C, int THREADS>
struct GeppLShared {
    GeppLHead<C> head[2][16];
    C pub[2][2 * NB];  // [parity]: the CTA's best row by absolute column
    C u[2][2 * NB];    // [parity]: the step's pivot row, columns > K (upper half zero)
    C zeros[2 * NB];
    typename GeppLKey<C>::type wkey[2][THREADS / 32];
    int wpos[2][THREADS / 32], wslot[2][THREADS / 32];
    int ipiv[NB];
    int moved;
};

struct GeppLCtx {
    int tid, lane, warp, half, slot, rank, cs, nbj, j;
    int *info;
};

template <typename C>
struct GeppLRow {
    C a[NB / 2];
    C lp;  // multiplier of the previous step, still to be applied to columns > K
    int pos;
    bool alive, valid;
};

// The lane with the largest key, then the lowest position (-1 when every key is 0), the same
// in every lane.  One reduction and one vote unless high words tie.
__device__ __forceinline__ int geppl_warp_best(unsigned long long key, int pos) {
    const unsigned hi = (unsigned)(key >> 32);
    const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
    bool top = key != 0ull && hi == mhi;
    unsigned bal = __ballot_sync(0xffffffffu, top);
    if (bal & (bal - 1)) {
        const unsigned lo = (unsigned)key;
        const unsigned mlo = __reduce_max_sync(0xffffffffu, top ? lo : 0u);
        top = top && lo == mlo;
        const unsigned pmin = __reduce_min_sync(0xffffffffu, top ? (unsigned)pos : 0xffffffffu);
        bal = __ballot_sync(0xffffffffu, top && (unsigned)pos == pmin);
    }
    return bal ? __ffs(bal) - 1 : -1;
}

__device__ __forceinline__ int geppl_warp_best(unsigned key, int pos) {
    const unsigned mk = __reduce_max_sync(0xffffffffu, key);
    const bool top = key != 0u && key == mk;
    unsigned bal = __ballot_sync(0xffffffffu, top);
    if (bal & (bal - 1)) {
        const unsigned pmin = __reduce_min_sync(0xffffffffu, top ? (unsigned)pos : 0xffffffffu);
        bal = __ballot_sync(0xffffffffu, top && (unsigned)pos == pmin);
    }
    return bal ? __ffs(bal) - 1 : -1;
}

// 1 / b with the components scaled by a power of two first (exact; no over- or underflow of
// |b|^2), one Newton reciprocal on the chain of every column.
__device__ __forceinline__ double2 geppl_recip(double2 b) {
    const int ex = max(__double2hiint(b.x) & 0x7ff00000, __double2hiint(b.y) & 0x7ff00000);
    // 2^-e of the larger component, kept normal at both ends of the range
    const double s = __hiloint2double(min(max(0x7fe00000 - ex, 0x00100000), 0x7fd00000), 0);
    const double br = b.x * s, bi = b.y * s;
    const double d = rcp_nr(fma(br, br, bi * bi)) * s;
    return make_double2(br * d, -bi * d);
}
__device__ __forceinline__ float2 geppl_recip(float2 b) { return crecip(b); }

template <int COUNT>
__device__ __forceinline__ void geppl_bar_sync(int id) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(COUNT) : "memory");
}
template <int COUNT>
__device__ __forceinline__ void geppl_bar_arrive(int id) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(COUNT) : "memory");
}

// The helper warp's column step: waits for the cluster barrier, then the winner's row,
// columns > K, with its pending update, into sh.u[H].  It may run one step ahead of a row
// warp still waiting for the row (the row warps arrive at the cluster barrier first), so the
// named barrier that announces the row alternates with the step's parity.
template <typename C, int H, int THREADS, bool SOLO>
__device__ __forceinline__ void geppl_helper(GeppLShared<C, THREADS> &sh, const GeppLCtx &cx, int K) {
    if (K >= cx.nbj) return;
    cg::cluster_group cluster = cg::this_cluster();
    if constexpr (SOLO) {
        geppl_bar_sync<THREADS + GEPPL_HELPER>(3);
    } else {
        gepp_arrive(false);
        gepp_wait();
    }
    if (K + 1 >= cx.nbj) return;
    unsigned long long k1 = 0ull;
    int p1 = 0x7fffffff;
    if (cx.lane < cx.cs) {
        k1 = sh.head[H][cx.lane].key;
        p1 = sh.head[H][cx.lane].pos;
    }
    const int wr = geppl_warp_best(k1, p1);
    const C *uprev = sh.u[H ^ 1];
    const int c0 = cx.lane, c1 = cx.lane + 32;
    C x0 = czero<C>(), x1 = czero<C>();
    if (wr >= 0) {
        const C *wrow = SOLO ? &sh.pub[H][0] : cluster.map_shared_rank(&sh.pub[H][0], wr);
        const C wlp = sh.head[H][wr].lp;
        if (c0 > K) x0 = wrow[c0];
        if (c1 > K) x1 = wrow[c1];
        if (K > 0) {
            if (c0 > K) cfms(x0, wlp, uprev[c0]);
            if (c1 > K) cfms(x1, wlp, uprev[c1]);
        }
    }
    sh.u[H][c0] = x0;
    sh.u[H][c1] = x1;
    __syncwarp();
    geppl_bar_arrive<THREADS + GEPPL_HELPER>(2 + 2 * H);
}

template <typename C, int H, int LIVE, int THREADS, bool SOLO>
__device__ __forceinline__ void geppl_col(GeppLRow<C> &st, GeppLShared<C, THREADS> &sh, C *__restrict__ retired,
                                          const GeppLCtx &cx, int t) {
    constexpr int WARPS = THREADS / 32, ROWS = THREADS / 2;
    const int K = 2 * t + H;
    if (K >= cx.nbj) return;
    cg::cluster_group cluster = cg::this_cluster();
    const C *uprev = sh.u[H ^ 1];

    // 1. the warp's best alive row for column K, then the CTA's
    using Key = typename GeppLKey<C>::type;
    Key key = 0;
    if (cx.half == H && st.alive) key = GeppLKey<C>::of(st.a[0]);
    const int wl = geppl_warp_best(key, st.pos);
    if (cx.lane == (wl < 0 ? 0 : wl)) {
        sh.wkey[H][cx.warp] = wl < 0 ? 0 : key;
        sh.wpos[H][cx.warp] = st.pos;
        sh.wslot[H][cx.warp] = cx.slot;
    }
    geppl_bar_sync<THREADS>(1);
    Key k8 = 0;
    int p8 = 0x7fffffff, s8 = 0;
    if (cx.lane < WARPS) {
        k8 = sh.wkey[H][cx.lane];
        p8 = sh.wpos[H][cx.lane];
        s8 = sh.wslot[H][cx.lane];
    }
    const int cw = geppl_warp_best(k8, p8);
    const int cslot = cw < 0 ? -1 : __shfl_sync(0xffffffffu, s8, cw);
    // its row published as it stands and its header pushed into every CTA by its warp (warp 0
    // pushes "no candidate" when the CTA has none)
    const int ow = cslot < 0 ? 0 : (2 * cslot) >> 5;
    if (cx.warp == ow) {
        if (cx.slot == cslot) {
#pragma unroll
            for (int q = 0; q < LIVE; ++q) sh.pub[H][2 * (q + t) + cx.half] = st.a[q];
        }
        const int l0 = cslot < 0 ? 0 : (2 * cslot) & 31;
        GeppLHead<C> hd;
        hd.piv = shfl_c(st.a[0], l0 + H);
        hd.next = H == 0 ? shfl_c(st.a[0], l0 + 1) : shfl_c(st.a[1], l0);
        hd.lp = shfl_c(st.lp, l0);
        hd.key = cw < 0 ? 0ull : (unsigned long long)__shfl_sync(0xffffffffu, k8, cw);
        hd.pos = __shfl_sync(0xffffffffu, p8, cw < 0 ? 0 : cw);
        hd.pad = 0;
        if (SOLO) {
            if (cx.lane == 0) sh.head[H][0] = hd;
        } else if (cx.lane < cx.cs) {
            *cluster.map_shared_rank(&sh.head[H][cx.rank], cx.lane) = hd;
        }
        __syncwarp();
    }
    if constexpr (!SOLO) gepp_arrive(cx.warp == ow);

    // 2. step K - 1's update of the columns > K while the other CTAs arrive
    if (K > 0) {
        geppl_bar_sync<THREADS + GEPPL_HELPER>(2 + 2 * (H ^ 1));
        // finished rows (multiplier 0) take a zero row instead of a branch around the updates
        // (the branch doubles the row registers)
        const C *uu = st.alive ? uprev : sh.zeros;
        if (H == 0 && cx.half == 1) cfms(st.a[0], st.lp, uu[2 * t + 1]);
#pragma unroll
        for (int q = 1; q < LIVE; ++q) cfms(st.a[q], st.lp, uu[2 * (q + t) + cx.half]);
    }
    __syncwarp();
    if constexpr (SOLO) geppl_bar_sync<THREADS + GEPPL_HELPER>(3);
    else gepp_wait();

    // 3. the winner (largest key, then lowest position); every candidate's reciprocal and
    //    column K + 1 meanwhile
    bool zero;
    int wp;
    C rp, un;
    {
        const GeppLHead<C> &hd = sh.head[H][cx.lane < cx.cs ? cx.lane : 0];
        const unsigned long long k1 = hd.key;
        const int p1 = hd.pos;
        C nx = hd.next;
        if (K > 0) cfms(nx, hd.lp, uprev[K + 1]);
        const C rpl = geppl_recip(hd.piv);
        if constexpr (SOLO) {
            zero = k1 <= 1ull;
            wp = k1 == 0ull ? K : p1;
            rp = rpl;
            un = k1 == 0ull ? czero<C>() : nx;
        } else {
            const int wr = geppl_warp_best(cx.lane < cx.cs ? k1 : 0ull, p1), src = wr < 0 ? 0 : wr;
            zero = __shfl_sync(0xffffffffu, k1, src) <= 1ull;  // no candidate, or 0: no elimination
            wp = wr < 0 ? K : __shfl_sync(0xffffffffu, p1, src);
            rp = shfl_c(rpl, src);
            un = wr < 0 ? czero<C>() : shfl_c(nx, src);
        }
    }
    if (cx.tid == 0 && cx.rank == 0) {
        sh.ipiv[K] = wp;
        if (zero) atomicCAS(cx.info, 0, cx.j + K + 1);
    }
    if (st.alive) {
        if (st.pos == wp) {
            st.alive = false;  // the pivot row: position K, its values final
            st.pos = K;
        } else if (st.pos == K) {
            st.pos = wp;
        }
    }
    C l = czero<C>();
    if (cx.half == H) l = zero ? st.a[0] : cmul(st.a[0], rp);
    const C lo = shfl_xor_c(l, 1);
    if (cx.half != H) l = lo;
    if (cx.half == H) retired[K * ROWS + cx.slot] = st.alive ? l : st.a[0];
    if (st.alive) {
        if (H == 0 && cx.half == 1) cfms(st.a[0], l, un);
        if (H == 1 && cx.half == 0) cfms(st.a[1], l, un);
        st.lp = l;
    } else {
        st.lp = czero<C>();
    }
}

template <typename C, int LIVE, int THREADS, bool SOLO>
__device__ __forceinline__ void geppl_phase(GeppLRow<C> &st, GeppLShared<C, THREADS> &sh, C *__restrict__ retired,
                                            const GeppLCtx &cx, int t0) {
#pragma unroll 1
    for (int t = t0; t < t0 + 8; ++t) {
        if (2 * t >= cx.nbj) return;  // the same in every thread
        geppl_col<C, 0, LIVE, THREADS, SOLO>(st, sh, retired, cx, t);
        geppl_col<C, 1, LIVE, THREADS, SOLO>(st, sh, retired, cx, t);
#pragma unroll
        for (int q = 0; q + 1 < LIVE; ++q) st.a[q] = st.a[q + 1];
        st.a[LIVE - 1] = czero<C>();
    }
}

// The panel (j, nbj) of A, rows j..n-1, on a cluster of gridDim.x CTAs (SOLO: one CTA, no
// cluster barriers), CTA c holding panel rows [c rpc, (c + 1) rpc) (rpc <= THREADS / 2).
// Dynamic smem: NB * THREADS / 2 elements (the retired columns, column-major by row slot).
// Outputs: the factored panel in place, ipiv (1-based, absolute), the first zero pivot in
// *info, *swapped, the panel's row moves (moves[0] = count, then destinations and,
// GEPP_MAX_MOVES entries on, sources, absolute rows in no particular order) and (complex64,
// pk.a_hi) the trailing update's packed L21 operand.
template <typename C, int THREADS, bool SOLO>
__global__ void __launch_bounds__(THREADS + GEPPL_HELPER, 1)
k_panel_gepp_loop(int n, C *__restrict__ A, int64_t lda, int j, int nbj, int rpc, int *__restrict__ ipiv,
                  int *__restrict__ info, int *__restrict__ swapped, int *__restrict__ moves, PanelPack pk) {
    constexpr int ROWS = THREADS / 2;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ GeppLShared<C, THREADS> sh;
    extern __shared__ __align__(16) unsigned char geppl_smem[];
    C *retired = reinterpret_cast<C *>(geppl_smem);
    GeppLCtx cx;
    cx.tid = threadIdx.x;
    cx.lane = cx.tid & 31;
    cx.warp = cx.tid >> 5;
    cx.half = cx.tid & 1;
    cx.slot = cx.tid >> 1;
    cx.rank = SOLO ? 0 : (int)cluster.block_rank();
    cx.cs = SOLO ? 1 : (int)cluster.num_blocks();
    cx.nbj = nbj;
    cx.j = j;
    cx.info = info;
    const int m = n - j;
    const bool helper = cx.tid >= THREADS;
    const int first = cx.rank * rpc + cx.slot;  // the row's place before the interchanges
    GeppLRow<C> st;
    st.pos = first;
    st.valid = !helper && cx.slot < rpc && st.pos < m;
    st.alive = st.valid;
    st.lp = czero<C>();
    if (!helper) {
#pragma unroll
        for (int q = 0; q < NB / 2; ++q) {
            const int c = 2 * q + cx.half;
            st.a[q] = (st.valid && c < nbj) ? A[(int64_t)(j + c) * lda + j + st.pos] : czero<C>();
        }
    }
    for (int e = cx.tid; e < 3 * 2 * NB; e += THREADS + GEPPL_HELPER)
        (e < 4 * NB ? &sh.u[0][0] : sh.zeros - 4 * NB)[e] = czero<C>();
    if (cx.tid == 0) sh.moved = 0;
    // every CTA's slots initialised before any CTA pushes into them
    if (SOLO) __syncthreads();
    else cluster.sync();
    if (helper) {
        for (int K = 0; K < nbj; K += 2) {
            geppl_helper<C, 0, THREADS, SOLO>(sh, cx, K);
            geppl_helper<C, 1, THREADS, SOLO>(sh, cx, K + 1);
        }
    } else {
        geppl_phase<C, 32, THREADS, SOLO>(st, sh, retired, cx, 0);
        geppl_phase<C, 24, THREADS, SOLO>(st, sh, retired, cx, 8);
        geppl_phase<C, 16, THREADS, SOLO>(st, sh, retired, cx, 16);
        geppl_phase<C, 8, THREADS, SOLO>(st, sh, retired, cx, 24);
        // the row moves: every row that changed its place, counted in CTA 0
        if (st.valid && cx.half == 0 && st.pos != first) {
            const int at = atomicAdd(SOLO ? &sh.moved : cluster.map_shared_rank(&sh.moved, 0), 1);
            if (at < GEPP_MAX_MOVES) {
                moves[1 + at] = j + st.pos;
                moves[1 + GEPP_MAX_MOVES + at] = j + first;
            }
        }
    }
    // every CTA has finished reading every other CTA's slots before any CTA exits; the rows'
    // final places may be in other CTAs' ranges, whose rows were all read at the start
    if (SOLO) __syncthreads();
    else cluster.sync();

    const int rest = m - nbj;
    if (st.valid) {
        const int d = st.pos;
        for (int c = cx.half; c < nbj; c += 2) A[(int64_t)(j + c) * lda + j + d] = retired[c * ROWS + cx.slot];
        if constexpr (sizeof(C) == sizeof(float2)) {
            if (pk.a_hi && d >= nbj) {
                const int mrow = d - nbj;
                for (int c = cx.half; c < NB; c += 2) {
                    float xr = 0.f, xi = 0.f;
                    if (c < nbj) {
                        const float2 x = *reinterpret_cast<const float2 *>(&retired[c * ROWS + cx.slot]);
                        xr = x.x;
                        xi = x.y;
                    }
                    pack_pair(pk.a_hi, pk.a_lo, tc_tile_offset(2 * mrow, 2 * c, pk.a_rows), xr, -xi);
                    pack_pair(pk.a_hi, pk.a_lo, tc_tile_offset(2 * mrow + 1, 2 * c, pk.a_rows), xi, xr);
                }
            }
        }
    }
    if (cx.rank != 0) return;
    if constexpr (sizeof(C) == sizeof(float2)) {
        if (pk.a_hi) {
            // padding rows of the packed operand past the panel's rows: zero
            const int pad_rows = pk.a_rows / 2;
            for (int e = cx.tid; e < (pad_rows - rest) * NB; e += THREADS + GEPPL_HELPER) {
                const int mr = rest + e / NB, cc = e % NB;
                pack_pair(pk.a_hi, pk.a_lo, tc_tile_offset(2 * mr, 2 * cc, pk.a_rows), 0.f, 0.f);
                pack_pair(pk.a_hi, pk.a_lo, tc_tile_offset(2 * mr + 1, 2 * cc, pk.a_rows), 0.f, 0.f);
            }
        }
    }
    // CTA 0: ipiv, the swapped flag and the number of row moves
    if (cx.tid < nbj) ipiv[j + cx.tid] = j + sh.ipiv[cx.tid] + 1;
    if (cx.tid == 0) {
        moves[0] = sh.moved;
        *swapped = sh.moved > 0;
    }
}

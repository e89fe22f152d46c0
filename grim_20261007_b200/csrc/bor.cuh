// Body-of-revolution PEC EFIE / MFIE / CFIE, per azimuthal mode.
//
// Stage 1  element-pair moments, mode-independent, for n = 0..mmax+1:
//   EFIE, from the modal Green's function G_n = int_{-pi}^{pi} e^{-jkR}/(4 pi R) cos(n xi) dxi:
//     A_ac  = sum T_a T_c rho rho' w w' G_n      DD_ac = sum D_a D_c w w' G_n
//     DT_ac = sum D_a T_c w w' G_n               TD_ac = sum T_a D_c w w' G_n
//     TT_ac = sum T_a T_c w w' G_n               (a, c in {0, 1}: the element's two tents)
//   MFIE (optional), from the four modal brackets K^n_uv = int F_uv(xi) e^{-j n xi} dxi
//   (uv = tt, tf, ft, ff; tt/ff even in xi, tf/ft odd):
//     B_uv,ac = sum T_a T_c rho rho' w w' K^n_uv
//   Layouts: mom[((e * ne + f) * (mmax + 2) + n) * 20 + slot],
//            momk[((e * ne + f) * (mmax + 2) + n) * 16 + 4 uv + 2 a + c], complex128.
//   The element pairs follow the reference's routing (bor/solver.py:1520-1580): far pairs
//   take 3 x 3 Gauss points and the uniform trapezoid rule in xi (k_bor_far, one CTA per
//   pair, three warps of three point pairs); near pairs take the host's point list -- graded cells for
//   self / adjacent pairs (bor/solver.py:718-806), a 12 x 12 Gauss rule for the others (:843)
//   -- and a composite rule on xi in [0, pi] using each integrand's parity (k_bor_near over
//   work items of at most BOR_NEAR_CHUNK point pairs, one warp per point pair, then
//   k_bor_near_reduce in a fixed order).
//
// Both kernels are bound by the FP64 pipe: per sample about 70 operations for the kernel
// values and, per order n, ten sums (G and the even brackets against cos n xi, the odd ones
// against sin n xi, re and im) plus four operations to turn e^{j n xi}.  A lane keeps the sums
// of MB orders, so that each value it reads from shared memory feeds MB of them (one order
// per thread: five 16-byte loads per ten sums, shared-memory bound at 32 % of the FP64 pipe).
// The far rule's samples are folded twice (xi -> -xi by parity in xi, xi -> pi - xi by parity
// in n), which leaves a quarter of the sums and half of the kernel values.  400-segment ogive,
// 42 orders, CFIE: far 30.9 -> 13.2 ms, near 41.4 -> 13.4 ms (near: 48 % of the FP64 pipe).
// Stage 2  k_bor_assemble: the reduced mode-m matrix alpha C EFIE + (1 - alpha) eta0
//   ((1/2) M - K), C = j k eta 2 pi, from the moments of the <= 4 element pairs touching
//   each node pair, with the pole treatment (inactive pole phi components, |m| = 1 pole t
//   component tied to phi by j m sign(t_rho)).
// Stage 3  k_bor_excitation: reduced right-hand sides alpha <W, E_inc> + (1 - alpha) eta0
//   <W, n x H_inc> (VV, HH per aspect) or far-field weights, with the phi integrals in
//   closed form through J_m (CUDA's jn).
// Reference: bor/solver.py:1769-1827 (assemble_mode), :1962 (assemble_mfie_mode),
// :2048 (rhs_mfie_mode), :2369-2440 (pole reduction), :2558-2608 (rhs_vv_hh_batch /
// farfield_vv_hh_batch), :4285-4301 (CFIE), bor/kernels.py:896,996 (MFIE brackets).
#pragma once
#include "common.cuh"
#include "hankel64.cuh"

#define BOR_FAR_ORDER 3
#define BOR_MAX_MODES 128
#define BOR_MAX_NXI 8192
#define BOR_SLOTS 20
#define BOR_KSLOTS 16
#define BOR_ALL_SLOTS (BOR_SLOTS + BOR_KSLOTS)
#define BOR_CHUNK 32        // samples a warp stages per pass (one per lane)
#define BOR_FAR_WARPS 3        // warps of a far CTA, three of the nine point pairs each
#define BOR_FAR_PAIRS (BOR_FAR_ORDER * BOR_FAR_ORDER)
#define BOR_NEAR_WARPS 8
#define BOR_NEAR_CHUNK 64   // point pairs per near work item
#define BOR_XI_CORE 20      // Gauss points of the near rule's sinh core
#define BOR_XI_PANEL 16     // Gauss points per doubling panel of the near rule
#define BOR_XI_WIDE 32      // Gauss points per panel of its uniform part

struct BorPt {
    double rho, z, w, T0, T1, D0, D1, tr, tz;
};

__device__ __forceinline__ BorPt bor_point(const double *nodes, int e, double s, double ws) {
    const double r0 = nodes[2 * e], z0 = nodes[2 * e + 1], r1 = nodes[2 * e + 2], z1 = nodes[2 * e + 3];
    const double dr = r1 - r0, dz = z1 - z0, L = sqrt(dr * dr + dz * dz);
    const double trho = dr / L;
    BorPt p;
    p.rho = r0 + s * dr;
    p.z = z0 + s * dz;
    p.w = ws * L;
    p.T0 = 1.0 - s;
    p.T1 = s;
    p.D0 = p.rho * (-1.0 / L) + p.T0 * trho;
    p.D1 = p.rho * (1.0 / L) + p.T1 * trho;
    p.tr = trho;
    p.tz = dz / L;
    return p;
}

// Far-pair xi sample count: a multiple of 32, of which the double fold needs four (xi = pi/2 is a
// sample and its own partner).
__device__ __forceinline__ int bor_nxi(double k, double rp, double rq, double r0, int mmax) {
    const double c = sqrt(rp * rq);
    const double v = 1.5 * (2.0 * k * c + mmax + 2) + 40.0 * c / fmax(r0, 1e-300) + 16.0;
    int n = 32 * (int)ceil(v / 32.0);
    return n > BOR_MAX_NXI ? BOR_MAX_NXI : n;
}

// Gauss-Legendre nodes/weights (orders 1..32) from the 2-D fill's constant tables.
__device__ __forceinline__ void gl_node(int q, int i, double &x, double &w) {
    x = c_gl_x[q * (q - 1) / 2 + i];
    w = c_gl_w[q * (q - 1) / 2 + i];
}

// Geometry of one point pair shared by every xi sample; the MFIE brackets as functions of
// h = 1 - cos xi and sin xi: tt = tt0 + h tt1, tf = tf1 sin xi, ft = ft1 sin xi, ff = ff0 + h ff1
// (cancellation-free forms).
struct BorPair {
    double k, d2, rr2;  // rr2 = 2 rho rho'
    double tt0, tt1, tf1, ft1, ff0, ff1;
};

__device__ __forceinline__ BorPair bor_pair(double k, const BorPt &p, const BorPt &q) {
    BorPair s;
    s.k = k;
    const double dr = p.rho - q.rho, dz = p.z - q.z;
    s.d2 = dr * dr + dz * dz;
    s.rr2 = 2.0 * p.rho * q.rho;
    const double X = p.tr * q.tz - p.tz * q.tr, D = p.tr * q.tr + p.tz * q.tz;
    const double A = p.tr * dr + p.tz * dz, N = -p.tz * dr + p.tr * dz;
    s.tt0 = A * X - D * N;
    s.tt1 = A * p.tz * q.tr + p.tr * q.rho * X + D * p.tz * q.rho + p.tr * q.tr * N;
    s.tf1 = -dz * (p.tr * p.tr + p.tz * p.tz);
    s.ft1 = q.rho * X + q.tr * N;
    s.ff0 = -N;
    s.ff1 = N - p.tz * q.rho;
    return s;
}

// One xi sample times weight wt: the Green's function g and (MFIE) the four brackets
// -p(R) [tt, tf, ft, ff], from sin(xi/2) and sin xi.  1/R from the hardware estimate and a
// third-order correction, R corrected to half an ulp.
template <bool MFIE>
__device__ __forceinline__ void bor_sample(const BorPair &s, double shalf, double sx, double wt, double2 &g,
                                           double2 (&F)[4]) {
    const double h = 2.0 * shalf * shalf;
    const double R2 = fma(s.rr2, h, s.d2);
    double ir;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(ir) : "d"(R2));
    const double e = fma(-R2 * ir, ir, 1.0);
    ir = fma(ir * e, fma(e, 0.375, 0.5), ir);
    double R = R2 * ir;
    R = fma(0.5 * ir, fma(-R, R, R2), R);
    const double kr = s.k * R;
    double sk, ck;
    gh_sincos(kr, sk, ck);
    const double a = wt * (1.0 / (4.0 * GRIM_PI)) * ir;
    g = make_double2(a * ck, -a * sk);
    if constexpr (MFIE) {
        const double pre = a * (ir * ir);
        // -(1 + j kR) e^{-jkR} / (4 pi R^3) times the weight
        const double pr = -pre * fma(kr, sk, ck), pi = pre * fma(-kr, ck, sk);
        const double tt = fma(h, s.tt1, s.tt0), tf = s.tf1 * sx, ft = s.ft1 * sx, ff = fma(h, s.ff1, s.ff0);
        F[0] = make_double2(pr * tt, pi * tt);
        F[1] = make_double2(pr * tf, pi * tf);
        F[2] = make_double2(pr * ft, pi * ft);
        F[3] = make_double2(pr * ff, pi * ff);
    }
}

// e^{2 pi j i / N}, 0 <= i < N: the quadrant exactly, then the polynomials.  One copy: k_bor_far
// waited for instructions a third of the time with it (and two kernel samples) inlined.
__device__ __noinline__ double2 bor_unit(int i, int N) {
    const int q = (4 * i + (N >> 1)) / N, rem = 4 * i - q * N;
    double sn, cs;
    gh_sincos_quadrant(rem * (0.5 * GRIM_PI / N), q, sn, cs);
    return make_double2(cs, sn);
}

// The 36 per-point-pair factors multiplying G_n (slots 0..19) or K^n_uv (slots 20..35).
__device__ __forceinline__ double bor_factor(const BorPt &p, const BorPt &q, int slot) {
    const int ac = slot & 3, a = ac >> 1, c = ac & 1;
    const double Ta = a ? p.T1 : p.T0, Tc = c ? q.T1 : q.T0;
    const double Da = a ? p.D1 : p.D0, Dc = c ? q.D1 : q.D0;
    const double ww = p.w * q.w;
    if (slot >= BOR_SLOTS) return Ta * Tc * (p.rho * q.rho * ww);
    switch (slot >> 2) {
    case 0: return Ta * Tc * (p.rho * q.rho * ww);
    case 1: return Da * Dc * ww;
    case 2: return Da * Tc * ww;
    case 3: return Ta * Dc * ww;
    default: return Ta * Tc * ww;
    }
}

// Lanes of a warp over the orders n < nm: blocks of MB orders, G = 32 / blocks lanes sharing a
// block (each every G-th sample).
__host__ __device__ constexpr int bor_far_blocks(int nm, int mb) { return 2 * (((nm + 1) / 2 + mb - 1) / mb); }
__host__ __device__ constexpr int bor_near_blocks(int nm, int mb) { return (nm + mb - 1) / mb; }
// Orders per lane: three (two CTAs of registers an SM), four where three need over 32 lanes.
__host__ __device__ constexpr int bor_mb(int nm) {
    return bor_far_blocks(nm, 3) <= 32 && bor_near_blocks(nm, 3) <= 32 ? 3 : 4;
}

// The lanes' sums over the groups g = 1.. of their block, added in order; group 0 holds them.
template <int COUNT>
__device__ __forceinline__ void bor_sum_groups(double2 (&v)[COUNT], int block, int blocks, int groups) {
#pragma unroll
    for (int i = 0; i < COUNT; ++i) {
        const double2 own = v[i];
        for (int g = 1; g < groups; ++g) {
            v[i].x += __shfl_sync(0xffffffffu, own.x, block + g * blocks);
            v[i].y += __shfl_sync(0xffffffffu, own.y, block + g * blocks);
        }
    }
}

// grid = (ne, ne), BOR_FAR_WARPS warps, warp w the point pairs 3 w .. 3 w + 2 of the element
// pair (nine warps leave 96 registers a thread, and the sums of MB orders spill); pairs with
// cls != 0 return at once.  A lane keeps MB orders of one parity (n = par + 2 i), whose
// folded samples are f(xi) +- f(pi - xi); e^{j n xi} is carried by rotation over G samples and
// re-anchored exactly every second chunk.
// dynamic smem: fold[warp][2 NV][BOR_CHUNK], sums[pair][nm][NV], fac[pair][nsl].
template <bool MFIE, int MB>
__global__ void __launch_bounds__(32 * BOR_FAR_WARPS, 4)
k_bor_far(int ne, const double *__restrict__ nodes, const unsigned char *__restrict__ cls, double k, int mmax,
          int nxi_cap, double2 *__restrict__ mom, double2 *__restrict__ momk) {
    constexpr int NV = MFIE ? 5 : 1, nsl = MFIE ? BOR_ALL_SLOTS : BOR_SLOTS;
    const int e = blockIdx.x, f = blockIdx.y;
    if (cls[(int64_t)e * ne + f] != 0) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int nm = mmax + 2, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    double2 *fold = reinterpret_cast<double2 *>(smem_raw) + warp * 2 * NV * BOR_CHUNK;
    double2 *sums = reinterpret_cast<double2 *>(smem_raw) + BOR_FAR_WARPS * 2 * NV * BOR_CHUNK;
    double *fac = reinterpret_cast<double *>(sums + BOR_FAR_PAIRS * nm * NV);
    const int blocks = bor_far_blocks(nm, MB), groups = 32 / blocks;
    const int block = lane % blocks, grp = lane / blocks, par = block & 1, n0 = par + 2 * MB * (block >> 1);
#pragma unroll 1
    for (int pp = warp * (BOR_FAR_PAIRS / BOR_FAR_WARPS); pp < (warp + 1) * (BOR_FAR_PAIRS / BOR_FAR_WARPS); ++pp) {
        double xo, wo, xs, wsq;
        gl_node(BOR_FAR_ORDER, pp / BOR_FAR_ORDER, xo, wo);
        gl_node(BOR_FAR_ORDER, pp % BOR_FAR_ORDER, xs, wsq);
        const BorPt p = bor_point(nodes, e, 0.5 * (xo + 1.0), 0.5 * wo);
        const BorPt q = bor_point(nodes, f, 0.5 * (xs + 1.0), 0.5 * wsq);
        for (int s = lane; s < nsl; s += 32) fac[pp * nsl + s] = bor_factor(p, q, s);
        const BorPair pr = bor_pair(k, p, q);
        const int N = min(bor_nxi(k, p.rho, q.rho, sqrt(pr.d2), mmax), nxi_cap);
        const double dxi = 2.0 * GRIM_PI / N;
        double2 acc[MB][NV], z[MB], rot[MB];
#pragma unroll
        for (int m = 0; m < MB; ++m) {
            // e^{j n dxi}; its powers: the lane's first sample (grp) and its step (groups)
            const double2 w = bor_unit((n0 + 2 * m) % N, N);
            double2 pw = make_double2(1.0, 0.0);
            z[m] = pw;
#pragma unroll 1
            for (int g = 0; g < groups; ++g) {
                if (g == grp) z[m] = pw;
                pw = cmul(pw, w);
            }
            rot[m] = pw;
#pragma unroll
            for (int v = 0; v < NV; ++v) acc[m][v] = make_double2(0.0, 0.0);
        }
        int i = grp < groups ? grp : 0x3fffffff;  // this lane's next folded sample
        const double2 *set = fold + par * NV * BOR_CHUNK;
        const int last = N / 4;
        for (int i0 = 0; i0 <= last; i0 += BOR_CHUNK) {
            // raw values at xi (side 0) and pi - xi (side 1) of the chunk's points: 2 cnt tasks (xi =
            // pi/2 is its own partner), then the folds in place -- even n: the sum of the even
            // functions and the difference of the odd ones; odd n: the other way round
            const int cnt = min(BOR_CHUNK, last + 1 - i0);
            __syncwarp();
#pragma unroll 1
            for (int task = lane; task < 2 * cnt; task += 32) {
                const int side = task >= cnt, at = side ? task - cnt : task, is = i0 + at;
                double2 val[5];
                if (side && is == last) {
#pragma unroll
                    for (int v = 0; v < NV; ++v) val[v] = make_double2(0.0, 0.0);
                } else {
                    const double2 u = bor_unit(side ? N / 2 - is : is, 2 * N);  // e^{j xi / 2}
                    double2 F[4];
                    bor_sample<MFIE>(pr, u.y, 2.0 * u.y * u.x, is == 0 ? dxi : 2.0 * dxi /* xi and -xi */, val[0], F);
#pragma unroll
                    for (int v = 0; v < 4; ++v) val[1 + v] = F[v];
                }
#pragma unroll
                for (int v = 0; v < NV; ++v) fold[(side * NV + v) * BOR_CHUNK + at] = val[v];
            }
            __syncwarp();
            if (lane < cnt) {
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    const bool odd = v == 2 || v == 3;
                    const double2 x = fold[v * BOR_CHUNK + lane], y = fold[(NV + v) * BOR_CHUNK + lane];
                    fold[v * BOR_CHUNK + lane] = odd ? csub(x, y) : cadd(x, y);
                    fold[(NV + v) * BOR_CHUNK + lane] = odd ? cadd(x, y) : csub(x, y);
                }
            }
            __syncwarp();
            const int iend = min(i0 + BOR_CHUNK, last + 1);
            if (i0 > 0 && (i0 & BOR_CHUNK) == 0 && i < iend) {
#pragma unroll
                for (int m = 0; m < MB; ++m)
                    z[m] = bor_unit((int)((unsigned)((n0 + 2 * m) * i) % (unsigned)N), N);
            }
            for (; i < iend; i += groups) {
                const int j = i - i0;
                const double2 v0 = set[j];
                double2 v1, v2, v3, v4;
                if constexpr (MFIE) {
                    v1 = set[BOR_CHUNK + j];
                    v2 = set[2 * BOR_CHUNK + j];
                    v3 = set[3 * BOR_CHUNK + j];
                    v4 = set[4 * BOR_CHUNK + j];
                }
#pragma unroll
                for (int m = 0; m < MB; ++m) {
                    const double2 c = z[m];
                    acc[m][0].x = fma(v0.x, c.x, acc[m][0].x);
                    acc[m][0].y = fma(v0.y, c.x, acc[m][0].y);
                    if constexpr (MFIE) {
                        acc[m][1].x = fma(v1.x, c.x, acc[m][1].x);
                        acc[m][1].y = fma(v1.y, c.x, acc[m][1].y);
                        acc[m][2].x = fma(v2.x, c.y, acc[m][2].x);
                        acc[m][2].y = fma(v2.y, c.y, acc[m][2].y);
                        acc[m][3].x = fma(v3.x, c.y, acc[m][3].x);
                        acc[m][3].y = fma(v3.y, c.y, acc[m][3].y);
                        acc[m][4].x = fma(v4.x, c.x, acc[m][4].x);
                        acc[m][4].y = fma(v4.y, c.x, acc[m][4].y);
                    }
                    z[m] = make_double2(c.x * rot[m].x - c.y * rot[m].y, c.x * rot[m].y + c.y * rot[m].x);
                }
            }
        }
#pragma unroll
        for (int m = 0; m < MB; ++m) {
            bor_sum_groups<NV>(acc[m], block, blocks, groups);
            const int n = n0 + 2 * m;
            if (grp == 0 && n < nm) {
#pragma unroll
                for (int v = 0; v < NV; ++v) sums[(pp * nm + n) * NV + v] = acc[m][v];
            }
        }
    }
    __syncthreads();
    const int64_t base = ((int64_t)e * ne + f) * nm;
    for (int i = t; i < nm * nsl; i += blockDim.x) {
        const int nn_ = i / nsl, slot = i - nn_ * nsl;
        const int v = slot < BOR_SLOTS ? 0 : 1 + ((slot - BOR_SLOTS) >> 2);
        double2 a = make_double2(0.0, 0.0);
#pragma unroll
        for (int q = 0; q < BOR_FAR_PAIRS; ++q) {
            const double fc = fac[q * nsl + slot];
            const double2 sv = sums[(q * nm + nn_) * NV + v];
            a.x += fc * sv.x;
            a.y += fc * sv.y;
        }
        if (slot < BOR_SLOTS) {
            mom[(base + nn_) * BOR_SLOTS + slot] = a;
        } else {
            // odd brackets: K = -j (sine sum)
            if (v == 2 || v == 3) a = make_double2(a.y, -a.x);
            momk[(base + nn_) * BOR_KSLOTS + slot - BOR_SLOTS] = a;
        }
    }
}

// Near-pair xi rule on [0, pi] for delta = R0 / c, span = 4 pi / (nmax + k c + 1) (two
// periods of the fastest oscillation): a sinh-mapped 20-point Gauss core on [0, a],
// a = min(4 delta, span, pi); 16-point panels [a 2^g, a 2^(g+1)] while a 2^g < span; then
// equal 32-point panels of at most four spans (eight periods, four points a period: the Gauss
// error of such an oscillation, (pi P/2)^65 / 65! at P = 8, is below 1e-19, and the nearest
// singularity, one span to the left, costs 2.6^-64) up to pi.
struct BorRule {
    double delta, span, a, vmax, top, wide;
    int geo, uni;
};

__device__ __forceinline__ BorRule bor_rule(double delta, double span) {
    BorRule r;
    r.delta = delta;
    r.span = span;
    r.a = fmin(fmin(4.0 * delta, span), GRIM_PI);
    r.vmax = asinh(r.a / delta);
    r.geo = 0;
    double top = r.a;
    while (top < span && top < GRIM_PI && r.geo < 2048) {
        top *= 2.0;
        ++r.geo;
    }
    r.top = top;
    r.uni = top < GRIM_PI ? (int)ceil((GRIM_PI - top) / (4.0 * span)) : 0;
    r.wide = r.uni > 0 ? (GRIM_PI - top) / r.uni : 0.0;
    return r;
}

__device__ __forceinline__ int bor_rule_count(const BorRule &r) {
    return BOR_XI_CORE + BOR_XI_PANEL * r.geo + BOR_XI_WIDE * r.uni;
}

// Gauss nodes and weights on [0, 1] of the rule's three orders, in shared memory (a constant
// table is read one address at a time).
struct BorGauss {
    double x[BOR_XI_CORE + BOR_XI_PANEL + BOR_XI_WIDE], w[BOR_XI_CORE + BOR_XI_PANEL + BOR_XI_WIDE];
};

__device__ __forceinline__ void bor_gauss_fill(BorGauss &g) {
    for (int i = threadIdx.x; i < BOR_XI_CORE + BOR_XI_PANEL + BOR_XI_WIDE; i += blockDim.x) {
        const int q = i < BOR_XI_CORE ? BOR_XI_CORE : (i < BOR_XI_CORE + BOR_XI_PANEL ? BOR_XI_PANEL : BOR_XI_WIDE);
        const int at = i - (q == BOR_XI_CORE ? 0 : (q == BOR_XI_PANEL ? BOR_XI_CORE : BOR_XI_CORE + BOR_XI_PANEL));
        double x, w;
        gl_node(q, at, x, w);
        g.x[i] = 0.5 * (x + 1.0);
        g.w[i] = 0.5 * w;
    }
}

// Node j of the rule: xi and weight (times 2 for the half range).
__device__ __forceinline__ void bor_rule_node(const BorRule &r, const BorGauss &g, int j, double &xi, double &w) {
    if (j < BOR_XI_CORE) {
        const double v = g.x[j] * r.vmax;
        xi = r.delta * sinh(v);
        w = r.delta * cosh(v) * g.w[j] * r.vmax;
    } else {
        double lo, len;
        int at;
        const int jp = j - BOR_XI_CORE, P = jp / BOR_XI_PANEL;
        if (P < r.geo) {
            at = BOR_XI_CORE + jp % BOR_XI_PANEL;
            lo = ldexp(r.a, P);
            len = fmin(ldexp(r.a, P + 1), GRIM_PI) - lo;
        } else {
            const int ju = jp - BOR_XI_PANEL * r.geo;
            at = BOR_XI_CORE + BOR_XI_PANEL + ju % BOR_XI_WIDE;
            lo = fma((double)(ju / BOR_XI_WIDE), r.wide, r.top);
            len = r.wide;
        }
        xi = fma(len, g.x[at], lo);
        w = len * g.w[at];
    }
    w *= 2.0;
}

struct BorItem {
    int e, f, r0, r1;  // element pair and its point-pair range in the rule table
};


// Stride of a sample's row of starting phases (not a multiple of 8: sixteen-byte words of
// eight rows in eight banks groups).
__host__ __device__ constexpr int bor_near_stride(int blocks) { return blocks % 8 == 0 ? blocks + 1 : blocks; }
// Complex words of a warp's staging area; its point pair's sums [nm][NV] reuse it.
__host__ __device__ constexpr int bor_near_area(int nm, int nv, int blocks) {
    return BOR_CHUNK * (nv + 1 + bor_near_stride(blocks)) > nm * nv ? BOR_CHUNK * (nv + 1 + bor_near_stride(blocks))
                                                                    : nm * nv;
}

// grid = number of near work items, at most BOR_NEAR_WARPS warps.  rule[3 i .. 3 i + 2] = (s, s', w).
// Writes the item's moments to part[item][n][slot] (nm x nsl complex).  Each warp takes its
// share of the point pairs: BOR_CHUNK samples at a time, one per lane with e^{j xi} and the phases
// e^{j n xi} at the start n of every block, then each lane the orders of its block.  After
// every round of one point pair a warp the CTA folds their sums into the item's moments.
// dynamic smem: area[warp], acc[nm][nsl], fac[warp][nsl], Gauss nodes.
template <bool MFIE, int MB>
__global__ void __launch_bounds__(32 * BOR_NEAR_WARPS, 2)
k_bor_near(const BorItem *__restrict__ items, const double *__restrict__ nodes, const double *__restrict__ rule,
           double k, int mmax, double2 *__restrict__ part) {
    constexpr int NV = MFIE ? 5 : 1, nsl = MFIE ? BOR_ALL_SLOTS : BOR_SLOTS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int nm = mmax + 2, t = threadIdx.x, lane = t & 31, warp = t >> 5, warps = blockDim.x >> 5;
    const int blocks = bor_near_blocks(nm, MB), groups = 32 / blocks, P = bor_near_stride(blocks);
    const int area = bor_near_area(nm, NV, blocks);
    double2 *areas = reinterpret_cast<double2 *>(smem_raw);
    double2 *smp = areas + warp * area;           // [NV][BOR_CHUNK]
    double2 *z1 = smp + NV * BOR_CHUNK;           // [BOR_CHUNK]
    double2 *zt = z1 + BOR_CHUNK;                 // [BOR_CHUNK][P]
    double2 *acc = areas + warps * area;           // [nm][nsl]
    double *fac = reinterpret_cast<double *>(acc + nm * nsl);
    BorGauss &gauss = *reinterpret_cast<BorGauss *>(fac + warps * nsl);
    const BorItem it = items[blockIdx.x];
    const int block = lane % blocks, grp = lane / blocks, n0 = block * MB;
    bor_gauss_fill(gauss);
    for (int i = t; i < nm * nsl; i += blockDim.x) acc[i] = make_double2(0.0, 0.0);
    __syncthreads();
    for (int base = it.r0; base < it.r1; base += warps) {
        const int ipp = base + warp;
        if (ipp < it.r1) {
            const BorPt p = bor_point(nodes, it.e, rule[3 * ipp], rule[3 * ipp + 2]);
            const BorPt q = bor_point(nodes, it.f, rule[3 * ipp + 1], 1.0);
            const BorPair pr = bor_pair(k, p, q);
            const double c = sqrt(p.rho * q.rho);
            const BorRule rl = bor_rule(sqrt(pr.d2) / c, 4.0 * GRIM_PI / ((mmax + 1) + k * c + 1.0));
            const int na = bor_rule_count(rl);
            for (int s = lane; s < nsl; s += 32) fac[warp * nsl + s] = bor_factor(p, q, s);
            double2 sum[MB][NV];
#pragma unroll
            for (int m = 0; m < MB; ++m)
#pragma unroll
                for (int v = 0; v < NV; ++v) sum[m][v] = make_double2(0.0, 0.0);
            for (int j0 = 0; j0 < na; j0 += BOR_CHUNK) {
                const int cnt = min(BOR_CHUNK, na - j0);
                __syncwarp();
                if (lane < cnt) {
                    double xi, w, sh, ch;
                    bor_rule_node(rl, gauss, j0 + lane, xi, w);
                    gh_sincos(0.5 * xi, sh, ch);
                    double2 g, F[4];
                    bor_sample<MFIE>(pr, sh, 2.0 * sh * ch, w, g, F);
                    smp[lane] = g;
                    if constexpr (MFIE) {
#pragma unroll
                        for (int v = 0; v < 4; ++v) smp[(1 + v) * BOR_CHUNK + lane] = F[v];
                    }
                    const double2 u = make_double2(1.0 - 2.0 * sh * sh, 2.0 * sh * ch);
                    z1[lane] = u;
                    double2 step = cmul(u, u), z = make_double2(1.0, 0.0);
                    step = MB == 4 ? cmul(step, step) : cmul(step, u);
                    for (int b = 0; b < blocks; ++b) {
                        zt[lane * P + b] = z;
                        z = cmul(z, step);
                    }
                }
                __syncwarp();
                if (grp < groups) {
                    for (int j = grp; j < cnt; j += groups) {
                        const double2 u = z1[j], v0 = smp[j];
                        double2 z = zt[j * P + block], v1, v2, v3, v4;
                        if constexpr (MFIE) {
                            v1 = smp[BOR_CHUNK + j];
                            v2 = smp[2 * BOR_CHUNK + j];
                            v3 = smp[3 * BOR_CHUNK + j];
                            v4 = smp[4 * BOR_CHUNK + j];
                        }
#pragma unroll
                        for (int m = 0; m < MB; ++m) {
                            sum[m][0].x = fma(v0.x, z.x, sum[m][0].x);
                            sum[m][0].y = fma(v0.y, z.x, sum[m][0].y);
                            if constexpr (MFIE) {
                                sum[m][1].x = fma(v1.x, z.x, sum[m][1].x);
                                sum[m][1].y = fma(v1.y, z.x, sum[m][1].y);
                                sum[m][2].x = fma(v2.x, z.y, sum[m][2].x);
                                sum[m][2].y = fma(v2.y, z.y, sum[m][2].y);
                                sum[m][3].x = fma(v3.x, z.y, sum[m][3].x);
                                sum[m][3].y = fma(v3.y, z.y, sum[m][3].y);
                                sum[m][4].x = fma(v4.x, z.x, sum[m][4].x);
                                sum[m][4].y = fma(v4.y, z.x, sum[m][4].y);
                            }
                            if (m + 1 < MB) z = cmul(z, u);
                        }
                    }
                }
            }
            __syncwarp();  // the samples are consumed: the sums take their place
#pragma unroll
            for (int m = 0; m < MB; ++m) {
                bor_sum_groups<NV>(sum[m], block, blocks, groups);
                if (grp == 0 && n0 + m < nm) {
#pragma unroll
                    for (int v = 0; v < NV; ++v) smp[(n0 + m) * NV + v] = sum[m][v];
                }
            }
        }
        __syncthreads();
        const int cnt = min(warps, it.r1 - base);
        for (int i = t; i < nm * nsl; i += blockDim.x) {
            const int n = i / nsl, slot = i - n * nsl, v = slot < BOR_SLOTS ? 0 : 1 + ((slot - BOR_SLOTS) >> 2);
            double2 a = make_double2(0.0, 0.0);
            for (int w = 0; w < cnt; ++w) {
                const double f = fac[w * nsl + slot];
                const double2 s = areas[w * area + n * NV + v];
                a.x = fma(f, s.x, a.x);
                a.y = fma(f, s.y, a.y);
            }
            // odd brackets: K = -j sum F sin(n xi)
            if (v == 2 || v == 3) a = make_double2(a.y, -a.x);
            acc[i].x += a.x;
            acc[i].y += a.y;
        }
        __syncthreads();
    }
    double2 *out = part + (int64_t)blockIdx.x * nm * nsl;
    for (int i = t; i < nm * nsl; i += blockDim.x) out[i] = acc[i];
}

// grid = number of near element pairs; pairs[i] = (e, f, first item, end item).
template <bool MFIE>
__global__ void k_bor_near_reduce(int ne, int mmax, const int4 *__restrict__ pairs, const double2 *__restrict__ part,
                                  double2 *__restrict__ mom, double2 *__restrict__ momk) {
    constexpr int nsl = MFIE ? BOR_ALL_SLOTS : BOR_SLOTS;
    const int nm = mmax + 2;
    const int4 pq = pairs[blockIdx.x];
    const int64_t base = ((int64_t)pq.x * ne + pq.y) * nm;
    for (int i = threadIdx.x; i < nm * nsl; i += blockDim.x) {
        double2 v = make_double2(0.0, 0.0);
        for (int it = pq.z; it < pq.w; ++it) {
            const double2 r = part[(int64_t)it * nm * nsl + i];
            v.x += r.x;
            v.y += r.y;
        }
        const int nn_ = i / nsl, slot = i - nn_ * nsl;
        if (slot < BOR_SLOTS) mom[(base + nn_) * BOR_SLOTS + slot] = v;
        else momk[(base + nn_) * BOR_KSLOTS + slot - BOR_SLOTS] = v;
    }
}

// grid = ceil(nred / 16) x ceil(nred / 16), block 16 x 16.  red_full[2*nred] lists, for
// every reduced function, up to two full components (t: node, phi: nn + node; -1 unused)
// and red_w[2*nred] their complex weights (1, or j m sign(t_rho) for a pole phi folded into
// the pole t function).  Each entry is sum over the components of conj(w_row) Z_full w_col
// with Z_full = alpha C EFIE + beta ((1/2) M - K) (beta = (1 - alpha) eta0; momk == nullptr
// for the EFIE alone, alpha = 1).  Bound by the moments' reads, 700 bytes of the mode's slots per
// element pair in 32-byte sectors (400 segments: 93 us; 105 with the element geometry derived
// in every thread).
__global__ void k_bor_assemble(int ne, int mmax, int m, double k, const double2 *__restrict__ mom,
                               const double2 *__restrict__ momk, double alpha, int nred,
                               const int *__restrict__ red_full, const double2 *__restrict__ red_w,
                               const double *__restrict__ nodes, double2 *__restrict__ Z, int64_t ldz) {
    const int r = blockIdx.x * 16 + threadIdx.x;  // row (test)
    const int c = blockIdx.y * 16 + threadIdx.y;  // column (source)
    const int nn = ne + 1;
    // tangent and length of the elements [component][before / after its node] of the tile's rows
    // and columns, once per tile
    __shared__ double geo[2][16][4][3];
    const int tid = threadIdx.y * 16 + threadIdx.x;
    if (tid < 128) {
        const int side = tid >> 6, at = (tid >> 2) & 15, which = tid & 3;
        const int q = (side ? blockIdx.y : blockIdx.x) * 16 + at;
        const int full = q < nred ? red_full[2 * q + (which >> 1)] : -1;
        const int e = full < 0 ? -1 : full % nn - 1 + (which & 1);
        if (e >= 0 && e < ne) {
            const double dr = nodes[2 * e + 2] - nodes[2 * e], dz = nodes[2 * e + 3] - nodes[2 * e + 1];
            const double L = hypot(dr, dz);
            geo[side][at][which][0] = dr / L;
            geo[side][at][which][1] = dz / L;
            geo[side][at][which][2] = L;
        }
    }
    __syncthreads();
    if (r >= nred || c >= nred) return;
    const int nm = mmax + 2;
    const int am = abs(m), am1 = abs(m - 1), ap1 = abs(m + 1);
    const double km2 = 1.0 / (k * k);
    const double C = k * 376.730313668 * 2.0 * GRIM_PI;  // C = j k eta 2 pi (times j below)
    const double beta = momk ? (1.0 - alpha) * 376.730313668 : 0.0;
    double2 total = make_double2(0.0, 0.0);
    for (int ri = 0; ri < 2; ++ri) {
        const int fr = red_full[2 * r + ri];
        if (fr < 0) continue;
        const double2 wr = red_w[2 * r + ri];
        const int ni = fr % nn, ci = fr / nn;  // node, component (0 t, 1 phi)
        for (int cj = 0; cj < 2; ++cj) {
            const int fc = red_full[2 * c + cj];
            if (fc < 0) continue;
            const double2 wc = red_w[2 * c + cj];
            const int nj = fc % nn, cc = fc / nn;
            double2 z = make_double2(0.0, 0.0), zk = z;
            double mass = 0.0;
            // element pairs (e, f) with e in {ni-1, ni}, f in {nj-1, nj}
            for (int de = 0; de < 2; ++de) {
                const int e = ni - 1 + de;
                if (e < 0 || e >= ne) continue;
                const int a = 1 - de;  // node ni is node index a of element e (e = ni-1 -> a = 1)
                const double *ge = geo[0][threadIdx.x][2 * ri + de];
                const double tre = ge[0], tze = ge[1];
                for (int df = 0; df < 2; ++df) {
                    const int f = nj - 1 + df;
                    if (f < 0 || f >= ne) continue;
                    const int b = 1 - df;
                    const double *gf = geo[1][threadIdx.y][2 * cj + df];
                    const double trf = gf[0], tzf = gf[1];
                    const int s = 2 * a + b;
                    const double2 *base = mom + ((int64_t)e * ne + f) * nm * BOR_SLOTS;
                    const double2 A0 = base[am * BOR_SLOTS + s];
                    const double2 Am1 = base[am1 * BOR_SLOTS + s];
                    const double2 Ap1 = base[ap1 * BOR_SLOTS + s];
                    const double2 Ac = make_double2(0.5 * (Am1.x + Ap1.x), 0.5 * (Am1.y + Ap1.y));
                    const double2 As = make_double2(0.5 * (Am1.x - Ap1.x), 0.5 * (Am1.y - Ap1.y));
                    const double2 DD = base[am * BOR_SLOTS + 4 + s];
                    const double2 DT = base[am * BOR_SLOTS + 8 + s];
                    const double2 TD = base[am * BOR_SLOTS + 12 + s];
                    const double2 TT = base[am * BOR_SLOTS + 16 + s];
                    double2 v;
                    if (ci == 0 && cc == 0) {
                        v.x = tre * trf * Ac.x + tze * tzf * A0.x - km2 * DD.x;
                        v.y = tre * trf * Ac.y + tze * tzf * A0.y - km2 * DD.y;
                    } else if (ci == 0 && cc == 1) {  // -j tre As - (j m / k^2) DT
                        v.x = tre * As.y + m * km2 * DT.y;
                        v.y = -tre * As.x - m * km2 * DT.x;
                    } else if (ci == 1 && cc == 0) {  // +j trf As + (j m / k^2) TD
                        v.x = -trf * As.y - m * km2 * TD.y;
                        v.y = trf * As.x + m * km2 * TD.x;
                    } else {                          // Ac - (m^2 / k^2) TT
                        v.x = Ac.x - (double)m * m * km2 * TT.x;
                        v.y = Ac.y - (double)m * m * km2 * TT.y;
                    }
                    z.x += v.x;
                    z.y += v.y;
                    if (momk) {
                        // K of quadrant uv (tt, tf, ft, ff); odd quadrants change sign with m
                        const int uv = 2 * ci + cc;
                        const double sg = (m < 0 && (uv == 1 || uv == 2)) ? -1.0 : 1.0;
                        const double2 kv =
                            momk[(((int64_t)e * ne + f) * nm + am) * BOR_KSLOTS + 4 * uv + s];
                        zk.x += sg * kv.x;
                        zk.y += sg * kv.y;
                        if (e == f && ci == cc) {
                            // mass 2 pi int rho T_a T_b dt on element e (3-point Gauss)
                            const double dre = nodes[2 * e + 2] - nodes[2 * e], Le = ge[2];
                            for (int ip = 0; ip < BOR_FAR_ORDER; ++ip) {
                                double xg, wg;
                                gl_node(BOR_FAR_ORDER, ip, xg, wg);
                                const double sq = 0.5 * (xg + 1.0);
                                const double rho = nodes[2 * e] + sq * dre;
                                const double Ta = a ? sq : 1.0 - sq, Tb = b ? sq : 1.0 - sq;
                                mass += 2.0 * GRIM_PI * (0.5 * wg * Le) * rho * Ta * Tb;
                            }
                        }
                    }
                }
            }
            // Z_full = alpha C j z + beta ((1/2) mass - 2 pi zk)
            double2 v = make_double2(-alpha * C * z.y, alpha * C * z.x);
            if (momk) {
                v.x += beta * (0.5 * mass - 2.0 * GRIM_PI * zk.x);
                v.y += beta * (-2.0 * GRIM_PI * zk.y);
            }
            // conj(wr) * v * wc
            const double2 t1 = make_double2(wr.x * v.x + wr.y * v.y, wr.x * v.y - wr.y * v.x);
            total.x += t1.x * wc.x - t1.y * wc.y;
            total.y += t1.x * wc.y + t1.y * wc.x;
        }
    }
    Z[(int64_t)c * ldz + r] = total;
}

// J_m(x) for any integer m (J_{-m} = (-1)^m J_m), through CUDA's jn.
__device__ __forceinline__ double jn_signed(int m, double x) {
    if (x == 0.0) return m == 0 ? 1.0 : 0.0;  // on-axis aspects: J_n(0) = delta_n0
    if (m >= 0) return jn(m, x);
    const double v = jn(-m, x);
    return ((-m) & 1) ? -v : v;
}

// J_{a-1}, J_a, J_{a+1} (a >= 0, J_{-1} = -J_1) at x >= 0 by Miller's backward recurrence
// f_{k-1} = (2 k / x) f_k - f_{k+1}, normalised by J_0 + 2 J_2 + 2 J_4 + ... = 1.  It starts
// where J falls below 1e-18 of the orders wanted: from order n = max(x, a + 1), J_{n + t (n/2)^(1/3)}
// follows Ai(t), and t = 16 is past 1e-18.  x up to BOR_MILLER_MAX (N steps a point).
#define BOR_MILLER_MAX 2000.0
__device__ __forceinline__ void bor_bessel3(int a, double x, double &jm1, double &j0, double &jp1) {
    if (x < 1e-8) {
        // the first term of the series: the next is below 3e-17 of it
        double p = 1.0;
        jm1 = 0.0;
        for (int i = 1; i <= a; ++i) {
            jm1 = p;
            p *= 0.5 * x / i;
        }
        j0 = p;
        jp1 = p * (0.5 * x / (a + 1));
        if (a == 0) jm1 = -jp1;
        return;
    }
    const double top = fmax(x, (double)(a + 1));
    int k = (int)(top + 16.0f * cbrtf(0.5f * (float)top)) + 6;
    k += (k ^ a) & 1;  // two steps a turn reach order a itself
    const double rx = 2.0 / x;
    double kr = k;
    double f1 = 0.0, f0 = 1e-280;        // orders k + 1, k
    double same = 0.0, other = 0.0;      // sums of the orders of a's parity, down to 1 or 2, and of the others
    double r0 = 0.0, r1 = 0.0, r2 = 0.0;  // orders a - 1, a, a + 1
    auto turn = [&](bool found) {
        same += f0;
        f1 = fma(kr * rx, f0, -f1);
        other += f1;
        f0 = fma((kr - 1.0) * rx, f1, -f0);
        kr -= 2.0;
        if ((__double2hiint(f0) & 0x7fffffff) > 0x5f000000) {  // about 2^497: small x, high orders
            constexpr double s = 1e-250;
            f1 *= s;
            f0 *= s;
            same *= s;
            other *= s;
            if (found) {
                r0 *= s;
                r1 *= s;
                r2 *= s;
            }
        }
    };
#pragma unroll 1
    for (; k > a; k -= 2) turn(false);
    r1 = f0;
    r2 = f1;
    r0 = fma(kr * rx, f0, -f1);
#pragma unroll 1
    for (; k > 1; k -= 2) turn(true);
    const double zero = k == 1 ? fma(rx, f0, -f1) : f0;  // order 0
    const double inv = 1.0 / fma(2.0, k == 1 ? other : same, zero);
    j0 = r1 * inv;
    jp1 = r2 * inv;
    jm1 = a == 0 ? -jp1 : r0 * inv;
}

// Per (aspect, Gauss point): J_m, J_{m-1}, J_{m+1} at k rho sin(theta) and the axial phase
// e^{j k z cos(theta)} -- evaluated once and shared by every row that the point touches.
// tab[((it * ne + e) * BOR_FAR_ORDER + ip) * 5 + {0..4}] = (J_m, J_{m-1}, J_{m+1}, cos, sin).
// One recurrence for the three orders: 400 segments, 361 aspects, k rho <= 25, 78 us a mode with
// three jn calls, 26 us (bound by the recurrence's FP64 steps, about 90 a point).
__global__ void k_bor_bessel(int ne, const double *__restrict__ nodes, double k, int m, int nth,
                             const double *__restrict__ th_deg, double *__restrict__ tab) {
    const int pidx = blockIdx.x * blockDim.x + threadIdx.x;
    const int it = blockIdx.y;
    if (pidx >= ne * BOR_FAR_ORDER || it >= nth) return;
    const int e = pidx / BOR_FAR_ORDER, ip = pidx % BOR_FAR_ORDER;
    double st, ct;
    sincospi(th_deg[it] / 180.0, &st, &ct);
    double xg, wg;
    gl_node(BOR_FAR_ORDER, ip, xg, wg);
    const double s = 0.5 * (xg + 1.0);
    const double r0 = nodes[2 * e], z0 = nodes[2 * e + 1];
    const double rho = r0 + s * (nodes[2 * e + 2] - r0), z = z0 + s * (nodes[2 * e + 3] - z0);
    const double x = k * rho * st;
    double *o = tab + ((int64_t)it * ne * BOR_FAR_ORDER + pidx) * 5;
    if (fabs(x) <= BOR_MILLER_MAX) {
        const int a = abs(m);
        double lo, mid, hi;
        bor_bessel3(a, fabs(x), lo, mid, hi);
        // J_n(-x) = J_{-n}(x) = (-1)^n J_n(x)
        const double even = a & 1 ? -1.0 : 1.0;
        if (x < 0.0) {
            mid *= even;
            lo *= -even;
            hi *= -even;
        }
        o[0] = m < 0 ? even * mid : mid;
        o[1] = m < 0 ? -even * hi : lo;
        o[2] = m < 0 ? -even * lo : hi;
    } else {  // NaN too
        o[0] = jn_signed(m, x);
        o[1] = jn_signed(m - 1, x);
        o[2] = jn_signed(m + 1, x);
    }
    double sp, cp;
    sincos(k * z * ct, &sp, &cp);
    o[3] = cp;
    o[4] = sp;
}

// Reduced excitation (far = 0) or far-field weights (far = 1) for mode m, from the
// k_bor_bessel table of the same (m, aspects).
// Columns: [VV theta_0..n-1, HH theta_0..n-1].  One thread per (reduced row, aspect), both
// polarisations from the same table entries and element geometry (a thread per column read
// and derived them twice: 37 us a mode at 400 segments, 361 aspects, now 20).
__global__ void k_bor_excitation(int ne, const double *__restrict__ nodes, int m, int nth,
                                 const double *__restrict__ th_deg, const double *__restrict__ tab, int far,
                                 double alpha, int nred, const int *__restrict__ red_full,
                                 const double2 *__restrict__ red_w, double2 *__restrict__ V, int64_t ldv) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const int it = blockIdx.y;
    if (r >= nred || it >= nth) return;
    const int nn = ne + 1;
    double st, ct;
    sincospi(th_deg[it] / 180.0, &st, &ct);
    // j^m, j^(m-1), j^(m+1) as unit complex numbers
    const int q0 = ((m % 4) + 4) % 4, qm = (((m - 1) % 4) + 4) % 4, qp = (((m + 1) % 4) + 4) % 4;
    const double2 u0 = make_double2(q0 == 0 ? 1 : (q0 == 2 ? -1 : 0), q0 == 1 ? 1 : (q0 == 3 ? -1 : 0));
    const double2 um = make_double2(qm == 0 ? 1 : (qm == 2 ? -1 : 0), qm == 1 ? 1 : (qm == 3 ? -1 : 0));
    const double2 up = make_double2(qp == 0 ? 1 : (qp == 2 ? -1 : 0), qp == 1 ? 1 : (qp == 3 ? -1 : 0));
    double2 total[2] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0)};  // VV, HH
    for (int ri = 0; ri < 2; ++ri) {
        const int fr = red_full[2 * r + ri];
        if (fr < 0) continue;
        const double2 w = red_w[2 * r + ri];
        const int node = fr % nn, comp = fr / nn;
        double2 sum[2] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
        for (int de = 0; de < 2; ++de) {
            const int e = node - 1 + de;
            if (e < 0 || e >= ne) continue;
            const int a = 1 - de;
            const double r0 = nodes[2 * e], dr = nodes[2 * e + 2] - r0, dz = nodes[2 * e + 3] - nodes[2 * e + 1];
            const double L = hypot(dr, dz), tr = dr / L, tz = dz / L;
            for (int ip = 0; ip < BOR_FAR_ORDER; ++ip) {
                double xg, wg;
                gl_node(BOR_FAR_ORDER, ip, xg, wg);
                const double s = 0.5 * (xg + 1.0);
                const double rho = r0 + s * dr, w = 0.5 * wg * L;
                const double T = a == 0 ? 1.0 - s : s;
                const double *tb = tab + (((int64_t)it * ne + e) * BOR_FAR_ORDER + ip) * 5;
                const double jm = tb[0], jm1 = tb[1], jp1 = tb[2];
                const double2 I0 = make_double2(2 * GRIM_PI * u0.x * jm, 2 * GRIM_PI * u0.y * jm);
                const double2 Ic = make_double2(GRIM_PI * (up.x * jp1 + um.x * jm1), GRIM_PI * (up.y * jp1 + um.y * jm1));
                // Is = -j pi (j^(m-1) J_{m-1} - j^(m+1) J_{m+1})
                const double2 dd = make_double2(um.x * jm1 - up.x * jp1, um.y * jm1 - up.y * jp1);
                double2 Is = make_double2(GRIM_PI * dd.y, -GRIM_PI * dd.x);
                if (far) Is = make_double2(-Is.x, -Is.y);
                // VV: the t and phi components of the first, HH: of the second
                const double2 tv = make_double2(tr * ct * Ic.x - tz * st * I0.x, tr * ct * Ic.y - tz * st * I0.y);
                const double2 pv = make_double2(-ct * Is.x, -ct * Is.y);
                const double2 th = make_double2(tr * Is.x, tr * Is.y);
                double2 ang[2] = {comp == 0 ? tv : pv, comp == 0 ? th : Ic};
                if (!far && alpha != 1.0) {
                    // eta0 <W, n x H_inc> (reference rhs_mfie_mode), weighted 1 - alpha
                    const double2 hm[2] = {comp == 0 ? Ic : make_double2(-tr * Is.x, -tr * Is.y),
                                           comp == 0 ? make_double2(ct * Is.x, ct * Is.y) : tv};
#pragma unroll
                    for (int p = 0; p < 2; ++p)
                        ang[p] = make_double2(alpha * ang[p].x + (1.0 - alpha) * hm[p].x,
                                              alpha * ang[p].y + (1.0 - alpha) * hm[p].y);
                }
                const double cp = tb[3], sp = tb[4];
                const double f = rho * w * T;
                const double2 ph = make_double2(cp * f, sp * f);
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    sum[p].x += ph.x * ang[p].x - ph.y * ang[p].y;
                    sum[p].y += ph.x * ang[p].y + ph.y * ang[p].x;
                }
            }
        }
        // rhs: conj(w) * sum (Q^H V);  far weights: w * sum (Q^T W)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            if (far) {
                total[p].x += w.x * sum[p].x - w.y * sum[p].y;
                total[p].y += w.x * sum[p].y + w.y * sum[p].x;
            } else {
                total[p].x += w.x * sum[p].x + w.y * sum[p].y;
                total[p].y += w.x * sum[p].y - w.y * sum[p].x;
            }
        }
    }
    V[(int64_t)it * ldv + r] = total[0];
    V[(int64_t)(nth + it) * ldv + r] = total[1];
}

// amp[col] += sum_r W[r, col] * X[r, col]  (one CTA per column, fixed-order reduction)
__global__ void k_bor_farfield_accumulate(int nred, int ncol, const double2 *__restrict__ W, int64_t ldw,
                                          const double2 *__restrict__ X, int64_t ldx, double2 *__restrict__ amp) {
    const int col = blockIdx.x;
    double re = 0.0, im = 0.0;
    for (int r = threadIdx.x; r < nred; r += blockDim.x) {
        const double2 w = W[(int64_t)col * ldw + r], x = X[(int64_t)col * ldx + r];
        re += w.x * x.x - w.y * x.y;
        im += w.x * x.y + w.y * x.x;
    }
    for (int off = 16; off > 0; off >>= 1) {
        re += __shfl_down_sync(0xffffffffu, re, off);
        im += __shfl_down_sync(0xffffffffu, im, off);
    }
    __shared__ double sr[32], si[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { sr[warp] = re; si[warp] = im; }
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        re = lane < nw ? sr[lane] : 0.0;
        im = lane < nw ? si[lane] : 0.0;
        for (int off = 16; off > 0; off >>= 1) {
            re += __shfl_down_sync(0xffffffffu, re, off);
            im += __shfl_down_sync(0xffffffffu, im, off);
        }
        if (lane == 0) {
            amp[col].x += re;
            amp[col].y += im;
        }
    }
}

// ---- mirror-symmetric bodies: even / odd halves of a mode system (reference
// bor/factor.py:37-116 MirrorSplit).  A body symmetric about a plane normal to the axis
// maps reduced unknown u to target[u] with sign[u] (J_t changes sign, J_phi does not).
// Pairs (p1 < p2 = target[p1], s = sign[p2]) and fixed unknowns (fe: sign +1, fo: sign -1)
// give, with r = 1/sqrt(2), the even half over (r (u_p1 + s u_p2), u_fe) and the odd half
// over (r (u_p1 - s u_p2), u_fo); when A = R A R they decouple exactly:
//   H[:k,:k] = (a[p1,p1] + s a[p2,p2] s +- (a[p1,p2] s + s a[p2,p1])) / 2
//   H[:k,k:] = (a[p1,f] +- s a[p2,f]) r,  H[k:,:k] = (a[f,p1] +- a[f,p2] s) r,  H[k:,k:] = a[f,f].
struct BorMirror {
    int k, nfe, nfo;
    const int *p1, *p2, *fe, *fo;
    const double *s;
};

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 cscale(double2 a, double f) { return make_double2(a.x * f, a.y * f); }

// grid over the (ke x ke) even and (ko x ko) odd halves; He, Ho column-major (ld ke, ko).
__global__ void k_bor_mirror_halves(BorMirror mr, const double2 *__restrict__ Z, int64_t ldz, double2 *__restrict__ He,
                                    double2 *__restrict__ Ho) {
    const int i = blockIdx.x * 16 + threadIdx.x, j = blockIdx.y * 16 + threadIdx.y;
    const int k = mr.k, ke = k + mr.nfe, ko = k + mr.nfo;
    const double r = 0.7071067811865475244;
    auto a = [&](int row, int col) { return Z[(int64_t)col * ldz + row]; };
    for (int parity = 0; parity < 2; ++parity) {
        const int m = parity ? ko : ke;
        if (i >= m || j >= m) continue;
        const double sg = parity ? -1.0 : 1.0;
        const int *fx = parity ? mr.fo : mr.fe;
        double2 v;
        if (i < k && j < k) {
            const int a1 = mr.p1[i], a2 = mr.p2[i], b1 = mr.p1[j], b2 = mr.p2[j];
            const double si = mr.s[i], sj = mr.s[j];
            const double2 common = cadd(a(a1, b1), cscale(a(a2, b2), si * sj));
            const double2 cross = cadd(cscale(a(a1, b2), sj), cscale(a(a2, b1), si));
            v = cscale(cadd(common, cscale(cross, sg)), 0.5);
        } else if (i < k) {
            const int f = fx[j - k];
            v = cscale(cadd(a(mr.p1[i], f), cscale(a(mr.p2[i], f), sg * mr.s[i])), r);
        } else if (j < k) {
            const int f = fx[i - k];
            v = cscale(cadd(a(f, mr.p1[j]), cscale(a(f, mr.p2[j]), sg * mr.s[j])), r);
        } else {
            v = a(fx[i - k], fx[j - k]);
        }
        (parity ? Ho : He)[(int64_t)j * m + i] = v;
    }
}

// max over entries of |a - (R A R)| and of |a| (two non-negative doubles, as ordered bits).
__global__ void k_bor_mirror_asym(int n, const double2 *__restrict__ Z, int64_t ldz, const int *__restrict__ target,
                                  const double *__restrict__ sign, unsigned long long *__restrict__ out) {
    const int i = blockIdx.x * 16 + threadIdx.x, j = blockIdx.y * 16 + threadIdx.y;
    double d = 0.0, m = 0.0;
    if (i < n && j < n) {
        const double2 a = Z[(int64_t)j * ldz + i];
        const double2 b = Z[(int64_t)target[j] * ldz + target[i]];
        const double f = sign[i] * sign[j];
        d = hypot(a.x - f * b.x, a.y - f * b.y);
        m = hypot(a.x, a.y);
    }
    for (int off = 16; off > 0; off >>= 1) {
        d = fmax(d, __shfl_down_sync(0xffffffffu, d, off));
        m = fmax(m, __shfl_down_sync(0xffffffffu, m, off));
    }
    if ((threadIdx.x + 16 * threadIdx.y) % 32 == 0) {
        atomicMax(out, (unsigned long long)__double_as_longlong(d));
        atomicMax(out + 1, (unsigned long long)__double_as_longlong(m));
    }
}

// Right-hand sides (n x nrhs, ld ldb) into the even (ke x nrhs) and odd (ko x nrhs) parts.
__global__ void k_bor_mirror_split(BorMirror mr, int nrhs, const double2 *__restrict__ B, int64_t ldb,
                                   double2 *__restrict__ Be, double2 *__restrict__ Bo) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
    const int k = mr.k, ke = k + mr.nfe, ko = k + mr.nfo;
    if (c >= nrhs) return;
    const double r = 0.7071067811865475244;
    const double2 *b = B + (int64_t)c * ldb;
    if (i < ke) {
        Be[(int64_t)c * ke + i] = i < k ? cscale(cadd(b[mr.p1[i]], cscale(b[mr.p2[i]], mr.s[i])), r) : b[mr.fe[i - k]];
    }
    if (i < ko) {
        Bo[(int64_t)c * ko + i] = i < k ? cscale(cadd(b[mr.p1[i]], cscale(b[mr.p2[i]], -mr.s[i])), r) : b[mr.fo[i - k]];
    }
}

// Solutions of the halves back to the n unknowns.
__global__ void k_bor_mirror_join(BorMirror mr, int nrhs, const double2 *__restrict__ Ye,
                                  const double2 *__restrict__ Yo, double2 *__restrict__ X, int64_t ldx) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
    const int k = mr.k, ke = k + mr.nfe, ko = k + mr.nfo;
    if (c >= nrhs) return;
    const double r = 0.7071067811865475244;
    double2 *x = X + (int64_t)c * ldx;
    const double2 *ye = Ye + (int64_t)c * ke, *yo = Yo + (int64_t)c * ko;
    if (i < k) {
        const double2 e = ye[i], o = yo[i];
        x[mr.p1[i]] = cscale(cadd(e, o), r);
        x[mr.p2[i]] = cscale(cadd(e, cscale(o, -1.0)), r * mr.s[i]);
    } else if (i < ke && i - k < mr.nfe) {
        x[mr.fe[i - k]] = ye[i];
    }
    if (i >= k && i < ko) x[mr.fo[i - k]] = yo[i];
}

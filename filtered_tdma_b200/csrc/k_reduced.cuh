// Reduced interface system of PaScaL's segmented solve, solved in registers
// with warp shuffles (the in-GPU replacement of the reference's all-to-all of
// reduced rows followed by a serial Thomas on 2P rows,
// libs/pascal_tdma/cpu/pascal_tdma.cpp:185-210).
//
// Row notation for sub-segment p of one system:
//   first: l0 xL(p-1) + xF(p) + u0 xL(p) = r0
//   last:  l1 xF(p) + xL(p) + u1 xF(p+1) = r1
// One cyclic-reduction level eliminates the first-row unknowns and leaves
//   a xL(p-1) + xL(p) + c xL(p+1) = d,
// which parallel cyclic reduction solves in log2(nseg) shuffle steps; the
// first-row unknowns follow from the first rows.
#pragma once

#include "btdma_common.cuh"

namespace btdma {

// One PCR row update of  l x_{i-dl} + x_i + u x_{i+dl} = r  with its
// neighbours (m: row i-dl, p: row i+dl).
__device__ __forceinline__ void pcr_step(double& l, double& u, double& r, double lm, double um,
                                         double rm, double lp, double up, double rp) {
    const double ib = rcp_nr(1.0 - l * um - u * lp);
    const double nl = -l * lm * ib;
    const double nu = -u * up * ib;
    r = (r - l * rm - u * rp) * ib;
    l = nl;
    u = nu;
}

// One system's reduced system over a group of W = 2^ceil(log2 nseg) <= 32
// consecutive lanes (lane p of the group holds sub-segment p; lanes with
// act == false carry identity rows).  Every lane of the warp must call it.
// Periodic systems (CYCLIC) need nseg to be a power of two.
template <bool CYCLIC>
__device__ __forceinline__ void reduced_solve_shfl(double l0, double u0, double r0, double l1,
                                                   double u1, double r1, int p, int nseg, int W,
                                                   bool act, double& xf, double& xl) {
    // next sub-segment's first row (zero past the end unless periodic)
    const int pn = (CYCLIC && p == nseg - 1) ? 0 : p + 1;
    double l0n = __shfl_sync(0xffffffffu, l0, pn, W);
    double u0n = __shfl_sync(0xffffffffu, u0, pn, W);
    double r0n = __shfl_sync(0xffffffffu, r0, pn, W);
    if (!CYCLIC && p + 1 >= nseg) l0n = u0n = r0n = 0.0;
    double al_ = 0, cl_ = 0, dl_ = 0;
    {
        const double ib = rcp_nr(1.0 - l1 * u0 - u1 * l0n);
        al_ = -l1 * l0 * ib;
        cl_ = -u1 * u0n * ib;
        dl_ = (r1 - l1 * r0 - u1 * r0n) * ib;
    }
    if (!act) al_ = cl_ = dl_ = 0.0;
    if (CYCLIC && nseg == 1) {
        xl = dl_ * rcp_nr(1.0 + al_ + cl_);
    } else {
        bool solved = false;
        xl = 0.0;
        for (int dl = 1; dl < nseg; dl <<= 1) {
            int im = p - dl, ip = p + dl;
            if (CYCLIC) {
                im = im < 0 ? im + nseg : im;
                ip = ip >= nseg ? ip - nseg : ip;
            }
            double lm = __shfl_sync(0xffffffffu, al_, im & (W - 1), W);
            double um = __shfl_sync(0xffffffffu, cl_, im & (W - 1), W);
            double rm = __shfl_sync(0xffffffffu, dl_, im & (W - 1), W);
            double lp = __shfl_sync(0xffffffffu, al_, ip & (W - 1), W);
            double up = __shfl_sync(0xffffffffu, cl_, ip & (W - 1), W);
            double rp = __shfl_sync(0xffffffffu, dl_, ip & (W - 1), W);
            if (!CYCLIC) {
                if (im < 0) lm = um = rm = 0.0;
                if (ip >= nseg) lp = up = rp = 0.0;
            }
            if (CYCLIC && 2 * dl == nseg) {
                // p-dl and p+dl are the same row j: 2x2 system in x_p, x_j
                const double si = al_ + cl_, sj = lm + um;
                xl = (dl_ - si * rm) * rcp_nr(1.0 - si * sj);
                solved = true;
            } else {
                pcr_step(al_, cl_, dl_, lm, um, rm, lp, up, rp);
            }
        }
        if (!solved) xl = dl_;
    }
    // x_first(p) = r0 - l0 xL(p-1) - u0 xL(p)
    const int pm = (CYCLIC && p == 0) ? nseg - 1 : p - 1;
    double xlm = __shfl_sync(0xffffffffu, xl, pm & (W - 1), W);
    if (!CYCLIC && p == 0) xlm = 0.0;
    xf = r0 - l0 * xlm - u0 * xl;
}

// Filtered's reduced system (FilteredTDMA v2, libs/filtered_tdma/cpu/
// filtered_tdma.cpp:217-238 with filtered_tdma_kernels.hpp's steps) in the
// lanes of reduced_solve_shfl: the sub-segments are grouped into segments of R
// consecutive lanes (R a power of two; the reference's ranks of m = 16 R rows).
// Inside a segment the system is solved exactly, with the two couplings to
// the neighbouring segments as parameters: three right-hand sides, y0 (the
// rows' own), yl (the left neighbour's last unknown = 1) and yr (the right
// neighbour's first unknown = 1), so every unknown is y0 + lam yl + rho yr.
// Across segments Filtered's approximation: the far couplings (a segment's
// first unknown's response to its right neighbour, its last unknown's to its
// left neighbour, of order rho^m) are dropped, which leaves one 2 x 2 system
// per interface (solve_interfaces, filtered_tdma_kernels.hpp:172-196):
//   f_k = y0F_k + yl F_k l_{k-1},  l_{k-1} = y0L_{k-1} + yr L_{k-1} f_k.
// lam and rho of each segment then come from its interfaces (0 outside the
// batch unless CYCLIC).  The J-row truncation of the correction is not
// applied: every row is back-substituted with the full correction, which costs
// nothing extra here; the result stays within Filtered's eps of the exact one.
template <bool CYCLIC>
__device__ __forceinline__ void reduced_solve_filtered(double l0, double u0, double r0, double l1,
                                                       double u1, double r1, int p, int nseg,
                                                       int W, int R, bool act, double& xf,
                                                       double& xl) {
    const unsigned FULL = 0xffffffffu;
    const int t = p & (R - 1);     // lane in the segment
    const int k0 = p - t;          // first lane of the segment
    const double l0s = t == 0 ? 0.0 : l0;  // couplings inside the segment only
    const double u1s = t == R - 1 ? 0.0 : u1;
    // the three right-hand sides of the first / last rows
    double a0 = r0, a1 = r1;
    double b0 = t == 0 ? -l0 : 0.0, b1 = 0.0;
    double c0 = 0.0, c1 = t == R - 1 ? -u1 : 0.0;
    // cyclic reduction: the next sub-segment's first row (inside the segment)
    const int pn = (p + 1) & (W - 1);
    const double l0n = __shfl_sync(FULL, l0, pn, W), u0n = __shfl_sync(FULL, u0, pn, W);
    const double a0n = __shfl_sync(FULL, a0, pn, W), b0n = __shfl_sync(FULL, b0, pn, W);
    const double c0n = __shfl_sync(FULL, c0, pn, W);
    const double ib = rcp_nr(1.0 - l1 * u0 - u1s * l0n);
    double al = -l1 * l0s * ib, cl = -u1s * u0n * ib;
    double da = (a1 - l1 * a0 - u1s * a0n) * ib;
    double db = (b1 - l1 * b0 - u1s * b0n) * ib;
    double dc = (c1 - l1 * c0 - u1s * c0n) * ib;
    if (!act) al = cl = da = db = dc = 0.0;
    // parallel cyclic reduction inside the segment
    for (int dl = 1; dl < R; dl <<= 1) {
        const bool vm = t - dl >= 0, vp = t + dl < R;
        const int im = (p - dl) & (W - 1), ip = (p + dl) & (W - 1);
        double lm = __shfl_sync(FULL, al, im, W), um = __shfl_sync(FULL, cl, im, W);
        double lp = __shfl_sync(FULL, al, ip, W), up = __shfl_sync(FULL, cl, ip, W);
        double am = __shfl_sync(FULL, da, im, W), ap = __shfl_sync(FULL, da, ip, W);
        double bm = __shfl_sync(FULL, db, im, W), bp = __shfl_sync(FULL, db, ip, W);
        double cm = __shfl_sync(FULL, dc, im, W), cp = __shfl_sync(FULL, dc, ip, W);
        if (!vm) lm = um = am = bm = cm = 0.0;
        if (!vp) lp = up = ap = bp = cp = 0.0;
        const double ibl = rcp_nr(1.0 - al * um - cl * lp);
        da = (da - al * am - cl * ap) * ibl;
        db = (db - al * bm - cl * bp) * ibl;
        dc = (dc - al * cm - cl * cp) * ibl;
        const double nl = -al * lm * ibl;
        cl = -cl * up * ibl;
        al = nl;
    }
    // last unknowns (da, db, dc); first unknowns from the first rows
    const int pm = (p - 1) & (W - 1);
    double xam = __shfl_sync(FULL, da, pm, W), xbm = __shfl_sync(FULL, db, pm, W);
    double xcm = __shfl_sync(FULL, dc, pm, W);
    if (t == 0) xam = xbm = xcm = 0.0;
    const double fa = a0 - l0s * xam - u0 * da;
    const double fb = b0 - l0s * xbm - u0 * db;
    const double fc = c0 - l0s * xcm - u0 * dc;
    // interface 2 x 2 at each segment's first lane: f_k and l_{k-1}, with
    // the previous segment's last lane's y0 and yr
    const int pl = (k0 - 1) & (W - 1);
    const double yl0 = __shfl_sync(FULL, da, pl, W), ylr = __shfl_sync(FULL, dc, pl, W);
    const bool left = CYCLIC || k0 > 0;
    double f = fa, lam = 0.0;
    if (left) {
        f = (fa + fb * yl0) * rcp_nr(1.0 - fb * ylr);
        lam = yl0 + ylr * f;
    }
    // every lane: lam of its segment (from its first lane) and rho (the next
    // segment's first lane's f)
    const int kn = (k0 + R) & (W - 1);
    const double lk = __shfl_sync(FULL, lam, k0, W);
    double rk = __shfl_sync(FULL, f, kn, W);
    if (!CYCLIC && k0 + R >= nseg) rk = 0.0;
    xf = fa + lk * fb + rk * fc;
    xl = da + lk * db + rk * dc;
}

// The reduced system of n consecutive sub-segments with their outer couplings as
// parameters, over the lanes of reduced_solve_shfl: lane p's unknowns are
//   xF(p) = f[0] + lam f[1] + rho f[2],  xL(p) = d[0] + lam d[1] + rho d[2]
// with lam the last unknown left of them and rho the first one right of them
// (reduced_solve_filtered's three right-hand sides, one segment of n lanes).
__device__ __forceinline__ void reduced_condense(double l0, double u0, double r0, double l1,
                                                 double u1, double r1, int p, int n, int W,
                                                 bool act, double (&f)[3], double (&d)[3]) {
    const unsigned FULL = 0xffffffffu;
    const bool first = p == 0, last = p == n - 1;
    const double l0s = first ? 0.0 : l0, u1s = last ? 0.0 : u1;  // couplings inside
    const double b0 = first ? -l0 : 0.0, c1 = last ? -u1 : 0.0;
    const int pn = (p + 1) & (W - 1);
    // the next sub-segment's first row (its b0 is 0: it is not the first)
    const double l0n = __shfl_sync(FULL, l0, pn, W), u0n = __shfl_sync(FULL, u0, pn, W);
    const double r0n = __shfl_sync(FULL, r0, pn, W);
    const double ib = rcp_nr(1.0 - l1 * u0 - u1s * l0n);
    double al = -l1 * l0s * ib, cl = -u1s * u0n * ib;
    double da = (r1 - l1 * r0 - u1s * r0n) * ib, db = -l1 * b0 * ib, dc = c1 * ib;
    if (!act) al = cl = da = db = dc = 0.0;
    for (int dl = 1; dl < n; dl <<= 1) {
        const bool vm = p - dl >= 0, vp = p + dl < n;
        const int im = (p - dl) & (W - 1), ip = (p + dl) & (W - 1);
        double lm = __shfl_sync(FULL, al, im, W), um = __shfl_sync(FULL, cl, im, W);
        double lp = __shfl_sync(FULL, al, ip, W), up = __shfl_sync(FULL, cl, ip, W);
        double am = __shfl_sync(FULL, da, im, W), ap = __shfl_sync(FULL, da, ip, W);
        double bm = __shfl_sync(FULL, db, im, W), bp = __shfl_sync(FULL, db, ip, W);
        double cm = __shfl_sync(FULL, dc, im, W), cp = __shfl_sync(FULL, dc, ip, W);
        if (!vm) lm = um = am = bm = cm = 0.0;
        if (!vp) lp = up = ap = bp = cp = 0.0;
        const double ibl = rcp_nr(1.0 - al * um - cl * lp);
        da = (da - al * am - cl * ap) * ibl;
        db = (db - al * bm - cl * bp) * ibl;
        dc = (dc - al * cm - cl * cp) * ibl;
        const double nl = -al * lm * ibl;
        cl = -cl * up * ibl;
        al = nl;
    }
    const int pm = (p - 1) & (W - 1);
    double xam = __shfl_sync(FULL, da, pm, W), xbm = __shfl_sync(FULL, db, pm, W);
    double xcm = __shfl_sync(FULL, dc, pm, W);
    if (first) xam = xbm = xcm = 0.0;
    f[0] = r0 - l0s * xam - u0 * da;
    f[1] = b0 - l0s * xbm - u0 * db;
    f[2] = -l0s * xcm - u0 * dc;
    d[0] = da;
    d[1] = db;
    d[2] = dc;
}

// The outer unknowns of n condensed blocks of one system, lane r of a group of W
// holding block r's first and last rows
//   F_r = f[0] + L_{r-1} f[1] + F_{r+1} f[2],  L_r = d[0] + L_{r-1} d[1] + F_{r+1} d[2]:
// lam = L_{r-1} and rho = F_{r+1} (0 outside the system unless CYCLIC).  Block by
// block, L_r = p + pl L_{-1} + s F_{r+1} and F_r = P + Pl L_{-1} + S F_{r+1};
// periodic systems close the chain with a 2 x 2 system in L_{-1} = L_{n-1} and
// F_n = F_0.  Every lane of the warp calls it.
template <bool CYCLIC>
__device__ __forceinline__ void reduced_outer(const double (&f)[3], const double (&d)[3], int r,
                                              int n, int W, double& lam, double& rho) {
    const unsigned FULL = 0xffffffffu;
    double P = f[0], S = f[2], p = d[0], s = d[2];
    double Pl = CYCLIC ? f[1] : 0.0, pl = CYCLIC ? d[1] : 0.0;  // of block 0
    for (int k = 1; k < n; ++k) {
        const double pm = __shfl_sync(FULL, p, k - 1, W), sm = __shfl_sync(FULL, s, k - 1, W);
        const double plm = CYCLIC ? __shfl_sync(FULL, pl, k - 1, W) : 0.0;
        if (r == k) {
            const double ib = rcp_nr(1.0 - f[1] * sm);
            P = (f[0] + f[1] * pm) * ib;
            S = f[2] * ib;
            p = d[0] + d[1] * (pm + sm * P);
            s = d[1] * sm * S + d[2];
            if constexpr (CYCLIC) {
                Pl = f[1] * plm * ib;
                pl = d[1] * (plm + sm * Pl);
            }
        }
    }
    double x = P, y = Pl, z = S;  // F_r = x + y L_{-1} + z F_n
    for (int k = n - 2; k >= 0; --k) {
        const double xn = __shfl_sync(FULL, x, k + 1, W);
        const double yn = CYCLIC ? __shfl_sync(FULL, y, k + 1, W) : 0.0;
        const double zn = CYCLIC ? __shfl_sync(FULL, z, k + 1, W) : 0.0;
        if (r == k) {
            x = P + S * xn;
            if constexpr (CYCLIC) {
                y = Pl + S * yn;
                z = S * zn;
            }
        }
    }
    double fr = x;
    double L0 = 0.0, Fn = 0.0;  // L_{-1}, F_n
    if constexpr (CYCLIC) {
        const double x0 = __shfl_sync(FULL, x, 0, W), y0 = __shfl_sync(FULL, y, 0, W);
        const double z0 = __shfl_sync(FULL, z, 0, W);
        const double pe = __shfl_sync(FULL, p, n - 1, W), ple = __shfl_sync(FULL, pl, n - 1, W);
        const double se = __shfl_sync(FULL, s, n - 1, W);
        const double id = rcp_nr((1.0 - z0) * (1.0 - ple) - y0 * se);
        Fn = (x0 * (1.0 - ple) + y0 * pe) * id;
        L0 = ((1.0 - z0) * pe + se * x0) * id;
        fr = x + y * L0 + z * Fn;
    }
    const int rm = (r - 1) & (W - 1), rp = (r + 1) & (W - 1);
    const double pm = __shfl_sync(FULL, p, rm, W), sm = __shfl_sync(FULL, s, rm, W);
    const double plm = CYCLIC ? __shfl_sync(FULL, pl, rm, W) : 0.0;
    const double fn = __shfl_sync(FULL, fr, rp, W);
    lam = r == 0 ? L0 : pm + plm * L0 + sm * fr;
    rho = r == n - 1 ? Fn : fn;
}

// The matrix steps of reduced_solve_shfl for one lane, written to lt[0 .. 5 +
// 3 * levels) (the lane table of a matrix shared by every system, see
// reduced_solve_rhs2).  Every lane of the warp calls it with the same nseg
// <= 32; lanes with act == false carry identity rows.
template <bool CYCLIC>
__device__ __forceinline__ void reduced_lane_table(double l0, double u0, double l1, double u1,
                                                   int p, int nseg, int W, bool act,
                                                   double* lt) {
    const int pn = (CYCLIC && p == nseg - 1) ? 0 : p + 1;
    double l0n = __shfl_sync(0xffffffffu, l0, pn, W);
    double u0n = __shfl_sync(0xffffffffu, u0, pn, W);
    const bool next = CYCLIC || p + 1 < nseg;
    if (!next) l0n = u0n = 0.0;
    const double ib = rcp_nr(1.0 - l1 * u0 - u1 * l0n);
    double al = act ? -l1 * l0 * ib : 0.0;
    double cl = act ? -u1 * u0n * ib : 0.0;
    if (lt) {
        lt[0] = act ? ib : 0.0;
        lt[1] = act ? l1 : 0.0;
        lt[2] = act && next ? u1 : 0.0;
        lt[3] = act ? l0 : 0.0;
        lt[4] = act ? u0 : 0.0;
    }
    if (CYCLIC && nseg == 1) {
        if (lt) {
            lt[5] = lt[6] = 0.0;
            lt[7] = rcp_nr(1.0 + al + cl);
        }
        return;
    }
    int v = 0;
    for (int dl = 1; dl < nseg; dl <<= 1, ++v) {
        int im = p - dl, ip = p + dl;
        if (CYCLIC) {
            im = im < 0 ? im + nseg : im;
            ip = ip >= nseg ? ip - nseg : ip;
        }
        double lm = __shfl_sync(0xffffffffu, al, im & (W - 1), W);
        double um = __shfl_sync(0xffffffffu, cl, im & (W - 1), W);
        double lp = __shfl_sync(0xffffffffu, al, ip & (W - 1), W);
        double up = __shfl_sync(0xffffffffu, cl, ip & (W - 1), W);
        const bool vm = CYCLIC || im >= 0, vp = CYCLIC || ip < nseg;
        if (!vm) lm = um = 0.0;
        if (!vp) lp = up = 0.0;
        double* lv = lt ? lt + 5 + 3 * v : nullptr;
        if (CYCLIC && 2 * dl == nseg) {
            // the 2x2 closing step: x_p = (r_p - (l + u) r_j) / (1 - (l + u)(l_j + u_j))
            const double si = al + cl;
            if (lv) {
                lv[0] = si;
                lv[1] = 0.0;
                lv[2] = rcp_nr(1.0 - si * (lm + um));
            }
            return;
        }
        const double ibl = rcp_nr(1.0 - al * um - cl * lp);
        if (lv) {
            lv[0] = vm ? al : 0.0;
            lv[1] = vp ? cl : 0.0;
            lv[2] = ibl;
        }
        const double nl = -al * lm * ibl;
        cl = -cl * up * ibl;
        al = nl;
    }
}

// reduced_solve_shfl for a batch whose systems share one matrix, two systems a lane (r0,
// r1 hold the first / last rows' values of both): lt is this lane's table from
// reduced_lane_table (entry k at lt[k * ls]), so only the right-hand sides travel (no
// reciprocals, arithmetic as in reduced_solve_shfl); the table entries are read once for
// both, and the two chains fill each other's latency.
template <bool CYCLIC>
__device__ __forceinline__ void reduced_solve_rhs2(double2 r0, double2 r1, int p, int nseg, int W,
                                                   const double* __restrict__ lt, int ls,
                                                   double& xf0, double& xl0, double& xf1,
                                                   double& xl1) {
    const unsigned FULL = 0xffffffffu;
    const int pn = ((CYCLIC && p == nseg - 1) ? 0 : p + 1) & (W - 1);
    const double na = __shfl_sync(FULL, r0.x, pn, W), nb = __shfl_sync(FULL, r0.y, pn, W);
    double ra, rb;
    {
        const double l1 = lt[1 * ls], u1 = lt[2 * ls], ib = lt[0];
        ra = (r1.x - l1 * r0.x - u1 * na) * ib;
        rb = (r1.y - l1 * r0.y - u1 * nb) * ib;
    }
    if (CYCLIC && nseg == 1) {
        ra *= lt[7 * ls];
        rb *= lt[7 * ls];
    } else {
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            const int dl = 1 << v;
            if (dl >= nseg) break;
            int im = p - dl, ip = p + dl;
            if (CYCLIC) {
                im = im < 0 ? im + nseg : im;
                ip = ip >= nseg ? ip - nseg : ip;
            }
            im &= W - 1;
            ip &= W - 1;
            const double ma = __shfl_sync(FULL, ra, im, W), mb = __shfl_sync(FULL, rb, im, W);
            const double pa = __shfl_sync(FULL, ra, ip, W), pb = __shfl_sync(FULL, rb, ip, W);
            const double l = lt[(5 + 3 * v) * ls], u = lt[(6 + 3 * v) * ls];
            const double ib = lt[(7 + 3 * v) * ls];
            ra = (ra - l * ma - u * pa) * ib;
            rb = (rb - l * mb - u * pb) * ib;
            if (CYCLIC && 2 * dl == nseg) break;
        }
    }
    const int pm = ((CYCLIC && p == 0) ? nseg - 1 : p - 1) & (W - 1);
    double ma = __shfl_sync(FULL, ra, pm, W), mb = __shfl_sync(FULL, rb, pm, W);
    if (!CYCLIC && p == 0) ma = mb = 0.0;
    const double l0 = lt[3 * ls], u0 = lt[4 * ls];
    xl0 = ra;
    xl1 = rb;
    xf0 = r0.x - l0 * ma - u0 * ra;
    xf1 = r0.y - l0 * mb - u0 * rb;
}

}  // namespace btdma

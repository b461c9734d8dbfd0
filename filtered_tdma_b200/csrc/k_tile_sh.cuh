// Tiled sweeps whose systems all share one matrix (heat ADI, channel momentum), for
// up to 32 sub-segments of 16 rows: the scheme of k_tile.cuh's shared-matrix modes
// (factor table, only right-hand sides travel) with two adjacent systems per
// thread.
//
//   * A thread owns sub-segment q of systems 2 p and 2 p + 1: every table entry it
//     reads from shared memory serves both, their D comes as one 16-byte load, and
//     mapped solutions leave as 16-byte stores.  (One system a thread spent 5
//     table loads a row beside its 6 FP64 operations.)
//   * Rows that are contiguous in the destination are stored straight from
//     registers, 32 bytes (four rows) at a time: whole sectors, no staging tile and
//     none of its two block barriers.
//   * The reduced solve takes two systems a lane (reduced_solve_rhs2).
//   * Finite check: an entry that is not finite makes every later one of its
//     back substitution not finite (x_k enters x_{k-1} times a finite factor, and
//     0 x Inf is NaN), so rows 1 and 0 of a sub-segment stand for all.
//
// Measured on B200 (k_tile.cuh's modes before / now): heat sweeps of 256 x 384 x 512, Z
// 339 / 286 us, Y 279 + 14 (its fold) / 185, X 199 / 140; momentum 256^3 209 / 167 for
// the three.  Z reads 2.25 cells a cell from L2, and SH_HEAT spills (120 bytes of stores,
// 156 of loads at 128 registers: both systems' 32 right-hand sides live through the
// stencil); X is at 90 % of the copy bandwidth.
// Wider groups alone did nothing for the old modes (X 199 -> 227 us at 32 systems); rows
// stored with single elements at their misaligned ends took X 250 us; 20 systems a group
// for the 24 sub-segments of Y (240 threads, 160-byte pieces) 195 us.
//
// MODE SH_ROWS   D in the sweep's layout [n_row][n_sys]; optional wall terms on the
//                first and last row (the heat step's fully implicit walls)
//      SH_FIELD  rows read from a ghosted field: boxes of SYS + 2 cells
//      SH_HEAT   the heat Z sweep: a group is 16 x SYS / 16 columns of cells, read in
//                boxes one cell wider on every side, and the right-hand side is
//                formed here from them
#pragma once

#include "btdma_common.cuh"
#include "k_reduced.cuh"
#include "k_tile.cuh"

namespace btdma {

enum ShMode { SH_ROWS = 0, SH_FIELD = 1, SH_HEAT = 2 };
// Stores of a solution: mapped rows in 16-byte pairs of systems, or one by one;
// contiguous rows on 32-byte boundaries, or with the first row of even / odd systems
// 24 / 8 bytes past one (a ghosted field's interior).
enum ShStore { SH_PAIR = 0, SH_ONE = 1, SH_LINE = 2, SH_LINE31 = 3 };

struct ShArgs {
    double* X;
    const double* gtab;  // factor table (tile_table_kernel)
    int n_sys, n_row, nseg, nst, n_groups;
    int xblk, xbs, xss, xrs;  // layout map of x, as TileArgs
    int fblk;                 // SH_FIELD / SH_HEAT: cells of a row of the field
    int pin;                  // SH_FIELD: row 0 of every system is x = 0
    // SH_ROWS walls (wall != 0): the first and last row get wall * ca[s % wblk + 1]
    // * cb[s / wblk + 1].  SH_HEAT: ca, cb, cc = cos(pi x), cos(pi y), cos(pi z).
    double wall;
    int wblk;
    const double *ca, *cb, *cc;
    double bx, by, bz, src;  // SH_HEAT: stencil bases and dt 3 pi^2
    int iy;
    unsigned* status;
};

// Rows per ring stage: 4, or 2 where a stage of heat boxes would leave no ring.
__host__ __device__ constexpr int sh_rps(int mode) { return mode == SH_HEAT ? 2 : 4; }
constexpr int SH_HX = 16;  // SH_HEAT: columns of a group in x
__host__ __device__ __forceinline__ int sh_cells(int sys, int mode) {  // of a row and sub-segment
    return mode == SH_ROWS ? sys
                           : (mode == SH_FIELD ? sys + 2 : (SH_HX + 2) * (sys / SH_HX + 2));
}
__host__ __device__ __forceinline__ int sh_stage_elems(int sys, int nseg, int mode) {
    const int e = sh_cells(sys, mode) * sh_rps(mode) * nseg;
    return (e + 15) / 16 * 16;  // boxes land on 128-byte boundaries
}
__host__ __device__ __forceinline__ int sh_threads(int sys, int nseg) {
    return (sys / 2 * nseg + 31) / 32 * 32;
}
// Ring, tables (rows: {inv, a inv}, pi, {alpha, gamma}; sub-segments: {r, r c0}),
// lane table, reduced rows [2][2][NSEG][SYS + 2] (double buffered), cos(pi
// z), mbarriers.
__host__ __device__ __forceinline__ size_t sh_smem_bytes(int sys, int nseg, int nst, int mode) {
    return sizeof(double) * ((size_t)nst * sh_stage_elems(sys, nseg, mode) +
                             (size_t)nseg * (TILE_MT * 5 + 2) + 32 * TILE_RED_LANE +
                             4ull * nseg * (sys + 2) +
                             (mode == SH_HEAT ? nseg * TILE_MT + 2 : 0)) +
           2ull * nst * sizeof(uint64_t) + 128;
}

__device__ __forceinline__ void st_global_4(double* p, double a, double b, double c, double d) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c),
                 "d"(d)
                 : "memory");
}
template <int SYS, bool CYCLIC, int MODE, int STORE>
__global__ void __launch_bounds__(TILE_MAX_THREADS, 1)
tile_sh_kernel(const __grid_constant__ CUtensorMap tm, const __grid_constant__ ShArgs args) {
    constexpr int M = TILE_MT;
    constexpr int RPS = sh_rps(MODE);
    constexpr int SPG = M / RPS;  // stages per group
    constexpr int NP = SYS / 2;   // pairs of systems
    constexpr int RP = SYS + 2;   // pitch of the reduced rows
    // cells of a box row, and box rows a sub-segment row has
    constexpr int CW = MODE == SH_ROWS ? SYS : (MODE == SH_FIELD ? SYS : SH_HX) + 2;
    constexpr int BY = MODE == SH_HEAT ? SYS / SH_HX + 2 : 1;
    extern __shared__ unsigned char smem_raw[];
    const int nseg = args.nseg, nst = args.nst;
    const int T = sh_threads(SYS, nseg);  // == blockDim.x
    const int W = tile_lanes(nseg);
    const int fstride = nseg * RP;
    const int sstride = sh_stage_elems(SYS, nseg, MODE);

    double* ring = reinterpret_cast<double*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    double2* tf = reinterpret_cast<double2*>(ring + (size_t)nst * sstride);  // {inv, a inv}
    double2* tb = tf + nseg * M;                                             // {alpha, gamma}
    double2* tr = tb + nseg * M;                                             // {r, r c0}
    double* tp = reinterpret_cast<double*>(tr + nseg);                       // pi
    double* lanes = tp + nseg * M;  // lane table [entry][lane]
    double* red = lanes + 32 * TILE_RED_LANE;
    double* czt = red + 4 * fstride;
    uint64_t* full =
        reinterpret_cast<uint64_t*>(czt + (MODE == SH_HEAT ? nseg * M + 2 : 0));
    uint64_t* empty = full + nst;

    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int nwarps = T / 32;
    const bool on = tid < NP * nseg;  // a last warp may be partly filled
    const int q = on ? tid / NP : 0;
    const int s = 2 * (on ? tid % NP : 0);

    if (tid == 0) {
        for (int i = 0; i < nst; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], nwarps);
        }
        fence_mbar_init();
    }
    for (int i = tid; i < nseg * M; i += T) {
        const double* g = args.gtab + (size_t)i * 5;
        tf[i] = make_double2(g[0], g[1]);
        tp[i] = g[2];
        tb[i] = make_double2(g[3], g[4]);
    }
    for (int i = tid; i < nseg; i += T) {
        const double* g = args.gtab + (size_t)args.n_row * 5 + (size_t)i * 6;
        tr[i] = make_double2(g[0], g[1]);
    }
    for (int i = tid; i < 32 * TILE_RED_LANE; i += T)
        lanes[(i % TILE_RED_LANE) * 32 + i / TILE_RED_LANE] =
            args.gtab[tile_red_offset(args.n_row) + i];
    if constexpr (MODE == SH_HEAT)
        for (int i = tid; i < args.n_row + 2; i += T) czt[i] = args.cc[i];
    __syncthreads();

    const int n_my = args.n_groups > (int)blockIdx.x
                         ? (args.n_groups - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x
                         : 0;
    const int total = n_my * SPG;
    const uint32_t stage_bytes = (uint32_t)(sh_cells(SYS, MODE) * RPS * nseg) * sizeof(double);
    auto issue = [&](int t) {  // one thread
        const int slot = t % nst;
        const int g = (int)blockIdx.x + (t / SPG) * (int)gridDim.x;
        const int s0 = g * SYS;
        const int k0 = (t % SPG) * RPS;
        double* dst = ring + (size_t)slot * sstride;
        mbar_expect_tx(&full[slot], stage_bytes);
        if constexpr (MODE == SH_ROWS)
            tma_load_3d(dst, &tm, s0, k0, 0, &full[slot]);
        else if constexpr (MODE == SH_FIELD)  // from the left neighbour (ghosted index ii)
            tma_load_4d(dst, &tm, s0 % args.fblk, s0 / args.fblk + 1, k0, 0, &full[slot]);
        else  // and from the row below
            tma_load_4d(dst, &tm, g % (args.fblk / SH_HX) * SH_HX,
                        g / (args.fblk / SH_HX) * (SYS / SH_HX), k0, 0, &full[slot]);
    };
    bool ok = true;
    if (tid == 0)
        for (int t = 0; t < nst && t < total; ++t) issue(t);

    double nonfinite = 0.0;  // becomes NaN if any solution entry is NaN or Inf
    int slot = 0, pslot = nst - 1;
    uint32_t phase = 0, pphase = 1;
    int t = 0, tw = 0;
    auto wait = [&]() {
        if (ok) ok = mbar_wait_bounded(&full[slot], phase, args.status);
    };
    const unsigned zero = (unsigned)args.n_sys >> 31;
    auto release = [&](unsigned bits) {  // and, one stage later, the slot's refill
        const unsigned z = loads_done(bits, zero);
        if (lane == 0) {
            mbar_arrive(&empty[slot] + z);
            if (t >= 1 && warp == tw && t - 1 + nst < total && ok) {
                ok = mbar_wait_bounded(&empty[pslot], pphase, args.status);
                if (ok) issue(t - 1 + nst);
            }
        }
        pslot = slot;
        pphase = phase;
        ++t;
        if (++tw == nwarps) tw = 0;
        if (++slot == nst) {
            slot = 0;
            phase ^= 1u;
        }
    };
    const double2* qf = tf + q * M;
    const double2* qb = tb + q * M;
    const double* qp = tp + q * M;

    for (int it = 0; it < n_my; ++it) {
        const int g = (int)blockIdx.x + it * (int)gridDim.x;
        int sys = g * SYS + s;  // the pair's first system
        int ii = 0, jj = 0;     // SH_HEAT: its cell
        if constexpr (MODE == SH_HEAT) {
            ii = g % (args.fblk / SH_HX) * SH_HX + s % SH_HX;
            jj = g / (args.fblk / SH_HX) * (SYS / SH_HX) + s / SH_HX;
            sys = jj * args.fblk + ii;
        }
        const bool valid = on && sys < args.n_sys;  // n_sys is even

        // ------------------------------------------------------ forward pass
        double e0[M], e1[M];  // delta of rows 1..M-1, then the solution
        double b0 = 0, b1 = 0, sd0 = 0, sd1 = 0;
        auto feed = [&](int k, double d0, double d1) {
            const double2 f = qf[k];
            if (k == 0) {
                b0 = d0 * f.x;
                b1 = d1 * f.x;
            } else if (k == 1) {
                sd0 = e0[1] = d0 * f.x;
                sd1 = e1[1] = d1 * f.x;
            } else {
                e0[k] = d0 * f.x - f.y * e0[k - 1];
                e1[k] = d1 * f.x - f.y * e1[k - 1];
                if (k <= M - 2) {
                    const double p = qp[k];
                    sd0 += p * e0[k];
                    sd1 += p * e1[k];
                }
            }
        };
        if constexpr (MODE == SH_HEAT) {
            // the 7-point right-hand side (the reference's rhs_kernel and build_lhs_z,
            // apps/heat_gpu/solve_theta.cu:121-202), ghosts computed where they are
            // read: a row is finished when the one above it is read; row 0 takes its
            // lower neighbour in the last stage, row M - 1 its upper one in the first
            // (from the neighbouring sub-segments' rows)
            const int ix = args.fblk;
            const double bx = args.bx, by = args.by, bz = args.bz;
            const double diag = 1.0 + (-2.0 * bx) + (-2.0 * by) + (-2.0 * bz);
            // the source term's x, y factors
            const double so0 = args.src * __ldg(args.ca + ii + 1) * __ldg(args.cb + jj + 1);
            const double so1 = args.src * __ldg(args.ca + ii + 2) * __ldg(args.cb + jj + 1);
            // whether the pair touches an x or y wall
            const bool edge = ii == 0 || ii + 2 == ix || jj == 0 || jj + 1 == args.iy;
            double first0 = 0, first1 = 0, pend0 = 0, pend1 = 0, pc0 = 0, pc1 = 0;
            double up0 = 0, up1 = 0, dn0 = 0, dn1 = 0;
#pragma unroll
            for (int j = 0; j < SPG; ++j) {
                wait();
                // box [sub-segment][row][y][x]: this pair's cells, y = 1 + s / 16
                const double* sb =
                    ring + (size_t)slot * sstride + (s / SH_HX + 1) * CW + s % SH_HX + 1;
                if (j == 0 && q + 1 < nseg) {
                    const double* p = sb + (q + 1) * RPS * BY * CW;
                    up0 = p[0];
                    up1 = p[1];
                }
                if (j == SPG - 1 && q > 0) {
                    const double* p = sb + ((q - 1) * RPS + RPS - 1) * BY * CW;
                    dn0 = p[0];
                    dn1 = p[1];
                }
                unsigned bits = 0;
                double tl[RPS], t0[RPS], t1[RPS], tr_[RPS], m0[RPS], m1[RPS], p0[RPS], p1[RPS];
#pragma unroll
                for (int r = 0; r < RPS; ++r) {
                    const double* p = sb + (q * RPS + r) * BY * CW;
                    tl[r] = p[-1];
                    t0[r] = p[0];
                    t1[r] = p[1];
                    tr_[r] = p[2];
                    m0[r] = p[-CW];
                    m1[r] = p[1 - CW];
                    p0[r] = p[CW];
                    p1[r] = p[1 + CW];
                    bits ^= word_of(tl[r]) ^ word_of(t0[r]) ^ word_of(t1[r]) ^ word_of(tr_[r]) ^
                            word_of(m0[r]) ^ word_of(m1[r]) ^ word_of(p0[r]) ^ word_of(p1[r]);
                }
                release(bits ^ word_of(up0) ^ word_of(up1) ^ word_of(dn0) ^ word_of(dn1));
#pragma unroll
                for (int r = 0; r < RPS; ++r) {
                    const int k = j * RPS + r;
                    const double cz = czt[q * M + k + 1];
                    const double a0 = t0[r], a1 = t1[r];
                    double lf = tl[r], rt = tr_[r];
                    double ya = m0[r], yb = m1[r], yc = p0[r], yd = p1[r];
                    if (edge) {  // ghosts of the x and y walls: 2 u - theta
                        const double c2 = -2.0 * cz, cy = __ldg(args.cb + jj + 1);
                        const double u0 = c2 * __ldg(args.ca + ii + 1);
                        const double u1 = c2 * __ldg(args.ca + ii + 2);
                        if (ii == 0) lf = c2 * cy - a0;
                        if (ii + 2 == ix) rt = c2 * cy - a1;
                        if (jj == 0) {
                            ya = u0 - a0;
                            yb = u1 - a1;
                        }
                        if (jj + 1 == args.iy) {
                            yc = u0 - a0;
                            yd = u1 - a1;
                        }
                    }
                    double v0 = (bx * a1 + bx * lf) + (by * yc + by * ya) + diag * a0 + so0 * cz;
                    double v1 = (bx * rt + bx * a0) + (by * yd + by * yb) + diag * a1 + so1 * cz;
                    if ((k == 0 && q == 0) || (k == M - 1 && q == nseg - 1)) {
                        // z walls: the ghost, and base * (ghost + cell) of the implicit fold
                        const double c2 = -2.0 * __ldg(args.cb + jj + 1);
                        const double g0 = c2 * __ldg(args.ca + ii + 1) - a0;
                        const double g1 = c2 * __ldg(args.ca + ii + 2) - a1;
                        v0 += bz * g0 + bz * (g0 + a0);
                        v1 += bz * g1 + bz * (g1 + a1);
                    }
                    if (k >= 1) {  // lower neighbour: the previous row
                        v0 += bz * pc0;
                        v1 += bz * pc1;
                    }
                    if (k == 0) {
                        first0 = v0;
                        first1 = v1;
                    } else {
                        if (k == 1) {  // row 0's upper neighbour
                            first0 += bz * a0;
                            first1 += bz * a1;
                        } else {
                            feed(k - 1, pend0 + bz * a0, pend1 + bz * a1);
                        }
                        pend0 = v0;
                        pend1 = v1;
                    }
                    pc0 = a0;
                    pc1 = a1;
                }
            }
            const bool top = q == nseg - 1, bot = q == 0;
            feed(M - 1, top ? pend0 : pend0 + bz * up0, top ? pend1 : pend1 + bz * up1);
            feed(0, bot ? first0 : first0 + bz * dn0, bot ? first1 : first1 + bz * dn1);
        } else {
            double w0 = 0, w1 = 0;  // wall terms of the first and last row
            if (MODE == SH_ROWS && args.wall != 0.0 && valid && (q == 0 || q == nseg - 1)) {
                const double cbv = args.wall * __ldg(args.cb + sys / args.wblk + 1);
                const int a = sys % args.wblk + 1;
                w0 = cbv * __ldg(args.ca + a);
                w1 = cbv * __ldg(args.ca + a + 1);
            }
#pragma unroll
            for (int j = 0; j < SPG; ++j) {
                wait();
                const double* sb = ring + (size_t)slot * sstride + (size_t)q * RPS * CW + s;
                double d0[RPS], d1[RPS];
                unsigned bits = 0;
#pragma unroll
                for (int r = 0; r < RPS; ++r) {
                    if constexpr (MODE == SH_ROWS) {
                        const double2 v = *reinterpret_cast<const double2*>(sb + r * CW);
                        d0[r] = v.x;
                        d1[r] = v.y;
                    } else {  // x = system + 1
                        d0[r] = sb[r * CW + 1];
                        d1[r] = sb[r * CW + 2];
                    }
                    bits ^= word_of(d0[r]) ^ word_of(d1[r]);
                }
                release(bits);
#pragma unroll
                for (int r = 0; r < RPS; ++r) {
                    const int k = j * RPS + r;
                    if (MODE == SH_ROWS && ((k == 0 && q == 0) || (k == M - 1 && q == nseg - 1))) {
                        d0[r] += w0;
                        d1[r] += w1;
                    }
                    if (MODE == SH_FIELD && k == 0 && args.pin != 0 && q == 0) d0[r] = d1[r] = 0.0;
                    feed(k, d0[r], d1[r]);
                }
            }
        }
        // double buffered: a slower warp may still read the last group's edge rows
        double* const rg = red + (it & 1) * 2 * fstride;
        if (on) {
            const double2 f = tr[q];
            double2* w = reinterpret_cast<double2*>(rg + q * RP + s);
            w[0] = make_double2(f.x * b0 - f.y * sd0, f.x * b1 - f.y * sd1);
            w[fstride / 2] = make_double2(e0[M - 1], e1[M - 1]);
        }
        __syncthreads();

        // ------------------------------------------------ reduced system
        {
            const int per_pass = T / W;  // pairs of systems per pass
            const int p = tid % W;
            for (int base = 0; base < NP; base += per_pass) {
                const int sp = base + tid / W;
                const bool act = sp < NP && p < nseg;
                double2* src = reinterpret_cast<double2*>(rg + p * RP + 2 * (act ? sp : 0));
                double2 ra = make_double2(0, 0), rb = ra;
                if (act) {
                    ra = src[0];
                    rb = src[fstride / 2];
                }
                double xf0, xl0, xf1, xl1;
                reduced_solve_rhs2<CYCLIC>(ra, rb, p, nseg, W, lanes + p, 32, xf0, xl0, xf1, xl1);
                if (act) {  // over the rows this thread has read
                    src[0] = make_double2(xf0, xf1);
                    src[fstride / 2] = make_double2(xl0, xl1);
                }
            }
        }
        __syncthreads();

        // --------------------------------------------------- back substitution
        {
            const double2* src = reinterpret_cast<const double2*>(rg + q * RP + s);
            const double2 xf = src[0], xl = src[fstride / 2];
            e0[M - 1] = xl.x;
            e1[M - 1] = xl.y;
#pragma unroll
            for (int k = M - 2; k >= 1; --k) {
                const double2 f = qb[k];
                e0[k] = e0[k] - f.x * xf.x - f.y * e0[k + 1];
                e1[k] = e1[k] - f.x * xf.y - f.y * e1[k + 1];
            }
            e0[0] = xf.x;
            e1[0] = xf.y;
            if (valid) {
                nonfinite = fma(e0[0], 0.0, fma(e1[0], 0.0, nonfinite));
                nonfinite = fma(e0[1], 0.0, fma(e1[1], 0.0, nonfinite));
                double* xp = args.X + (ptrdiff_t)(sys / args.xblk) * (ptrdiff_t)args.xbs +
                             (ptrdiff_t)(sys % args.xblk) * (ptrdiff_t)args.xss +
                             (ptrdiff_t)(q * M) * (ptrdiff_t)args.xrs;
                if constexpr (STORE == SH_LINE) {
#pragma unroll
                    for (int k = 0; k < M; k += 4) {
                        st_global_4(xp + k, e0[k], e0[k + 1], e0[k + 2], e0[k + 3]);
                        st_global_4(xp + args.xss + k, e1[k], e1[k + 1], e1[k + 2], e1[k + 3]);
                    }
                } else if constexpr (STORE == SH_LINE31) {
                    // even systems: rows 1..16, row 16 the next sub-segment's first; odd
                    // ones: rows -1..14, row -1 the previous sub-segment's last
                    const bool top = q + 1 == nseg;
                    const double nx = top ? 0.0 : src[RP / 2].x;
                    const double pv = q == 0 ? 0.0 : src[fstride / 2 - RP / 2].y;
                    if (q == 0) xp[0] = e0[0];
#pragma unroll
                    for (int k = 1; k + 4 < M; k += 4)
                        st_global_4(xp + k, e0[k], e0[k + 1], e0[k + 2], e0[k + 3]);
                    if (!top) {
                        st_global_4(xp + M - 3, e0[M - 3], e0[M - 2], e0[M - 1], nx);
                    } else {
#pragma unroll
                        for (int k = M - 3; k < M; ++k) xp[k] = e0[k];
                    }
                    xp += args.xss;
                    if (q != 0) {
                        st_global_4(xp - 1, pv, e1[0], e1[1], e1[2]);
                    } else {
#pragma unroll
                        for (int k = 0; k < 3; ++k) xp[k] = e1[k];
                    }
#pragma unroll
                    for (int k = 3; k + 4 < M; k += 4)
                        st_global_4(xp + k, e1[k], e1[k + 1], e1[k + 2], e1[k + 3]);
                    if (top) xp[M - 1] = e1[M - 1];
                } else {
#pragma unroll
                    for (int k = 0; k < M; ++k) {
                        if constexpr (STORE == SH_PAIR) {
                            *reinterpret_cast<double2*>(xp) = make_double2(e0[k], e1[k]);
                        } else {
                            xp[0] = e0[k];
                            xp[args.xss] = e1[k];
                        }
                        xp += args.xrs;
                    }
                }
            }
        }
    }
    if (nonfinite != 0.0) raise_status(args.status, ST_NONFINITE);  // NaN != 0
    if (!ok && tid == 0)  // a wait gave up: in-flight copies get a bounded chance to land
        for (int i = 0; i < nst; ++i) mbar_wait_bounded(&full[i], 0, nullptr, 1u << 8);
}

}  // namespace btdma

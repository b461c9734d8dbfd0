// Wall-normal solve of the channel flow's FFT Poisson equation: one thread solves the
// real and the imaginary part of a mode's sub-segment, whose matrix (generated from
// the row tables and the mode's shift) is eliminated once for both.
//
// The working set is a few tens of MB (in L2), so the time is latency: rounds of
// (load, row recurrences, reduced system, back substitution) per SM.  Hence groups of
// NP modes that fill 256 threads (a part's 16 rows of state twice fill 239 registers),
// sized so that the rounds come out even, and each group's rows in one TMA box, the
// next group's already on its way (two buffers).  The general tiled kernel treated the
// parts as separate systems: every matrix twice, four rounds instead of three.
// Measured on B200 (with the 10 us copy of the right-hand side before it): 128 x 128 x
// 192 40 -> 25 us, 186 x 98 x 272 72 -> 42 us.  Sub-segments of 8 rows, two CTAs a SM,
// took 29.5 us, and lost accuracy (1.1e-12 against 4e-13) to the longer reduced system.
//
// Per mode m and row k:  a_k x_{k-1} - (a_k + c_k + lambda_m) x_k + c_k x_{k+1} = d_k
// (mode 0's row 0 pinned to 0 when asked).  Elimination and reduced system are those
// of k_tile.cuh / reduced_solve_shfl.
#pragma once

#include "btdma_common.cuh"
#include "k_reduced.cuh"
#include "k_tile.cuh"

namespace btdma {

constexpr int POIS_THREADS = 256;

struct PoisArgs {
    double* X;  // complex [nz][n_modes]
    const double* ga;
    const double* gc;
    const double* lam;
    int nz, n_modes, pin;
    int np, nseg, n_groups;  // modes a group, sub-segments, groups
    unsigned* status;
};

// Two boxes [NSEG][M][2 NP], reduced rows [8][NSEG][NP + 1], row tables {a, c}.
__host__ __device__ __forceinline__ size_t pois_box_elems(int np, int nz) {
    return ((size_t)2 * np * nz + 15) / 16 * 16;
}
__host__ __device__ __forceinline__ size_t pois_smem_bytes(int np, int nseg, int nz) {
    return sizeof(double) *
               (2 * pois_box_elems(np, nz) + 8ull * nseg * (np + 1) + 2ull * nz + 2) +
           2 * sizeof(uint64_t) + 128;
}

// reduced_solve_shfl (not periodic) for two right-hand sides of one matrix.
__device__ __forceinline__ void reduced_solve_pair(double l0, double u0, double l1, double u1,
                                                   double2 r0, double2 r1, int p, int nseg, int W,
                                                   bool act, double2& xf, double2& xl) {
    const unsigned FULL = 0xffffffffu;
    const int pn = (p + 1) & (W - 1);
    double l0n = __shfl_sync(FULL, l0, pn, W), u0n = __shfl_sync(FULL, u0, pn, W);
    double na = __shfl_sync(FULL, r0.x, pn, W), nb = __shfl_sync(FULL, r0.y, pn, W);
    if (p + 1 >= nseg) l0n = u0n = na = nb = 0.0;
    const double ib = rcp_nr(1.0 - l1 * u0 - u1 * l0n);
    double al = -l1 * l0 * ib, cl = -u1 * u0n * ib;
    double da = (r1.x - l1 * r0.x - u1 * na) * ib, db = (r1.y - l1 * r0.y - u1 * nb) * ib;
    if (!act) al = cl = da = db = 0.0;
    for (int dl = 1; dl < nseg; dl <<= 1) {
        const bool vm = p - dl >= 0, vp = p + dl < nseg;
        const int im = (p - dl) & (W - 1), ip = (p + dl) & (W - 1);
        double lm = __shfl_sync(FULL, al, im, W), um = __shfl_sync(FULL, cl, im, W);
        double ma = __shfl_sync(FULL, da, im, W), mb = __shfl_sync(FULL, db, im, W);
        double lp = __shfl_sync(FULL, al, ip, W), up = __shfl_sync(FULL, cl, ip, W);
        double pa = __shfl_sync(FULL, da, ip, W), pb = __shfl_sync(FULL, db, ip, W);
        if (!vm) lm = um = ma = mb = 0.0;
        if (!vp) lp = up = pa = pb = 0.0;
        const double ibl = rcp_nr(1.0 - al * um - cl * lp);
        da = (da - al * ma - cl * pa) * ibl;
        db = (db - al * mb - cl * pb) * ibl;
        const double nl = -al * lm * ibl;
        cl = -cl * up * ibl;
        al = nl;
    }
    const int pm = (p - 1) & (W - 1);
    double ma = __shfl_sync(FULL, da, pm, W), mb = __shfl_sync(FULL, db, pm, W);
    if (p == 0) ma = mb = 0.0;
    xl = make_double2(da, db);
    xf = make_double2(r0.x - l0 * ma - u0 * da, r0.y - l0 * mb - u0 * db);
}

__global__ void __launch_bounds__(POIS_THREADS, 1)
poisson_kernel(const __grid_constant__ CUtensorMap tm, const PoisArgs args) {
    constexpr int M = TILE_MT;
    extern __shared__ unsigned char smem_raw[];
    const int np = args.np, nseg = args.nseg, nz = args.nz;
    const int T = blockDim.x;
    const int W = tile_lanes(nseg);
    const int RP = np + 1, fstride = nseg * RP;
    const int box = (int)pois_box_elems(np, nz);
    double* buf = reinterpret_cast<double*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    double2* tab = reinterpret_cast<double2*>(buf + 2 * (size_t)box);  // {a, c} a row
    double* red = reinterpret_cast<double*>(tab + nz + 1);
    uint64_t* full = reinterpret_cast<uint64_t*>(red + 8 * fstride);
    const int tid = threadIdx.x;
    const bool on = tid < np * nseg;
    const int q = on ? tid / np : 0;
    const int m = on ? tid - q * np : 0;

    if (tid == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        fence_mbar_init();
    }
    for (int i = tid; i < nz; i += T) tab[i] = make_double2(args.ga[i], args.gc[i]);
    __syncthreads();
    const int n_my = args.n_groups > (int)blockIdx.x
                         ? (args.n_groups - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x
                         : 0;
    auto issue = [&](int it) {  // one thread
        const int g = (int)blockIdx.x + it * (int)gridDim.x;
        mbar_expect_tx(&full[it & 1], (uint32_t)(2 * np * nz) * sizeof(double));
        tma_load_3d(buf + (size_t)(it & 1) * box, &tm, g * 2 * np, 0, 0, &full[it & 1]);
    };
    bool ok = true;
    if (tid == 0)
        for (int it = 0; it < 2 && it < n_my; ++it) issue(it);

    double nonfinite = 0.0;
    for (int it = 0; it < n_my; ++it) {
        const int mode = ((int)blockIdx.x + it * (int)gridDim.x) * np + m;
        const bool valid = on && mode < args.n_modes;
        const double lam = valid ? __ldg(args.lam + mode) : 0.0;
        if (ok) ok = mbar_wait_bounded(&full[it & 1], (it >> 1) & 1, args.status);

        // ------------------------------------------------------ forward pass
        double al[M], ga[M], e0[M], e1[M];  // rows 1..M-1 used
        {
            const double2* d = reinterpret_cast<const double2*>(buf + (size_t)(it & 1) * box) +
                               (size_t)q * M * np + m;
            double ab0 = 0, cb0 = 0, pi = 1.0, sa = 0, s0 = 0, s1 = 0;
            double2 b0 = make_double2(0, 0);
#pragma unroll
            for (int k = 0; k < M; ++k) {
                const double2 t = tab[q * M + k];
                double2 v = d[k * np];
                double a = t.x, c = t.y, b = -(t.x + t.y) - lam;
                if (k == 0) {
                    if (args.pin != 0 && q == 0 && mode == 0) {
                        a = c = v.x = v.y = 0.0;
                        b = 1.0;
                    }
                    const double ib = rcp_nr(b);
                    ab0 = a * ib;
                    cb0 = c * ib;
                    b0 = make_double2(v.x * ib, v.y * ib);
                } else if (k == 1) {
                    const double ib = rcp_nr(b);
                    sa = al[1] = a * ib;
                    ga[1] = c * ib;
                    s0 = e0[1] = v.x * ib;
                    s1 = e1[1] = v.y * ib;
                } else {
                    const double inv = rcp_nr(b - a * ga[k - 1]);
                    ga[k] = c * inv;
                    al[k] = -a * al[k - 1] * inv;
                    e0[k] = (v.x - a * e0[k - 1]) * inv;
                    e1[k] = (v.y - a * e1[k - 1]) * inv;
                    if (k <= M - 2) {
                        pi = -ga[k - 1] * pi;
                        sa += pi * al[k];
                        s0 += pi * e0[k];
                        s1 += pi * e1[k];
                    }
                }
            }
            const double r = rcp_nr(1.0 - cb0 * sa);
            if (on) {
                double* w = red + q * RP + m;
                w[0 * fstride] = r * ab0;
                w[1 * fstride] = r * cb0 * (-ga[M - 2] * pi);
                w[2 * fstride] = al[M - 1];
                w[3 * fstride] = ga[M - 1];
                w[4 * fstride] = r * (b0.x - cb0 * s0);
                w[5 * fstride] = r * (b0.y - cb0 * s1);
                w[6 * fstride] = e0[M - 1];
                w[7 * fstride] = e1[M - 1];
            }
        }
        __syncthreads();  // every row of the box has been used
        if (tid == 0 && it + 2 < n_my && ok) issue(it + 2);

        // ------------------------------------------------ reduced system
        {
            const int per_pass = T / W;
            const int p = tid % W;
            for (int base = 0; base < np; base += per_pass) {
                const int sp = base + tid / W;
                const bool act = sp < np && p < nseg;
                double* src = red + (act ? p * RP + sp : 0);
                double l0 = 0, u0 = 0, l1 = 0, u1 = 0;
                double2 r0 = make_double2(0, 0), r1 = r0;
                if (act) {
                    l0 = src[0 * fstride];
                    u0 = src[1 * fstride];
                    l1 = src[2 * fstride];
                    u1 = src[3 * fstride];
                    r0 = make_double2(src[4 * fstride], src[5 * fstride]);
                    r1 = make_double2(src[6 * fstride], src[7 * fstride]);
                }
                double2 xf, xl;
                reduced_solve_pair(l0, u0, l1, u1, r0, r1, p, nseg, W, act, xf, xl);
                if (act) {
                    src[4 * fstride] = xf.x;
                    src[5 * fstride] = xf.y;
                    src[6 * fstride] = xl.x;
                    src[7 * fstride] = xl.y;
                }
            }
        }
        __syncthreads();

        // --------------------------------------------------- back substitution
        {
            const double* src = red + q * RP + m;
            const double2 xf = make_double2(src[4 * fstride], src[5 * fstride]);
            double2 x = make_double2(src[6 * fstride], src[7 * fstride]);
            if (valid) {
                const size_t row = (size_t)args.n_modes;
                double2* xp = reinterpret_cast<double2*>(args.X) + (size_t)(q * M + M - 1) * row +
                              mode;
                *xp = x;
#pragma unroll
                for (int k = M - 2; k >= 1; --k) {
                    x.x = e0[k] - al[k] * xf.x - ga[k] * x.x;
                    x.y = e1[k] - al[k] * xf.y - ga[k] * x.y;
                    xp -= row;
                    *xp = x;
                }
                // a row that is not finite makes every later one so: row 1 stands for all
                nonfinite = fma(x.x, 0.0, fma(x.y, 0.0, nonfinite));
                nonfinite = fma(xf.x, 0.0, fma(xf.y, 0.0, nonfinite));
                xp -= row;
                *xp = xf;
            }
        }
    }
    if (nonfinite != 0.0) raise_status(args.status, ST_NONFINITE);  // NaN != 0
    if (!ok && tid == 0)
        for (int i = 0; i < 2; ++i) mbar_wait_bounded(&full[i], 0, nullptr, 1u << 8);
}

}  // namespace btdma

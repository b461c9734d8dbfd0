// The wide solve (k_tile_wide.cuh) for periodic FP64 systems of any length: those
// whose rows are not 32 x a power of two, which the wide kernel's identity rows
// would cut open.  Sub-segment length and systems per CTA are chosen at run time.
//
//   rows      ASYNC = false: sub-segments of m <= 32 rows, the last one shorter
//             (a tensor map and a TMA box of its own); the ring is that of
//             k_tile_wide.cuh, the boxes of a stage issued by eight lanes.
//             ASYNC = true (FP64): sub-segments of floor / ceil(n_row / NSEG)
//             rows; each thread copies its own rows (cp.async, 8 bytes) into its
//             own column of the ring, so neither the row stride nor the row
//             count has to suit a tensor map (odd n_sys), and no barrier guards
//             the ring: a refill waits for the thread's own loads only.  (One
//             cp.async.bulk per row piece instead, which wants no map either, was
//             measured at 50 cycles a piece: 262144 x 512 in 2.9 ms against 1.1 ms.)
//   cluster   as in k_tile_wide.cuh.
//
// Needs NSC <= 16 sub-segments of 3 to 32 rows per CTA, in one CTA a power of two.
// The TMA form needs an even n_sys and 16-byte aligned arrays.
// Measured on B200 (us, segment kernels / now): TMA 65536 x 192 176 / 105, 48268 x 85
// 83 / 46, 20000 x 700 818 / 199; cp.async 48269 x 85 141 / 60, 4589 x 1537 3813 / 119
// (P = 4, and 16 above 250 rows).  Every form spills (248 to 400 bytes of stores at 128
// registers: run-time lengths keep both ends of every row block alive).
#pragma once

#include <cooperative_groups.h>

#include "btdma_common.cuh"
#include "k_reduced.cuh"
#include "k_tile_wide.cuh"

namespace btdma {

constexpr int ANY_ASYNC_NST = 6;  // ring stages of the cp.async form

// Tensor maps of A, B, C, D: boxes of NSC sub-segments, of NSC - 1, and of the
// last sub-segment when it is shorter than the others.
struct AnyMaps {
    CUtensorMap full[4], less[4], tail[4];
};

struct AnyArgs {
    const double* in[4];  // A, B, C, D (read through them by the cp.async form)
    double* X;
    int n_sys, n_row;
    int sys;       // systems per CTA, a multiple of 16
    int nsc, cl;   // sub-segments per CTA, CTAs per system
    int m;         // rows of a sub-segment (the longest)
    int nst;       // ring stages
    int n_groups;  // groups of sys systems
    unsigned* status;
};

// Threads of a CTA: whole warps.
__host__ __device__ __forceinline__ int any_threads(int sys, int nsc) {
    return (sys * nsc + 31) / 32 * 32;
}
// Shared memory: ring, reduced rows [6][NSC][SYS + 1], published rows [2][6][SYS]
// and outer unknowns [2][SYS] (clusters), mbarriers, the tensor-memory address.
__host__ __device__ __forceinline__ size_t any_smem_bytes(int sys, int nsc, int cl, int nst,
                                                          int elem) {
    const size_t t = any_threads(sys, nsc);
    return (size_t)nst * 4 * tile_rps(elem) * t * elem + 6ull * nsc * (sys + 1) * sizeof(double) +
           (cl > 1 ? 14ull * sys * sizeof(double) : 0) + (2ull * nst + 2) * sizeof(uint64_t) + 16 +
           128;
}

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// Running state of one sub-segment's forward pass (row 0, scaled by its pivot, waits
// in the thread's own slot of the reduced rows).
struct AnyFwd {
    double pi, sa, sd;     // running products of the reduced first row
    double alp, gap, dep;  // alpha, gamma, delta of the previous row
};

// Row k of a sub-segment (wide_row with a run-time length; any k >= 2 stands for
// the rest): `inner` unless it is the last row; pi ends as pi_{length - 1}.  Reciprocals
// are correctly rounded, so that pivots of the whole FP64 range are served, as these
// shapes always were (rcp_nr: 48268 x 85 44.2 us against 45.6, 4589 x 1537 114 / 119;
// the wide kernel's watched pass spilled twice as much here and took 49 / 122).
__device__ __forceinline__ void any_row(AnyFwd& f, int k, bool inner, double a, double b,
                                        double cc, double d, bool on, double* w, int fstride) {
    if (k == 0) {
        const double ib = Exact64::rcp(b);
        if (on) {
            w[0 * fstride] = a * ib;
            w[1 * fstride] = cc * ib;
            w[2 * fstride] = d * ib;
        }
    } else if (k == 1) {
        const double ib = Exact64::rcp(b);
        f.alp = a * ib;
        f.gap = cc * ib;
        f.dep = d * ib;
        f.pi = 1.0;
        f.sa = f.alp;
        f.sd = f.dep;
    } else {
        const double inv = Exact64::rcp(b - a * f.gap);
        const double g = cc * inv;
        const double e = (d - a * f.dep) * inv;
        const double l = -a * f.alp * inv;
        f.pi = -f.gap * f.pi;
        if (inner) {
            f.sa += f.pi * l;
            f.sd += f.pi * e;
        }
        f.alp = l;
        f.gap = g;
        f.dep = e;
    }
}

template <bool ASYNC, bool CLUSTER>
__global__ void __launch_bounds__(TILE_MAX_THREADS, 1)
tile_any_kernel(const __grid_constant__ AnyMaps maps, const __grid_constant__ AnyArgs args) {
    namespace cg = cooperative_groups;
    using TIN = double;
    constexpr int TR = WIDE_TROWS, M = WIDE_M;
    constexpr int RPS = tile_rps((int)sizeof(TIN));
    extern __shared__ unsigned char smem_raw[];
    const int S = args.sys, nsc = args.nsc, nst = ASYNC ? ANY_ASYNC_NST : args.nst;
    const int cl = CLUSTER ? args.cl : 1;
    const int T = any_threads(S, nsc);    // == blockDim.x
    const int cols = ASYNC ? T : S * nsc;  // columns of a ring stage
    const int W = tile_lanes(nsc);
    const int RP = S + 1;
    const int fstride = nsc * RP;
    const int m = args.m;
    const int spg = (m + RPS - 1) / RPS;  // stages per group
    const int sstride = 4 * RPS * cols;   // elements per stage

    TIN* ring = reinterpret_cast<TIN*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    double* red = reinterpret_cast<double*>(ring + (size_t)nst * sstride);
    double* pub = red + 6 * fstride;               // [2][6][S]
    double* outer = pub + (CLUSTER ? 12 * S : 0);  // [2][S]
    uint64_t* full = reinterpret_cast<uint64_t*>(outer + (CLUSTER ? 2 * S : 0));
    uint64_t* empty = full + nst;
    uint64_t* xbar = empty + nst;  // [2]: the peers' published rows of a group
    uint32_t* tslot = reinterpret_cast<uint32_t*>(xbar + 2);

    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int nwarps = T / 32;
    const bool on = tid < S * nsc;  // a last warp may be partly filled
    const int q = on ? tid / S : 0;
    const int s = on ? tid - q * S : 0;
    const int c = CLUSTER ? (int)cg::this_cluster().block_rank() : 0;
    const int cid = CLUSTER ? (int)blockIdx.x / cl : (int)blockIdx.x;
    const int ncid = CLUSTER ? (int)gridDim.x / cl : (int)gridDim.x;
    const size_t ns = (size_t)args.n_sys;
    const unsigned zero = (unsigned)args.n_sys >> 31;  // see loads_done
    // this thread's rows of every system it takes
    int r0, mlen;
    if constexpr (ASYNC) {
        seg_range(args.n_row, nsc * cl, c * nsc + q, r0, mlen);
    } else {
        r0 = (c * nsc + q) * m;
        mlen = min(m, args.n_row - r0);
    }
    const int wlo = __reduce_min_sync(0xffffffffu, mlen);  // rows every lane of the warp has

    if (tid == 0) {
        for (int i = 0; i < nst; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], nwarps);
        }
        mbar_init(&xbar[0], cl);
        mbar_init(&xbar[1], cl);
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(tslot, (uint32_t)wide_tmem_cols(nwarps));
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if constexpr (CLUSTER) tile_cluster_sync(cl);  // the peers' mbarriers are ready
    const uint32_t tcol = *static_cast<volatile uint32_t*>(tslot) + ((uint32_t)(warp & 3) << 21) +
                          (uint32_t)(warp >> 2) * WIDE_TCOLS;

    const int n_my = args.n_groups > cid ? (args.n_groups - cid + ncid - 1) / ncid : 0;
    const int total = n_my * spg;

    // TMA form, stage t by one warp: lanes 0..3 the boxes of A, B, C, D, lanes 4..7
    // those of a shorter last sub-segment
    auto issue = [&](int t, int islot) {
        const int it = t / spg;
        const int k0 = (t - it * spg) * RPS;
        const int f = lane & 3;
        const bool tailed = (c + 1) * nsc * m > args.n_row;
        if (lane == 0) mbar_expect_tx(&full[islot], (uint32_t)sstride * sizeof(TIN));
        __syncwarp();
        if (lane < 4 ? !tailed || nsc > 1 : tailed && lane < 8) {
            const bool tl = lane >= 4;
            const CUtensorMap* mp =
                tl ? &maps.tail[f] : (tailed ? &maps.less[f] : &maps.full[f]);
            TIN* dst = ring + (size_t)islot * sstride + (f * cols + (tl ? S * (nsc - 1) : 0)) * RPS;
            tma_load_3d(dst, mp, (cid + it * ncid) * S, k0, tl ? 0 : c * nsc, &full[islot]);
        }
    };
    // cp.async form, every thread for its own rows: the next stage to request (group ig,
    // row ik of the sub-segment) into its column at dst
    int ig = 0, ik = 0;
    auto request = [&](TIN* dst) {
        if (ig < n_my) {
            const int isys = (cid + ig * ncid) * S + s;
            if (on && isys < args.n_sys) {
                const size_t o = (size_t)(r0 + ik) * ns + isys;
#pragma unroll
                for (int r = 0; r < RPS; ++r) {
                    if (ik + r < mlen) {
#pragma unroll
                        for (int f = 0; f < 4; ++f)
                            cp_async8(dst + (f * RPS + r) * cols, args.in[f] + o + r * ns);
                    }
                }
            }
            ik += RPS;
            if (ik >= m) {
                ik = 0;
                ++ig;
            }
        }
        cp_async_commit();
    };
    bool ok = true;
    if constexpr (ASYNC) {
        for (int t = 0; t < ANY_ASYNC_NST - 1; ++t) request(ring + (size_t)t * sstride + tid);
    } else if (warp == 0) {
        for (int t = 0; t < nst && t < total; ++t) issue(t, t);
    }

    const int toff = ASYNC ? tid : q * RPS * S + s;
    const int rstep = ASYNC ? cols : S;  // between the rows of a stage
    TIN* st = ring + toff;
    // cp.async form: this thread's column of the slot read one stage ago.  The values
    // read there are taken into the address, so that the copies into it are issued
    // after those loads have completed (see loads_done; a thread's own loads suffice,
    // nobody else reads its column).
    TIN* pst = st + (size_t)(nst - 1) * sstride;
    int slot = 0;
    uint32_t phase = 0;
    int t = 0;
    auto fetch = [&](double (&a2)[RPS], double (&b2)[RPS], double (&c2)[RPS], double (&d2)[RPS]) {
        if constexpr (ASYNC)
            cp_async_wait<ANY_ASYNC_NST - 2>();
        else if (ok)
            ok = mbar_wait_bounded_spin(&full[slot], phase, args.status);
        unsigned bits = 0;
#pragma unroll
        for (int r = 0; r < RPS; ++r) {
            a2[r] = st[0 * RPS * cols + r * rstep];
            b2[r] = st[1 * RPS * cols + r * rstep];
            c2[r] = st[2 * RPS * cols + r * rstep];
            d2[r] = st[3 * RPS * cols + r * rstep];
            bits ^= word_of(a2[r]) ^ word_of(b2[r]) ^ word_of(c2[r]) ^ word_of(d2[r]);
        }
        if constexpr (ASYNC) {
            request(pst);
            pst = st + (bits & zero);
        } else {
            const unsigned z = loads_done(bits, zero);
            if (lane == 0) mbar_arrive(&empty[slot] + z);
            // one stage later the warp whose turn it is refills the slot of stage
            // t - 1 with stage t - 1 + nst, once every warp has released it
            const int ps = slot == 0 ? nst - 1 : slot - 1;
            if (warp == (nwarps >= nst ? ps : ps % nwarps) && t >= 1 && t - 1 + nst < total) {
                if (ok)
                    ok = mbar_wait_bounded_spin(&empty[ps], slot == 0 ? phase ^ 1u : phase,
                                                args.status);
                if (ok) issue(t - 1 + nst, ps);
            }
            ++t;
        }
        st += sstride;
        if (++slot == nst) {
            slot = 0;
            phase ^= 1u;
            st = ring + toff;
        }
    };

    double nonfinite = 0.0;
    for (int it = 0; it < n_my; ++it) {
        const int g = cid + it * ncid;
        const int sys = g * S + s;
        const bool valid = on && sys < args.n_sys;

        // ------------------------------------------------------ forward pass
        double al[M - TR], ga[M - TR], de[M - TR];  // rows TR .. M - 1
        {
            AnyFwd f = {};
            double ta[4], tg[4], td[4];  // a 4-row block
            // rows kb .. kb + 3 (first: kb = 0); whole: every lane has them and the
            // row after
            auto block = [&](int kb, bool first, bool whole) {
#pragma unroll
                for (int j = 0; j < 4 / RPS; ++j) {
                    if (whole || kb + j * RPS < m) {
                        double a2[RPS], b2[RPS], c2[RPS], d2[RPS];
                        fetch(a2, b2, c2, d2);
#pragma unroll
                        for (int r = 0; r < RPS; ++r) {
                            const int k = kb + j * RPS + r;
                            if (whole || k < mlen)
                                any_row(f, first ? j * RPS + r : 4, whole || k < mlen - 1, a2[r],
                                        b2[r], c2[r], d2[r], on, red + q * RP + s, fstride);
                            ta[j * RPS + r] = f.alp;
                            tg[j * RPS + r] = f.gap;
                            td[j * RPS + r] = f.dep;
                        }
                    }
                }
            };
            auto rows = [&](int kb, bool first) {
                if (kb + 4 < wlo)
                    block(kb, first, true);
                else
                    block(kb, first, false);
            };
            auto keep = [&](int kb) { tmem_store_rows(tcol + kb * 6, ta, tg, td); };
            rows(0, true);
            keep(0);
#pragma unroll 1
            for (int kb = 4; kb < TR && kb < m; kb += 4) {
                rows(kb, false);
                keep(kb);
            }
#pragma unroll
            for (int kb = TR; kb < M; kb += 4) {
                if (kb < m) {
                    rows(kb, false);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        al[kb - TR + r] = ta[r];
                        ga[kb - TR + r] = tg[r];
                        de[kb - TR + r] = td[r];
                    }
                }
            }
            if (on) {
                double* w = red + q * RP + s;
                const double cb0 = w[fstride], rr = rcp_nr(1.0 - cb0 * f.sa);
                w[0 * fstride] = rr * w[0];
                w[1 * fstride] = rr * cb0 * f.pi;
                w[2 * fstride] = rr * (w[2 * fstride] - cb0 * f.sd);
                w[3 * fstride] = f.alp;
                w[4 * fstride] = f.gap;
                w[5 * fstride] = f.dep;
            }
        }
        __syncthreads();

        // ------------------------------------------------ reduced system
        double x_first, x_last;
        {
            const int per_pass = T / W;  // systems per pass
            const int p = tid % W;
            double* pb = pub + (it & 1) * 6 * S;
            for (int base = 0; base < S; base += per_pass) {
                const int sp = base + tid / W;
                const bool act = sp < S && p < nsc;
                double l0 = 0, u0 = 0, b0 = 0, l1 = 0, u1 = 0, b1 = 0;
                double* src = red + p * RP + sp;
                if (act) {
                    l0 = src[0 * fstride];
                    u0 = src[1 * fstride];
                    b0 = src[2 * fstride];
                    l1 = src[3 * fstride];
                    u1 = src[4 * fstride];
                    b1 = src[5 * fstride];
                }
                if constexpr (CLUSTER) {
                    double f[3], d[3];
                    reduced_condense(l0, u0, b0, l1, u1, b1, p, nsc, W, act, f, d);
                    if (act) {  // over the fields this thread has read
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            src[i * fstride] = f[i];
                            src[(3 + i) * fstride] = d[i];
                            if (p == 0) pb[i * S + sp] = f[i];
                            if (p == nsc - 1) pb[(3 + i) * S + sp] = d[i];
                        }
                    }
                } else {
                    double xf, xl;
                    reduced_solve_shfl<true>(l0, u0, b0, l1, u1, b1, p, nsc, W, act, xf,
                                               xl);
                    if (act) {
                        src[0] = xf;
                        src[fstride] = xl;
                    }
                }
            }
            if constexpr (CLUSTER) {
                __syncthreads();  // the CTA's rows are published
                if (tid < cl) mbar_arrive_cluster(&xbar[it & 1], tid);
                if (ok) ok = mbar_wait_cluster(&xbar[it & 1], (it >> 1) & 1, args.status);
                // the outer unknowns of every CTA of a system, one lane a CTA
                const int WC = tile_lanes(cl);
                const int per = T / WC;
                const int r = tid % WC;
                for (int base = 0; base < S; base += per) {
                    const int sp = base + tid / WC;
                    double f[3] = {0, 0, 0}, d[3] = {0, 0, 0};
                    if (sp < S && r < cl) {
                        const double* src = cg::this_cluster().map_shared_rank(pb, r) + sp;
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            f[i] = src[i * S];
                            d[i] = src[(3 + i) * S];
                        }
                    }
                    double lam, rho;
                    reduced_outer<true>(f, d, r, cl, WC, lam, rho);
                    if (sp < S && r == c) {
                        outer[sp] = lam;
                        outer[S + sp] = rho;
                    }
                }
            }
            __syncthreads();
            const double* src = red + q * RP + s;
            if constexpr (CLUSTER) {
                const double lam = outer[s], rho = outer[S + s];
                x_first = src[0] + lam * src[1 * fstride] + rho * src[2 * fstride];
                x_last = src[3 * fstride] + lam * src[4 * fstride] + rho * src[5 * fstride];
            } else {
                x_first = src[0];
                x_last = src[fstride];
            }
        }

        // --------------------------------------------- back substitution
        double* xp = args.X + (size_t)(r0 + mlen - 1) * ns + sys;
        double xn = x_last;
        auto put = [&](double x) {
            if (valid) {
                *xp = x;
                nonfinite = fma(x, 0.0, nonfinite);
            }
            xp -= ns;
        };
        put(x_last);
#pragma unroll
        for (int k = M - 2; k >= TR; --k) {
            if (k < mlen - 1) {
                xn = de[k - TR] - al[k - TR] * x_first - ga[k - TR] * xn;
                put(xn);
            }
        }
        tmem_wait_st();
#pragma unroll
        for (int k0 = TR - 4; k0 >= 0; k0 -= 4) {
            if (k0 < m) {
                uint32_t wa[8], wg[8], wd[8];
                tmem_load_rows(tcol + k0 * 6, wa, wg, wd);
#pragma unroll
                for (int r = 3; r >= 0; --r) {
                    if (k0 + r == 0) continue;  // row 0 is x_first
                    if (k0 + r < mlen - 1) {
                        xn = tmem_word(wd, r) - tmem_word(wa, r) * x_first -
                             tmem_word(wg, r) * xn;
                        put(xn);
                    }
                }
            }
        }
        put(x_first);
    }
    if (nonfinite != 0.0) raise_status(args.status, ST_NONFINITE);
    if constexpr (!ASYNC) {
        if (!ok && warp == 0)  // a wait gave up: in-flight copies get a bounded chance to land
            for (int i = 0; i < nst; ++i) mbar_wait_bounded(&full[i], 0, nullptr, 1u << 8);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0)
        tmem_dealloc(*static_cast<volatile uint32_t*>(tslot), (uint32_t)wide_tmem_cols(nwarps));
    if constexpr (CLUSTER) tile_cluster_sync(cl);  // peers may still read this CTA's rows
}

}  // namespace btdma

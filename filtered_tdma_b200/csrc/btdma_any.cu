// Launch planning of the periodic any-length tiled solve (k_tile_any.cuh).
#include "btdma_host.cuh"
#include "k_tile_any.cuh"

namespace {

struct AnyPlan {
    int sys = 0, nsc = 0, cl = 0, m = 0, nst = 0;
    bool async = false;
};

template <bool ASYNC, bool CLUSTER>
int launch_any(const AnyMaps& maps, const AnyArgs& a, cudaStream_t st) {
    return launch_tmem<tile_any_kernel<ASYNC, CLUSTER>, CLUSTER>(
        any_threads(a.sys, a.nsc), any_smem_bytes(a.sys, a.nsc, a.cl, a.nst, 8), a.cl,
        a.n_groups, st, maps, a);
}

// The fewest CTAs a system, then the fewest sub-segments, of at most 32 rows (one
// CTA: a power of two of them); as many systems as fill 512 threads, halved while
// at most half the SMs have a CTA.
AnyPlan any_plan(int n_row, int n_sys, bool tma) {
    AnyPlan p;
    const int cl0 = (n_row + 511) / 512;
    if (tma) {  // the last sub-segment takes what the others leave: at least 3 rows
        for (int cl = cl0; cl <= 8 && !p.nsc; ++cl)
            for (int nsc = (n_row + 32 * cl - 1) / (32 * cl); nsc <= 16; ++nsc) {
                const int nseg = cl * nsc, m = (n_row + nseg - 1) / nseg;
                if (m < 4 || n_row - (nseg - 1) * m < 3) continue;
                if (cl == 1 && (nsc & (nsc - 1)) != 0) continue;
                p.nsc = nsc;
                p.cl = cl;
                p.m = m;
                break;
            }
    }
    if (!p.nsc) {
        if (cl0 > 8) return p;
        p.async = true;
        p.cl = cl0;
        p.nsc = (n_row + 32 * p.cl - 1) / (32 * p.cl);
        if (p.cl == 1) p.nsc = tile_lanes(p.nsc);
        p.m = (n_row + p.cl * p.nsc - 1) / (p.cl * p.nsc);
        if (n_row / (p.cl * p.nsc) < 3) return AnyPlan();
    }
    int sys = std::min(256, 512 / p.nsc / 16 * 16);
    while (sys % 32 == 0 && sys / 2 * p.nsc >= 128 &&
           2ll * p.cl * ((n_sys + sys - 1) / sys) <= num_sms())
        sys /= 2;
    const size_t cap = (size_t)max_smem_optin();
    int nst = p.async ? ANY_ASYNC_NST : TILE_MAX_NST;
    while (!p.async && nst >= 3 && any_smem_bytes(sys, p.nsc, p.cl, nst, 8) > cap) --nst;
    while (p.async && sys > 16 && any_smem_bytes(sys, p.nsc, p.cl, nst, 8) > cap) sys -= 16;
    if (nst < 3 || any_smem_bytes(sys, p.nsc, p.cl, nst, 8) > cap) return AnyPlan();
    p.nst = nst;
    p.sys = sys;
    return p;
}

}  // namespace

int tile_any_solve(const double* A, const double* B, const double* C, const double* D, double* X,
                   int n_sys, int n_row, unsigned* status, cudaStream_t st, int n_plan) {
    const double* src[4] = {A, B, C, D};
    bool tma = n_plan % 2 == 0;
    for (const double* p : src) tma = tma && tma_ok(p, n_sys);
    const AnyPlan p = any_plan(n_row, n_sys, tma);
    if (p.sys == 0) return 0;
    AnyMaps maps = {};
    AnyArgs a = {};
    const int nseg = p.nsc * p.cl;
    const int tail = n_row - (nseg - 1) * p.m;  // rows of the last sub-segment
    for (int i = 0; i < 4; ++i) {
        a.in[i] = src[i];
        if (p.async) continue;
        const bool cut = tail < p.m;
        const int nf = cut ? nseg - 1 : nseg;  // sub-segments of m rows
        if ((!cut || p.cl > 1) &&
            !make_tile_map(&maps.full[i], src[i], n_sys, nf, p.sys, p.nsc, 8, 4, p.m))
            return 0;
        if (cut && p.nsc > 1 &&
            !make_tile_map(&maps.less[i], src[i], n_sys, nf, p.sys, p.nsc - 1, 8, 4, p.m))
            return 0;
        if (cut && !make_tile_map(&maps.tail[i], src[i] + (size_t)nf * p.m * n_sys, n_sys, 1,
                                  p.sys, 1, 8, 4, tail))
            return 0;
    }
    a.X = X;
    a.n_sys = n_sys;
    a.n_row = n_row;
    a.sys = p.sys;
    a.nsc = p.nsc;
    a.cl = p.cl;
    a.m = p.m;
    a.nst = p.nst;
    a.n_groups = (n_sys + p.sys - 1) / p.sys;
    a.status = status;
    int rc;
    if (p.async)
        rc = p.cl > 1 ? launch_any<true, true>(maps, a, st) : launch_any<true, false>(maps, a, st);
    else
        rc = p.cl > 1 ? launch_any<false, true>(maps, a, st)
                      : launch_any<false, false>(maps, a, st);
    return rc == BTDMA_OK ? 1 : rc;
}

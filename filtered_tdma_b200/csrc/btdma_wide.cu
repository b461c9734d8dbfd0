// Launch planning of the wide solve's general form (k_tile_wide.cuh, GEN): row
// counts that 32 does not divide, odd n_sys, systems over a cluster's CTAs.
#include "btdma_host.cuh"

namespace {

struct WidePlan {
    int sys = 0, nsc = 0, cl = 0, nst = 0;
};

template <int SYS, bool CYCLIC, typename TIN, bool CLUSTER, bool WATCH>
int launch_wide(const WideMapsGen& maps, const TileArgs& a, const WideGen& gen, cudaStream_t st) {
    const bool odd = sizeof(TIN) == 8 && (a.n_sys & 1) != 0;
    return launch_tmem<tile_wide_kernel<SYS, CYCLIC, TIN, false, true, CLUSTER, WATCH>, CLUSTER>(
        SYS * a.nseg, tile_wide_smem_bytes(SYS, a.nseg, a.nst, (int)sizeof(TIN), odd, a.cl),
        a.cl, a.n_groups, st, maps, a, gen);
}

template <bool CYCLIC, typename TIN, bool WATCH>
int launch_wide_plan(int sys, const WideMapsGen& maps, const TileArgs& a, const WideGen& gen,
                     cudaStream_t st) {
    if (a.cl > 1) return launch_wide<32, CYCLIC, TIN, true, WATCH>(maps, a, gen, st);
    switch (sys) {
        case 256: return launch_wide<256, CYCLIC, TIN, false, WATCH>(maps, a, gen, st);
        case 128: return launch_wide<128, CYCLIC, TIN, false, WATCH>(maps, a, gen, st);
        case 64: return launch_wide<64, CYCLIC, TIN, false, WATCH>(maps, a, gen, st);
        case 16: return launch_wide<16, CYCLIC, TIN, false, WATCH>(maps, a, gen, st);
        default: return launch_wide<32, CYCLIC, TIN, false, WATCH>(maps, a, gen, st);
    }
}

// watch: FP64 shapes the narrow kernel does not take.
template <bool CYCLIC, typename TIN>
int launch_wide_plan(int sys, const WideMapsGen& maps, const TileArgs& a, const WideGen& gen,
                     bool watch, cudaStream_t st) {
    if constexpr (sizeof(TIN) == 8) {
        if (watch) return launch_wide_plan<CYCLIC, TIN, true>(sys, maps, a, gen, st);
    }
    return launch_wide_plan<CYCLIC, TIN, false>(sys, maps, a, gen, st);
}

// The widest group that fills 512 threads, halved while at most half the SMs have
// a CTA (as tile_wide_plan).  Where the narrow kernel takes the shape too, it keeps
// the batches that leave the SMs idle even so: B200, us, narrow / this one,
//   65536 x 240 161 / 107, 65536 x 272 222 / 143, 65536 x 400 276 / 181
//   8192 x 176 23.3 / 15.4, 4096 x 272 17.5 / 13.8, 4096 x 240 12.3 / 11.6
//   4096 x 176 9.6 / 12.0, 2048 x 272 9.5 / 13.7, 16384 x 48 9.2 / 11.1
//   clusters: 4096 x 1024 58 / 43, 2048 x 2048 63 / 44, 4096 x 4096 290 / 165,
//   256 x 4096 32 / 20, but 1024 x 1024 14.8 / 18.4 and 512 x 2048 16.1 / 18.7
// Against the segment kernels (row counts 16 does not divide, odd n_sys) this one
// is faster but for small batches of short segments (kept there by solve_impl):
//   2048 x 250 19.5 / 10.6, 2049 x 250 50 / 12.2, 22585 x 512 5109 / 91,
//   62500 x 250 285 / 110.
WidePlan wide_gen_plan(int n_row, int n_plan, bool cyclic, int elem, bool odd, bool narrow) {
    WidePlan p;
    const int nseg = (n_row + WIDE_M - 1) / WIDE_M;
    int cl = (nseg + 15) / 16;
    if (cyclic) {  // whole sub-segments, as many in every CTA
        if (n_row % WIDE_M) return p;
        while (cl <= 8 && nseg % cl) ++cl;
        if (cl == 1 && (nseg & (nseg - 1)) != 0) return p;
    }
    if (cl > 8) return p;
    const int nsc = (nseg + cl - 1) / cl;
    if (cl > 1 && nsc < 8) return p;
    int sys = cl > 1 || nsc > 8 ? 32 : (nsc > 4 ? 64 : (nsc > 2 || odd ? 128 : 256));
    auto idle = [&] { return 2ll * cl * ((n_plan + sys - 1) / sys) <= num_sms(); };
    if (cl > 1) {
        if (narrow && n_row <= 2048 && idle()) return p;
    } else {
        const int min_threads = narrow ? 256 : 128;
        while (idle() && sys > 16) {
            if (sys / 2 * nsc < min_threads || sys / 2 * nsc % 32 != 0 || (narrow && nsc <= 2)) {
                if (narrow) return p;
                break;
            }
            sys /= 2;
        }
    }
    const int per_sm = std::max(1, TILE_MAX_THREADS / (sys * nsc));
    const size_t cap = std::min((size_t)max_smem_optin(),
                                (size_t)max_smem_per_sm() / per_sm - 1024);
    int nst = TILE_MAX_NST;
    while (nst >= 3 && tile_wide_smem_bytes(sys, nsc, nst, elem, odd, cl) > cap) --nst;
    if (nst < 3) return p;
    p.sys = sys;
    p.nsc = nsc;
    p.cl = cl;
    p.nst = nst;
    return p;
}

// Boxes of SYS systems x a stage's rows x nsc sub-segments of rows (a tensor of
// nseg sub-segments); odd n_sys: of pairs of rows.
bool wide_map(CUtensorMap* map, const void* ptr, int n_sys, int rows, int nseg, int sys, int nsc,
              int elem, bool odd) {
    if (!odd) return make_tile_map(map, ptr, n_sys, nseg, sys, nsc, elem, 4, rows);
    auto fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {2 * (cuuint64_t)n_sys, (cuuint64_t)rows / 2, (cuuint64_t)nseg};
    if (rows == 1) {  // a single row
        dims[0] = (cuuint64_t)n_sys;
        dims[1] = 1;
    }
    const cuuint64_t pair = 2 * (cuuint64_t)n_sys * sizeof(double);
    cuuint64_t strides[2] = {pair, pair * dims[1]};
    cuuint32_t box[3] = {(cuuint32_t)sys + 2, 1, (cuuint32_t)nsc};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<void*>(ptr), dims, strides, box,
              estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

template <typename TIN>
int tile_wide_gen(const TIN* A, const TIN* B, const TIN* C, const TIN* D, double* X, int n_sys,
                  int n_row, bool cyclic, unsigned* status, cudaStream_t st, bool narrow,
                  int n_plan) {
    const int elem = (int)sizeof(TIN);
    const TIN* src[4] = {A, B, C, D};
    for (const TIN* p : src)
        if ((reinterpret_cast<uintptr_t>(p) & 15) != 0) return 0;
    const bool odd = elem == 8 && n_sys % 2 != 0;
    if (!odd && ((size_t)n_sys * elem) % 16 != 0) return 0;
    const WidePlan p = wide_gen_plan(n_row, n_plan, cyclic, elem, odd, narrow);
    if (p.sys == 0) return 0;
    WideMapsGen maps = {};
    WideGen gen = {};
    const int nseg = (n_row + WIDE_M - 1) / WIDE_M;
    int nfull = nseg;  // sub-segments of the main boxes
    if (!cyclic) {
        nfull = nseg - 1;
        gen.tail = n_row - nfull * WIDE_M;
        gen.nl = nfull - (p.cl - 1) * p.nsc;
    } else {
        gen.nl = p.nsc;
    }
    for (int f = 0; f < 4; ++f) {
        if constexpr (sizeof(TIN) == 8) gen.in[f] = src[f];
        if ((cyclic || p.cl > 1) &&
            !wide_map(&maps.full[f], src[f], n_sys, WIDE_M, nfull, p.sys, p.nsc, elem, odd))
            return 0;
        if (cyclic) continue;
        if (gen.nl > 0 &&
            !wide_map(&maps.less[f], src[f], n_sys, WIDE_M, nfull, p.sys, gen.nl, elem, odd))
            return 0;
        const TIN* tp = src[f] + (size_t)nfull * WIDE_M * n_sys;
        const int rows = gen.tail - (f == 2 ? 1 : 0);  // C's last row is not read
        const int units = odd ? rows / 2 : rows;
        if (units == 0) gen.empty |= 1 << f;
        if (!wide_map(&maps.tail[f], tp, n_sys, units == 0 ? (odd ? 2 : 1) : (odd ? 2 * units : rows),
                      1, p.sys, p.nsc - gen.nl, elem, odd))
            return 0;
        if (odd && rows % 2 &&
            !wide_map(&maps.last[f], tp + (size_t)(rows - 1) * n_sys, n_sys, 1, 1, p.sys,
                      p.nsc - gen.nl, elem, odd))
            return 0;
    }
    TileArgs a = {};
    a.X = X;
    a.n_sys = n_sys;
    a.n_row = n_row;
    a.nseg = p.nsc;
    a.cl = p.cl;
    a.nst = p.nst;
    a.n_groups = (n_sys + p.sys - 1) / p.sys;
    a.status = status;
    const int rc = cyclic ? launch_wide_plan<true, TIN>(p.sys, maps, a, gen, !narrow, st)
                          : launch_wide_plan<false, TIN>(p.sys, maps, a, gen, !narrow, st);
    return rc == BTDMA_OK ? 1 : rc;
}

template int tile_wide_gen<double>(const double*, const double*, const double*, const double*,
                                   double*, int, int, bool, unsigned*, cudaStream_t, bool, int);
template int tile_wide_gen<float>(const float*, const float*, const float*, const float*, double*,
                                  int, int, bool, unsigned*, cudaStream_t, bool, int);

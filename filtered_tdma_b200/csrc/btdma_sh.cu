// Launch planning of the shared-matrix sweeps with two systems a thread
// (k_tile_sh.cuh).
#include "btdma_host.cuh"

namespace {

struct ShPlan {
    int sys = 0, nseg = 0, nst = 0;
};

ShPlan sh_plan(const ShArgs& a, int mode, bool cyclic) {
    ShPlan p;
    if (a.n_row % TILE_MT != 0 || a.n_sys % 2 != 0) return p;
    const int nseg = a.n_row / TILE_MT;
    if (nseg > 32 || (cyclic && (nseg & (nseg - 1)) != 0)) return p;
    int sys = nseg > 16 && mode != SH_HEAT ? 16 : 32;  // SH_HEAT: always 32
    // SH_FIELD: a group stays in one row of cells; SH_HEAT: whole 16 x sys / 16 blocks
    if (mode == SH_FIELD && a.fblk % sys != 0) sys = 16;
    if (mode == SH_FIELD && a.fblk % sys != 0) return p;
    if (mode == SH_HEAT && (a.fblk % SH_HX != 0 || a.iy % (sys / SH_HX) != 0)) return p;
    const int T = sh_threads(sys, nseg);
    // an equal share of the SM per resident CTA (128 registers a thread)
    int per_sm = std::max(1, 65536 / (T * 128));
    int nst = 0;
    for (; per_sm >= 1 && nst < 3; --per_sm) {
        const size_t cap =
            std::min((size_t)max_smem_optin(), (size_t)max_smem_per_sm() / per_sm - 1024);
        nst = TILE_MAX_NST_CONST;
        while (nst >= 3 && sh_smem_bytes(sys, nseg, nst, mode) > cap) --nst;
    }
    if (nst < 3) return p;
    p.sys = sys;
    p.nseg = nseg;
    p.nst = nst;
    return p;
}

template <int SYS, bool CYCLIC, int MODE, int STORE>
int launch_sh(const CUtensorMap& tm, const ShArgs& a, cudaStream_t st) {
    auto kern = tile_sh_kernel<SYS, CYCLIC, MODE, STORE>;
    static bool attr_done = false;
    if (!attr_done) {
        CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                max_smem_optin()));
        attr_done = true;
    }
    const int threads = sh_threads(SYS, a.nseg);
    const size_t smem = sh_smem_bytes(SYS, a.nseg, a.nst, MODE);
    int nb = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, threads, smem));
    const int grid = std::min(num_sms() * std::max(1, nb), a.n_groups);
    kern<<<grid, threads, smem, st>>>(tm, a);
    CK(cudaGetLastError());
    return 1;
}

template <int SYS, int MODE>
int launch_sh_store(const CUtensorMap& tm, const ShArgs& a, bool cyclic, int store,
                    cudaStream_t st) {
    if constexpr (MODE == SH_ROWS) {
        switch (store * 2 + (cyclic ? 1 : 0)) {
            case SH_PAIR * 2: return launch_sh<SYS, false, MODE, SH_PAIR>(tm, a, st);
            case SH_PAIR * 2 + 1: return launch_sh<SYS, true, MODE, SH_PAIR>(tm, a, st);
            case SH_LINE * 2: return launch_sh<SYS, false, MODE, SH_LINE>(tm, a, st);
            case SH_LINE * 2 + 1: return launch_sh<SYS, true, MODE, SH_LINE>(tm, a, st);
            case SH_LINE31 * 2: return launch_sh<SYS, false, MODE, SH_LINE31>(tm, a, st);
            case SH_LINE31 * 2 + 1: return launch_sh<SYS, true, MODE, SH_LINE31>(tm, a, st);
            case SH_ONE * 2 + 1: return launch_sh<SYS, true, MODE, SH_ONE>(tm, a, st);
            default: return launch_sh<SYS, false, MODE, SH_ONE>(tm, a, st);
        }
    } else if constexpr (MODE == SH_FIELD) {
        return store == SH_PAIR ? launch_sh<SYS, false, MODE, SH_PAIR>(tm, a, st)
                                : launch_sh<SYS, false, MODE, SH_ONE>(tm, a, st);
    } else {  // into the library's own buffer
        return store == SH_PAIR ? launch_sh<SYS, false, MODE, SH_PAIR>(tm, a, st) : 0;
    }
}

// 4-D view of a ghosted field (x, y, row of the sub-segment, sub-segment) from plane
// k = 1: boxes of cells + 2 x rows cells x a stage's rows x nseg.
bool field_map(CUtensorMap* map, const double* q, int nx, int ny, int nseg, int cells, int rows,
               int rps) {
    auto fn = encode_fn();
    if (!fn) return false;
    const size_t rx = (size_t)nx + 2, plane = rx * ((size_t)ny + 2);
    cuuint64_t dims[4] = {(cuuint64_t)rx, (cuuint64_t)ny + 2, (cuuint64_t)TILE_MT,
                          (cuuint64_t)nseg};
    cuuint64_t strides[3] = {rx * sizeof(double), plane * sizeof(double),
                             (cuuint64_t)TILE_MT * plane * sizeof(double)};
    cuuint32_t box[4] = {(cuuint32_t)cells + 2, (cuuint32_t)rows, (cuuint32_t)rps,
                         (cuuint32_t)nseg};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, const_cast<double*>(q + plane), dims,
              strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

int try_sh(int mode, const double* src, int nx, int ny, ShArgs a, bool cyclic, cudaStream_t st) {
    if (!tma_ok(src, 2)) return 0;
    const ShPlan p = sh_plan(a, mode, cyclic);
    if (p.sys == 0) return 0;
    if (a.xblk <= 0) {  // x in D's layout
        a.xblk = a.n_sys;
        a.xbs = 0;
        a.xss = 1;
        a.xrs = a.n_sys;
    }
    a.nseg = p.nseg;
    a.nst = p.nst;
    a.n_groups = (a.n_sys + p.sys - 1) / p.sys;
    CUtensorMap tm;
    const int rps = sh_rps(mode);
    if (mode == SH_ROWS ? !make_tile_map(&tm, src, a.n_sys, p.nseg, p.sys, p.nseg, 8, 1)
                        : !field_map(&tm, src, nx, ny, p.nseg, mode == SH_HEAT ? SH_HX : p.sys,
                                           mode == SH_HEAT ? p.sys / SH_HX + 2 : 1, rps))
        return 0;
    const int off = (int)(reinterpret_cast<uintptr_t>(a.X) / sizeof(double) & 3);
    int store = SH_ONE;
    if (a.xrs == 1) {
        if (a.xbs % 4 == 0 && a.xss % 2 == 0 && a.xblk % 2 == 0) {
            const int odd = (off + a.xss) & 3;  // where the odd systems' rows start
            if (off == 0 && odd == 0) store = SH_LINE;
            if (off == 3 && odd == 1) store = SH_LINE31;
        }
    } else if (a.xss == 1 && off % 2 == 0 && a.xbs % 2 == 0 && a.xrs % 2 == 0 &&
               a.xblk % 2 == 0) {
        store = SH_PAIR;
    }
    if (a.xblk % 2 != 0) return 0;  // a pair of systems shares a block of the map
    if (p.sys == 32) {
        if (mode == SH_ROWS) return launch_sh_store<32, SH_ROWS>(tm, a, cyclic, store, st);
        if (mode == SH_FIELD) return launch_sh_store<32, SH_FIELD>(tm, a, cyclic, store, st);
        return launch_sh_store<32, SH_HEAT>(tm, a, cyclic, store, st);
    }
    if (mode == SH_ROWS) return launch_sh_store<16, SH_ROWS>(tm, a, cyclic, store, st);
    return launch_sh_store<16, SH_FIELD>(tm, a, cyclic, store, st);
}

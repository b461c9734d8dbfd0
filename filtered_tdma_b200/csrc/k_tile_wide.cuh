// Wide variant of the register-tiled segmented solve (k_tile.cuh): sub-segments
// of 32 rows, whose elimination state is held partly in registers (12 rows) and
// partly in tensor memory (20 rows), so a CTA takes twice the systems and every row
// of a TMA box is twice as wide in HBM.
//
// Why: the DRAM serves a stream of row pieces (SYS x element bytes, rows a full
// row of the batch apart) at a rate that grows with the piece width: 64-byte
// pieces reach about half the bandwidth of 128-byte ones, 128-byte pieces about
// three quarters of 256-byte ones.  The tiled kernel keeps the state of all its
// rows in registers (24 bytes a row), which caps it at 16 systems of 512 rows
// per SM.  The SM's 256 KB of tensor memory is per-thread storage too: a warp
// reads and writes its own quarter of the lanes (tcgen05.st / tcgen05.ld, 32
// lanes x 32-bit columns), one 120-column slice per warp holding WIDE_TROWS = 20
// rows' alpha, gamma and delta of each thread.  With it a CTA takes 32 systems of 512
// rows.  (16 rows there left 56 to 128 bytes of spills.)
//
//   forward   thread (s, q) = system s, rows 32 q .. 32 q + 31: the pass of
//             k_tile.cuh over 32 rows; the state of rows 0..19 moves to tensor
//             memory four rows at a time, rows 20..31 stay in registers.
//   reduced   one system per group of W lanes (reduced_solve_shfl), half as
//             many rows as with 16-row sub-segments.
//   back      rows 31..20 from registers, then rows 19..0 from tensor memory.
//
// The ring is that of k_tile.cuh (full / empty mbarriers per stage, refills
// issued by a rotating producer warp), with unhinted polls.  A, B, C, D are
// read once.
// Needs NSEG = n_row / 32 <= 16 (periodic: a power of two), n_sys * elem a
// multiple of 16 bytes and 16-byte aligned arrays; SYS = 16 (NSEG = 16) to 256
// systems, so that a CTA has 256 to 512 threads.
//
// Measured on B200 (262144 x 512), every pass on another batch: FP64 0.85 ms, FP32
// storage 0.62 ms, 98 % and 80 % of the copy bandwidth at the algorithmic 40 / 24
// bytes a row (before, with half the rows eliminated a second time from L2: 1.16 / 0.87
// ms; the DRAM moved 1.15x the bytes and each row's arithmetic ran 1.5 times).
// Launched back to back, on one batch or two in turn, 0.81 and 0.53 ms.  Bound by DRAM;
// with 6 / 5 / 4 ring stages of 32 KB it takes 0.811 / 0.815 / 0.857 ms so.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "btdma_common.cuh"
#include "k_reduced.cuh"
#include "k_tile.cuh"

namespace btdma {

constexpr int WIDE_M = 32;      // rows per sub-segment (per thread)
constexpr int WIDE_TROWS = 20;  // rows whose state goes to tensor memory (the first ones)
constexpr int WIDE_TCOLS = WIDE_TROWS * 6;  // columns of a warp: 3 doubles a row

// The general form (GEN) takes any n_row and odd n_sys, and with CLUSTER systems
// longer than a CTA holds:
//   tail      the sub-segment with the system's last rows arrives by boxes of its
//             own (rows past the end are zero-filled; there B becomes 1, which
//             leaves identity rows, x = 0).  C's boxes end one row earlier, so the
//             unused coupling of the last row is 0 whatever the array holds.
//   odd       with an odd n_sys every other row is 8 bytes off TMA's 16: rows are
//             taken in pairs, as a row of 2 n_sys elements whose stride suits
//             TMA, the odd row from x = n_sys + first system - 1 (even), in boxes
//             two elements wider.
//   cluster   CL CTAs each own NSC consecutive sub-segments of the same systems.
//             A CTA solves its own reduced system with its two outer couplings as
//             parameters (reduced_condense): its first and last unknown become
//             linear in the left neighbour's last and the right neighbour's first
//             unknown.  These six numbers a system are published in shared memory
//             (double buffered); every CTA signals its peers' mbarriers once a
//             group, reads all CL of them and eliminates over the CTAs in lane
//             registers (reduced_outer).
struct WideMaps {
    CUtensorMap full[4];  // A, B, C, D: boxes of the CTA's sub-segments
};
struct WideMapsGen {
    CUtensorMap full[4];
    CUtensorMap less[4];  // the last CTA: its sub-segments before the tail one
    CUtensorMap tail[4];  // the tail one (and all-identity ones after it)
    CUtensorMap last[4];  // odd n_sys: the tail's unpaired last row
};
struct WideGen {
    int tail;   // rows of the tail sub-segment (0: periodic, none)
    int nl;     // sub-segments before it in the last CTA
    int empty;  // bit f: array f has no (pair of) rows in the tail's box
    const double* in[4];  // A, B, C, D (FP64), for passes with PIV_EXACT
};

// Elements of a ring stage; odd n_sys: a box per array and row of NSC pieces of
// SYS + 2, the tail's box on a 128-byte boundary of its own.
__host__ __device__ __forceinline__ int wide_odd_box(int sys, int nseg) {
    return (nseg * (sys + 2) + 15) / 16 * 16 + 16;
}
__host__ __device__ __forceinline__ int wide_stage_elems(int sys, int nseg, int elem, bool odd) {
    return odd ? 8 * wide_odd_box(sys, nseg) : 4 * tile_rps(elem) * sys * nseg;
}
// Shared memory: ring + reduced rows (6 x NSEG x (SYS + 1) doubles; x_first /
// x_last reuse fields 0 and 1) + published rows [2][6][SYS] and outer unknowns
// [2][SYS] (clusters) + mbarriers + the tensor-memory address.
__host__ __device__ __forceinline__ size_t tile_wide_smem_bytes(int sys, int nseg, int nst,
                                                                int elem, bool odd = false,
                                                                int cl = 1) {
    return (size_t)nst * wide_stage_elems(sys, nseg, elem, odd) * elem +
           6ull * nseg * (sys + 1) * sizeof(double) + (cl > 1 ? 14ull * sys * sizeof(double) : 0) +
           (2ull * nst + 2) * sizeof(uint64_t) + 16 + 128;
}

// ------------------------------------------------------------- tensor memory
// Columns a CTA of `warps` warps allocates (a power of two >= 32).
__host__ __device__ __forceinline__ int wide_tmem_cols(int warps) {
    int c = 32;
    while (c < (warps + 3) / 4 * WIDE_TCOLS) c <<= 1;
    return c;
}
// Shared memory a CTA of a cluster asks for when it needs `smem` bytes and `cols` columns:
// at least half the SM's (sm_bytes, of which every resident CTA takes 1 KB more than it
// asks for), and more than half with more than 256 columns.  So such a CTA has no other
// cluster's CTA, of any launch, beside it, and others at most one, whose columns (powers
// of two) fit wherever they lie.  Without it two clusters, of two launches on two streams,
// could each have a CTA in tmem_alloc, which waits without a limit, for the columns of a
// CTA that waits at its cluster's barrier for the other one's peer.  (CTAs without a
// cluster wait for nobody once they have their columns: they only delay.)
__host__ __device__ __forceinline__ size_t wide_cluster_smem(size_t smem, int cols,
                                                             size_t sm_bytes) {
    const size_t least = sm_bytes / 2 - 1024 + (cols > 256 ? 128 : 0);
    return smem > least ? smem : least;
}
// tcgen05's .sync.aligned instructions need every lane of the warp at the same
// instruction, and callers come from per-lane branches (stores of systems past the
// batch, rows past a tail): each of these wrappers converges the warp itself.
//
// One warp; the address of the columns is written to *dst (shared memory).  The
// call waits while another CTA on the SM holds the columns.
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t cols) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(dst)),
                 "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols)
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
    __syncwarp();
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// 4 rows' alpha, gamma and delta of every lane to 24 columns of the warp's lanes.
__device__ __forceinline__ void tmem_store_rows(uint32_t addr, const double (&al)[4],
                                                const double (&ga)[4], const double (&de)[4]) {
    __syncwarp();
    auto put = [](uint32_t at, const double (&v)[4]) {
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(
                at),
            "r"(__double2loint(v[0])), "r"(__double2hiint(v[0])), "r"(__double2loint(v[1])),
            "r"(__double2hiint(v[1])), "r"(__double2loint(v[2])), "r"(__double2hiint(v[2])),
            "r"(__double2loint(v[3])), "r"(__double2hiint(v[3]))
            : "memory");
    };
    put(addr, al);
    put(addr + 8, ga);
    put(addr + 16, de);
}
// The 24 columns back into registers; the wait passes them through, so that no use
// of them moves above it.
__device__ __forceinline__ void tmem_load_rows(uint32_t addr, uint32_t (&u)[8], uint32_t (&v)[8],
                                               uint32_t (&w)[8]) {
    __syncwarp();
    auto get = [](uint32_t at, uint32_t (&r)[8]) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
              "=r"(r[7])
            : "r"(at)
            : "memory");
    };
    get(addr, u);
    get(addr + 8, v);
    get(addr + 16, w);
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(u[0]), "+r"(u[1]), "+r"(u[2]), "+r"(u[3]), "+r"(u[4]), "+r"(u[5]),
                   "+r"(u[6]), "+r"(u[7]), "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]),
                   "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(w[0]), "+r"(w[1]),
                   "+r"(w[2]), "+r"(w[3]), "+r"(w[4]), "+r"(w[5]), "+r"(w[6]), "+r"(w[7])
                 :
                 : "memory");
}
__device__ __forceinline__ double tmem_word(const uint32_t (&w)[8], int i) {
    return __hiloint2double((int)w[2 * i + 1], (int)w[2 * i]);
}

// One arrival on the mbarrier at the same shared-memory offset in CTA `rank` of
// the cluster, releasing this thread's (and, after a block barrier, the CTA's)
// earlier writes to the cluster.
__device__ __forceinline__ void mbar_arrive_cluster(uint64_t* bar, int rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(bar)),
                 "r"(rank));
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
static __device__ __noinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity,
                                                      unsigned* status) {
    for (uint32_t it = 0; it < (1u << 22); ++it) {
        if (mbar_try_wait_cluster(bar, parity)) return true;
        if (status && (it & 1023u) == 1023u &&
            (*reinterpret_cast<volatile unsigned*>(status) & ST_TIMEOUT))
            return false;
    }
    raise_status(status, ST_TIMEOUT);
    return false;
}

// Running state of one sub-segment's forward pass (rows 0 .. M-1).
struct WideFwd {
    double ab0, cb0, db0;  // row 0 scaled by its pivot
    double pi, sa, sd;     // running products of the reduced first row
    double alp, gap, dep;  // alpha, gamma, delta of the previous row
    double gm2;            // gamma of row M-2
};

// The reciprocals of a forward pass.  rcp_nr wants normal pivots with normal reciprocals,
// as the narrow kernel's.  Row counts and batches outside that kernel's keep the whole FP64
// range, as the segment kernels they ran on: PIV_WATCH notes pivots of 2^1017 and more (one above
// 2^1022 would pass with a reciprocal of 0), subnormal and infinite ones leave NaN, and a
// warp with such a system takes its rows again from global memory with PIV_EXACT, where
// that system's lanes use correctly rounded reciprocals.  (B200, 62500 x 250: 110 us
// unwatched, 112 watched; correctly rounded ones throughout, or a check and a branch a
// row, 114, and 4 to 8 % over clusters, where the watch costs at most 1.)
enum Pivots { PIV_NORMAL = 0, PIV_WATCH = 1, PIV_EXACT = 2 };
struct PivotWatch {
    bool big = false;    // PIV_WATCH: a pivot of 2^1017 or more
    bool exact = false;  // PIV_EXACT: this lane's system needs it
};
template <int PIV>
__device__ __forceinline__ double wide_rcp(double x, PivotWatch& pw) {
    if constexpr (PIV == PIV_WATCH)
        pw.big |= (__double2hiint(x) & 0x7f800000) == 0x7f800000;
    double r = rcp_nr(x);
    if constexpr (PIV == PIV_EXACT) {
        if (pw.exact) r = Exact64::rcp(x);
    }
    return r;
}
// Whether a sub-segment's pass met a pivot outside rcp_nr's range (or NaN in the data); d0
// and dep: the right-hand sides of its row 0, whose chain ends there, and its last row.
__device__ __forceinline__ bool pivots_out_of_range(const PivotWatch& pw, double d0, double dep) {
    return pw.big || isnan(d0) || isnan(dep);
}
// Row k of the forward pass (the expressions of k_tile.cuh's loop, FP64).
template <int PIV>
__device__ __forceinline__ void wide_row(WideFwd& f, int k, double a, double b, double cc,
                                         double d, PivotWatch& pw) {
    constexpr int M = WIDE_M;
    if (k == 0) {
        const double ib = wide_rcp<PIV>(b, pw);
        f.ab0 = a * ib;
        f.cb0 = cc * ib;
        f.db0 = d * ib;
    } else if (k == 1) {
        const double ib = wide_rcp<PIV>(b, pw);
        f.alp = a * ib;
        f.gap = cc * ib;
        f.dep = d * ib;
        f.pi = 1.0;
        f.sa = f.alp;
        f.sd = f.dep;
    } else {
        const double inv = wide_rcp<PIV>(b - a * f.gap, pw);
        const double g = cc * inv;
        const double e = (d - a * f.dep) * inv;
        const double l = -a * f.alp * inv;
        if (k <= M - 2) {
            f.pi = -f.gap * f.pi;
            f.sa += f.pi * l;
            f.sd += f.pi * e;
        }
        if (k == M - 2) f.gm2 = g;
        f.alp = l;
        f.gap = g;
        f.dep = e;
    }
}

// The two reduced rows of a finished sub-segment into red[f][q][s].
__device__ __forceinline__ void wide_reduced(const WideFwd& f, double* w, int fstride) {
    const double pi_last = -f.gm2 * f.pi;
    const double r0 = rcp_nr(1.0 - f.cb0 * f.sa);
    w[0 * fstride] = r0 * f.ab0;
    w[1 * fstride] = r0 * f.cb0 * pi_last;
    w[2 * fstride] = r0 * (f.db0 - f.cb0 * f.sd);
    w[3 * fstride] = f.alp;
    w[4 * fstride] = f.gap;
    w[5 * fstride] = f.dep;
}

// FILT: Filtered's reduced system (as tile_f64_kernel's FILT; the mode's segment
// length counts 32-row sub-segments here).  WATCH: pivots of the whole FP64 range.
template <int SYS, bool CYCLIC, typename TIN, bool FILT = false, bool GEN = false,
          bool CLUSTER = false, bool WATCH = false>
__global__ void __launch_bounds__(TILE_MAX_THREADS, 1)
tile_wide_kernel(const __grid_constant__ std::conditional_t<GEN, WideMapsGen, WideMaps> maps,
                 const TileArgs args, const WideGen gen) {
    namespace cg = cooperative_groups;
    static_assert(!FILT || !GEN, "Filtered segments are whole sub-segments");
    static_assert(!CLUSTER || GEN, "clusters run the general form");
    static_assert(!WATCH || (GEN && sizeof(TIN) == 8), "reads FP64 arrays by their pointers");
    constexpr int M = WIDE_M, TR = WIDE_TROWS;
    constexpr int RPS = tile_rps((int)sizeof(TIN));
    constexpr int SPG = M / RPS;  // stages per group
    constexpr int RP = SYS + 1;
    constexpr bool PAD = GEN && !CYCLIC;
    constexpr int PIV = WATCH ? PIV_WATCH : PIV_NORMAL;
    // a closed gate: nothing to do (TILE_MODE_GATE_ZERO: open while *gate == 0); every
    // CTA reads the same word
    if (!GEN && args.gate != nullptr &&
        ((*static_cast<const volatile unsigned*>(args.gate) == 0u) !=
         ((args.mode & TILE_MODE_GATE_ZERO) != 0)))
        return;
    extern __shared__ unsigned char smem_raw[];
    const int nseg = args.nseg, nst = args.nst;  // nseg: sub-segments of this CTA
    const int cl = CLUSTER ? args.cl : 1;
    const int T = SYS * nseg;  // == blockDim.x, whole warps
    const int W = tile_lanes(nseg);
    const int fstride = nseg * RP;
    const bool odd = GEN && sizeof(TIN) == 8 && (args.n_sys & 1) != 0;
    const int bx = odd ? wide_odd_box(SYS, nseg) : 0;

    TIN* ring = reinterpret_cast<TIN*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    const int sstride = odd ? 8 * bx : 4 * RPS * T;  // elements per stage
    double* red = reinterpret_cast<double*>(ring + (size_t)nst * sstride);
    double* pub = red + 6 * fstride;                 // [2][6][SYS]
    double* outer = pub + (CLUSTER ? 12 * SYS : 0);  // [2][SYS]
    uint64_t* full = reinterpret_cast<uint64_t*>(outer + (CLUSTER ? 2 * SYS : 0));
    uint64_t* empty = full + nst;
    uint64_t* xbar = empty + nst;  // [2]: the peers' published rows of a group
    uint32_t* tslot = reinterpret_cast<uint32_t*>(xbar + 2);

    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int nwarps = T / 32;
    const int s = tid % SYS;
    const int q = tid / SYS;
    const size_t ns = (size_t)args.n_sys;
    const unsigned zero = (unsigned)args.n_sys >> 31;  // see loads_done
    const int c = CLUSTER ? (int)cg::this_cluster().block_rank() : 0;
    const int cid = CLUSTER ? (int)blockIdx.x / cl : (int)blockIdx.x;
    const int ncid = CLUSTER ? (int)gridDim.x / cl : (int)gridDim.x;
    const int r0 = (c * nseg + q) * M;  // first row of the sub-segment
    // PAD: rows of the sub-segment that the system has (<= 0: none)
    const int mlen = PAD ? args.n_row - r0 : M;
    const bool tailed = PAD && c == cl - 1;
    const int nmain = tailed ? gen.nl : nseg;  // sub-segments of the main boxes

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
    // this warp's lanes (its quarter) and columns
    const uint32_t tcol = *static_cast<volatile uint32_t*>(tslot) + ((uint32_t)(warp & 3) << 21) +
                          (uint32_t)(warp >> 2) * WIDE_TCOLS;

    const int filt_r = FILT ? (args.mode >> TILE_MODE_FILT_SHIFT) & 255 : 0;  // lanes a segment
    const int n_my = args.n_groups > cid
                         ? (args.n_groups - cid + ncid - 1) / ncid
                         : 0;
    const int total = n_my * SPG;
    const uint32_t stage_bytes =
        odd ? 8u * nseg * (SYS + 2) * sizeof(TIN) : (uint32_t)sstride * sizeof(TIN);

    // Stage t: one thread, or (GEN) a warp: lane = array + 4 (tail) + 8 (odd row).
    auto issue = [&](int t) {
        const int slot = t % nst;
        const int g0 = (cid + (t / SPG) * ncid) * SYS;
        const int k0 = (t % SPG) * RPS;
        TIN* dst = ring + (size_t)slot * sstride;
        if constexpr (GEN) {
            if (lane == 0) mbar_expect_tx(&full[slot], stage_bytes);
            __syncwarp();
            const int f = lane & 3, tl = (lane >> 2) & 1, par = lane >> 3;
            if (par > (odd ? 1 : 0) || (tl ? !tailed : nmain == 0)) return;
            const CUtensorMap* mp = tl ? &maps.tail[f] : (tailed ? &maps.less[f] : &maps.full[f]);
            int x = g0, y = odd ? k0 >> 1 : k0, z = tl ? 0 : c * nseg;
            if (odd) {
                dst += (f * 2 + par) * bx + (tl ? (nmain * (SYS + 2) + 15) / 16 * 16 : 0);
                if (par) x += args.n_sys - 1;
            } else {
                dst += f * RPS * T + (tl ? nmain * RPS * SYS : 0);
            }
            if (tl) {
                const int rows = gen.tail - (f == 2 ? 1 : 0);  // C: not its last row
                if (odd && !par && (rows & 1) && y == rows >> 1) {
                    mp = &maps.last[f];
                    y = 0;
                } else {
                    y += (gen.empty >> f) & 1;  // nothing there: past the map's one row
                }
            }
            tma_load_3d(dst, mp, x, y, z, &full[slot]);
        } else {
            mbar_expect_tx(&full[slot], stage_bytes);
            tma_load_3d(dst + 0 * RPS * T, &maps.full[0], g0, k0, 0, &full[slot]);
            tma_load_3d(dst + 1 * RPS * T, &maps.full[1], g0, k0, 0, &full[slot]);
            tma_load_3d(dst + 2 * RPS * T, &maps.full[2], g0, k0, 0, &full[slot]);
            tma_load_3d(dst + 3 * RPS * T, &maps.full[3], g0, k0, 0, &full[slot]);
        }
    };
    bool ok = true;
    if (GEN ? warp == 0 : tid == 0)
        for (int t = 0; t < nst && t < total; ++t) issue(t);

    // this thread's rows of a stage: array f, row r at st + f * fstep + r * rstep
    const int toff = odd ? (q < nmain ? q * (SYS + 2)
                                      : (nmain * (SYS + 2) + 15) / 16 * 16 +
                                            (q - nmain) * (SYS + 2)) + s
                         : q * RPS * SYS + s;
    const int rstep = odd ? bx + 1 : SYS;
    const int fstep = odd ? 2 * bx : RPS * T;
    const TIN* st = ring + toff;
    int slot = 0;
    uint32_t phase = 0;
    int pslot = nst - 1;
    uint32_t pphase = 1;
    int t = 0;
    int tw = 0;
    // Next stage's RPS rows of this thread's sub-segment (widened), then the
    // release of the slot and, one stage later, its refill.
    auto fetch = [&](double (&a2)[RPS], double (&b2)[RPS], double (&c2)[RPS], double (&d2)[RPS]) {
        if (ok) ok = mbar_wait_bounded_spin(&full[slot], phase, args.status);
        unsigned bits = 0;
#pragma unroll
        for (int r = 0; r < RPS; ++r) {
            const TIN va = st[0 * fstep + r * rstep], vb = st[1 * fstep + r * rstep];
            const TIN vc = st[2 * fstep + r * rstep], vd = st[3 * fstep + r * rstep];
            bits ^= word_of(va) ^ word_of(vb) ^ word_of(vc) ^ word_of(vd);
            a2[r] = (double)va;
            b2[r] = (double)vb;
            c2[r] = (double)vc;
            d2[r] = (double)vd;
        }
        const unsigned z = loads_done(bits, zero);
        if constexpr (GEN) {
            if (lane == 0) mbar_arrive(&empty[slot] + z);
            if (warp == tw && t >= 1 && t - 1 + nst < total) {
                if (ok) ok = mbar_wait_bounded_spin(&empty[pslot], pphase, args.status);
                if (ok) issue(t - 1 + nst);
                __syncwarp();
            }
        } else if (lane == 0) {
            mbar_arrive(&empty[slot] + z);
            if (t >= 1 && warp == tw && t - 1 + nst < total && ok) {
                ok = mbar_wait_bounded_spin(&empty[pslot], pphase, args.status);
                if (ok) issue(t - 1 + nst);
            }
        }
        pslot = slot;
        pphase = phase;
        ++t;
        if (++tw == nwarps) tw = 0;
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
        const int sys = g * SYS + s;
        const bool valid = sys < args.n_sys;

        // ------------------------------------------------------ forward pass
        double al[M - TR], ga[M - TR], de[M - TR];  // rows TR .. M - 1
        {
            WideFwd f = {};
            PivotWatch pw;
            double ta[4], tg[4], td[4];  // rows of the 4-row block going to tensor memory
#pragma unroll
            for (int j = 0; j < SPG; ++j) {
                double a2[RPS], b2[RPS], c2[RPS], d2[RPS];
                fetch(a2, b2, c2, d2);
#pragma unroll
                for (int r = 0; r < RPS; ++r) {
                    const int k = j * RPS + r;
                    if constexpr (PAD) b2[r] = k < mlen ? b2[r] : 1.0;
                    wide_row<PIV>(f, k, a2[r], b2[r], c2[r], d2[r], pw);
                    if (k < TR) {
                        ta[k % 4] = f.alp;
                        tg[k % 4] = f.gap;
                        td[k % 4] = f.dep;
                    } else {
                        al[k - TR] = f.alp;
                        ga[k - TR] = f.gap;
                        de[k - TR] = f.dep;
                    }
                }
                const int kn = (j + 1) * RPS;
                if (kn <= TR && kn % 4 == 0) {
                    tmem_store_rows(tcol + (kn - 4) * 6, ta, tg, td);
                }
            }
            if constexpr (PIV == PIV_WATCH) {
                pw.exact = valid && pivots_out_of_range(pw, f.db0, f.dep);
                if (__builtin_expect(__any_sync(0xffffffffu, pw.exact), 0)) {
                    f = {};
                    // rows k .. k + 3 of the pass; a row past the system's end is an
                    // identity row, and its last row has no coupling below (PAD)
                    auto rows4 = [&](int k, bool first, bool last) {
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            double v[4] = {0.0, 1.0, 0.0, 0.0};
                            if (valid && k + r < mlen) {
                                const size_t o = (size_t)(r0 + k + r) * ns + sys;
#pragma unroll
                                for (int i = 0; i < 4; ++i)
                                    if (!PAD || i != 2 || r0 + k + r + 1 < args.n_row)
                                        v[i] = gen.in[i][o];
                            }
                            wide_row<PIV_EXACT>(f, first ? r : (last ? M - 4 + r : 4), v[0], v[1],
                                                v[2], v[3], pw);
                            ta[r] = f.alp;
                            tg[r] = f.gap;
                            td[r] = f.dep;
                        }
                    };
                    rows4(0, true, false);
                    tmem_store_rows(tcol, ta, tg, td);
#pragma unroll 1
                    for (int k = 4; k < TR; k += 4) {
                        rows4(k, false, false);
                        tmem_store_rows(tcol + k * 6, ta, tg, td);
                    }
#pragma unroll
                    for (int k = TR; k < M; k += 4) {
                        rows4(k, false, k == M - 4);
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            al[k - TR + r] = ta[r];
                            ga[k - TR + r] = tg[r];
                            de[k - TR + r] = td[r];
                        }
                    }
                }
            }
            if constexpr (PAD) f.ab0 = r0 == 0 ? 0.0 : f.ab0;  // no row above the first
            wide_reduced(f, red + q * RP + s, fstride);
        }
        __syncthreads();

        // ------------------------------------------------ reduced system
        {
            const int per_pass = T / W;  // systems per pass
            const int p = tid % W;
            double* pb = pub + (it & 1) * 6 * SYS;
            for (int base = 0; base < SYS; base += per_pass) {
                const int sp = base + tid / W;
                const bool act = sp < SYS && p < nseg;
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
                    reduced_condense(l0, u0, b0, l1, u1, b1, p, nseg, W, act, f, d);
                    if (act) {  // over the fields this thread has read
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            src[i * fstride] = f[i];
                            src[(3 + i) * fstride] = d[i];
                            if (p == 0) pb[i * SYS + sp] = f[i];
                            if (p == nseg - 1) pb[(3 + i) * SYS + sp] = d[i];
                        }
                    }
                } else {
                    double xf, xl;
                    if constexpr (FILT)
                        reduced_solve_filtered<CYCLIC>(l0, u0, b0, l1, u1, b1, p, nseg, W, filt_r,
                                                       act, xf, xl);
                    else
                        reduced_solve_shfl<CYCLIC>(l0, u0, b0, l1, u1, b1, p, nseg, W, act, xf,
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
                const int r = tid % WC;
                for (int base = 0; base < SYS; base += T / WC) {
                    const int sp = base + tid / WC;
                    double f[3] = {0, 0, 0}, d[3] = {0, 0, 0};
                    if (sp < SYS && r < cl) {
                        const double* src = cg::this_cluster().map_shared_rank(pb, r) + sp;
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            f[i] = src[i * SYS];
                            d[i] = src[(3 + i) * SYS];
                        }
                    }
                    double lam, rho;
                    reduced_outer<CYCLIC>(f, d, r, cl, WC, lam, rho);
                    if (sp < SYS && r == c) {
                        outer[sp] = lam;
                        outer[SYS + sp] = rho;
                    }
                }
            }
        }
        __syncthreads();

        // ------------------------------------------------ back substitution
        double x_first, x_last;
        {
            const double* src = red + q * RP + s;
            if constexpr (CLUSTER) {
                const double lam = outer[s], rho = outer[SYS + s];
                x_first = src[0] + lam * src[1 * fstride] + rho * src[2 * fstride];
                x_last = src[3 * fstride] + lam * src[4 * fstride] + rho * src[5 * fstride];
            } else {
                x_first = src[0];
                x_last = src[fstride];
            }
        }
        double* xp = args.X + (size_t)(r0 + M - 1) * ns + sys;
        double xn = x_last;
        // systems past the batch are zero-filled (0 / 0 pivots): nothing of them
        // is stored or counted
        auto put = [&](int k, double x) {
            if (valid && (!PAD || k < mlen)) {
                *xp = x;
                nonfinite = fma(x, 0.0, nonfinite);
            }
            xp -= ns;
        };
        put(M - 1, x_last);
#pragma unroll
        for (int k = M - 2; k >= TR; --k) {
            xn = de[k - TR] - al[k - TR] * x_first - ga[k - TR] * xn;
            put(k, xn);
        }
        tmem_wait_st();
#pragma unroll
        for (int k0 = TR - 4; k0 >= 0; k0 -= 4) {
            uint32_t wa[8], wg[8], wd[8];
            tmem_load_rows(tcol + k0 * 6, wa, wg, wd);
#pragma unroll
            for (int r = 3; r >= 0; --r) {
                if (k0 + r == 0) continue;  // row 0 is x_first
                xn = tmem_word(wd, r) - tmem_word(wa, r) * x_first - tmem_word(wg, r) * xn;
                put(k0 + r, xn);
            }
        }
        put(0, x_first);
    }
    if (nonfinite != 0.0) raise_status(args.status, ST_NONFINITE);
    if (!ok && (GEN ? warp == 0 : tid == 0))
        for (int i = 0; i < nst; ++i) mbar_wait_bounded(&full[i], 0, nullptr, 1u << 8);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0)
        tmem_dealloc(*static_cast<volatile uint32_t*>(tslot), (uint32_t)wide_tmem_cols(nwarps));
    if constexpr (CLUSTER) tile_cluster_sync(cl);  // peers may still read this CTA's rows
}

}  // namespace btdma

// CUDA kernels and their launchers, one instantiation per storage format
// (tcym_kern_su{2,3}_f{32,64}*.cu).
//
// A thread takes a site, a site pair (FP32 formats with even nz), one of its directions or
// one of its links (the FP64 step: tasks of a tile, tcym_march.cuh).  Reductions are
// deterministic: each block writes a partial record (FP64) and the last block to finish sums
// the records in block order, so a result never depends on scheduling.
#pragma once

#include <cuda_runtime.h>

#include "tcym_march.cuh"
#include "tcym_site.cuh"

namespace tcym {

// partial record of one block: 9 sums and 3 maxima
enum : int {
    P_ESQ0 = 0, P_BSQ0 = 3, P_GSQ = 6, P_USQ = 7, P_EDB = 8, P_GMAX = 9, P_GABS = 10, P_UMAX = 11, P_WIDTH = 12
};
// device result block (doubles), written by finish_record
enum : int {
    R_ESQ0 = 0, R_BSQ0 = 3, R_GMAX = 6, R_GRMS = 7, R_GABS = 8, R_UMAX = 9, R_URMS = 10, R_EDB = 11,
    R_NCS = 12, R_NCS_COMP = 13, R_NONFINITE = 14,
    R_TICKET = 15,  // an integer: blocks of the running reduction that are done (0 between reductions)
    R_WIDTH = 16
};

#ifndef TCYM_SU2_THREADS
#define TCYM_SU2_THREADS 128
#endif
constexpr int kThreadsSU2 = TCYM_SU2_THREADS;
constexpr int kThreadsSU3 = 128;
constexpr int kRedThreads = 256;
// Resident blocks per SM requested for the per-site step and the checkerboard flow
// (register cap = 65536 / (blocks * threads)).
template <int FMT> constexpr int min_blocks_for() {
    return Fmt<FMT>::NA == 8 ? 4 : (FMT == FMT_SU2_F32 ? 8 : 1);
}

template <int FMT> constexpr int threads_for() { return Fmt<FMT>::NA == 3 ? kThreadsSU2 : kThreadsSU3; }

// The paired step (FP32 formats, even nz): one thread per site pair, 128 per
// block; resident blocks per SM requested (register cap 65536 / (blocks * 128)).
constexpr int kThreadsPair = 128;
// 1: blocks away from the seam run a copy of the step without the lane-swap
// tests; 0: one copy, the swaps decided per load
#ifndef TCYM_PAIR_SEAM_SPLIT
#define TCYM_PAIR_SEAM_SPLIT 1
#endif
// SU(3): 4 blocks (128 registers, no spills) measured 0.331 ms per 128^3 step
// against 0.342 ms at 3 (166 registers)
#ifndef TCYM_SU3_PAIR_MINBLOCKS
#define TCYM_SU3_PAIR_MINBLOCKS 4
#endif
// SU(2): 7 blocks (72 registers, a 4-byte spill) measured 0.090 ms per 128^3
// step against 0.094 ms at 6 (80 registers) and 0.107 ms at 5 (96, no spill)
#ifndef TCYM_SU2_PAIR_MINBLOCKS
#define TCYM_SU2_PAIR_MINBLOCKS 7
#endif
template <int FMT> constexpr int pair_min_blocks_for() {
    return Fmt<FMT>::NA == 8 ? TCYM_SU3_PAIR_MINBLOCKS : TCYM_SU2_PAIR_MINBLOCKS;
}
// L2 prefetch at the start of a block of the linear paired step: bit 0 the
// block's own field lines, bit 1 the lines of U_0, U_1 one pair-plane up in z
#ifndef TCYM_PAIR_PREFETCH
#define TCYM_PAIR_PREFETCH 0
#endif

// The lines a block of the linear paired step (pairs [p0, p0 + kThreadsPair))
// reads first from DRAM: its own fields, loaded only when each direction's
// update needs them, and the links U_0, U_1 of the pairs one step up in z,
// which its plaquettes read before the block owning them runs.  Each thread
// issues a few L2 prefetches (hints: no registers held, nothing waits on them),
// all inside the field and link arrays.  Planes: SU(3) FP32 links 6 x 16 B per
// pair and direction, fields 4 x 16 B; SU(2) FP32 links 2 x 16 B, fields 3 x 8 B.
template <int FMT>
__device__ __forceinline__ void prefetch_pair_block(const Geom &g, const void *Uin, const void *E, int64_t p0, int what) {
    constexpr bool su3 = Fmt<FMT>::NA == 8;
    constexpr int LP = su3 ? 6 : 2, LB = 16;   // link planes per direction, bytes per pair
    constexpr int EP = su3 ? 4 : 3, EB = su3 ? 16 : 8;
    constexpr int e_lines = 3 * EP * (kThreadsPair * EB / 128);
    constexpr int z_lines = 2 * LP * (kThreadsPair * LB / 128);
    const int64_t Vh = g.V >> 1;
    const int64_t sz = (int64_t)g.nx * g.ny;
    int64_t pz = p0 + sz;  // one pair-plane up; from the last plane, the seam's partner plane 0
    if (pz >= Vh) pz -= Vh;
    for (int i = threadIdx.x; i < e_lines + z_lines; i += kThreadsPair) {
        const char *addr = nullptr;
        if (i < e_lines) {
            if (!(what & 1)) continue;
            constexpr int per = kThreadsPair * EB / 128;
            const int plane = i / per;
            const int64_t q = p0 + (int64_t)(i % per) * (128 / EB);
            if (q < Vh) addr = static_cast<const char *>(E) + ((int64_t)plane * Vh + q) * EB;
        } else {
            if (!(what & 2)) continue;
            constexpr int per = kThreadsPair * LB / 128;
            const int j = i - e_lines;
            const int plane = j / per;  // direction plane / LP, component plane % LP
            const int64_t q = pz + (int64_t)(j % per) * (128 / LB);
            if (q < Vh) addr = static_cast<const char *>(Uin) + ((int64_t)plane * Vh + q) * LB;
        }
        if (addr) asm volatile("prefetch.global.L2 [%0];" ::"l"(addr));
    }
}

inline int grid_for(int64_t n, int threads) {
    int64_t b = (n + threads - 1) / threads;
    return (int)(b < 1 ? 1 : b);
}

template <class T> StepCoef<T> coef_cast(const StepCoef<double> &c) {
    StepCoef<T> r;
    r.mode = c.mode;
    r.seed = c.seed;
    r.step = c.step;
    for (int i = 0; i < 3; ++i) {
        r.fc[i] = (T)c.fc[i]; r.cnu[i] = (T)c.cnu[i]; r.uc[i] = (T)c.uc[i];
        r.damp[i] = (T)c.damp[i]; r.kick[i] = (T)c.kick[i];
    }
    return r;
}

// ------------------------------------------------------------------ kernels
// shared-memory slots of the plaquette projections (site_step, site_step_pair)
template <int FMT> constexpr int plaq_slots() { return 3 * Fmt<FMT>::NA; }

// the per-site step (FP32 with odd nz, FP64 by step_tile; DO_U false: the E update alone),
// sites [s0, s1)
template <int FMT, bool DO_U>
__global__ void __launch_bounds__(threads_for<FMT>(), min_blocks_for<FMT>()) k_step(Geom g, const void *Uin, void *Uout, void *E,
                                                             StepCoef<typename Fmt<FMT>::T> c, int64_t s0, int64_t s1) {
    __shared__ typename Fmt<FMT>::T sm[plaq_slots<FMT>() * threads_for<FMT>()];
    const int64_t s = s0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= s1) return;
    site_step<Fmt<FMT>, DO_U>(g, Uin, Uout, E, c, s, 0, sm + threadIdx.x, threads_for<FMT>());
}

// One block of the FP64 step (tcym_march.cuh): phases 1 and 2 of each of its planes.
template <class F, bool DO_U>
__device__ __forceinline__ void march_block(const Geom &g, const void *Uin, void *Uout, void *E,
                                            const StepCoef<typename F::T> &c, const MarchTile &t, const SiteRange &r,
                                            int64_t block, uint64_t step_add) {
    extern __shared__ __align__(16) unsigned char march_sh[];
    const March<F> m(g, Uin, t, r, block, march_sh);
    const int tid = threadIdx.x, nt = blockDim.x;
    m.setup(tid, nt);
    __syncthreads();
    for (int z = m.z0; z < m.z1; ++z) {
        m.projections(z, tid, nt);
        __syncthreads();
        m.template links<DO_U>(z, tid, nt, Uout, E, c, r, step_add);
        __syncthreads();
    }
}
// Resident blocks of kMarchThreads per SM: two at 128 registers for SU(3) (FP64 keeps 24
// bytes of spills; at one block, 255 registers, the FP64 unit is not kept busy), three for SU(2).
template <int FMT> constexpr int march_min_blocks() { return Fmt<FMT>::NA == 8 ? 2 : 3; }
// DO_U: the whole step, the new links into Uout; else the E update alone
template <int FMT, bool DO_U>
__global__ void __launch_bounds__(kMarchThreads, march_min_blocks<FMT>())
    k_march(Geom g, const void *Uin, void *Uout, void *E, StepCoef<typename Fmt<FMT>::T> c, MarchTile t, SiteRange r) {
    march_block<Fmt<FMT>, DO_U>(g, Uin, Uout, E, c, t, r, blockIdx.x, 0);
}
template <int FMT> __global__ void __launch_bounds__(128) k_update_u(Geom g, void *U, const void *E,
                                                                     StepCoef<typename Fmt<FMT>::T> c) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s < g.V) site_update_u<Fmt<FMT>>(g, U, E, c, s);
}

// one thread per site pair (FP32 formats, even nz); blocks touching the seam
// take the lane-swapping loads
// TILED = false: the linear mapping, compiled apart so its index arithmetic
// stays as light as the kernel's register budget wants
template <int FMT, bool TILED>
__global__ void __launch_bounds__(kThreadsPair, pair_min_blocks_for<FMT>())
    k_step_pair(Geom g, const void *Uin, void *Uout, void *E, StepCoef<float> c, Tile t) {
    __shared__ f2 sm[plaq_slots<FMT>() * kThreadsPair];
    int64_t p;
    bool seam;
    if constexpr (TILED) {
        if (!tile_pair(g, t, blockIdx.x, threadIdx.x, p, seam)) return;
    } else {
        const int64_t p0 = ((int64_t)blockIdx.x + t.b0) * kThreadsPair;
        if (TCYM_PAIR_PREFETCH) prefetch_pair_block<FMT>(g, Uin, E, p0, TCYM_PAIR_PREFETCH);
        p = p0 + threadIdx.x;
        if (p >= (g.V >> 1)) return;
        seam = pairs_touch_seam(g, p0, kThreadsPair);
    }
#if TCYM_PAIR_SEAM_SPLIT
    if (seam) site_step_pair<Fmt<FMT>, true>(g, Uin, Uout, E, c, p, 0, sm + threadIdx.x, kThreadsPair);
    else site_step_pair<Fmt<FMT>, false>(g, Uin, Uout, E, c, p, 0, sm + threadIdx.x, kThreadsPair);
#else
    site_step_pair<Fmt<FMT>, true>(g, Uin, Uout, E, c, p, 0, sm + threadIdx.x, kThreadsPair);
#endif
}

// The paired step of a small lattice: a pair's three plaquettes, then its three links, by
// three threads (warps 0, 1, 2 of a block of 32 pairs), the same arithmetic a third as
// long.  Below about a wave of such blocks a step is the latency of one thread's work:
// SU(3) at 24^3 13.4 us by k_step_pair on GB300.  split_step(): the lattices that take it.
constexpr int kSplitPairs = 32;
template <int FMT>
__global__ void __launch_bounds__(3 * kSplitPairs, Fmt<FMT>::NA == 8 ? 5 : 8)
    k_step_split(Geom g, const void *Uin, void *Uout, void *E, StepCoef<float> c) {
    using F = Fmt<FMT>;
    __shared__ f2 sm[plaq_slots<FMT>() * kSplitPairs];
    const int mu = threadIdx.x / kSplitPairs, i = threadIdx.x - mu * kSplitPairs;
    const int64_t p0 = (int64_t)blockIdx.x * kSplitPairs, Vh = g.V >> 1;
    const int64_t p = p0 + i < Vh ? p0 + i : Vh - 1;  // a thread past the end repeats the last pair's plaquette
    const PairNbhd nb(g, p);
    const bool seam = pairs_touch_seam(g, p0, kSplitPairs);
    if (seam) pair_plaquette<F, true>(g, nb, Uin, mu, p, sm + i, kSplitPairs);
    else pair_plaquette<F, false>(g, nb, Uin, mu, p, sm + i, kSplitPairs);
    __syncthreads();
    if (p0 + i >= Vh) return;
    if (seam) pair_link<F, true>(g, nb, Uin, Uout, E, c, c, mu, p, 0, sm + i, kSplitPairs);
    else pair_link<F, false>(g, nb, Uin, Uout, E, c, c, mu, p, 0, sm + i, kSplitPairs);
}

// Checkerboard sub-sweep of (parity, mu): the sites of the parity, for even extents,
// t -> (x, row) with x of the right parity
template <class T> struct FlowCoefT {
    T fc[3], cn[3], uc[3];
};
template <int FMT>
__global__ void __launch_bounds__(threads_for<FMT>(), min_blocks_for<FMT>()) k_flow_cb(Geom g, void *U, int parity, int mu,
                                                                FlowCoefT<typename Fmt<FMT>::T> c) {
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.V / 2) return;
    const int hx = g.nx / 2;
    int64_t row = t / hx;
    int xh = (int)(t - row * hx);
    int y = (int)(row % g.ny), z = (int)(row / g.ny);
    int x = 2 * xh + ((y + z + parity) & 1);
    int64_t s = x + (int64_t)g.nx * row;
    link_flow<Fmt<FMT>>(g, U, mu, c.fc, c.cn, c.uc, s);
}
// FP32 pair storage with nz / 2 even (a pair's sites have one parity): a thread per pair,
// a block a tile of 8 pairs of the parity x 4 rows x 4 planes, or of other powers of two where
// that leaves fewer threads idle (cb_tile).  It waits for links from
// L2 (13 of them a thread), of which the tile finds its neighbours' in L1.  A sweep (six
// sub-sweeps) on GB300: SU(2) 96^3 149 us per site (one lane of every pair vector, twice the
// sectors), 92 us by pairs in index order, 76 us by tiles; SU(3) 96^3 522 / 258 / 256 us.
// (16 x 4 x 2: 75 and 250 us, but half idle at nx = 16.)
template <int FMT>
__global__ void __launch_bounds__(kThreadsPair, Fmt<FMT>::NA == 8 ? 4 : 8)
    k_flow_cb_pair(Geom g, void *U, int parity, int mu, FlowCoefT<float> c, CbTile t) {
    const int i = threadIdx.x, nzh = g.nz >> 1;
    const int xh = (blockIdx.x << t.lx) + (i & ((1 << t.lx) - 1));
    const int y = (blockIdx.y << t.ly) + (i >> t.lx & ((1 << t.ly) - 1));
    const int z0 = blockIdx.z << t.lz, z = z0 + (i >> (t.lx + t.ly));
    if (2 * xh >= g.nx || y >= g.ny || z >= nzh) return;
    const int64_t p = 2 * xh + ((y + z + parity) & 1) + (int64_t)g.nx * (y + (int64_t)g.ny * z);
    // block-uniform: does the block hold a plane next to the seam?
    if (z0 == 0 || z0 + (1 << t.lz) >= nzh) pair_link_flow<Fmt<FMT>, true>(g, U, mu, c.fc, c.cn, c.uc, p);
    else pair_link_flow<Fmt<FMT>, false>(g, U, mu, c.fc, c.cn, c.uc, p);
}

// Reductions.  On GB300 a warp's FP64 add takes 16 cycles of its SM's one FP64 unit, so
// a block's record (up to 12 values) is summed with as few as the tree allows: every
// thread's values go to shared memory, a warp takes a value, adds its 256/32 columns and
// finishes by shuffles, 12 warp-adds a value where a shuffle tree in every warp took 48.
// Only the slots a kernel fills (USED) are reduced.  The last block to finish sums the
// blocks' records in block order and writes the result, so a reduction is one launch
// (a second one cost 5 to 10 us); the order of every sum depends on the launch's shape
// alone.
constexpr unsigned kUsedSample = (1u << P_ESQ0) * 7u | (1u << P_BSQ0) * 7u | 1u << P_EDB;
constexpr unsigned kUsedGauss = 1u << P_GSQ | 1u << P_GMAX | 1u << P_GABS;
constexpr unsigned kUsedAll = (1u << P_WIDTH) - 1u;
constexpr int used_count(unsigned used) { return used == 0 ? 0 : (int)(used & 1u) + used_count(used >> 1); }
// the slot of the q-th used value
__device__ __forceinline__ int used_slot(unsigned used, int q) {
    for (; q > 0; --q) used &= used - 1;
    return __ffs((int)used) - 1;
}
__device__ __forceinline__ double slot_op(int k, double a, double b) { return k < P_GMAX ? a + b : fmax(a, b); }
__device__ __forceinline__ double warp_op(int k, double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = slot_op(k, v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// The block's record from its threads' values, the used slots only, one after the other
// (COMPACT) or each in its place; own: of these the ones that the block fills (the others of
// its record are not written); sh: used_count(USED) * NT doubles.
template <unsigned USED, int NT, bool COMPACT>
__device__ __forceinline__ void block_record(const double *v, double *sh, double *record, unsigned own = USED) {
    constexpr int NQ = used_count(USED);
    const int lane = threadIdx.x & 31;
    int q = 0;
#pragma unroll
    for (int k = 0; k < P_WIDTH; ++k)
        if (USED >> k & 1) {
            if (own >> k & 1) sh[q * NT + threadIdx.x] = v[k];
            ++q;
        }
    __syncthreads();
    for (q = threadIdx.x >> 5; q < NQ; q += NT / 32) {
        const int k = used_slot(USED, q);
        if (!(own >> k & 1)) continue;
        double r = sh[q * NT + lane];
#pragma unroll
        for (int i = 1; i < NT / 32; ++i) r = slot_op(k, r, sh[q * NT + lane + 32 * i]);
        r = warp_op(k, r);
        if (lane == 0) record[COMPACT ? q : k] = r;
    }
}

// What the summed records become.
struct Finish {
    double *result;              // the result block
    double *ctl;                 // a restore's control block (finish_record), else nullptr
    double inv_v, na_v, three_v; // 1 / V, na V, 3 V
    double ncs_dt;               // N_CS advances by ncs_dt E.B / (8 pi^2) (0: it stays)
    double tol;                  // restore: the stopping rule of iteration `it`
    int it, check;
};
inline Finish make_finish(double *result, int na, int64_t V, double ncs_dt, double *ctl = nullptr, double tol = 0.0,
                          int it = 0, bool check = false) {
    return Finish{result, ctl, 1.0 / (double)V, (double)na * (double)V, 3.0 * (double)V, ncs_dt, tol, it, check ? 1 : 0};
}

// The totals t[0..P_WIDTH) into the result block, by the block's first warps: the
// divisions and roots (hundreds of cycles each) side by side.  A restore (f.ctl): a
// non-finite reduction sets ctl[1] and stops it after this iteration; with `check` (the
// deviation the reference tests, GaussRestore.cpp:150), a signed maximum <= tol stops it.
__device__ __forceinline__ void finish_record(const double *t, const Finish &f, double *edb = nullptr,
                                              double *ncs = nullptr) {
    double *res = f.result;
    const int i = threadIdx.x;
    if (i < 6) res[R_ESQ0 + i] = t[P_ESQ0 + i] * f.inv_v;  // E^2 and B^2: the same order in both
    else if (i == 6) res[R_GMAX] = t[P_GMAX];
    else if (i == 7) res[R_GABS] = t[P_GABS];
    else if (i == 8) res[R_UMAX] = t[P_UMAX];
    else if (i == 32) res[R_GRMS] = sqrt(t[P_GSQ] / f.na_v);
    else if (i == 64) res[R_URMS] = sqrt(t[P_USQ] / f.three_v);
    else if (i == 96) {
        bool bad = false;
        for (int k = 0; k < P_WIDTH; ++k) bad |= !isfinite(t[k]);
        res[R_EDB] = t[P_EDB];
        bad |= res[R_NONFINITE] != 0.0;
        res[R_NONFINITE] = bad ? 1.0 : 0.0;
        double sum = res[R_NCS];
        if (f.ncs_dt != 0.0) {
            // Kahan: sum += ncs_dt * E.B / (8 pi^2) with running compensation
            const double inv8pi2 = 0.125 / (3.14159265358979323846 * 3.14159265358979323846);
            const double y = f.ncs_dt * t[P_EDB] * inv8pi2 - res[R_NCS_COMP];
            const double s = sum + y;
            res[R_NCS_COMP] = (s - sum) - y;
            res[R_NCS] = sum = s;
        }
        if (edb) *edb = t[P_EDB];
        if (ncs) *ncs = sum;
        if (f.ctl) {
            const double gmax = t[P_GMAX];
            bad |= !(gmax == gmax);
            if (bad) f.ctl[1] = 1.0;
            if (bad || (f.check && gmax <= f.tol)) f.ctl[0] = fmin(f.ctl[0], (double)(f.it + 1));
        }
    }
}

// The totals of `blocks` records into t[0..P_WIDTH): thread i takes the records i, i + NT,
// ..., all slots' loads in flight together (a warp a slot, one load after the other, waited
// 10 us for the 1024 records of a 64^3 lattice), then the block's columns are summed as any
// block's.  own(b): the slots that record b holds; sh: used_count(USED) * NT doubles.
template <unsigned USED> struct AllSlots {
    __device__ unsigned operator()(unsigned) const { return USED; }
};
template <unsigned USED, int NT, bool COMPACT, class OWN = AllSlots<USED>>
__device__ __forceinline__ void sum_records(const double *partial, int blocks, double *sh, double *t,
                                            const OWN &own = OWN()) {
    constexpr int NQ = used_count(USED);
    double v[P_WIDTH];
#pragma unroll
    for (int k = 0; k < P_WIDTH; ++k) v[k] = 0.0;  // every slot's sum or maximum starts at 0
#pragma unroll 4
    for (int b = threadIdx.x; b < blocks; b += NT) {
        const unsigned filled = own(b);
        int q = 0;
#pragma unroll
        for (int k = 0; k < P_WIDTH; ++k)
            if (USED >> k & 1) {
                if (filled >> k & 1) v[k] = slot_op(k, v[k], __ldcg(&partial[COMPACT ? (int64_t)b * NQ + q : (int64_t)b * P_WIDTH + k]));
                ++q;
            }
    }
    if (threadIdx.x < P_WIDTH) t[threadIdx.x] = 0.0;
    block_record<USED, NT, false>(v, sh, t);
    __syncthreads();
}

// The end of a reduction kernel of NT >= 128 threads a block: this block's record, and
// in the last block the result.
template <unsigned USED, int NT, class OWN = AllSlots<USED>>
__device__ __forceinline__ void reduce_and_finish(const double *v, double *partial, const Finish &f,
                                                  const OWN &own = OWN()) {
    static_assert(NT >= 128, "finish_record spreads over four warps");
    __shared__ double sh[used_count(USED) * NT], total[P_WIDTH];
    __shared__ int last;
    const unsigned block = blockIdx.x + gridDim.x * blockIdx.y, blocks = gridDim.x * gridDim.y;
    block_record<USED, NT, true>(v, sh, partial + (int64_t)block * used_count(USED), own(block));
    __threadfence();  // the record before the ticket
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned *ticket = reinterpret_cast<unsigned *>(f.result + R_TICKET);
        last = atomicAdd(ticket, 1u) == blocks - 1;
        if (last) *ticket = 0;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (f.ctl && (double)f.it >= f.ctl[0]) return;  // a deviation past the restore's stop: the result stays
    sum_records<USED, NT, true>(partial, blocks, sh, total, own);
    finish_record(total, f);
}
// the record alone (callers that sum the records in a launch of their own)
__device__ __forceinline__ void block_partial(const double *vals, double *partial) {
    __shared__ double sh[used_count(kUsedGauss) * kRedThreads];
    double *record = partial + (int64_t)blockIdx.x * P_WIDTH;
    if (threadIdx.x < P_WIDTH) record[threadIdx.x] = 0.0;
    __syncthreads();
    block_record<kUsedGauss, kRedThreads, false>(vals, sh, record);
}

// FULL: the Gauss and unitarity slots are filled too
template <int FMT, bool FULL>
__global__ void __launch_bounds__(kRedThreads) k_observables(Geom g, const void *U, const void *E, int mask,
                                                             double *partial, Finish fin) {
    using F = Fmt<FMT>;
    double v[P_WIDTH];
#pragma unroll
    for (int k = 0; k < P_WIDTH; ++k) v[k] = 0.0;
    v[P_GMAX] = 0.0;  // signed maximum starts at 0 (GaussLawViolation.cpp:17,44)
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < g.V; s += (int64_t)gridDim.x * blockDim.x) {
        SiteObs<F> o;
        site_observables<F>(g, U, E, mask, s, o);
        for (int m = 0; m < 3; ++m) { v[P_ESQ0 + m] += o.esq[m]; v[P_BSQ0 + m] += o.bsq[m]; }
        for (int a = 0; a < F::NA; ++a) {
            v[P_GSQ] += o.g[a] * o.g[a];
            v[P_GMAX] = fmax(v[P_GMAX], o.g[a]);
            v[P_GABS] = fmax(v[P_GABS], fabs(o.g[a]));
        }
        for (int m = 0; m < 3; ++m) { v[P_USQ] += o.un[m] * o.un[m]; v[P_UMAX] = fmax(v[P_UMAX], o.un[m]); }
        v[P_EDB] += o.edotb;
    }
    reduce_and_finish<FULL ? kUsedAll : kUsedSample, kRedThreads>(v, partial, fin);
}

// Storage units (Unit): pairs for the FP32 formats with even nz, sites for FP64.
template <int FMT> constexpr bool unit_pairs() { return Fmt<FMT>::PAIRED; }

// The observables of a lattice in storage units: the N_CS sample (mask OBS_EDOTB: E^2,
// plaquette B^2, clover E.B) and, FULL (OBS_ALL), the Gauss and unitarity violations.  A
// thread takes a unit and a direction (blockIdx.y; FULL: 3 is the violations), so a small
// lattice has three or four times its units in threads.  The sample's sums over components
// run in the storage's precision, those of all observables in FP64 (FieldSums, ViolationSums), and
// everything across units in FP64.  SU(3) FP64 is bound by its multiply-adds (0.87 ms at 48^3),
// the others wait for L2.  All observables, with the call, on GB300, one thread a site / by unit
// and direction: SU(3) FP64 16^3 375 / 75 us, 48^3 1074 / 949; SU(2) FP64 16^3 91 / 38, 48^3 224 /
// 199; SU(3) FP32 16^3 86 / 30, 64^3 412 / 145, 128^3 2792 / 973; SU(2) FP32 64^3 147 / 74, 128^3
// 640 / 309.  SU(3) by two blocks of 255 registers: three of 168 spill (FP64 48^3 997 us).
constexpr int kThreadsObs = 128;
// a unit's contribution to its direction's sums
template <class T> __device__ __forceinline__ double lanes_sum(T x) { return (double)x; }
template <> __device__ __forceinline__ double lanes_sum<f2>(f2 x) { return (double)x.v.x + (double)x.v.y; }
__device__ __forceinline__ double lanes_max(double x, double m) { return fmax(m, x); }
__device__ __forceinline__ float lanes_max(f2 x, float m) { return fmaxf(m, fmaxf(x.v.x, x.v.y)); }
// the slots of a block's record: those of its direction, or the violations' (a block of 128
// sites that summed all 12 spent a tenth of a small FP64 lattice's time on zeros)
struct UnitSlots {
    unsigned blocks;  // of a direction
    __device__ unsigned operator()(unsigned b) const {
        const unsigned mu = b / blocks;
        return mu < 3 ? (1u << P_ESQ0 | 1u << P_BSQ0) << mu | 1u << P_EDB
                      : 1u << P_GSQ | 1u << P_USQ | 1u << P_GMAX | 1u << P_GABS | 1u << P_UMAX;
    }
};
template <int FMT, bool FULL>
__global__ void __launch_bounds__(kThreadsObs, Fmt<FMT>::NA == 8 ? 2 : 4)
    k_obs_units(Geom g, const void *U, const void *E, double *partial, Finish fin) {
    using F = Fmt<FMT>;
    using UN = Unit<F, unit_pairs<FMT>()>;
    using T = typename UN::T;
    const int mu = blockIdx.y;
    const int64_t n = UN::count(g), step = (int64_t)gridDim.x * blockDim.x;
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double es = 0.0, bs = 0.0, edb = 0.0, gsq = 0.0, usq = 0.0, gmax = 0.0, gabs = 0.0;
    typename UN::C umax = 0;
    if constexpr (FULL) {
        if (mu < 3) {
            FieldSums<T, F::NA> sums;
            for (int again = 0; again < 2; ++again) {
                bs = 0.0;
                for (int64_t i = i0; i < n; i += step) {
                    T e[F::NA], et[F::NA], b[F::NA], bsq;
                    unit_clover<F, unit_pairs<FMT>()>(g, U, E, i, mu, e, et, b, bsq);
                    if (again) sums.add64(e, et, b);
                    else sums.add(e, et, b);
                    bs += lanes_sum(bsq);
                }
                if (again || sums.exact()) break;
            }
            es = sums.sq;
            edb = sums.dot;
        } else {
            ViolationSums<T, F::NA> sums;
            for (int again = 0; again < 2; ++again) {
                usq = 0.0;
                for (int64_t i = i0; i < n; i += step) {
                    WideSum<T> s[F::NA];
                    unit_gauss<F, unit_pairs<FMT>()>(g, U, E, i, s);
                    if (again) sums.add64(s);
                    else sums.add(s);
                    const UN u(g, i);
#pragma unroll 1
                    for (int d = 0; d < 3; ++d) {
                        const T un = UN::G::unitarity_square(u.link(U, d, 0));
                        usq += lanes_sum(un);
                        umax = lanes_max(un, umax);
                    }
                }
                if (again || sums.exact()) break;
            }
            gsq = sums.sq;
            gmax = sums.most;
            gabs = sums.mag;
        }
    } else {
        for (int64_t i = i0; i < n; i += step) {
            T esq, bsq;
            edb += lanes_sum(unit_sample<F, unit_pairs<FMT>()>(g, U, E, i, mu, esq, bsq));
            es += lanes_sum(esq);
            bs += lanes_sum(bsq);
        }
    }
    double v[P_WIDTH];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        v[P_ESQ0 + k] = k == mu ? es : 0.0;
        v[P_BSQ0 + k] = k == mu ? bs : 0.0;
    }
    v[P_EDB] = edb;
    v[P_GSQ] = gsq;
    v[P_USQ] = usq;
    v[P_GMAX] = gmax;
    v[P_GABS] = gabs;
    v[P_UMAX] = sqrt((double)umax);
    reduce_and_finish<FULL ? kUsedAll : kUsedSample, kThreadsObs>(v, partial, fin, UnitSlots{gridDim.x});
}

// Gauss violation into the FP64 scratch G[a*V + s]; partial maxima as for observables.
template <int FMT>
__device__ __forceinline__ void gauss_compute_block(const Geom &g, const void *U, const void *E, double *G,
                                                    double *v) {
    using F = Fmt<FMT>;
#pragma unroll
    for (int k = 0; k < P_WIDTH; ++k) v[k] = 0.0;
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < g.V; s += (int64_t)gridDim.x * blockDim.x) {
        double gv[F::NA];
        site_gauss<F>(g, U, E, s, gv);
        for (int a = 0; a < F::NA; ++a) {
            G[a * g.V + s] = gv[a];
            v[P_GSQ] += gv[a] * gv[a];
            v[P_GMAX] = fmax(v[P_GMAX], gv[a]);
            v[P_GABS] = fmax(v[P_GABS], fabs(gv[a]));
        }
    }
}
template <int FMT>
__global__ void __launch_bounds__(kRedThreads) k_gauss_compute(Geom g, const void *U, const void *E, double *G,
                                                               double *partial) {
    double v[P_WIDTH];
    gauss_compute_block<FMT>(g, U, E, G, v);
    block_partial(v, partial);
}

template <int FMT>
__global__ void __launch_bounds__(threads_for<FMT>()) k_gauss_update(Geom g, const void *U, void *E, const double *G,
                                                                     double gam) {
    int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= g.V) return;
    site_gauss_update<Fmt<FMT>>(g, U, E, G, gam, s);
}

// The same two kernels for iteration `it` of a restore whose control block
// holds, in ctl[0], the first iteration that is not to run (the last block of the
// deciding reduction lowers it, when every block has read it): a kernel of a later iteration returns at once,
// so the host can queue many iterations between its checks.
template <int FMT>
__global__ void __launch_bounds__(kRedThreads) k_gauss_compute_it(Geom g, const void *U, const void *E, double *G,
                                                                  double *partial, Finish fin) {
    if ((double)fin.it >= fin.ctl[0]) return;  // the same value for every thread of the grid
    double v[P_WIDTH];
    gauss_compute_block<FMT>(g, U, E, G, v);
    reduce_and_finish<kUsedGauss, kRedThreads>(v, partial, fin);
}
template <int FMT>
__global__ void __launch_bounds__(threads_for<FMT>()) k_gauss_update_it(Geom g, const void *U, void *E, const double *G,
                                                                        double gam, const double *ctl, int it) {
    if ((double)it >= ctl[0]) return;
    int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= g.V) return;
    site_gauss_update<Fmt<FMT>>(g, U, E, G, gam, s);
}

// The restore by units (FP32 with even nz in site pairs, FP64): a thread a unit forms the
// deviation (k_deviation); FP32 pairs then do a sub-step's update and the next deviation in
// one pass over the links, from the fields Ein and G Gin into Eout and Gout (k_restore_next),
// FP64 updates with a thread a unit and direction (k_restore, blockIdx.y).  FP32 is bound by
// memory and launches, FP64 by its multiply-adds, of which one pass does half as many again
// (each neighbour's update a second time).  An iteration of three sub-steps on GB300, one pass
// / two: SU(3) FP32 32^3 46 / 58 us, 64^3 133 / 120, 128^3 702 / 786; SU(2) FP32 32^3 36 / 46, 128^3
// 275 / 355; FP64 48^3 SU(3) 960 / 669, SU(2) 234 / 185.
constexpr int kThreadsRestore = 128;
template <int FMT> using UnitG = typename Unit<Fmt<FMT>, unit_pairs<FMT>()>::T;
// a unit's violation into G and its thread's sums v
template <int FMT, class C>
__device__ __forceinline__ void take_deviation(const UnitG<FMT> *gv, UnitG<FMT> *G, int64_t n, int64_t i, C &gsq, C &gmax,
                                               C &gabs) {
#pragma unroll
    for (int a = 0; a < Fmt<FMT>::NA; ++a) {
        G[a * n + i] = gv[a];
        if constexpr (unit_pairs<FMT>()) {
            const float x = gv[a].v.x, y = gv[a].v.y;
            gsq = fmaf(x, x, fmaf(y, y, gsq));
            gmax = fmaxf(gmax, fmaxf(x, y));
            gabs = fmaxf(gabs, fmaxf(fabsf(x), fabsf(y)));
        } else {
            gsq = fma(gv[a], gv[a], gsq);
            gmax = fmax(gmax, gv[a]);
            gabs = fmax(gabs, fabs(gv[a]));
        }
    }
}
__device__ __forceinline__ void finish_deviation(double gsq, double gmax, double gabs, double *partial, const Finish &fin) {
    double v[P_WIDTH];
#pragma unroll
    for (int k = 0; k < P_WIDTH; ++k) v[k] = 0.0;
    v[P_GSQ] = gsq;
    v[P_GMAX] = gmax;
    v[P_GABS] = gabs;
    reduce_and_finish<kUsedGauss, kThreadsRestore>(v, partial, fin);
}
// the deviation in iteration fin.it: a launch of an iteration past the stop returns at once
template <int FMT>
__global__ void __launch_bounds__(kThreadsRestore, 4)
    k_deviation(Geom g, const void *U, const void *E, UnitG<FMT> *G, double *partial, Finish fin) {
    using F = Fmt<FMT>;
    using RU = Unit<F, unit_pairs<FMT>()>;
    if ((double)fin.it >= fin.ctl[0]) return;  // the same value for every thread of the grid
    const int64_t n = RU::count(g);
    typename RU::C gsq = 0, gmax = 0, gabs = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        UnitG<FMT> gv[F::NA];
        unit_deviation<F, unit_pairs<FMT>()>(g, U, E, i, gv);
        take_deviation<FMT>(gv, G, n, i, gsq, gmax, gabs);
    }
    finish_deviation(gsq, gmax, gabs, partial, fin);
}
template <int FMT>
__global__ void __launch_bounds__(kThreadsRestore, 4)
    k_restore(Geom g, const void *U, void *E, const UnitG<FMT> *G, double gam, const double *ctl, int it) {
    using RU = Unit<Fmt<FMT>, unit_pairs<FMT>()>;
    if ((double)it >= ctl[0]) return;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < RU::count(g)) unit_restore<Fmt<FMT>, unit_pairs<FMT>()>(g, U, E, G, (typename RU::C)gam, i, blockIdx.y);
}
// The update belongs to iteration `it`, the deviation to fin.it; a deviation past the stop
// leaves the result of the last one.  (SU(3): three blocks of 168 registers; four spill, 809 us
// at 128^3.)
template <int FMT>
__global__ void __launch_bounds__(kThreadsRestore, Fmt<FMT>::NA == 8 ? 3 : 4)
    k_restore_next(Geom g, const void *U, const void *Ein, void *Eout, const UnitG<FMT> *Gin, UnitG<FMT> *Gout, float gam,
                   int it, double *partial, Finish fin) {
    using F = Fmt<FMT>;
    if ((double)it >= fin.ctl[0]) return;
    const int64_t n = Unit<F, true>::count(g);
    float gsq = 0, gmax = 0, gabs = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        UnitG<FMT> gv[F::NA];
        unit_restore_next<F, true>(g, U, Ein, Eout, Gin, gam, i, gv);
        take_deviation<FMT>(gv, Gout, n, i, gsq, gmax, gabs);
    }
    finish_deviation(gsq, gmax, gabs, partial, fin);
}

template <int FMT> __global__ void k_set_zero(Geom g, void *U, void *E) {
    int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s < g.V) site_set_zero<Fmt<FMT>>(g, U, E, s);
}
template <int FMT> __global__ void k_gaussian_efield(Geom g, void *E, double sigma, uint64_t seed, uint64_t step) {
    int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s < g.V) site_gaussian_efield<Fmt<FMT>>(g, E, sigma, seed, s, step);
}
template <int FMT> __global__ void k_random_links(Geom g, void *U, double sigma, uint64_t seed) {
    int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s < g.V) site_random_links<Fmt<FMT>>(g, U, sigma, seed, s);
}
template <int FMT> __global__ void k_block(Geom gs, Geom gd, const void *Us, void *Ud) {
    int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s < gd.V) site_block<Fmt<FMT>>(gs, gd, Us, Ud, s);
}
template <int FMT> __global__ void k_reunitarize(Geom g, void *U) {
    int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s < g.V) site_reunitarize<Fmt<FMT>>(g, U, s);
}
// FP32 storage: one thread per pair and direction (blockIdx.y)
template <int FMT> __global__ void __launch_bounds__(128) k_reunitarize_pair(Geom g, void *U) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < pair_sites(g.V)) pair_reunitarize<Fmt<FMT>>(U, g.V, blockIdx.y, p);
}
template <int FMT>
__global__ void k_geodesic(Geom g, const void *Uold, const void *Unew, double c, void *Umid, void *Emid) {
    int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s < g.V) site_geodesic<Fmt<FMT>>(g, Uold, Unew, c, Umid, Emid, s);
}
// Sites [s0, s0 + n) between the reference's AoS FP64 arrays and the device
// layout.  A block takes kAosSites sites: their AoS records (SU(3): 432 + 192 B a
// site) pass through shared memory, so that the AoS side is read or written by
// consecutive threads at consecutive addresses; each thread then converts one link.
constexpr int kAosSites = 64, kAosThreads = 192;
template <int FMT> constexpr int aos_link_doubles() { return Fmt<FMT>::NA == 3 ? 4 : 18; }
template <int FMT> constexpr size_t aos_smem() {
    return sizeof(double) * kAosSites * 3 * (aos_link_doubles<FMT>() + Fmt<FMT>::NA);
}
template <int FMT>
__global__ void __launch_bounds__(kAosThreads)
    k_from_aos(Geom g, void *U, void *E, const double *Ua, const double *Ea, int64_t s0, int64_t n) {
    using F = Fmt<FMT>;
    constexpr int NMD = aos_link_doubles<FMT>(), NA = F::NA;
    extern __shared__ double aos_sh[];
    double *su = aos_sh, *se = aos_sh + kAosSites * 3 * NMD;
    const int64_t b0 = s0 + (int64_t)blockIdx.x * kAosSites;
    const int ns = (int)(n - (b0 - s0) < kAosSites ? n - (b0 - s0) : kAosSites);
    if (Ua)
        for (int i = threadIdx.x; i < ns * 3 * NMD; i += blockDim.x) su[i] = Ua[b0 * 3 * NMD + i];
    if (Ea)
        for (int i = threadIdx.x; i < ns * 3 * NA; i += blockDim.x) se[i] = Ea[b0 * 3 * NA + i];
    __syncthreads();
    const int l = threadIdx.x, site = l / 3, mu = l - 3 * site;
    if (site >= ns) return;
    site_link_from_aos<F>(g, U, E, Ua ? su : nullptr, Ea ? se : nullptr, site, b0 + site, mu);
}
template <int FMT>
__global__ void __launch_bounds__(kAosThreads)
    k_to_aos(Geom g, const void *U, const void *E, double *Ua, double *Ea, int64_t s0, int64_t n) {
    using F = Fmt<FMT>;
    constexpr int NMD = aos_link_doubles<FMT>(), NA = F::NA;
    extern __shared__ double aos_sh[];
    double *su = aos_sh, *se = aos_sh + kAosSites * 3 * NMD;
    const int64_t b0 = s0 + (int64_t)blockIdx.x * kAosSites;
    const int ns = (int)(n - (b0 - s0) < kAosSites ? n - (b0 - s0) : kAosSites);
    const int l = threadIdx.x, site = l / 3, mu = l - 3 * site;
    if (site < ns) site_link_to_aos<F>(g, U, E, Ua ? su : nullptr, Ea ? se : nullptr, site, b0 + site, mu);
    __syncthreads();
    if (Ua)
        for (int i = threadIdx.x; i < ns * 3 * NMD; i += blockDim.x) Ua[b0 * 3 * NMD + i] = su[i];
    if (Ea)
        for (int i = threadIdx.x; i < ns * 3 * NA; i += blockDim.x) Ea[b0 * 3 * NA + i] = se[i];
}

// ------------------------------------------------------------------ launchers
template <int FMT> struct Launch {
    using F = Fmt<FMT>;
    using T = typename F::T;
    static constexpr int FMT_ID = FMT;
    static constexpr int TPB = threads_for<FMT>();

    // One fused step (E and links).  t: the block tiling of the paired step (FP32
    // formats with even nz), m: of the FP64 step.
    static cudaError_t step(const Geom &g, const void *Uin, void *Uout, void *E, const StepCoef<double> &cd, const Tile &t,
                            const MarchTile &m, cudaStream_t st) {
        if constexpr (F::PAIRED) {
            if (paired_step(g)) {
                const StepCoef<T> c = coef_cast<T>(cd);
                const unsigned blocks = (unsigned)tile_blocks(g, t);
                if (!t.tx && split_step(g))
                    k_step_split<FMT><<<grid_for(g.V >> 1, kSplitPairs), 3 * kSplitPairs, 0, st>>>(g, Uin, Uout, E, c);
                else if (t.tx) k_step_pair<FMT, true><<<blocks, kThreadsPair, 0, st>>>(g, Uin, Uout, E, c, t);
                else k_step_pair<FMT, false><<<blocks, kThreadsPair, 0, st>>>(g, Uin, Uout, E, c, t);
                return cudaGetLastError();
            }
        }
        return step_sites<true>(g, Uin, Uout, E, cd, m, SiteRange{0, g.nz, 0, g.V}, st);
    }
    // the E update alone, per site
    static cudaError_t update_e(const Geom &g, const void *U, void *E, const StepCoef<double> &cd, const MarchTile &m,
                                cudaStream_t st) {
        return step_sites<false>(g, U, nullptr, E, cd, m, SiteRange{0, g.nz, 0, g.V}, st);
    }
    static cudaError_t update_u(const Geom &g, void *U, const void *E, const StepCoef<double> &cd, cudaStream_t st) {
        k_update_u<FMT><<<grid_for(g.V, 128), 128, 0, st>>>(g, U, E, coef_cast<T>(cd));
        return cudaGetLastError();
    }
    // the sites of r (r.z0, r.z1: its planes), per site
    template <bool DO_U>
    static cudaError_t step_sites(const Geom &g, const void *Uin, void *Uout, void *E, const StepCoef<double> &cd,
                                  const MarchTile &m, const SiteRange &r, cudaStream_t st) {
        const StepCoef<T> c = coef_cast<T>(cd);
        if constexpr (!F::PAIRED) {
            if (m.tx != 0) {
                const unsigned blocks = (unsigned)march_blocks(m, r.z1 - r.z0);
                k_march<FMT, DO_U><<<blocks, m.threads, march_smem<F>(m), st>>>(g, Uin, Uout, E, c, m, r);
                return cudaGetLastError();
            }
        }
        k_step<FMT, DO_U><<<grid_for(r.s1 - r.s0, TPB), TPB, 0, st>>>(g, Uin, Uout, E, c, r.s0, r.s1);
        return cudaGetLastError();
    }
    // Lattices whose paired step spreads a pair over three threads (k_step_split): up to
    // about a wave of its blocks on GB300's 152 multiprocessors (5 of 32 SU(3) pairs each, 8 of
    // SU(2)'s).  Per step by k_step_pair / k_step_split on GB300: SU(3)
    // 16^3 13.4 / 8.2 us, 24^3 13.4 / 8.3, 32^3 14.4 / 12.3, 48^3 23.7 / 26.6; SU(2) 16^3 to
    // 32^3 8.2 / 6.2 us, 48^3 10.3 / 10.3.
    static bool split_step(const Geom &g) { return (g.V >> 1) <= (F::NA == 8 ? 25000 : 33000); }
    // Does step() take the paired kernel (one thread per site pair)?
    static bool paired_step(const Geom &g) { return F::PAIRED && g.nz % 2 == 0; }
    // One fused step (E and links) of the storage indices [i0, i1) only: site
    // pairs when paired_step(g), else sites; i0 a multiple of 128 for pairs.
    // The linear block mapping.
    static cudaError_t step_range(const Geom &g, const void *Uin, void *Uout, void *E, const StepCoef<double> &cd,
                                  int64_t i0, int64_t i1, const MarchTile &m, cudaStream_t st) {
        if (i1 <= i0) return cudaSuccess;
        if constexpr (F::PAIRED) {
            if (paired_step(g)) {
                Tile t{0, 0, 0, 0, 0, (int)(i0 / kThreadsPair)};
                const unsigned blocks = (unsigned)((i1 - i0 + kThreadsPair - 1) / kThreadsPair);
                k_step_pair<FMT, false><<<blocks, kThreadsPair, 0, st>>>(g, Uin, Uout, E, coef_cast<T>(cd), t);
                return cudaGetLastError();
            }
        }
        const int64_t plane = (int64_t)g.nx * g.ny;
        return step_sites<true>(g, Uin, Uout, E, cd, m,
                           SiteRange{(int)(i0 / plane), (int)((i1 + plane - 1) / plane), i0, i1}, st);
    }
    static cudaError_t flow_cb(const Geom &g, void *U, int parity, int mu, const double *fc, const double *cn,
                               const double *uc, cudaStream_t st) {
        FlowCoefT<T> c;
        for (int i = 0; i < 3; ++i) { c.fc[i] = (T)fc[i]; c.cn[i] = (T)cn[i]; c.uc[i] = (T)uc[i]; }
        if constexpr (F::PAIRED) {
            if (cb_pairs(g, F::NA == 8)) {
                const CbTile t = cb_tile(g);
                const dim3 grid((unsigned)grid_for(g.nx / 2, 1 << t.lx), (unsigned)grid_for(g.ny, 1 << t.ly),
                                (unsigned)grid_for(g.nz / 2, 1 << t.lz));
                k_flow_cb_pair<FMT><<<grid, kThreadsPair, 0, st>>>(g, U, parity, mu, c, t);
                return cudaGetLastError();
            }
        }
        k_flow_cb<FMT><<<grid_for(g.V / 2, TPB), TPB, 0, st>>>(g, U, parity, mu, c);
        return cudaGetLastError();
    }
    static int reduce_grid(const Geom &g, int max_blocks) {
        int b = grid_for(g.V, kRedThreads);
        return b < max_blocks ? b : max_blocks;
    }
    // the observables `mask` into fin's result block; max_blocks: records in `partial`
    static cudaError_t observables(const Geom &g, const void *U, const void *E, int mask, double *partial,
                                   int max_blocks, const Finish &fin, cudaStream_t st) {
        if ((mask == OBS_EDOTB || mask == OBS_ALL) && (!F::PAIRED || g.nz % 2 == 0)) {
            const int need = grid_for(Unit<F, unit_pairs<FMT>()>::count(g), kThreadsObs);
            if (mask == OBS_ALL) {  // at most max_blocks records
                const int x = need < max_blocks / 4 ? need : max_blocks / 4;
                k_obs_units<FMT, true><<<dim3((unsigned)x, 4), kThreadsObs, 0, st>>>(g, U, E, partial, fin);
            } else {
                const int x = need < max_blocks / 3 ? need : max_blocks / 3;
                k_obs_units<FMT, false><<<dim3((unsigned)x, 3), kThreadsObs, 0, st>>>(g, U, E, partial, fin);
            }
            return cudaGetLastError();
        }
        const int blocks = reduce_grid(g, max_blocks);
        if (mask & (OBS_GAUSS | OBS_UNIT))
            k_observables<FMT, true><<<blocks, kRedThreads, 0, st>>>(g, U, E, mask, partial, fin);
        else
            k_observables<FMT, false><<<blocks, kRedThreads, 0, st>>>(g, U, E, mask, partial, fin);
        return cudaGetLastError();
    }
    // The restore.  Does a sub-step update and form the next deviation in one launch?
    static bool restore_fused(const Geom &g) { return F::PAIRED && g.nz % 2 == 0; }
    // bytes of one G buffer of the fused restore
    static size_t restore_g_bytes(const Geom &g) { return sizeof(f2) * F::NA * (size_t)(g.V >> 1); }
    // the deviation G of E, in iteration fin.it: by units, or per site (FP32, odd nz; G: na V doubles)
    static cudaError_t restore_deviation(const Geom &g, const void *U, const void *E, void *G, double *partial,
                                         int max_blocks, const Finish &fin, cudaStream_t st) {
        if constexpr (F::PAIRED) {
            if (g.nz % 2) {
                k_gauss_compute_it<FMT><<<reduce_grid(g, max_blocks), kRedThreads, 0, st>>>(
                    g, U, E, static_cast<double *>(G), partial, fin);
                return cudaGetLastError();
            }
        }
        // max_blocks is 8 a multiprocessor.  FP64: 3 (a grid of 4 would hold every register for
        // the whole launch, and the request loop's ticks wait for its blocks: 2.0 ms a tick
        // beside a 128^3 preparation, against 0.24 ms alone)
        const int need = grid_for(Unit<F, unit_pairs<FMT>()>::count(g), kThreadsRestore);
        const int most = F::PAIRED ? max_blocks : max_blocks / 8 * 3;
        k_deviation<FMT><<<need < most ? need : most, kThreadsRestore, 0, st>>>(g, U, E, static_cast<UnitG<FMT> *>(G),
                                                                                partial, fin);
        return cudaGetLastError();
    }
    // the update by it in iteration `it` (not fused)
    static cudaError_t restore_update(const Geom &g, const void *U, void *E, const void *G, double gam, const double *ctl,
                                      int it, cudaStream_t st) {
        if constexpr (F::PAIRED) {
            k_gauss_update_it<FMT><<<grid_for(g.V, TPB), TPB, 0, st>>>(g, U, E, static_cast<const double *>(G), gam, ctl, it);
        } else {
            k_restore<FMT><<<dim3((unsigned)grid_for(g.V, kThreadsRestore), 3), kThreadsRestore, 0, st>>>(
                g, U, E, static_cast<const UnitG<FMT> *>(G), gam, ctl, it);
        }
        return cudaGetLastError();
    }
    // both (fused)
    static cudaError_t restore_step(const Geom &g, const void *U, const void *Ein, void *Eout, const void *Gin, void *Gout,
                                    double gam, int it, double *partial, int max_blocks, const Finish &fin,
                                    cudaStream_t st) {
        if constexpr (F::PAIRED) {
            const int need = grid_for(g.V >> 1, kThreadsRestore);
            k_restore_next<FMT><<<need < max_blocks ? need : max_blocks, kThreadsRestore, 0, st>>>(
                g, U, Ein, Eout, static_cast<const UnitG<FMT> *>(Gin), static_cast<UnitG<FMT> *>(Gout), (float)gam, it,
                partial, fin);
            return cudaGetLastError();
        }
        return cudaErrorInvalidValue;
    }
    static cudaError_t set_zero(const Geom &g, void *U, void *E, cudaStream_t st) {
        k_set_zero<FMT><<<grid_for(g.V, 256), 256, 0, st>>>(g, U, E);
        return cudaGetLastError();
    }
    static cudaError_t gaussian_efield(const Geom &g, void *E, double sigma, uint64_t seed, uint64_t step,
                                       cudaStream_t st) {
        k_gaussian_efield<FMT><<<grid_for(g.V, 128), 128, 0, st>>>(g, E, sigma, seed, step);
        return cudaGetLastError();
    }
    static cudaError_t random_links(const Geom &g, void *U, double sigma, uint64_t seed, cudaStream_t st) {
        k_random_links<FMT><<<grid_for(g.V, 128), 128, 0, st>>>(g, U, sigma, seed);
        return cudaGetLastError();
    }
    static cudaError_t geodesic(const Geom &g, const void *Uold, const void *Unew, double c, void *Umid, void *Emid,
                                cudaStream_t st) {
        k_geodesic<FMT><<<grid_for(g.V, 128), 128, 0, st>>>(g, Uold, Unew, c, Umid, Emid);
        return cudaGetLastError();
    }
    // the blocked links of gs on gd (half the even extents)
    static cudaError_t block(const Geom &gs, const Geom &gd, const void *Us, void *Ud, cudaStream_t st) {
        k_block<FMT><<<grid_for(gd.V, 128), 128, 0, st>>>(gs, gd, Us, Ud);
        return cudaGetLastError();
    }
    static cudaError_t reunitarize(const Geom &g, void *U, cudaStream_t st) {
        if constexpr (F::PAIRED)
            k_reunitarize_pair<FMT><<<dim3((unsigned)grid_for(pair_sites(g.V), 128), 3), 128, 0, st>>>(g, U);
        else
            k_reunitarize<FMT><<<grid_for(g.V, 128), 128, 0, st>>>(g, U);
        return cudaGetLastError();
    }
    // sites [s0, s0 + n) (n < 0: all)
    static cudaError_t from_aos(const Geom &g, void *U, void *E, const double *Ua, const double *Ea, cudaStream_t st,
                                int64_t s0 = 0, int64_t n = -1) {
        if (n < 0) n = g.V - s0;
        k_from_aos<FMT><<<grid_for(n, kAosSites), kAosThreads, aos_smem<FMT>(), st>>>(g, U, E, Ua, Ea, s0, n);
        return cudaGetLastError();
    }
    static cudaError_t to_aos(const Geom &g, const void *U, const void *E, double *Ua, double *Ea, cudaStream_t st,
                              int64_t s0 = 0, int64_t n = -1) {
        if (n < 0) n = g.V - s0;
        k_to_aos<FMT><<<grid_for(n, kAosSites), kAosThreads, aos_smem<FMT>(), st>>>(g, U, E, Ua, Ea, s0, n);
        return cudaGetLastError();
    }
};

// Sum the block partials in block order and write the result block; optionally
// advance the Kahan-compensated N_CS by ncs_dt * E.B / (8 pi^2).
cudaError_t finalize_obs(const double *partial, int blocks, int na, int64_t V, double ncs_dt, double *result,
                         cudaStream_t st);
// loads k_finalize's code now (with lazy module loading it would load at its first launch)
cudaError_t preload_finalize();
}  // namespace tcym

// The FP64 step in blocks that share their plaquettes.  (The FP32 formats step in site
// pairs, site_step_pair, or for odd nz per site, site_step: there the step waits for links
// from L2 more than for arithmetic, and sharing the plaquettes measured slower: SU(3)
// pairs 55 us a 64^3 step against 49, single sites 319 us against 257 at 96 x 96 x 95.)
//
// The force on U_mu(x) sums, over nu != mu, the plaquette above the link (corner x)
// minus the one below it (corner x - nu) carried to x.  With P_{mu nu}(y) the
// plaquette that starts and ends at y, the loop below the link, run from x, is
// U_nu^-1(x-nu) P_{mu nu}(x-nu) U_nu(x-nu), and proj(V^-1 P V) = Ad(V^-1) proj(P)
// for a group element V.  So with p_{mu nu}(y) = proj(P_{mu nu}(y)) the reference's
// bracket (Dynamics.cpp:184-188) is
//   f_mu(x) = sum_nu c_nu [ p_{mu nu}(x) - Ad(U_nu^-1(x-nu)) p_{mu nu}(x-nu) ],
// and a step needs three plaquettes a site, each projected once and used by four links,
// and six rotations of an algebra vector, where the staple form takes three plaquettes,
// six lower staples and three more projections a site.  FP64 is bound by its
// multiply-adds (1.2 TFLOP/s on GB300): SU(3) about 2650 a site against 3230.
// Links may be a little off the group (copied from FP32 storage, loaded with few digits).  For
// SU(2) the identity holds for any quaternion V.  For SU(3) it is off by V's deviation eps (E
// by 0.6 eps of a dt = 0.05 step, where staples whose third rows follow from the first two are
// off by 1.2 eps), so plaquettes are whole products and Ad(V^-1) is taken as V^dagger p V.
//
// A block owns a tx x ty tile of a z-plane and walks zl planes up in z.  Per plane, phase
// 1 forms the projections of the tile and of the row and column just below it in x and
// y, phase 2 moves the tile's links; both spread (site, direction) tasks over the
// block's threads, with a barrier between, so that a small lattice has three times the
// threads of one site each.  The projections carried up in z stay in shared memory from
// one plane to the next (before the first plane they are formed from its links), so only
// the row and column are formed twice, by neighbouring blocks.  Every projection is the
// same arithmetic on the same links wherever it is formed: a result does not depend on
// the tiling.
#pragma once

#include "tcym_site.cuh"

namespace tcym {

// How the blocks cover the sites: tx x ty tiles of a plane, zl planes a block (tx 0: a
// lattice that steps faster by sites, site_step).
struct MarchTile {
    int tx, ty, tiles_x, tiles_y, zl, threads;
};
// The sites of a launch: planes [z0, z1), and of these the sites [s0, s1).
struct SiteRange {
    int z0, z1;
    int64_t s0, s1;
};
TCYM_HD int64_t march_blocks(const MarchTile &t, int planes) {
    return (int64_t)t.tiles_x * t.tiles_y * ((planes + t.zl - 1) / t.zl);
}
constexpr int kMarchThreads = 224;  // largest block: the 192 + 32 tasks of an 8 x 8 tile's phase 1
constexpr int kMarchSites = 64;     // largest tile
// A site of the tile or of its halo row or column: x + nx y, its slot among the
// projections, and the wraps of its neighbours.
struct MarchSite {
    int idx, flags;
};
enum : int { MS_SLOT = 0xfff, MS_XLAST = 1 << 12, MS_YLAST = 1 << 13, MS_XFIRST = 1 << 14, MS_YFIRST = 1 << 15,
             MS_XWRAP = 1 << 16, MS_YWRAP = 1 << 17 };
// shared memory of a block: three projections a site (and of the halo row and column),
// the two carried up from the plane below, and the table of sites
template <class F> TCYM_HD size_t march_smem(const MarchTile &t) {
    const int slots = (t.tx + 1) * (t.ty + 1), sites = t.tx * t.ty;
    return sizeof(typename F::T) * F::NA * (3 * slots + 2 * sites) + sizeof(MarchSite) * (sites + t.tx + t.ty);
}

template <class F> struct March {
    using T = typename F::T;
    using G = typename F::G;
    using Mat = typename F::Mat;
    static constexpr int NA = F::NA;

    const void *U;
    int64_t V;
    int nx, ny, nz, plane;
    int w, h, S, hx, hy;  // the tile: its extents, its sites, those of its halo column (x) and row (y)
    int x0, y0, stride, slots, sites;
    int z0, z1;           // planes of the block
    T *p, *below;
    MarchSite *info;

    TCYM_HD March(const Geom &g, const void *Uin, const MarchTile &t, const SiteRange &r, int64_t block, void *smem)
        : U(Uin), V(g.V), nx(g.nx), ny(g.ny), nz(g.nz), plane(g.nx * g.ny) {
        const int per = t.tiles_x * t.tiles_y;
        const int chunk = (int)(block / per), b = (int)(block - (int64_t)chunk * per);
        const int by = b / t.tiles_x, bx = b - by * t.tiles_x;
        x0 = bx * t.tx;
        y0 = by * t.ty;
        w = t.tx < nx - x0 ? t.tx : nx - x0;
        h = t.ty < ny - y0 ? t.ty : ny - y0;
        S = w * h;
        hx = w == nx ? 0 : h;  // a tile as wide as the lattice holds its own x neighbours
        hy = h == ny ? 0 : w;
        stride = t.tx + 1;
        slots = stride * (t.ty + 1);
        sites = t.tx * t.ty;
        z0 = r.z0 + chunk * t.zl;
        z1 = z0 + t.zl < r.z1 ? z0 + t.zl : r.z1;
        p = static_cast<T *>(smem);
        below = p + 3 * NA * slots;
        info = reinterpret_cast<MarchSite *>(below + 2 * NA * sites);
    }

    // the table: the tile's sites row by row, the halo row y0 - 1, the halo column x0 - 1
    TCYM_HD void setup(int tid, int nt) const {
        for (int e = tid; e < S + hy + hx; e += nt) {
            int lx, ly;
            if (e < S) { ly = e / w; lx = e - ly * w; }
            else if (e < S + hy) { ly = -1; lx = e - S; }
            else { lx = -1; ly = e - S - hy; }
            const int x = x0 + lx < 0 ? nx - 1 : x0 + lx, y = y0 + ly < 0 ? ny - 1 : y0 + ly;
            int f = (ly + 1) * stride + lx + 1;
            if (x == nx - 1) f |= MS_XLAST;
            if (y == ny - 1) f |= MS_YLAST;
            if (x == 0) f |= MS_XFIRST;
            if (y == 0) f |= MS_YFIRST;
            if (hx == 0 && lx == 0) f |= MS_XWRAP;
            if (hy == 0 && ly == 0) f |= MS_YWRAP;
            info[e] = MarchSite{x + nx * y, f};
        }
    }

    // p_{k,k+1} over kLoopScale at plane z
    TCYM_HD void plaquette(int k, MarchSite u, int z, T *pr) const {
        const int nu = k == 2 ? 0 : k + 1;
        const int64_t at = (int64_t)z * plane + u.idx;
        const int64_t ax = at + (u.flags & MS_XLAST ? 1 - nx : 1);
        const int64_t ay = at + (u.flags & MS_YLAST ? nx - plane : nx);
        const int64_t az = z == nz - 1 ? (int64_t)u.idx : at + plane;
        // P = [U_k(x) U_nu(x+k)] [U_nu(x) U_k(x+nu)]^dag
        const Mat a = F::load(U, V, k, at);
        const Mat b = F::load(U, V, nu, k == 0 ? ax : (k == 1 ? ay : az));
        const Mat t1 = G::template mulx<false, false>(a, b);
        const Mat c = F::load(U, V, nu, at);
        const Mat d = F::load(U, V, k, nu == 0 ? ax : (nu == 1 ? ay : az));
        const Mat t2 = G::template mulx<false, false>(c, d);
        G::loop_proj(t1, t2, pr);
    }

    // Phase 1 at plane z: tasks by plaquette plane (yz, zx, xy over the tile; xy and yz
    // over the halo row; xy and zx over the halo column), on the block's first plane
    // after the tile's yz and zx of the plane below, carried up.
    TCYM_HD void projections(int z, int tid, int nt) const {
        const int pro = z == z0 ? 2 * S : 0, total = pro + 3 * S + 2 * (hx + hy);
#pragma unroll 1
        for (int j = tid; j < total; j += nt) {
            int i = j < pro ? j : j - pro;
            int k, e;
            if (i < 3 * S) {
                const int q = (i >= S) + (i >= 2 * S);
                k = q == 2 ? 0 : q + 1;
                e = i - q * S;
            } else if ((i -= 3 * S) < 2 * hy) {
                k = i >= hy;
                e = S + (i >= hy ? i - hy : i);
            } else {
                i -= 2 * hy;
                k = i >= hx ? 2 : 0;
                e = S + hy + (i >= hx ? i - hx : i);
            }
            const MarchSite u = info[e];
            const int zp = j >= pro ? z : (z == 0 ? nz - 1 : z - 1);
            T pr[NA];
            plaquette(k, u, zp, pr);
            T *dst;
            int step;
            if (j < pro) {
                T t[NA];
                G::carry(F::load(U, V, 2, (int64_t)zp * plane + u.idx), pr, t);
                dst = below + (k - 1) * NA * sites + e;
                step = sites;
#pragma unroll
                for (int a = 0; a < NA; ++a) pr[a] = t[a];
            } else {
                dst = p + k * NA * slots + (u.flags & MS_SLOT);
                step = slots;
            }
#pragma unroll
            for (int a = 0; a < NA; ++a) dst[a * step] = pr[a];
        }
    }

    // Phase 2 at plane z: the force, E and (DO_U) the new link of every (site, direction)
    // of the tile in [s0, s1), and the projections carried up to the next plane.
    template <bool DO_U>
    TCYM_HD void links(int z, int tid, int nt, void *Uout, void *E, const StepCoef<T> &c, const SiteRange &r,
                       uint64_t step_add) const {
#pragma unroll 1
        for (int j = tid; j < 3 * S; j += nt) {
            const int mu = (j >= S) + (j >= 2 * S);
            const int e = j - mu * S;
            const MarchSite u = info[e];
            const int64_t at = (int64_t)z * plane + u.idx;
            T f[NA];
#pragma unroll
            for (int a = 0; a < NA; ++a) f[a] = T(0);
#pragma unroll 1
            for (int s = 0; s < 2; ++s) {
                // nu = mu + 1: +c p_{mu,mu+1}; nu = mu + 2: -c p_{mu+2,mu}
                int nu = mu + 1 + s;
                nu = nu >= 3 ? nu - 3 : nu;
                const int k = s ? nu : mu;
                const T ck = T(s ? -G::kLoopScale : G::kLoopScale) * sel3(c.cnu, nu);
                const T *own = p + k * NA * slots + (u.flags & MS_SLOT);
                // in x and y: the neighbour's projection carried here; in z: the one
                // carried up before, and this plane's own carried up for the next
                int from = 0;
                int64_t src = at;
                if (nu == 1) {
                    from = u.flags & MS_YWRAP ? (h - 1) * stride : -stride;
                    src += u.flags & MS_YFIRST ? plane - nx : -nx;
                }
                if (nu == 0) {
                    from = u.flags & MS_XWRAP ? w - 1 : -1;
                    src += u.flags & MS_XFIRST ? nx - 1 : -1;
                }
                T q[NA], t[NA];
#pragma unroll
                for (int a = 0; a < NA; ++a) q[a] = own[a * slots + from];
                G::carry(F::load(U, V, nu, src), q, t);
                if (nu == 2) {
                    T *b = below + (k - 1) * NA * sites + e;  // no other task's
#pragma unroll
                    for (int a = 0; a < NA; ++a) {
                        f[a] = fma(ck, q[a] - b[a * sites], f[a]);
                        b[a * sites] = t[a];
                    }
                } else {
#pragma unroll
                    for (int a = 0; a < NA; ++a) f[a] = fma(ck, own[a * slots] - t[a], f[a]);
                }
            }
            if (at < r.s0 || at >= r.s1) continue;
            T ev[NA];
            F::load_e(E, V, mu, at, ev);
            const T fc = sel3(c.fc, mu);
            if (c.mode == MODE_LANGEVIN) {
                T xi[NA];
                normals<T, NA>(c.seed, STREAM_NOISE, c.step + step_add, (uint32_t)at, (uint32_t)mu, xi);
                const T damp = sel3(c.damp, mu), kick = sel3(c.kick, mu);
#pragma unroll
                for (int a = 0; a < NA; ++a) ev[a] = ev[a] + fma(kick, xi[a], fma(-damp, ev[a], fc * f[a]));
            } else if (c.mode == MODE_FLOW) {
#pragma unroll
                for (int a = 0; a < NA; ++a) ev[a] = fc * f[a];
            } else {
#pragma unroll
                for (int a = 0; a < NA; ++a) ev[a] = fma(fc, f[a], ev[a]);
            }
            F::store_e(E, V, mu, at, ev);
            if (DO_U) F::store(Uout, V, mu, at, G::iexp_mul(sel3(c.uc, mu), ev, F::load(U, V, mu, at)));
        }
    }
};

// The blocks' cost, in multiply-adds of whole warps: phase 1's plaquettes (310 for SU(3) in
// FP64) and phase 2's links (572, of which E alone 350) of each plane, and the first plane's
// extra 2 S plaquettes with their rotations (454).
inline double march_warps(double n) { return 32.0 * (int)((n + 31) / 32); }
inline double march_plane(int S, int halo, bool links) {
    return 310 * march_warps(3 * S + 2 * halo) + (links ? 572 : 350) * march_warps(3 * S);
}
inline double march_first(int S) { return 454 * march_warps(2 * S); }
// The tiling of a lattice that has the share `sms` of a device's multiprocessors, alone or among
// others (an ensemble's members).  Its cost model is the work of the busiest multiprocessor, that
// with the most blocks: alone these are full ones, among others two of them, the rest the
// average block.  Fewer than six warps on it leave its FP64 unit idle in proportion, and every plane adds
// the latency of its two phases (as 6000 multiply-adds).  Blocks walk up to 16 planes, among
// others 8 (the launch's tail).
// Measured on GB300, FP64 per step, the rule's choice / 16 x 8 tiles of 8 planes: SU(3)
// 16^3 43 / 678 us, 48^3 587 / 714 us; SU(2) 16^3 12 / 140 us.
inline MarchTile march_tile(const Geom &g, double sms, bool alone, double *least = nullptr, bool links = true) {
    MarchTile best{};
    double cost = 0;
    for (int tx = g.nx < 16 ? g.nx : 16; tx > 0; --tx) {
        const int nx = (g.nx + tx - 1) / tx;
        if ((g.nx + nx - 1) / nx != tx) continue;  // as many smaller tiles do
        if (tx < 4 && best.tx) break;
        const int most = kMarchSites / tx;
        for (int ty = g.ny < most ? g.ny : most; ty > 0; --ty) {
            const int ny = (g.ny + ty - 1) / ty;
            if ((g.ny + ny - 1) / ny != ty) continue;
            if (tx * ty < 16 && best.tx) break;
            const int halo = (tx == g.nx ? 0 : ty) + (ty == g.ny ? 0 : tx), S = tx * ty;
            const double plane = march_plane(S, halo, links), first = march_first(S);
            double planes = 0, firsts = 0;  // of all tiles, ragged ones as they are
            for (int i = 0; i < 2; ++i)
                for (int j = 0; j < 2; ++j) {
                    const int w = i ? g.nx - tx * (nx - 1) : tx, h = j ? g.ny - ty * (ny - 1) : ty;
                    const double n = (double)(i ? 1 : nx - 1) * (j ? 1 : ny - 1);
                    planes += n * march_plane(w * h, (w == g.nx ? 0 : h) + (h == g.ny ? 0 : w), links);
                    firsts += n * march_first(w * h);
                }
            for (int zl = 1; zl <= g.nz && zl <= (alone ? 16 : 8); ++zl) {
                const int chunks = (g.nz + zl - 1) / zl;
                const double blocks = (double)nx * ny * chunks, per_sm = ceil(blocks / sms);
                const int tasks = 3 * S + 2 * halo + (zl == 1 ? 2 * S : 0);
                const int threads = tasks > kMarchThreads ? kMarchThreads : (tasks + 31) / 32 * 32;
                const double warps = per_sm * threads / 32, block = zl * plane + first;
                double c = per_sm * block;
                if (!alone && per_sm > 2) c = 2 * block + (per_sm - 2) * (g.nz * planes + chunks * firsts) / blocks;
                c = c * (warps < 6 ? 6 / warps : 1) + 6000.0 * zl;
                if (!best.tx || c < cost) {
                    cost = c;
                    best = MarchTile{tx, ty, nx, ny, zl, threads};
                }
            }
        }
    }
    if (least) *least = cost;
    return best;
}
// The cost of a step (links) or of the E update alone by sites (site_step in blocks of 128), by
// the same measure.
inline double sites_cost(int64_t V, double sms, bool links = true) {
    return (links ? 3150.0 : 2400.0) * 128 * ceil((double)((V + 127) / 128) / sms);
}
// The step of a lattice alone: by tiles, or by sites (tx 0) where that costs less: extents that
// the tiles fit badly, in waves of blocks that are nearly full.  By sites / by tiles, us a step
// on GB300, SU(3) 18 x 28 x 34 109 / 119, 26^3 109 / 150, 33 x 20 x 27 109 / 148, 24^3 109 / 105,
// 28^3 209 / 158, 48^3 619 / 587; SU(2) 26^3 25 / 33, 28^3 43 / 33.  E alone: SU(3) 32^3 162 / 165, 48^3
// 476 / 450; of SU(2), where tiles must cost a tenth less (its few operations weigh their
// barriers more), 32^3 33 / 36, 36^3 46 / 52, 40^3 60 / 58.
inline MarchTile step_tile(const Geom &g, double sms, bool su3, bool links) {
    double least;
    MarchTile t = march_tile(g, sms, true, &least, links);
    if (sites_cost(g.V, sms, links) * (su3 || links ? 1 : 0.9) < least) t.tx = 0;
    return t;
}

}  // namespace tcym

// TEST-ONLY host build of the per-site device code (not part of libtcym.so).
//
// Compiled by nvcc for the host only (no kernels), it runs the exact
// __host__ __device__ site functions the CUDA kernels call, in a loop over
// sites, on host arrays in the device storage layout.  tests/ use it to check
// the device arithmetic (both FP64 and FP32 formats) against the FP64 oracle
// on machines without a GPU.
#include <cstdint>
#include <cstring>
#include <vector>

#include "tcym_pipeline.h"
#include "tcym_march.cuh"

using namespace tcym;

namespace {

StepCoef<double> coef(int mode, double dt, double gamma, double T, uint64_t seed, uint64_t step) {
    // unit spacings (the same folding as tcym_coef in tcym_capi.cu)
    StepCoef<double> c;
    std::memset(&c, 0, sizeof(c));
    c.mode = mode;
    c.seed = seed;
    c.step = step;
    for (int mu = 0; mu < 3; ++mu) {
        c.fc[mu] = mode == MODE_FLOW ? -2.0 : -2.0 * dt;
        c.cnu[mu] = 1.0;
        c.uc[mu] = -dt;
        if (mode == MODE_LANGEVIN) {
            c.damp[mu] = gamma * dt;
            c.kick[mu] = std::sqrt(gamma) * std::sqrt(dt) * std::sqrt(2.0 * T);
        }
    }
    return c;
}

template <class T> StepCoef<T> cast(const StepCoef<double> &c) {
    StepCoef<T> r;
    r.mode = c.mode; r.seed = c.seed; r.step = c.step;
    for (int i = 0; i < 3; ++i) {
        r.fc[i] = (T)c.fc[i]; r.cnu[i] = (T)c.cnu[i]; r.uc[i] = (T)c.uc[i];
        r.damp[i] = (T)c.damp[i]; r.kick[i] = (T)c.kick[i];
    }
    return r;
}

template <int FMT> struct H {
    using F = Fmt<FMT>;
    using T = typename F::T;
    // pairs: 0 per-site step; 1 + tx: the paired step with tiling tx (0: linear)
    static void step(const Geom &g, const void *Uin, void *Uout, void *E, const StepCoef<double> &cd, int doE,
                     int doU, int pairs) {
        StepCoef<T> c = cast<T>(cd);
        if constexpr (F::PAIRED) {
            // the device's paired step, block by block and thread by thread as the kernel runs it
            if (pairs && doE && doU && g.nz % 2 == 0) {
                const Tile t = make_tile(g, pairs - 1);
                for (int64_t b = 0; b < tile_blocks(g, t); ++b)
                    for (int tid = 0; tid < 128; ++tid) {
                        int64_t p;
                        bool seam;
                        if (!tile_pair(g, t, b, tid, p, seam)) continue;
                        f2 sm[3 * F::NA];
                        if (seam) site_step_pair<F, true>(g, Uin, Uout, E, c, p, 0, sm, 1);
                        else site_step_pair<F, false>(g, Uin, Uout, E, c, p, 0, sm, 1);
                    }
                return;
            }
        }
        if (!doE) {
            for (int64_t s = 0; s < g.V; ++s) site_update_u<F>(g, Uout, E, c, s);
            return;
        }
        sites(g, Uin, Uout, E, c, doU, SiteRange{0, g.nz, 0, g.V});
    }
    // the per-site step as Launch::step_sites runs it
    static void sites(const Geom &g, const void *Uin, void *Uout, void *E, const StepCoef<T> &c, bool doU,
                      const SiteRange &r) {
        const MarchTile t = step_tile(g, 152, F::NA == 8, doU);
        if (!F::PAIRED && t.tx != 0) {
            march(g, Uin, Uout, E, c, doU, r, t);
            return;
        }
        T sm[3 * F::NA];
        for (int64_t s = r.s0; s < r.s1; ++s) {
            if (doU) site_step<F, true>(g, Uin, Uout, E, c, s, 0, sm, 1);
            else site_step<F, false>(g, Uin, Uout, E, c, s, 0, sm, 1);
        }
    }
    // the device's FP64 step, block by block, phase by phase and thread by thread
    static void march(const Geom &g, const void *Uin, void *Uout, void *E, const StepCoef<T> &c, bool doU,
                      const SiteRange &r, const MarchTile &t) {
        std::vector<unsigned char> sm(march_smem<F>(t));
        for (int64_t b = 0; b < march_blocks(t, r.z1 - r.z0); ++b) {
            const March<F> m(g, Uin, t, r, b, sm.data());
            for (int i = 0; i < t.threads; ++i) m.setup(i, t.threads);
            for (int z = m.z0; z < m.z1; ++z) {
                for (int i = 0; i < t.threads; ++i) m.projections(z, i, t.threads);
                for (int i = 0; i < t.threads; ++i) {
                    if (doU) m.template links<true>(z, i, t.threads, Uout, E, c, r, 0);
                    else m.template links<false>(z, i, t.threads, Uout, E, c, r, 0);
                }
            }
        }
    }
    // one fused step of the storage indices [i0, i1) as Launch::step_range runs it: the
    // paired step's linear blocks from block i0 / 128 (Tile::b0), or sites
    static void step_range(const Geom &g, const void *Uin, void *Uout, void *E, const StepCoef<double> &cd,
                           int64_t i0, int64_t i1) {
        StepCoef<T> c = cast<T>(cd);
        if constexpr (F::PAIRED) {
            if (g.nz % 2 == 0) {
                const Tile t{0, 0, 0, 0, 0, (int)(i0 / 128)};
                for (int64_t b = 0; b < (i1 - i0 + 127) / 128; ++b)
                    for (int tid = 0; tid < 128; ++tid) {
                        int64_t p;
                        bool seam;
                        if (!tile_pair(g, t, b, tid, p, seam)) continue;
                        f2 sm[3 * F::NA];
                        if (seam) site_step_pair<F, true>(g, Uin, Uout, E, c, p, 0, sm, 1);
                        else site_step_pair<F, false>(g, Uin, Uout, E, c, p, 0, sm, 1);
                    }
                return;
            }
        }
        const int64_t plane = (int64_t)g.nx * g.ny;
        sites(g, Uin, Uout, E, c, true, SiteRange{(int)(i0 / plane), (int)((i1 + plane - 1) / plane), i0, i1});
    }
    static void flow_cb(const Geom &g, void *U, double dtau, int nsweeps) {
        const T fc[3] = {T(-2), T(-2), T(-2)}, cn[3] = {T(1), T(1), T(1)}, uc[3] = {T(-dtau), T(-dtau), T(-dtau)};
        if constexpr (F::PAIRED) {
            if (g.nz % 4 == 0) {  // pairs of one parity, as the device takes them (small SU(2) lattices apart)
                const int64_t plane = (int64_t)g.nx * g.ny, Vh = g.V >> 1;
                for (int k = 0; k < 6 * nsweeps; ++k)
                    for (int64_t p = 0; p < Vh; ++p) {
                        Nbhd nb(g, p);
                        if (nb.parity() != k / 3 % 2) continue;
                        if (p < plane || p >= Vh - plane) pair_link_flow<F, true>(g, U, k % 3, fc, cn, uc, p);
                        else pair_link_flow<F, false>(g, U, k % 3, fc, cn, uc, p);
                    }
                return;
            }
        }
        for (int sw = 0; sw < nsweeps; ++sw)
            for (int p = 0; p < 2; ++p)
                for (int mu = 0; mu < 3; ++mu)
                    for (int64_t s = 0; s < g.V; ++s) {
                        Nbhd nb(g, s);
                        if (nb.parity() == p) link_flow<F>(g, U, mu, fc, cn, uc, s);
                    }
    }
    // E^2, plaquette B^2 and clover E.B of an FP64 site by the units' code, in place of site_observables'
    static void sample_units(const Geom &g, const void *U, const void *E, int64_t s, SiteObs<F> &o) {
        if constexpr (!F::PAIRED) {
            o.edotb = 0;
            for (int mu = 0; mu < 3; ++mu) o.edotb += unit_sample<F, false>(g, U, E, s, mu, o.esq[mu], o.bsq[mu]);
            WideSum<double> gv[F::NA];
            unit_gauss<F, false>(g, U, E, s, gv);
            for (int a = 0; a < F::NA; ++a) o.g[a] = lane64(gv[a], 0);
        }
    }
    static void observables(const Geom &g, const void *U, const void *E, int mask, double *out) {
        double esq[3] = {0, 0, 0}, bsq[3] = {0, 0, 0}, gsq = 0, usq = 0, edb = 0, gmax = 0, gabs = 0, umax = 0;
        for (int64_t s = 0; s < g.V; ++s) {
            SiteObs<F> o;
            site_observables<F>(g, U, E, mask, s, o);
            if (mask == OBS_ALL) sample_units(g, U, E, s, o);
            for (int m = 0; m < 3; ++m) { esq[m] += o.esq[m]; bsq[m] += o.bsq[m]; usq += o.un[m] * o.un[m]; umax = std::fmax(umax, o.un[m]); }
            for (int a = 0; a < F::NA; ++a) { gsq += o.g[a] * o.g[a]; gmax = std::fmax(gmax, o.g[a]); gabs = std::fmax(gabs, std::fabs(o.g[a])); }
            edb += o.edotb;
        }
        const double V = (double)g.V;
        for (int m = 0; m < 3; ++m) { out[3 + m] = esq[m] / V; out[6 + m] = bsq[m] / V; }
        out[1] = 0.5 * (out[3] + out[4] + out[5]);
        out[2] = 0.5 * (out[6] + out[7] + out[8]);
        out[0] = out[1] + out[2];
        out[9] = gmax;
        out[10] = std::sqrt(gsq / (F::NA * V));
        out[11] = umax;
        out[12] = std::sqrt(usq / (3 * V));
        out[13] = edb;
        out[14] = 0;
        out[15] = gabs;
    }
    // the N_CS sample through the paired code (FP32 pair storage, even nz): the
    // E^2, plaquette B^2 and clover E.B slots of observables(); false if not paired
    static bool edotb_pair(const Geom &g, const void *U, const void *E, double *out) {
        if constexpr (F::PAIRED) {
            if (g.nz % 2) return false;
            double esq[3] = {0, 0, 0}, bsq[3] = {0, 0, 0}, edb = 0;
            const int64_t Vh = g.V >> 1;
            for (int64_t p = 0; p < Vh; ++p)
                for (int mu = 0; mu < 3; ++mu) {
                    f2 e2, b2;
                    const f2 d = unit_sample<F, true>(g, U, E, p, mu, e2, b2);
                    esq[mu] += (double)e2.v.x + (double)e2.v.y;
                    bsq[mu] += (double)b2.v.x + (double)b2.v.y;
                    edb += (double)d.v.x + (double)d.v.y;
                }
            const double V = (double)g.V;
            for (int k = 0; k < 16; ++k) out[k] = 0;
            for (int m = 0; m < 3; ++m) { out[3 + m] = esq[m] / V; out[6 + m] = bsq[m] / V; }
            out[1] = 0.5 * (out[3] + out[4] + out[5]);
            out[2] = 0.5 * (out[6] + out[7] + out[8]);
            out[0] = out[1] + out[2];
            out[13] = edb;
            return true;
        }
        return false;
    }
    static void iexp_aos(double c, const double *alpha, double *out) {
        T e[F::NA];
        for (int a = 0; a < F::NA; ++a) e[a] = (T)alpha[a];
        auto m = F::G::iexp((T)c, e);
        if constexpr (F::NA == 3) {
            for (int k = 0; k < 4; ++k) out[k] = (double)m.q[k];
        } else {
            for (int i = 0; i < 3; ++i)
                for (int j = 0; j < 3; ++j) {
                    out[2 * (i + 3 * j)] = (double)m.m[i][j].re;
                    out[2 * (i + 3 * j) + 1] = (double)m.m[i][j].im;
                }
        }
    }
    // A with exp(i c A^a t^a) = V, V given in the reference AoS link layout
    static void ilog_aos(double c, const double *v, double *out) {
        typename F::G::Mat m;
        if constexpr (F::NA == 3) {
            for (int k = 0; k < 4; ++k) m.q[k] = (T)v[k];
        } else {
            for (int i = 0; i < 3; ++i)
                for (int j = 0; j < 3; ++j) m.m[i][j] = cx<T>{(T)v[2 * (i + 3 * j)], (T)v[2 * (i + 3 * j) + 1]};
        }
        T o[F::NA];
        F::G::ilog((T)c, m, o);
        for (int a = 0; a < F::NA; ++a) out[a] = (double)o[a];
    }
    // the Gauss violation of every site by the pairs' code, out[s * NA + a]
    static bool gauss_pair(const Geom &g, const void *U, const void *E, double *out) {
        if constexpr (F::PAIRED) {
            if (g.nz % 2) return false;
            const int64_t Vh = g.V >> 1;
            for (int64_t p = 0; p < Vh; ++p) {
                WideSum<f2> gv[F::NA];
                unit_gauss<F, true>(g, U, E, p, gv);
                for (int a = 0; a < F::NA; ++a) {
                    out[p * F::NA + a] = lane64(gv[a], 0);
                    out[(p + Vh) * F::NA + a] = lane64(gv[a], 1);
                }
            }
            return true;
        }
        return false;
    }
    // the same site by site, as the other formats measure it
    static void gauss_sites(const Geom &g, const void *U, const void *E, double *out) {
        for (int64_t s = 0; s < g.V; ++s) {
            SiteObs<F> o;
            site_observables<F>(g, U, E, OBS_GAUSS, s, o);
            for (int a = 0; a < F::NA; ++a) out[s * F::NA + a] = o.g[a];
        }
    }
    static void geodesic(const Geom &g, const void *Uold, const void *Unew, double c, void *Umid, void *Emid) {
        for (int64_t s = 0; s < g.V; ++s) site_geodesic<F>(g, Uold, Unew, c, Umid, Emid, s);
    }
    static void reunitarize(const Geom &g, void *U) {
        if constexpr (F::PAIRED) {
            for (int64_t p = 0; p < pair_sites(g.V); ++p)
                for (int mu = 0; mu < 3; ++mu) pair_reunitarize<F>(U, g.V, mu, p);
        } else {
            for (int64_t s = 0; s < g.V; ++s) site_reunitarize<F>(g, U, s);
        }
    }
    // the FP64 projection whatever the storage
    static void reunitarize_fp64(const Geom &g, void *U) {
        for (int64_t s = 0; s < g.V; ++s) site_reunitarize<F>(g, U, s);
    }
    // the restore by units as tcym_gauss_restore runs it: one pass a sub-step for pairs, two for FP64
    template <bool PAIR> static int restore_units(const Geom &g, const void *U, void *E, double tol, int maxit) {
        using RU = Unit<F, PAIR>;
        using RT = typename RU::T;
        using C = typename RU::C;
        const int64_t n = RU::count(g);
        const size_t ebytes = sizeof(C) * 3 * (PAIR ? 2 * n : n) * F::NA;
        std::vector<RT> G0(F::NA * n), G1(F::NA * n);
        std::vector<char> E1(ebytes);
        RT *G[2] = {G0.data(), G1.data()};
        void *Eb[2] = {E, E1.data()};
        const double gam[3] = {7.0 / 24.0, 7.0 / 48.0, 7.0 / 72.0};
        double gmax = 0;
        RT gv[F::NA];
        auto take = [&](int64_t i, RT *out) {
            for (int a = 0; a < F::NA; ++a) {
                out[a * n + i] = gv[a];
                if constexpr (PAIR) gmax = std::fmax(gmax, std::fmax((double)gv[a].v.x, (double)gv[a].v.y));
                else gmax = std::fmax(gmax, (double)gv[a]);
            }
        };
        auto deviation = [&]() {
            gmax = 0;
            for (int64_t i = 0; i < n; ++i) {
                unit_deviation<F, PAIR>(g, U, E, i, gv);
                take(i, G[0]);
            }
        };
        deviation();
        int it = 0, sub = 0;
        double last = gmax;
        while (it < maxit && last > tol) {
            for (int k = 0; k < 3; ++k) {
                if constexpr (PAIR) {
                    gmax = 0;
                    for (int64_t i = 0; i < n; ++i) {
                        unit_restore_next<F, PAIR>(g, U, Eb[sub], Eb[1 - sub], G[sub], (C)gam[k], i, gv);
                        take(i, G[1 - sub]);
                    }
                    sub ^= 1;
                    if (k == 1) last = gmax;  // the third deviation
                } else {
                    deviation();
                    if (k == 2) last = gmax;
                    for (int mu = 0; mu < 3; ++mu)
                        for (int64_t i = 0; i < n; ++i) unit_restore<F, PAIR>(g, U, E, G[0], (C)gam[k], i, mu);
                }
            }
            ++it;
        }
        if (sub) std::memcpy(E, E1.data(), ebytes);
        return it;
    }
    static int gauss_restore(const Geom &g, const void *U, void *E, double tol, int maxit) {
        if constexpr (!F::PAIRED) return restore_units<false>(g, U, E, tol, maxit);
        if constexpr (F::PAIRED)
            if (g.nz % 2 == 0) return restore_units<true>(g, U, E, tol, maxit);
        std::vector<double> G((size_t)F::NA * g.V);
        const double gam[3] = {7.0 / 24.0, 7.0 / 48.0, 7.0 / 72.0};
        auto dev = [&]() {
            double m = 0;
            for (int64_t s = 0; s < g.V; ++s) {
                double gv[F::NA];
                site_gauss<F>(g, U, E, s, gv);
                for (int a = 0; a < F::NA; ++a) { G[a * g.V + s] = gv[a]; m = std::fmax(m, gv[a]); }
            }
            return m;
        };
        double gmax = dev();
        int it = 0;
        while (it < maxit && gmax > tol) {
            for (int k = 0; k < 3; ++k) {
                gmax = dev();
                for (int64_t s = 0; s < g.V; ++s) site_gauss_update<F>(g, U, E, G.data(), gam[k], s);
            }
            ++it;
        }
        return it;
    }
};

Geom geom(const int *n) { return Geom{n[0], n[1], n[2], (int64_t)n[0] * n[1] * n[2]}; }

#define HC_DISPATCH(fmt, body)                                  \
    switch (fmt) {                                              \
        case FMT_SU2_F32: { using HH = H<FMT_SU2_F32>; body; } break; \
        case FMT_SU2_F64: { using HH = H<FMT_SU2_F64>; body; } break; \
        case FMT_SU3_F32: { using HH = H<FMT_SU3_F32>; body; } break; \
        case FMT_SU3_F64: { using HH = H<FMT_SU3_F64>; body; } break; \
        default: return -1;                                     \
    }

// E.E and (E + E').B / 4, summed over `count` pairs at a time as a thread of the device sums
// them, of n pairs' components e[pair][component][lane]
template <int NA> void pair_sums(int64_t n, int64_t count, const float *e, const float *et, const float *b, double *out) {
    for (int64_t i0 = 0; i0 < n; i0 += count) {
        FieldSums<f2, NA> sums;
        for (int again = 0; again < 2; ++again) {
            for (int64_t i = i0; i < i0 + count && i < n; ++i) {
                f2 x[NA], y[NA], z[NA];
                for (int a = 0; a < NA; ++a) {
                    const int64_t j = 2 * (i * NA + a);
                    x[a] = f2(e[j], e[j + 1]); y[a] = f2(et[j], et[j + 1]); z[a] = f2(b[j], b[j + 1]);
                }
                if (again) sums.add64(x, y, z);
                else sums.add(x, y, z);
            }
            if (again || sums.exact()) break;
        }
        out[2 * (i0 / count)] = sums.sq;
        out[2 * (i0 / count) + 1] = sums.dot;
    }
}
// sum of squares, largest component and largest magnitude (from 0 on) of n pairs' violations,
// each the sum of k FP32 terms t[pair][component][term][lane]
template <int NA> void violation_sums(int64_t n, int64_t count, int k, const float *t, double *out) {
    for (int64_t i0 = 0; i0 < n; i0 += count) {
        ViolationSums<f2, NA> sums;
        for (int again = 0; again < 2; ++again) {
            for (int64_t i = i0; i < i0 + count && i < n; ++i) {
                WideSum<f2> s[NA];
                for (int a = 0; a < NA; ++a) {
                    s[a] = WideSum<f2>(f2(0.0));
                    for (int j = 0; j < k; ++j) {
                        const float *x = t + 2 * ((i * NA + a) * k + j);
                        s[a].add(f2(x[0], x[1]));
                    }
                }
                if (again) sums.add64(s);
                else sums.add(s);
            }
            if (again || sums.exact()) break;
        }
        double *o = out + 3 * (i0 / count);
        o[0] = sums.sq; o[1] = sums.most; o[2] = sums.mag;
    }
}

}  // namespace

extern "C" {

int hc_from_aos(int fmt, const int *n, const double *Ua, const double *Ea, void *U, void *E) {
    Geom g = geom(n);
    HC_DISPATCH(fmt, for (int64_t s = 0; s < g.V; ++s) site_from_aos<HH::F>(g, U, E, Ua, Ea, s));
    return 0;
}
// sites [s0, s0 + cnt) of full AoS arrays into the storage
int hc_from_aos_range(int fmt, const int *n, const double *Ua, const double *Ea, void *U, void *E, int64_t s0,
                      int64_t cnt) {
    Geom g = geom(n);
    HC_DISPATCH(fmt, for (int64_t s = s0; s < s0 + cnt; ++s) site_from_aos<HH::F>(g, U, E, Ua, Ea, s));
    return 0;
}
// one leapfrog step of the storage indices [i0, i1) (site pairs when the format pairs and nz is even)
int hc_step_range(int fmt, const int *n, const void *Uin, void *Uout, void *E, double dt, int64_t i0, int64_t i1) {
    Geom g = geom(n);
    StepCoef<double> c = coef(MODE_LEAPFROG, dt, 0, 0, 0, 0);
    HC_DISPATCH(fmt, HH::step_range(g, Uin, Uout, E, c, i0, i1));
    return 0;
}
int hc_to_aos(int fmt, const int *n, const void *U, const void *E, double *Ua, double *Ea) {
    Geom g = geom(n);
    HC_DISPATCH(fmt, for (int64_t s = 0; s < g.V; ++s) site_to_aos<HH::F>(g, U, E, Ua, Ea, s));
    return 0;
}
// pairs: 0 the per-site step; 1 + tx: the paired step where the device takes it (FP32
// formats, even nz, fused step) with block tiling tx (0: linear)
int hc_step(int fmt, const int *n, const void *Uin, void *Uout, void *E, int mode, double dt, double gamma, double T,
            uint64_t seed, uint64_t step, int doE, int doU, int pairs) {
    Geom g = geom(n);
    StepCoef<double> c = coef(mode, dt, gamma, T, seed, step);
    HC_DISPATCH(fmt, HH::step(g, Uin, Uout, E, c, doE, doU, pairs));
    return 0;
}
// one leapfrog step in blocks that share their plaquettes, with the tiling tx x ty, zl planes a block, `threads` threads
// (tx 0: the rule for a device of `threads` multiprocessors, 0: among others)
int hc_march(int fmt, const int *n, const void *Uin, void *Uout, void *E, double dt, int tx, int ty, int zl,
             int threads) {
    Geom g = geom(n);
    StepCoef<double> c = coef(MODE_LEAPFROG, dt, 0, 0, 0, 0);
    const MarchTile t = tx ? MarchTile{tx, ty, (g.nx + tx - 1) / tx, (g.ny + ty - 1) / ty, zl, threads} : march_tile(g, threads > 0 ? threads : 0.5, threads > 0);
    HC_DISPATCH(fmt, HH::march(g, Uin, Uout, E, cast<HH::T>(c), true, SiteRange{0, g.nz, 0, g.V}, t));
    return 0;
}
// does the FP64 step (links) or E update of a lattice alone on `sms` multiprocessors go by sites?
int hc_by_sites(const int *n, int sms, int su3, int links) { return step_tile(geom(n), sms, su3 != 0, links != 0).tx == 0; }
// the checkerboard tiles of a lattice, their shape in out[3]; returns whether an FP32 lattice
// goes by pairs
int hc_cb_tile(const int *n, int su3, int *out) {
    Geom g = geom(n);
    const CbTile t = cb_tile(g);
    out[0] = 1 << t.lx; out[1] = 1 << t.ly; out[2] = 1 << t.lz;
    return cb_pairs(g, su3 != 0);
}
int hc_flow_cb(int fmt, const int *n, void *U, double dtau, int nsweeps) {
    Geom g = geom(n);
    HC_DISPATCH(fmt, HH::flow_cb(g, U, dtau, nsweeps));
    return 0;
}
int hc_observables(int fmt, const int *n, const void *U, const void *E, int mask, double *out) {
    Geom g = geom(n);
    HC_DISPATCH(fmt, HH::observables(g, U, E, mask, out));
    return 0;
}
int hc_edotb_pair(int fmt, const int *n, const void *U, const void *E, double *out) {
    Geom g = geom(n);
    int ok = 0;
    HC_DISPATCH(fmt, ok = HH::edotb_pair(g, U, E, out));
    return ok;
}
// n pairs in groups of `count` (pair_sums, violation_sums)
int hc_pair_sums(int na, int64_t n, int64_t count, const float *e, const float *et, const float *b, double *out) {
    if (na == 3) pair_sums<3>(n, count, e, et, b, out);
    else pair_sums<8>(n, count, e, et, b, out);
    return 0;
}
int hc_violation_sums(int na, int64_t n, int64_t count, int k, const float *t, double *out) {
    if (na == 3) violation_sums<3>(n, count, k, t, out);
    else violation_sums<8>(n, count, k, t, out);
    return 0;
}
// the Gauss violation of every site, by pairs (0: the storage holds none) or site by site
int hc_gauss(int fmt, const int *n, const void *U, const void *E, int pairs, double *out) {
    Geom g = geom(n);
    int ok = 1;
    HC_DISPATCH(fmt, {
        if (pairs) ok = HH::gauss_pair(g, U, E, out);
        else HH::gauss_sites(g, U, E, out);
    });
    return ok;
}
int hc_gauss_restore(int fmt, const int *n, const void *U, void *E, double tol, int maxit) {
    Geom g = geom(n);
    int it = 0;
    HC_DISPATCH(fmt, it = HH::gauss_restore(g, U, E, tol, maxit));
    return it;
}
int hc_reunitarize(int fmt, const int *n, void *U) {
    Geom g = geom(n);
    HC_DISPATCH(fmt, HH::reunitarize(g, U));
    return 0;
}
int hc_reunitarize_fp64(int fmt, const int *n, void *U) {
    Geom g = geom(n);
    HC_DISPATCH(fmt, HH::reunitarize_fp64(g, U));
    return 0;
}
// Block of the links of extents n into Ub (extents n / 2, the same format)
int hc_block(int fmt, const int *n, const void *U, void *Ub) {
    const Geom gs = geom(n);
    const int h[3] = {n[0] / 2, n[1] / 2, n[2] / 2};
    const Geom gd = geom(h);
    HC_DISPATCH(fmt, for (int64_t s = 0; s < gd.V; ++s) site_block<HH::F>(gs, gd, U, Ub, s));
    return 0;
}
int hc_init(int fmt, const int *n, void *U, void *E, int what, double sigma, uint64_t seed) {
    Geom g = geom(n);
    HC_DISPATCH(fmt, for (int64_t s = 0; s < g.V; ++s) {
        if (what == 0) site_set_zero<HH::F>(g, U, E, s);
        else if (what == 1) site_gaussian_efield<HH::F>(g, E, sigma, seed, s);
        else site_random_links<HH::F>(g, U, sigma, seed, s);
    });
    return 0;
}
int hc_ilog(int fmt, double c, const double *v, double *out) {
    HC_DISPATCH(fmt, HH::ilog_aos(c, v, out));
    return 0;
}
int hc_geodesic(int fmt, const int *n, const void *Uold, const void *Unew, double c, void *Umid, void *Emid) {
    Geom g = geom(n);
    HC_DISPATCH(fmt, HH::geodesic(g, Uold, Unew, c, Umid, Emid));
    return 0;
}
// exp(i c t^a alpha^a) in the format's precision, returned in the reference AoS link layout
int hc_iexp(int fmt, double c, const double *alpha, double *out) {
    HC_DISPATCH(fmt, HH::iexp_aos(c, alpha, out));
    return 0;
}
// the host-resident step's pipeline for N units in planes of P, chunk size C:
// its chunk bounds (at most cap written) and the issue order, kinds[i] (0
// upload, 1 step) of chunks[i]; returns the number of operations
int64_t hc_pipeline_schedule(int64_t N, int64_t P, int64_t C, int64_t *bounds, int64_t bcap, int *kinds,
                             int64_t *chunks, int64_t cap) {
    const std::vector<int64_t> b = pipeline_bounds(N, P, C);
    for (int64_t i = 0; i < (int64_t)b.size() && i < bcap; ++i) bounds[i] = b[i];
    int64_t n = 0;
    pipeline_schedule(b, P, [&](int op, int64_t j) {
        if (n < cap) { kinds[n] = op; chunks[n] = j; }
        ++n;
    });
    return n;
}
double hc_normal(uint64_t seed, uint32_t stream, uint64_t step, uint32_t site, uint32_t mu, uint32_t a, int single) {
    double z0, z1;
    if (single) {
        float f0, f1;
        normal_pair<float>(seed, stream, step, site, mu, a >> 1, &f0, &f1);
        z0 = f0; z1 = f1;
    } else {
        normal_pair<double>(seed, stream, step, site, mu, a >> 1, &z0, &z1);
    }
    return (a & 1) ? z1 : z0;
}

}  // extern "C"

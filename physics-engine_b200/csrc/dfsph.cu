// Divergence-free SPH (crates/pe-fluid/src/dfsph.rs) on the cell-sorted state
// of a World whose grid cell is the kernel's support radius.
//
// Slot state: pos = (x, psi), vel = (v, rho), acc = (v*, warm-start kappa of
// the density solver), nout = (n_out, warm-start kappa of the divergence
// solver), bf = boundary reaction, p = the density solver's kappa (the
// reference's pressure diagnostic). All of it moves with the re-sort.
//
// Lists: a fluid slot's visit list holds its fluid neighbours in support and
// every boundary candidate of the 27 (9) neighbour cells, as the reference's
// lists do: the reaction weights (dfsph.rs:498-518) range over every boundary
// candidate, in or out of the support. Fluid candidates out of the support add
// +-0 and are left out; the solver's neighbour count (dfsph.rs:281-296), which
// counts every candidate, takes them from the union size the list build records.
//
// Boundary reactions: the reference scatters, for fluid i in ascending index,
// F_b(i) wt_ij / sum_j wt_ij onto each boundary candidate j. The neighbour
// relation of the cell grid is symmetric, so a boundary slot gathers the same
// terms from its fluid candidates in ascending original index (its "lower"
// list), which is the reference's order of additions.
//
// The solvers' average errors are sequential sums in original index order
// (dfsph.rs:552-569, 604-616) of non-negative terms, and only their comparison
// with the tolerance is used. Any summation order of n non-negative terms lies
// within gamma_(n-1) = (n-1)u / (1 - (n-1)u) (relative) of the exact sum, so a
// parallel sum S brackets the sequential one in S (1 +- 2 gamma / (1 - gamma)).
// When the whole bracket, divided by the fluid count, falls on one side of the
// tolerance, that is the reference's decision; otherwise the terms (scattered
// to original order) are summed sequentially by one thread. Either way the
// convergence decision is the reference's bit for bit. Compiled with
// --fmad=false.
#include <algorithm>
#include <cmath>
#include <limits>
#include <type_traits>

#include "dfsph.cuh"
#include "lane_group.cuh"
#include "list_iter.cuh"

namespace pe {

namespace {

constexpr uint32_t kDfThreads = 128;

inline uint32_t blocks_for(uint64_t n, uint32_t t) { return (uint32_t)((n + t - 1) / t); }

__device__ __forceinline__ bool is_boundary(const StateBufs& s, uint32_t i) { return s.flags[i] & kFlagBoundary; }

// particles.rs:126 boundary_sees_fluid (un-oriented samples see everything)
__device__ __forceinline__ bool sees(const DfsphConst& k, const double4& xb, const double4& nb, bool oriented,
                                     const double4& xf) {
    if (!oriented) return true;
    const double n2 = nb.x * nb.x + nb.y * nb.y + nb.z * nb.z;
    if (n2 <= 0.0) return true;
    const double eps = k.eps_h * sqrt(fmax(n2, 0.0));
    const double d = (xf.x - xb.x) * nb.x + (xf.y - xb.y) * nb.y + (xf.z - xb.z) * nb.z;
    return d > -eps;
}

// A candidate beyond the kernel's support adds an exact +-0 to the gradient
// and kernel sums (W and grad W vanish there); those sums skip it. The margin
// on far2 keeps the test conservative under rounding.
struct Offset {
    double x, y, z, r2;
    __device__ __forceinline__ Offset(const double4& xi, const double4& xj)
        : x(xj.x - xi.x), y(xj.y - xi.y), z(xj.z - xi.z), r2(x * x + y * y + z * z) {}
    __device__ __forceinline__ bool far(const DfsphConst& k) const { return r2 > k.far2; }
};

struct TwoStates {
    double4 x, v;
};

// dfsph.rs:309-323 neighbour_mass_for
__device__ __forceinline__ double nmass(const DfsphConst& k, const StateBufs& s, uint32_t e, const double4& xj,
                                        const double4& xi) {
    if (!(e & kEntryBoundary)) return k.mass;
    const uint32_t j = e & kEntrySlotMask;
    const bool oriented = e & kEntryOriented;
    return sees(k, xj, oriented ? s.nout[j] : make_double4(0, 0, 0, 0), oriented, xi) ? k.rho0 * xj.w : 0.0;
}

// What a pair contributes to a solver's passes besides velocities and pressures
// depends on the positions alone, which stay as they are through a solver's
// iterations (twelve error and twelve pressure passes a step at 46,620 particles).
// So the alpha pass keeps it beside the lists, at an entry's index into the pool:
// of a fluid slot's entry the scale of grad W, of a boundary slot's the
// reaction's weight; kSkip where the pair adds nothing (grad W's scale and the
// weight are never negative). Lists beyond the buffer are computed as they go.
constexpr double kSkip = -1.0;

// The reaction's weight of a fluid particle and a boundary sample (dfsph.rs:497)
__device__ __forceinline__ double reaction_weight(double r2) {
    return fmin(quot_any(1.0, fmax(sqrt(r2), 1e-9)), 1e6);
}

// Entry p's place in the buffer (a list that does not fit: any)
__device__ __forceinline__ double kept_value(const ListBufs& l, bool fits, const uint32_t* p) {
    return __ldg(l.wpair + (fits ? p - l.pool : 0));
}

// Scale of grad W and mass of entry e; false if the pair adds nothing.
template <bool KEPT>
__device__ __forceinline__ bool pair_scale(const DfsphConst& k, const StateBufs& s, uint32_t e, const double4& xi,
                                           const double4& xj, const Offset& o, bool fits, double kept, double* mj,
                                           double* sc) {
    if (KEPT && fits) {
        *mj = (e & kEntryBoundary) ? k.rho0 * xj.w : k.mass;
        *sc = kept;
        return !(kept < 0.0);
    }
    if (o.far(k)) return false;
    *mj = nmass(k, s, e, xj, xi);
    if (*mj == 0.0) return false;
    *sc = kfn_grad_scale(k.kf, o.r2);
    return true;
}

// dfsph.rs:718-735: boundary forces cleared, v* = v + g dt (2-D: z = 0)
__global__ void k_df_begin(uint32_t n, DfsphConst k, double dt, StateBufs s) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double4 f = s.bf[i];
    f.x = 0.0;
    f.y = 0.0;
    f.z = 0.0;
    s.bf[i] = f;
    const double4 v = s.vel[i];
    double4 a = s.acc[i];
    if (is_boundary(s, i)) {
        a.x = v.x;
        a.y = v.y;
        a.z = v.z;
    } else {
        const double gx = k.gx * dt, gy = k.gy * dt, gz = k.gz * dt;
        a.x = v.x + gx;
        a.y = v.y + gy;
        a.z = k.dim == 2 ? 0.0 : v.z + gz;
    }
    s.acc[i] = a;
}

// The pair passes run G lanes a slot (lane_group.cuh, df_lanes): a group's lanes
// compute the terms of G consecutive entries, added in entry order, a skipped
// entry as +0. Every lane of a warp stays to the end of each walk.

// dfsph.rs:382-416 XSPH on v* (fluid neighbours)
template <int G>
__global__ void __launch_bounds__(kDfThreads) k_df_xsph(uint32_t n, DfsphConst k, StateBufs s, ListBufs l,
                                                       double4* __restrict__ dv) {
    extern __shared__ __align__(16) double s_words[];
    const LaneGroup<G> g;
    const uint32_t i = g.slot;
    const bool fluid = i < n && !is_boundary(s, i);
    if (i < n && !fluid && g.sub == 0) dv[i] = make_double4(0.0, 0.0, 0.0, 0.0);
    if (!__any_sync(kFullWarp, fluid)) return;
    ListRef lr{l.pool, 0u, 0u};
    double4 xi = make_double4(0.0, 0.0, 0.0, 0.0), vi = xi;
    double rho_i = 0.0;
    if (fluid) {
        lr = list_ref(l, i, kListVisit);
        xi = s.pos[i];
        vi = s.acc[i];
        rho_i = s.vel[i].w;
    }
    struct Neighbour {
        double4 x, v;
        double rho;
    };
    OrderedSum<G, 3> c(s_words + g.warp * OrderedSum<G, 3>::kDoubles, g, 0.0);
    group_for_each<G>(
        lr, g,
        [&](uint32_t e, const uint32_t*) {
            const uint32_t j = e & kEntrySlotMask;
            return Neighbour{gather4(s.pos + j), gather4(s.acc + j), s.vel[j].w};
        },
        [&](bool has, uint32_t e, const Neighbour& d, const uint32_t*) {
            double t[3] = {0.0, 0.0, 0.0};
            const Offset o(xi, d.x);
            if (has && !(e & kEntryBoundary) && !o.far(k)) {
                const double wij = kfn_w_r2(k.kf, o.r2);
                const double rho_bar = 0.5 * (rho_i + d.rho);
                const double f = quot_any(k.mass, fmax(rho_bar, 1e-12)) * wij;
                t[0] = (d.v.x - vi.x) * f;
                t[1] = (d.v.y - vi.y) * f;
                t[2] = (d.v.z - vi.z) * f;
            }
            c.add(t);
        });
    double r[3];
    c.totals(r);
    if (fluid && g.sub == 0) dv[i] = make_double4(r[0] * k.xsph_eps, r[1] * k.xsph_eps, r[2] * k.xsph_eps, 0.0);
}

__global__ void k_df_xsph_apply(uint32_t n, StateBufs s, const double4* __restrict__ dv) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || is_boundary(s, i)) return;
    double4 a = s.acc[i];
    const double4 d = dv[i];
    a.x = a.x + d.x;
    a.y = a.y + d.y;
    a.z = a.z + d.z;
    s.acc[i] = a;
}

// kappa = the warm-start accumulator (which 0: density, acc.w; 1: divergence, nout.w)
__global__ void k_df_warm_load(uint32_t n, DfsphConst k, int which, StateBufs s, double* __restrict__ kappa,
                               double* __restrict__ kr) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double kap = which ? s.nout[i].w : s.acc[i].w;
    kappa[i] = kap;
    kr[i] = is_boundary(s, i) ? 0.0 / k.rho0 : kap / fmax(s.vel[i].w, 1e-12);
}

__global__ void k_df_warm_zero(uint32_t n, int which, StateBufs s) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (which) s.nout[i].w = 0.0;
    else s.acc[i].w = 0.0;
}

// dfsph.rs:326-351 density_derivative of slot i with v* (every lane of the
// group gets it; fluid: the group has a slot to do)
template <int G, bool KEPT>
__device__ __forceinline__ double density_rate(const DfsphConst& k, const StateBufs& s, const ListBufs& l,
                                               const LaneGroup<G>& g, bool fluid, double* words) {
    const uint32_t i = g.slot;
    ListRef lr{l.pool, 0u, 0u};
    double4 xi = make_double4(0.0, 0.0, 0.0, 0.0), vi = xi;
    if (fluid) {
        lr = list_ref(l, i, kListVisit);
        xi = s.pos[i];
        vi = s.acc[i];
    }
    struct Neighbour {
        double4 x, v;
        double kept;
    };
    const bool fits = KEPT && w_fits(l, lr);
    OrderedSum<G, 1> drho(words, g, 0.0);
    group_for_each<G>(
        lr, g,
        [&](uint32_t e, const uint32_t* p) {
            const uint32_t j = e & kEntrySlotMask;
            return Neighbour{gather4(s.pos + j), gather4(((e & kEntryBoundary) ? s.vel : s.acc) + j),
                             KEPT ? kept_value(l, fits, p) : 0.0};
        },
        [&](bool has, uint32_t e, const Neighbour& d, const uint32_t*) {
            double t[1] = {0.0}, mj, sc;
            const Offset o(xi, d.x);
            if (has && pair_scale<KEPT>(k, s, e, xi, d.x, o, fits, d.kept, &mj, &sc)) {
                const double gx = o.x * sc, gy = o.y * sc, gz = o.z * sc;
                const double wx = vi.x - d.v.x, wy = vi.y - d.v.y, wz = vi.z - d.v.z;
                t[0] = mj * (wx * gx + wy * gy + wz * gz);
            }
            drho.add(t);
        });
    double r[1];
    drho.totals(r);
    return r[0];
}

// One error pass of a solver (dfsph.rs:552-569 density, 604-616 divergence):
// kappa, the warm-start accumulation, the pressure diagnostic and the error
// term of each particle in original order.
template <int G, bool KEPT>
__global__ void __launch_bounds__(kDfThreads) k_df_error(uint32_t n, DfsphConst k, int divergence, double dt,
                                                        double dt2, StateBufs s, ListBufs l,
                                                        const double* __restrict__ alpha, double* __restrict__ kappa,
                                                        double* __restrict__ kr, double* __restrict__ err_orig) {
    extern __shared__ __align__(16) double s_words[];
    const LaneGroup<G> g;
    const uint32_t i = g.slot;
    const bool fluid = i < n && !is_boundary(s, i);
    if (i < n && !fluid && g.sub == 0) {
        kappa[i] = 0.0;
        kr[i] = 0.0 / k.rho0;  // dfsph.rs:462-469: kj = 0, rho_j = rho0
        err_orig[s.orig[i]] = 0.0;
    }
    if (!__any_sync(kFullWarp, fluid)) return;
    const double drho = density_rate<G, KEPT>(k, s, l, g, fluid, s_words + g.warp * OrderedSum<G, 1>::kDoubles);
    if (!fluid || g.sub != 0) return;
    const uint32_t o = s.orig[i];
    double kap, e;
    if (!divergence) {
        const double rho_star = s.vel[i].w + dt * drho;
        const double err = fmax(rho_star - k.rho0, 0.0);
        e = err / k.rho0;
        kap = k.omega * err / dt2 * alpha[i];
        s.p[i] = kap;  // dfsph.rs:761 p = kappa after the step
        if (k.warm_start) s.acc[i].w = s.acc[i].w + kap;
    } else {
        const double d = fmax(drho, 0.0);
        e = d / k.rho0;
        kap = k.omega * (1.0 / dt) * d * alpha[i];
        if (k.warm_start) s.nout[i].w = s.nout[i].w + kap;
    }
    kappa[i] = kap;
    // dfsph.rs:436, 470: kappa / max(rho, 1e-12), the same quotient the
    // reference forms for every pair, formed once
    kr[i] = kap / fmax(s.vel[i].w, 1e-12);
    err_orig[o] = e;
}

// Partial sums of v (any order: only bounds are taken from them).
constexpr uint32_t kSumBlocks = 148, kSumThreads = 256;

__global__ void __launch_bounds__(kSumThreads) k_df_partial_sums(uint32_t n, const double* __restrict__ v,
                                                                double* __restrict__ part) {
    __shared__ double red[kSumThreads];
    double s = 0.0;
    for (uint32_t i = blockIdx.x * kSumThreads + threadIdx.x; i < n; i += kSumBlocks * kSumThreads) s += v[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (uint32_t o = kSumThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void __launch_bounds__(kSumThreads) k_df_final_sum(const double* __restrict__ part,
                                                             double* __restrict__ out) {
    __shared__ double red[kSumThreads];
    red[threadIdx.x] = threadIdx.x < kSumBlocks ? part[threadIdx.x] : 0.0;
    __syncthreads();
    for (uint32_t o = kSumThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = red[0];
}

// Sequential sum in original index order (the reference's accumulation order).
__global__ void k_df_serial_sum(uint32_t n, const double* __restrict__ v, double* __restrict__ out) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    double s = 0.0;
    for (uint32_t i = 0; i < n; ++i) s += v[i];
    *out = s;
}

// dfsph.rs:422-530, fluid side: dv from kappa, the cap, the reaction total and
// weight sum, v* += dv.
template <int G, bool KEPT>
__global__ void __launch_bounds__(kDfThreads) k_df_pressure_fluid(uint32_t n, DfsphConst k, double dt,
                                                                 double inv_dt, StateBufs s, ListBufs l,
                                                                 const double* __restrict__ kr,
                                                                 const double* __restrict__ wsum,
                                                                 double4* __restrict__ react) {
    extern __shared__ __align__(16) double s_words[];
    const LaneGroup<G> g;
    const uint32_t i = g.slot;
    const bool fluid = i < n && !is_boundary(s, i);
    if (!__any_sync(kFullWarp, fluid)) return;
    ListRef lr{l.pool, 0u, 0u};
    double4 xi = make_double4(0.0, 0.0, 0.0, 0.0);
    double kri = 0.0;  // ki / rho_i
    if (fluid) {
        lr = list_ref(l, i, kListVisit);
        xi = s.pos[i];
        kri = kr[i];
    }
    // the sums over all neighbours, and over the boundary ones (exchanged only
    // in rounds that have one)
    double* const words = s_words + g.warp * 2u * OrderedSum<G, 3>::kDoubles;
    OrderedSum<G, 3> all(words, g, 0.0), bnd(words + OrderedSum<G, 3>::kDoubles, g, 0.0);
    struct Neighbour {
        double4 x;
        double kr, kept;
    };
    const bool fits = KEPT && w_fits(l, lr);
    group_for_each<G>(
        lr, g,
        [&](uint32_t e, const uint32_t* p) {
            const uint32_t j = e & kEntrySlotMask;
            return Neighbour{gather4(s.pos + j), __ldg(kr + j), KEPT ? kept_value(l, fits, p) : 0.0};
        },
        [&](bool has, uint32_t e, const Neighbour& d, const uint32_t*) {
            double t[3] = {0.0, 0.0, 0.0}, tb[3] = {0.0, 0.0, 0.0}, mj, sc;
            bool b = false;
            const Offset o(xi, d.x);
            if (has && pair_scale<KEPT>(k, s, e, xi, d.x, o, fits, d.kept, &mj, &sc)) {
                const double coeff = mj * (kri + d.kr);  // mj (ki / rho_i + kj / rho_j)
                t[0] = (o.x * sc) * coeff;
                t[1] = (o.y * sc) * coeff;
                t[2] = (o.z * sc) * coeff;
                b = e & kEntryBoundary;
                if (b) {
                    tb[0] = t[0];
                    tb[1] = t[1];
                    tb[2] = t[2];
                }
            }
            all.add(t);
            if (__any_sync(kFullWarp, b)) bnd.add(tb);
        });
    double ra[3], rb[3];
    all.totals(ra);
    bnd.totals(rb);
    double dx = ra[0], dy = ra[1], dz = ra[2], bx = rb[0], by = rb[1], bz = rb[2];
    dx = dx * (-dt);
    dy = dy * (-dt);
    dz = dz * (-dt);
    bx = bx * (-dt);
    by = by * (-dt);
    bz = bz * (-dt);
    double scale = 1.0;
    if (k.dv_cap > 0.0) {
        const double s2 = dx * dx + dy * dy + dz * dz;
        if (s2 > k.dv_cap * k.dv_cap) {
            scale = k.dv_cap / sqrt(s2);
            dx = dx * scale;
            dy = dy * scale;
            dz = dz * scale;
        }
    }
    bx = bx * scale;
    by = by * scale;
    bz = bz * scale;
    if (!fluid || g.sub != 0) return;
    double4 rec = make_double4(0.0, 0.0, 0.0, 0.0);
    if (bx * bx + by * by + bz * bz > 0.0) {
        const double ws = wsum[i];  // the weights of its visible samples
        if (ws > 0.0) {
            const double m = -k.mass * inv_dt;
            rec = make_double4(bx * m, by * m, bz * m, ws);
        }
    }
    react[i] = rec;
    double4 a = s.acc[i];
    a.x = a.x + dx;
    a.y = a.y + dy;
    a.z = k.dim == 2 ? 0.0 : a.z + dz;
    s.acc[i] = a;
}

// The boundary slots' half of what is kept: the reaction's weight of each fluid candidate.
template <int G>
__global__ void __launch_bounds__(kDfThreads) k_df_boundary_weights(uint32_t n, DfsphConst k, StateBufs s, ListBufs l) {
    const LaneGroup<G> g;
    const uint32_t j = g.slot;
    ListRef lr{l.pool, 0u, 0u};
    double4 xj = make_double4(0.0, 0.0, 0.0, 0.0), nj = xj;
    bool oriented = false;
    if (j < n && is_boundary(s, j)) {
        lr = list_ref(l, j, kListLower);
        xj = s.pos[j];
        oriented = s.flags[j] & kFlagOriented;
        if (oriented) nj = s.nout[j];
    }
    const bool fits = w_fits(l, lr);
    if (!fits && g.sub == 0) atomicOr(l.w_short, 1u);
    group_for_each<G>(
        lr, g, [&](uint32_t e, const uint32_t*) { return gather4(s.pos + (e & kEntrySlotMask)); },
        [&](bool has, uint32_t, const double4& xi, const uint32_t* p) {
            if (has && fits)
                l.wpair[p - l.pool] = sees(k, xj, nj, oriented, xi) ? reaction_weight(Offset(xi, xj).r2) : kSkip;
        });
}

// dfsph.rs:508-517, boundary side: the reaction shares of the fluid
// candidates, in ascending original index.
template <int G, bool KEPT>
__global__ void __launch_bounds__(kDfThreads) k_df_pressure_boundary(uint32_t n, DfsphConst k, StateBufs s,
                                                                    ListBufs l, const double4* __restrict__ react) {
    extern __shared__ __align__(16) double s_words[];
    const LaneGroup<G> g;
    const uint32_t j = g.slot;
    const bool bound = j < n && is_boundary(s, j);
    if (!__any_sync(kFullWarp, bound)) return;
    ListRef lr{l.pool, 0u, 0u};
    double4 xj = make_double4(0.0, 0.0, 0.0, 0.0), nj = xj, f = xj;
    bool oriented = false;
    if (bound) {
        lr = list_ref(l, j, kListLower);
        xj = s.pos[j];
        f = s.bf[j];
        oriented = s.flags[j] & kFlagOriented;
        if (oriented) nj = s.nout[j];
    }
    struct Neighbour {
        double4 rec;
        double kept;
    };
    const bool fits = KEPT && w_fits(l, lr);
    const double start[3] = {f.x, f.y, f.z};
    OrderedSum<G, 3> sum(s_words + g.warp * OrderedSum<G, 3>::kDoubles, g, start);
    group_for_each<G>(
        lr, g,
        [&](uint32_t e, const uint32_t* p) {
            return Neighbour{gather4(react + (e & kEntrySlotMask)), KEPT ? kept_value(l, fits, p) : 0.0};
        },
        [&](bool has, uint32_t e, const Neighbour& d, const uint32_t*) {
            const double4& rec = d.rec;
            double t[3] = {0.0, 0.0, 0.0};
            bool adds = has && rec.w > 0.0;
            double wt = d.kept;
            if (adds && !fits) {
                const double4 xi = s.pos[e & kEntrySlotMask];
                wt = sees(k, xj, nj, oriented, xi) ? reaction_weight(Offset(xi, xj).r2) : kSkip;
            }
            adds = adds && !(wt < 0.0);
            if (adds) {
                const double sh = quot_any(wt, rec.w);
                t[0] = rec.x * sh;
                t[1] = rec.y * sh;
                t[2] = rec.z * sh;
            }
            if (__any_sync(kFullWarp, adds)) sum.add(t);
        });
    double r[3];
    sum.totals(r);
    if (bound && g.sub == 0) s.bf[j] = make_double4(r[0], r[1], r[2], f.w);
}

// dfsph.rs:742-748 x += v* dt (fluid; 2-D: z = 0)
__global__ void k_df_advect(uint32_t n, int dim, double dt, StateBufs s) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || is_boundary(s, i)) return;
    double4 p = s.pos[i];
    const double4 a = s.acc[i];
    p.x = p.x + a.x * dt;
    p.y = p.y + a.y * dt;
    p.z = dim == 2 ? 0.0 : p.z + a.z * dt;
    s.pos[i] = p;
}

// dfsph.rs:668-715
__global__ void k_df_free_slip(uint32_t n, DfsphConst k, StateBufs s) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || is_boundary(s, i)) return;
    double4 x = s.pos[i], v = s.acc[i];
    if (k.has_slip[0] && x.x < k.slip[0]) {
        x.x = k.slip[0];
        if (v.x < 0.0) v.x = 0.0;
    }
    if (k.has_slip[1] && x.y < k.slip[1]) {
        x.y = k.slip[1];
        if (v.y < 0.0) v.y = 0.0;
    }
    if (k.has_slip[2] && x.x > k.slip[2]) {
        x.x = k.slip[2];
        if (v.x > 0.0) v.x = 0.0;
    }
    if (k.has_slip[3] && x.y > k.slip[3]) {
        x.y = k.slip[3];
        if (v.y > 0.0) v.y = 0.0;
    }
    s.pos[i] = x;
    s.acc[i] = v;
}

// dfsph.rs:214-244 density with the oriented-boundary filter
template <int G>
__global__ void __launch_bounds__(kDfThreads) k_df_density(uint32_t n, DfsphConst k, StateBufs s, ListBufs l) {
    extern __shared__ __align__(16) double s_words[];
    const LaneGroup<G> g;
    const uint32_t i = g.slot;
    const bool fluid = i < n && !is_boundary(s, i);
    if (i < n && !fluid && g.sub == 0) s.vel[i].w = k.rho0;
    if (!__any_sync(kFullWarp, fluid)) return;
    ListRef lr{l.pool, 0u, 0u};
    double4 xi = make_double4(0.0, 0.0, 0.0, 0.0);
    if (fluid) {
        lr = list_ref(l, i, kListVisit);
        xi = s.pos[i];
    }
    OrderedSum<G, 1> rho(s_words + g.warp * OrderedSum<G, 1>::kDoubles, g, k.rho_self);
    group_for_each<G>(
        lr, g, [&](uint32_t e, const uint32_t*) { return gather4(s.pos + (e & kEntrySlotMask)); },
        [&](bool has, uint32_t e, const double4& xj, const uint32_t*) {
            double t[1] = {0.0};
            const Offset o(xi, xj);
            if (has && !o.far(k)) {
                const double wij = kfn_w_r2(k.kf, o.r2);
                if (!(e & kEntryBoundary)) {
                    t[0] = k.mass * wij;
                } else {
                    const uint32_t j = e & kEntrySlotMask;
                    const bool oriented = e & kEntryOriented;
                    if (sees(k, xj, oriented ? s.nout[j] : make_double4(0, 0, 0, 0), oriented, xi))
                        t[0] = k.rho0 * xj.w * wij;
                }
            }
            rho.add(t);
        });
    double r[1];
    rho.totals(r);
    if (fluid && g.sub == 0) s.vel[i].w = fmax(r[0], 1e-12);
}

// dfsph.rs:252-307 alpha = rho / max(|sum m grad W|^2 + sum |m grad W|^2, floor)
// (alpha null: left as it is). Also fills wsum, the sum of a fluid particle's
// reaction weights, and what is kept of its pairs (l.wpair not null).
template <int G>
__global__ void __launch_bounds__(kDfThreads) k_df_alpha(uint32_t n, DfsphConst k, StateBufs s, ListBufs l,
                                                        double* __restrict__ alpha, double* __restrict__ wsum) {
    extern __shared__ __align__(16) double s_words[];
    const LaneGroup<G> g;
    const uint32_t i = g.slot;
    const bool fluid = i < n && !is_boundary(s, i);
    if (alpha && i < n && !fluid && g.sub == 0) alpha[i] = 0.0;
    if (!__any_sync(kFullWarp, fluid)) return;
    ListRef lr{l.pool, 0u, 0u};
    double4 xi = make_double4(0.0, 0.0, 0.0, 0.0);
    bool keep = false;
    if (fluid) {
        lr = list_ref(l, i, kListVisit);
        xi = s.pos[i];
        if (l.wpair) {
            keep = w_fits(l, lr);
            if (!keep && g.sub == 0) atomicOr(l.w_short, 1u);
        }
    }
    double* const words = s_words + g.warp * (OrderedSum<G, 4>::kDoubles + OrderedSum<G, 1>::kDoubles);
    OrderedSum<G, 4> sum(words, g, 0.0);  // m grad W, |m grad W|^2
    OrderedSum<G, 1> weights(words + OrderedSum<G, 4>::kDoubles, g, 0.0);
    uint32_t nb_all = 0, nb_kept = 0;
    group_for_each<G>(
        lr, g, [&](uint32_t e, const uint32_t*) { return gather4(s.pos + (e & kEntrySlotMask)); },
        [&](bool has, uint32_t e, const double4& xj, const uint32_t* p) {
            double t[4] = {0.0, 0.0, 0.0, 0.0}, w[1] = {0.0};
            const bool bnd = has && (e & kEntryBoundary);
            if (has) {
                const Offset o(xi, xj);
                double mj = k.mass, sc = kSkip;
                if (bnd) {
                    const bool oriented = e & kEntryOriented;
                    const bool seen = sees(k, xj, oriented ? s.nout[e & kEntrySlotMask] : make_double4(0, 0, 0, 0),
                                           oriented, xi);
                    mj = seen ? k.rho0 * xj.w : 0.0;
                    if (seen) w[0] = reaction_weight(o.r2);
                    nb_all += 1u;
                    nb_kept += mj != 0.0 ? 1u : 0u;
                }
                if (!(bnd && mj == 0.0) && !o.far(k)) {
                    sc = kfn_grad_scale(k.kf, o.r2);
                    t[0] = (o.x * sc) * mj;
                    t[1] = (o.y * sc) * mj;
                    t[2] = (o.z * sc) * mj;
                    t[3] = t[0] * t[0] + t[1] * t[1] + t[2] * t[2];
                }
                if (keep) l.wpair[p - l.pool] = mj == 0.0 ? kSkip : sc;
            }
            sum.add(t);
            if (__any_sync(kFullWarp, bnd)) weights.add(w);
        });
    nb_all = g.sum(nb_all);
    nb_kept = g.sum(nb_kept);
    double r[4], ws[1];
    sum.totals(r);
    weights.totals(ws);
    if (!fluid || g.sub != 0) return;
    wsum[i] = ws[0];
    if (!alpha) return;
    // every fluid candidate but i itself, and the boundary ones of non-zero mass
    const uint32_t nn = (l.ncand[i] - 1u - nb_all) + nb_kept;
    if (nn < 2) {
        alpha[i] = 0.0;
        return;
    }
    const double denom = fmax(r[0] * r[0] + r[1] * r[1] + r[2] * r[2] + r[3], k.denom_floor);
    alpha[i] = s.vel[i].w / denom;
}

// dfsph.rs:755-765 v = v* (2-D: z = 0)
__global__ void k_df_finish(uint32_t n, int dim, StateBufs s) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || is_boundary(s, i)) return;
    double4 v = s.vel[i];
    const double4 a = s.acc[i];
    v.x = a.x;
    v.y = a.y;
    v.z = dim == 2 ? 0.0 : a.z;
    s.vel[i] = v;
}

__global__ void k_df_export_orig(uint32_t n, const uint32_t* __restrict__ orig, const double* __restrict__ src,
                                 double* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[orig[i]] = src[i];
}

// Calls f(integral_constant<int, G>) for the lanes a slot of the pair passes.
template <class F>
void with_df_lanes(uint32_t lanes, F&& f) {
    if (lanes == 1) f(std::integral_constant<int, 1>{});
    else if (lanes == 8) f(std::integral_constant<int, 8>{});
    else f(std::integral_constant<int, 32>{});
}

template <int G, int K>
size_t df_smem(uint32_t sums = 1) {
    return (size_t)sums * (kDfThreads / 32u) * OrderedSum<G, K>::kDoubles * sizeof(double);
}

template <int G>
uint32_t df_blocks(uint32_t n) {
    return blocks_for((uint64_t)n * G, kDfThreads);
}

}  // namespace

DfsphSolver::DfsphSolver(const DfsphParams& prm, const WorldConfig& cfg, int dim, double rest_density, double mass,
                         double h, uint64_t n, const double* x, const double* v, const uint8_t* kind,
                         const double* psi, const double* n_out)
    : prm_(prm) {
    // dfsph.rs:139-152: diameter defaults to h; 2-D particles are planar
    if (prm_.particle_diameter <= 0.0) prm_.particle_diameter = h;
    std::vector<double> xs(x, x + 3 * n), vs;
    if (v) vs.assign(v, v + 3 * n);
    else vs.assign(3 * n, 0.0);
    if (dim == 2)
        for (uint64_t i = 0; i < n; ++i) {
            xs[3 * i + 2] = 0.0;
            vs[3 * i + 2] = 0.0;
        }
    for (uint64_t i = 0; i < n; ++i) n_fluid_ += kind[i] == 0;
    n_ = n;
    set_lanes(0);
    WorldParams wp{};
    wp.kernel = 0;
    wp.eos_rest_density = rest_density;
    wp.eos_sound_speed = 1.0;
    wp.eos_gamma = 7.0;
    for (int a = 0; a < 3; ++a) wp.gravity[a] = prm.gravity[a];
    WorldConfig wc = cfg;
    wc.precision = 0;
    wc.use_graph = 0;
    wc.pair_weights = 0;
    w_.reset(new World(wp, wc, dim, rest_density, mass, h, n, xs.data(), vs.data(), kind, psi, n_out, nullptr, 1,
                       kernel_support(prm.kernel, h)));
    w_->list_keep_boundary_ = true;
    w_->lists_outlive_poll_ = true;  // a step begins with the lists the last one ended with
    w_->refresh_step_const();
    const size_t N = std::max<uint64_t>(n, 1);
    alpha_ = w_->alloc<double>(N);
    wsum_ = w_->alloc<double>(N);
    kappa_ = w_->alloc<double>(N);
    kr_ = w_->alloc<double>(N);
    dv_ = w_->alloc<double4>(N);
    react_ = w_->alloc<double4>(N);
    err_orig_ = w_->alloc<double>(N);
    sum_ = w_->alloc<double>(1);
    part_ = w_->alloc<double>(kSumBlocks);
    w_->check(cudaMallocHost(&sum_host_, sizeof(double)), "pinned");
    refresh_const();
    // dfsph.rs:177-179
    rebuild();
    density_and_alpha();
    // The buffer of the kept pairs is made by the first pass that fills it (as the
    // first guess of the list pool's and again as the sized pool's it made up a
    // tenth of the creation of a world of 46,620 particles).
    w_->pair_w_on_ = true;
    w_->check(cudaStreamSynchronize(w_->st_), "dfsph init");
}

DfsphSolver::~DfsphSolver() {
    if (sum_host_) cudaFreeHost(sum_host_);
}

void DfsphSolver::set_lanes(uint32_t lanes) {
    if (lanes != 0 && lanes != 1 && lanes != 8 && lanes != 32) throw std::invalid_argument("lanes per slot");
    df_lanes_ = df_lanes_boundary_ = lanes;
    if (lanes == 0) {
        df_lanes_ = dfsph_lanes(n_fluid_, n_);
        df_lanes_boundary_ = dfsph_boundary_lanes(n_fluid_, n_);
    }
}

void DfsphSolver::rebuild_neighbours() { rebuild(); }

void DfsphSolver::compute_density() {
    World& w = *w_;
    const uint32_t n = (uint32_t)w.n_;
    if (!n) return;
    with_df_lanes(df_lanes_, [&](auto gc) {
        constexpr int G = decltype(gc)::value;
        k_df_density<G><<<df_blocks<G>(n), kDfThreads, df_smem<G, 1>(), w.st_>>>(n, kc_, w.cur_, w.lists_);
    });
    w.launches_ += 1;
}

void DfsphSolver::compute_alpha() { alpha_pass(alpha_); }

// alpha (unless null) and what the solvers' passes read of the pairs
void DfsphSolver::alpha_pass(double* alpha) {
    World& w = *w_;
    const uint32_t n = (uint32_t)w.n_;
    if (!n) return;
    w.make_pair_weights();
    if (w.lists_.wpair && !w.w_short_cleared_)
        w.check(cudaMemsetAsync(&w.sc_->w_short, 0, sizeof(uint32_t), w.st_), "memset");
    w.w_short_cleared_ = false;
    with_df_lanes(df_lanes_, [&](auto gc) {
        constexpr int G = decltype(gc)::value;
        constexpr int K = G < 4 ? 1 : 4;
        k_df_alpha<G><<<df_blocks<G>(n), kDfThreads, df_smem<G, K>() + df_smem<G, 1>(), w.st_>>>(
            n, kc_, w.cur_, w.lists_, alpha, wsum_);
    });
    w.launches_ += 1;
    if (w.lists_.wpair) {
        with_df_lanes(df_lanes_boundary_, [&](auto gc) {
            constexpr int G = decltype(gc)::value;
            k_df_boundary_weights<G><<<df_blocks<G>(n), kDfThreads, 0, w.st_>>>(n, kc_, w.cur_, w.lists_);
        });
        w.launches_ += 1;
    }
    w.w_valid_ = true;
}

// Before a solver: the positions may have been set, or moved by the slip planes, since alpha's pass.
void DfsphSolver::keep_pairs() {
    w_->make_pair_weights();
    if (!w_->w_valid_) alpha_pass(nullptr);
}

// Calls f(integral_constant<int, G>, bool_constant<KEPT>)
template <class F>
void DfsphSolver::with_pairs(uint32_t lanes, F&& f) {
    with_df_lanes(lanes, [&](auto gc) {
        if (w_->lists_.wpair) f(gc, std::true_type{});
        else f(gc, std::false_type{});
    });
}

double DfsphSolver::mean_density_error() {
    World& w = *w_;
    const uint64_t n = w.n_;
    std::vector<double> rho(n);
    std::vector<uint8_t> kind(n);
    if (n) {
        w.get_scalar(0, rho.data());
        w.get_kind(kind.data());
    }
    double s = 0.0;
    uint64_t c = 0;
    for (uint64_t i = 0; i < n; ++i)
        if (kind[i] == 0) {
            s += std::fabs(rho[i] - w.rho0_) / w.rho0_;
            c += 1;
        }
    return c == 0 ? 0.0 : s / (double)c;
}

double DfsphSolver::v_max() {
    World& w = *w_;
    const uint64_t n = w.n_;
    std::vector<double> v(3 * n);
    std::vector<uint8_t> kind(n);
    if (n) {
        w.get_vec(1, v.data());
        w.get_kind(kind.data());
    }
    double m = 0.0;
    for (uint64_t i = 0; i < n; ++i)
        if (kind[i] == 0) m = std::fmax(m, v[3 * i] * v[3 * i] + v[3 * i + 1] * v[3 * i + 1] + v[3 * i + 2] * v[3 * i + 2]);
    return std::sqrt(m);
}

void DfsphSolver::set_params(const DfsphParams& p) {
    if (kernel_support(p.kernel, w_->h_) != kernel_support(prm_.kernel, w_->h_))
        throw std::invalid_argument("the support radius is fixed at creation");
    prm_ = p;
    if (prm_.particle_diameter <= 0.0) prm_.particle_diameter = w_->h_;
    refresh_const();
}

void DfsphSolver::refresh_const() {
    DfsphConst& k = kc_;
    const World& w = *w_;
    w_->w_valid_ = false;  // what is kept of the pairs is the parameters' too
    k.dim = w.dim_;
    k.kf = make_kernel_fn(prm_.kernel, w.h_, w.dim_);
    k.mass = w.mass_;
    k.rho0 = w.rho0_;
    // dfsph.rs:225 rho = mass * w(kern, 0.0, h, dim)
    double w0;
    switch (prm_.kernel) {
        case kCubic: w0 = k.kf.alpha * (1.0 - 1.5 * 0.0 * 0.0 + 0.75 * 0.0 * 0.0 * 0.0); break;
        case kWendland: w0 = k.kf.alpha * 1.0 * 1.0 * 1.0 * 1.0 * (2.0 * 0.0 + 1.0); break;
        case kPoly6: {
            const double t = w.h_ * w.h_ - 0.0 * 0.0;
            w0 = k.kf.alpha * t * t * t;
            break;
        }
        default: {
            const double t = w.h_ - 0.0;
            w0 = k.kf.alpha * t * t * t;
            break;
        }
    }
    k.rho_self = k.mass * w0;
    k.eps_h = 0.15 * w.h_;
    // dfsph.rs:260-267
    const double h_safe = std::fmax(w.h_, 1e-12);
    const double char_grad = w.dim_ == 2 ? k.mass / (h_safe * h_safe * h_safe)
                                         : k.mass / (h_safe * h_safe * h_safe * h_safe);
    k.denom_floor = std::fmax(1e-6 * char_grad * char_grad, 1e-12);
    k.xsph_eps = prm_.xsph_epsilon;
    k.gx = prm_.gravity[0];
    k.gy = prm_.gravity[1];
    k.gz = prm_.gravity[2];
    k.omega = prm_.solver_omega;
    k.dv_cap = prm_.max_velocity_correction;
    k.warm_start = prm_.warm_start;
    {
        const double far = kernel_support(prm_.kernel, w.h_) * (1.0 + 1e-9);
        k.far2 = far * far;
    }
    for (int a = 0; a < 4; ++a) {
        k.has_slip[a] = prm_.has_slip[a];
        k.slip[a] = prm_.slip[a];
    }
}

void DfsphSolver::rebuild() {
    World& w = *w_;
    w.build_grid(nullptr, nullptr, true);
    w.ensure_lists(false);  // visit lists (fluid) and ascending fluid lists (boundary)
}

void DfsphSolver::density_and_alpha() {
    compute_density();
    compute_alpha();
}

void DfsphSolver::pressure_update(double dt, bool /*divergence*/) {
    World& w = *w_;
    const uint32_t n = (uint32_t)w.n_;
    const double inv_dt = 1.0 / std::fmax(dt, 1e-12);
    with_pairs(df_lanes_, [&](auto gc, auto kept) {
        constexpr int G = decltype(gc)::value;
        constexpr int K = G < 3 ? 1 : 3;
        k_df_pressure_fluid<G, decltype(kept)::value>
            <<<df_blocks<G>(n), kDfThreads, df_smem<G, K>(2), w.st_>>>(n, kc_, dt, inv_dt, w.cur_, w.lists_, kr_, wsum_,
                                                                      react_);
    });
    with_pairs(df_lanes_boundary_, [&](auto gc, auto kept) {
        constexpr int G = decltype(gc)::value;
        constexpr int K = G < 3 ? 1 : 3;
        k_df_pressure_boundary<G, decltype(kept)::value>
            <<<df_blocks<G>(n), kDfThreads, df_smem<G, K>(), w.st_>>>(n, kc_, w.cur_, w.lists_, react_);
    });
    w.launches_ += 2;
}

double DfsphSolver::solve_error(double dt, bool divergence) {
    World& w = *w_;
    const uint32_t n = (uint32_t)w.n_;
    with_pairs(df_lanes_, [&](auto gc, auto kept) {
        constexpr int G = decltype(gc)::value;
        k_df_error<G, decltype(kept)::value><<<df_blocks<G>(n), kDfThreads, df_smem<G, 1>(), w.st_>>>(
            n, kc_, divergence ? 1 : 0, dt, dt * dt, w.cur_, w.lists_, alpha_, kappa_, kr_, err_orig_);
    });
    k_df_partial_sums<<<kSumBlocks, kSumThreads, 0, w.st_>>>(n, err_orig_, part_);
    k_df_final_sum<<<1, kSumThreads, 0, w.st_>>>(part_, sum_);
    w.launches_ += 3;
    // the sequential sum's terms are kept until the decision is known: the
    // pressure update does not touch them
    pressure_update(dt, divergence);
    w.check(cudaMemcpyAsync(sum_host_, sum_, sizeof(double), cudaMemcpyDeviceToHost, w.st_), "dfsph error");
    w.check(cudaStreamSynchronize(w.st_), "dfsph error");
    const double tol = divergence ? prm_.divergence_error_tol : prm_.density_error_tol;
    const double cnt = n_fluid_ > 0 ? (double)n_fluid_ : 1.0;
    const double S = *sum_host_;
    const double u = std::ldexp(1.0, -53);
    const double nm1 = n > 1 ? (double)(n - 1) : 0.0;
    const double gam = nm1 * u / (1.0 - nm1 * u);
    // generous outward margin for the bracket's own roundings
    const double delta = (2.0 * gam / (1.0 - gam)) * S * (1.0 + 1e-6) + 4.0 * std::numeric_limits<double>::denorm_min();
    const double hi = (S + delta) / cnt, lo = std::fmax(S - delta, 0.0) / cnt;
    if (std::isfinite(S) && hi <= tol) return S / cnt;            // the sequential average is <= tol too
    if (std::isfinite(S) && lo > tol && lo == lo) return S / cnt;  // and > tol here
    // within the bracket's width of the tolerance (or non-finite): the sequential sum decides
    k_df_serial_sum<<<1, 32, 0, w.st_>>>(n, err_orig_, sum_);
    w.launches_ += 1;
    w.check(cudaMemcpyAsync(sum_host_, sum_, sizeof(double), cudaMemcpyDeviceToHost, w.st_), "dfsph error");
    w.check(cudaStreamSynchronize(w.st_), "dfsph error");
    ++serial_sums_;
    double avg = *sum_host_;
    if (n_fluid_ > 0) avg /= (double)n_fluid_;
    return avg;
}

uint64_t DfsphSolver::correct_density_error(double dt) {
    World& w = *w_;
    const uint32_t n = (uint32_t)w.n_;
    const uint32_t nb = blocks_for(n, kDfThreads);
    keep_pairs();
    if (prm_.warm_start) {
        k_df_warm_load<<<nb, kDfThreads, 0, w.st_>>>(n, kc_, 0, w.cur_, kappa_, kr_);
        w.launches_ += 1;
        pressure_update(dt, false);
    }
    k_df_warm_zero<<<nb, kDfThreads, 0, w.st_>>>(n, 0, w.cur_);
    w.launches_ += 1;
    uint64_t iters = 0;
    for (;;) {
        const double avg = solve_error(dt, false);
        iters += 1;
        err_density_ = avg;
        if ((avg <= prm_.density_error_tol && iters >= 2) || iters >= prm_.max_density_iters) break;
    }
    return iters;
}

uint64_t DfsphSolver::correct_divergence_error(double dt) {
    World& w = *w_;
    const uint32_t n = (uint32_t)w.n_;
    const uint32_t nb = blocks_for(n, kDfThreads);
    keep_pairs();
    if (prm_.warm_start) {
        k_df_warm_load<<<nb, kDfThreads, 0, w.st_>>>(n, kc_, 1, w.cur_, kappa_, kr_);
        w.launches_ += 1;
        pressure_update(dt, true);
    }
    k_df_warm_zero<<<nb, kDfThreads, 0, w.st_>>>(n, 1, w.cur_);
    w.launches_ += 1;
    uint64_t iters = 0;
    for (;;) {
        const double avg = solve_error(dt, true);
        iters += 1;
        err_divergence_ = avg;
        if ((avg <= prm_.divergence_error_tol && iters >= 1) || iters >= prm_.max_divergence_iters) break;
    }
    return iters;
}

void DfsphSolver::free_slip() {
    if (!prm_.has_slip[0] && !prm_.has_slip[1] && !prm_.has_slip[2] && !prm_.has_slip[3]) return;
    World& w = *w_;
    const uint32_t n = (uint32_t)w.n_;
    k_df_free_slip<<<blocks_for(n, kDfThreads), kDfThreads, 0, w.st_>>>(n, kc_, w.cur_);
    w.launches_ += 1;
    w.w_valid_ = false;  // positions on the planes have moved
}

void DfsphSolver::step(double dt_in) {
    World& w = *w_;
    const uint32_t n = (uint32_t)w.n_;
    const double dt = std::fmax(dt_in, 1e-12);
    last_dt_ = dt;
    if (n == 0) {
        w.t_ += dt;
        return;
    }
    const uint32_t nb = blocks_for(n, kDfThreads);
    cudaStream_t st = w.st_;
    k_df_begin<<<nb, kDfThreads, 0, st>>>(n, kc_, dt, w.cur_);
    w.launches_ += 1;
    if (prm_.xsph_epsilon != 0.0) {
        with_df_lanes(df_lanes_, [&](auto gc) {
            constexpr int G = decltype(gc)::value;
            k_df_xsph<G><<<df_blocks<G>(n), kDfThreads, df_smem<G, (G < 3 ? 1 : 3)>(), st>>>(n, kc_, w.cur_, w.lists_,
                                                                                            dv_);
        });
        k_df_xsph_apply<<<nb, kDfThreads, 0, st>>>(n, w.cur_, dv_);
        w.launches_ += 2;
    }
    it_density_ = correct_density_error(dt);
    k_df_advect<<<nb, kDfThreads, 0, st>>>(n, w.dim_, dt, w.cur_);
    w.launches_ += 1;
    free_slip();
    rebuild();
    density_and_alpha();
    it_divergence_ = correct_divergence_error(dt);
    free_slip();
    k_df_finish<<<nb, kDfThreads, 0, st>>>(n, w.dim_, w.cur_);
    w.launches_ += 1;
    w.check(cudaGetLastError(), "dfsph step");
    w.t_ += dt;
    a_adv_set_ = true;
}

double DfsphSolver::suggest_dt() {
    World& w = *w_;
    const uint64_t n = w.n_;
    std::vector<double> v(3 * n);
    std::vector<uint8_t> kind(n);
    if (n) {
        w.get_vec(1, v.data());
        w.get_kind(kind.data());
    }
    const double g2 = prm_.gravity[0] * prm_.gravity[0] + prm_.gravity[1] * prm_.gravity[1] +
                      prm_.gravity[2] * prm_.gravity[2];
    double vmax = 0.0, amax = 0.0;
    for (uint64_t i = 0; i < n; ++i) {
        if (kind[i] != 0) continue;
        vmax = std::fmax(vmax, v[3 * i] * v[3 * i] + v[3 * i + 1] * v[3 * i + 1] + v[3 * i + 2] * v[3 * i + 2]);
        amax = std::fmax(amax, a_adv_set_ ? g2 : 0.0);
    }
    vmax = std::sqrt(vmax);
    amax = std::sqrt(amax);
    const double d = std::fmax(prm_.particle_diameter, 1e-12);
    const double dt_v = prm_.cfl_lambda * d / std::fmax(vmax, 1e-6);
    // cfl.rs:36 suggested_dt(h, 0, vmax, max(amax, 1e-6), {cfl_lambda, 0.25})
    const double am = std::fmax(amax, 1e-6);
    const double dv2 = prm_.cfl_lambda * w.h_ / std::fmax(0.0 + vmax, 1e-12);
    const double df2 = am > 1e-12 ? 0.25 * std::sqrt(w.h_ / am) : std::numeric_limits<double>::infinity();
    const double dt_f = std::fmin(dv2, df2);
    const double r = std::fmin(dt_v, dt_f);
    return r < 1e-6 ? 1e-6 : (r > 1e-2 ? 1e-2 : r);
}

double DfsphSolver::step_adaptive() {
    a_adv_set_ = true;  // dfsph.rs:774 compute_nonpressure_accel
    const double dt = prm_.adaptive_dt ? suggest_dt() : std::fmax(last_dt_, 1e-4);
    step(dt);
    return dt;
}

void DfsphSolver::run(double dt, uint64_t steps) {
    for (uint64_t s = 0; s < steps; ++s) {
        step(dt);
        if ((s + 1) % 16 == 0) w_->status();
    }
}

void DfsphSolver::get_alpha(double* out) {
    World& w = *w_;
    const uint32_t n = (uint32_t)w.n_;
    if (!n) return;
    k_df_export_orig<<<blocks_for(n, 256), 256, 0, w.st_>>>(n, w.cur_.orig, alpha_, err_orig_);
    w.check(cudaMemcpyAsync(out, err_orig_, sizeof(double) * n, cudaMemcpyDeviceToHost, w.st_), "alpha");
    w.check(cudaStreamSynchronize(w.st_), "alpha");
}

}  // namespace pe

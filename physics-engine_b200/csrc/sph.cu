// The f64 SPH passes of the WCSPH step, one thread per cell-sorted slot.
//
// Each pass walks the slot's neighbour list and reproduces the reference's
// floating-point sequence exactly (compiled with --fmad=false):
//   density   — wcsph.rs:117-154 (visiting order)
//   pressure  — wcsph.rs:157-178, eos.rs:59-80, viscosity.rs:89
//   forces    — wcsph.rs:181-259 + the kick/drift of wcsph.rs:332-342
//   xsph      — wcsph.rs:283-323
//
// Force-order argument. The reference accumulates a[i] by a symmetric
// scatter: for each fluid i in ascending index, for each neighbour j in
// visiting order, a fluid j > i adds f to a[i] and subtracts it from a[j].
// Hence the final a[k] is the sequence
//     0  -  f(i1,k) - f(i2,k) - ...      (fluid i < k, ascending i)
//        +  f(k,j) ...                   (fluid j > k and boundary j, visiting order)
//        +  g.
// Every factor of f(i,k) is symmetric in (i,k) bit for bit (sums commute,
// (-a)(-b) = ab exactly) except grad W, which flips sign exactly, so
// f(i,k) = -f(k,i) bitwise and x - f(i,k) = x + f(k,i). A gather that adds
// f(k,i) over the "lower" list (ascending original index) and then f(k,j)
// over the visiting-order list, skipping entries flagged lower, therefore
// yields the reference's bits. Pairs outside the support contribute +-0,
// which leaves a sum that started at +0 unchanged, so the lists may omit them.
#include <algorithm>
#include <type_traits>

#include "pe_math.cuh"
#include "wcsph_device.cuh"
#include "sph_pair.cuh"
#include "list_iter.cuh"
#include "lane_group.cuh"

namespace pe {

namespace {

constexpr int kThreads = 128;
// Visit entries compacted per chunk in the force pass. 64 rather than 32: the
// warp's pair loop runs to the fullest lane of each chunk, and the spread of
// the kept counts shrinks relative to their mean as the chunk grows (forces
// 3.32 -> 3.17 ms at 1M). 64 x 4 bytes per thread is 32 KB per 128-thread
// CTA, which still leaves the pass register-limited (five CTAs per SM).
constexpr uint32_t kCompact = 64;

inline uint32_t blocks_for(uint64_t n, uint32_t t) { return (uint32_t)((n + t - 1) / t); }

struct PosVel {
    double4 x, v;
};

__device__ __forceinline__ void prefetch_l1(const void* p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// Bound by the L1's data path (76 % of its wavefronts with two 16-byte loads a
// gathered position, one 4-byte load an entry and a 16-byte store every other
// W), then by fixed latencies. Rows of four entries are read, and their W
// stored, in one access each, and a position is one 32-byte load: 1410 ->
// 1105 us at 1M (the FP64 issue alone would take ~0.5 ms). Held to 80
// registers (six CTAs of 128 threads an SM) with the data one entry ahead;
// two ahead takes 95 registers and 1125 us, 64 registers spill and take 1527.
template <bool CUBIC>
__global__ void __launch_bounds__(kMaxPassThreads, 3) k_density(uint32_t n, StepConst k, StateBufs s,
                                                      ListBufs l) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (s.flags[i] & kFlagBoundary) {
        s.vel[i].w = k.rho0;  // wcsph.rs:127
        return;
    }
    const double4 xi = s.pos[i];
    double rho = k.rho_self;  // 0.0 + mass * W(0)
    const ListRef vr = list_ref(l, i, kListVisit);
    // W of entry t kept at the entry's pool index for the XSPH pass, a row of
    // four in one 32-byte store; wrow walks the slot's rows
    bool keep_w = false;
    if (l.wpair) {
        keep_w = w_fits(l, vr);
        if (!keep_w) atomicOr(l.w_short, 1u);
    }
    double* wrow = keep_w ? l.wpair + (vr.p - l.pool) : nullptr;
    double w4[4] = {0.0, 0.0, 0.0, 0.0};
    for_each_row<1>(
        vr, [&](uint32_t e) { return gather4(s.pos + (e & kEntrySlotMask)); }, [](uint32_t) {},
        [&](uint32_t q, uint32_t e, const double4& xj) {
            const uint32_t j = e & kEntrySlotMask;
            const double dx = xj.x - xi.x, dy = xj.y - xi.y, dz = xj.z - xi.z;
            const double wij = w_of_r2<CUBIC>(dx * dx + dy * dy + dz * dz, k);
            w4[q] = wij;
            if ((e & kEntryOriented) && !sees_fluid(k, xj, s.nout[j], xi.x, xi.y, xi.z)) return;
            // fluid: mass * W; boundary: (rho0 * psi_j) * W (wcsph.rs:143-148)
            const double f = (e & kEntryBoundary) ? k.rho0 * xj.w : k.mass;
            rho += f * wij;
        },
        [&](uint32_t) {
            if (keep_w) {
                store4(wrow, w4);
                wrow += vr.step;
            }
        });
    rho = fmax(rho, 1e-12);  // wcsph.rs:152 (f64::max)
    s.vel[i].w = rho;
    // keep the cached p / rho^2 consistent with the new rho (the reference
    // divides the stored p by the current rho in every force pair)
    s.pos[i].w = s.p[i] / (rho * rho);
}

// max |v|^2 of each tank's fluid (viscosity.rs:89-100), as u64 bits: a warp
// whose lanes all belong to one tank reduces first, a warp across a tank
// boundary lets each lane add its own value.
__global__ void k_vmax(uint32_t n, Tanks tk, StateBufs s) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    double m = 0.0;
    uint32_t t = 0xffffffffu;
    if (i < n) {
        t = tk.slot_tank[i];
        if (!(s.flags[i] & kFlagBoundary)) {
            double4 v = s.vel[i];
            double q = v.x * v.x + v.y * v.y + v.z * v.z;
            if (q > m) m = q;  // viscosity.rs:91-96 (NaN never exceeds m)
        }
    }
    unsigned long long b = __double_as_longlong(m);
    const uint32_t t0 = __shfl_sync(0xffffffffu, t, 0);
    if (i >= n) t = t0;  // idle lanes carry lane 0's tank and a zero
    if (__all_sync(0xffffffffu, t == t0)) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            unsigned long long x = __shfl_xor_sync(0xffffffffu, b, o);
            b = x > b ? x : b;
        }
        // Non-negative doubles order like their bit patterns.
        if ((threadIdx.x & 31u) == 0 && b != 0ull && t0 != 0xffffffffu) atomicMax(&tk.vmax2[t0], b);
    } else if (b != 0ull && i < n) {
        atomicMax(&tk.vmax2[t], b);
    }
}

__global__ void k_pressure(uint32_t n, StepConst k, Tanks tk, StateBufs s) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // compute_pressure (wcsph.rs:158-169): c = max(c, 10 * v_max), persisted
    // per tank. Every thread of a tank derives the same c; re-reading an
    // already-updated c gives the same value (the update is idempotent), so
    // the write by the tank's first slot is race-free in effect.
    const uint32_t t = tk.slot_tank[i];
    double c = tk.c[t];
    if (k.adapt_sound_speed) {
        double vmax = sqrt(__longlong_as_double((long long)tk.vmax2[t]));
        double min_c = 10.0 * fmax(vmax, 0.0);
        c = c < min_c ? min_c : c;
    }
    if (i == tk.desc[t].slot_begin) tk.c[t] = c;
    if (s.flags[i] & kFlagBoundary) {
        s.p[i] = 0.0;
        return;
    }
    double rho = s.vel[i].w;
    double ratio = rho / k.eos_rho0;
    double b = k.eos_rho0 * c * c / k.eos_gamma;
    double pw = k.gamma_is_int ? pow_int_dd(ratio, k.gamma_int) : pow(ratio, k.eos_gamma);
    double p = b * (pw - 1.0);
    s.p[i] = p;
    s.pos[i].w = p / (rho * rho);  // p_i / (rho_i * rho_i), used by every pair of i
}

// Pressure + Monaghan viscosity force of fluid pair (k, j), seen from k:
// rx = x_j - x_k (wcsph.rs:219), pi_ij(x_k, x_j, v_k, v_j, rho_k, rho_j).
template <bool CUBIC, bool BETA0>
__device__ __forceinline__ void fluid_pair(const StepConst& kc, bool fast, double nac, const double4& xk, const double4& vk,
                                           const double4& xj, const double4& vj, double (&f)[3]) {
    const double rx = xj.x - xk.x, ry = xj.y - xk.y, rz = xj.z - xk.z;
    const double r2 = rx * rx + ry * ry + rz * rz;
    // viscosity.rs:51-73 with r_ij = x_k - x_j, v_ij = v_k - v_j. Evaluated for
    // every pair and selected, so that approaching and receding pairs do not
    // split the warp; a receding pair's value is discarded (pi = 0 exactly).
    // x_k - x_j is exactly -(x_j - x_k) (round to nearest is symmetric), so
    // |x_k - x_j|^2 is r2 bit for bit and v_ij . (x_k - x_j) is -(v_ij . r)
    // up to the sign of a zero, which only ever selects pi = 0.
    const double wx = vk.x - vj.x, wy = vk.y - vj.y, wz = vk.z - vj.z;
    const double vr = -(wx * rx + wy * ry + wz * rz);
    const double rho_bar = 0.5 * (vk.w + vj.w);
    const double d2 = r2 + kc.eps_h2;
    double sc, pic;
    double r = 0.0, y = 0.0;
    bool block = fast && moderate(r2) && moderate(rho_bar) && moderate_or_zero(vr);
    if (block) {
        y = sqrt_rn(r2, &r);
        block = divisor_ok(r) && divisor_ok(d2) && divisor_ok(rho_bar);
    }
    if (block) {
        const double dwdr = CUBIC ? dwdr_cubic_block(r, kc) : kern_dwdr(r, kc);
        sc = quot_rn(-dwdr, r, recip_refine(r, y));
        const double mu = quot_rn(kc.h * vr, d2, recip_rn(d2));
        // With beta = 0 the beta mu^2 term is a signed zero, which leaves the
        // nonzero nac * mu of an approaching pair (mu < 0) unchanged.
        const double num = BETA0 ? nac * mu : nac * mu + kc.visc_beta * mu * mu;
        pic = quot_rn(num, rho_bar, recip_rn(rho_bar));
    } else {
        r = sqrt(r2);
        if (r < 1e-30) return;
        sc = -kdwdr<CUBIC>(r, kc) / r;
        const double mu = kc.h * vr / d2;
        const double num = BETA0 ? nac * mu : nac * mu + kc.visc_beta * mu * mu;
        pic = num / rho_bar;
    }
    const double gx = rx * sc, gy = ry * sc, gz = rz * sc;
    const double press = xk.w + xj.w;  // p_k/rho_k^2 + p_j/rho_j^2
    const double mp = -kc.mass * press;
    const double pi = vr >= 0.0 ? 0.0 : pic;
    const double mv = -kc.mass * pi;
    f[0] = gx * mp + gx * mv;
    f[1] = gy * mp + gy * mv;
    f[2] = gz * mp + gz * mv;
}

// Akinci boundary pressure of fluid k against boundary sample j (wcsph.rs:244-255).
template <bool CUBIC>
__device__ __forceinline__ void boundary_pair(const StepConst& kc, const double4& xk, const double4& xj,
                                              bool oriented, const double4* nout, uint32_t j, double (&f)[3]) {
    double rx = xj.x - xk.x, ry = xj.y - xk.y, rz = xj.z - xk.z;
    double sc;
    if (!grad_scale<CUBIC>(rx * rx + ry * ry + rz * rz, kc, &sc)) return;
    if (oriented && !sees_fluid(kc, xj, nout[j], xk.x, xk.y, xk.z)) return;
    double gx = rx * sc, gy = ry * sc, gz = rz * sc;
    double m = -(kc.rho0 * xj.w) * xk.w;  // -(rho0 psi_j) * p_k/rho_k^2
    f[0] = gx * m;
    f[1] = gy * m;
    f[2] = gz * m;
}

template <bool INTEGRATE, int DIM, bool CUBIC, bool BETA0>
__global__ void __launch_bounds__(kMaxPassThreads) k_forces(uint32_t n, StepConst kc, Tanks tk,
                                                            StateBufs s, ListBufs l, double dt,
                                                            double4* __restrict__ pos_next,
                                                            double4* __restrict__ vel_next,
                                                            const double4* __restrict__ st_a) {
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    if (s.flags[k] & kFlagBoundary) return;
    const double c0 = tk.c[tk.slot_tank[k]];
    const double nac = -kc.visc_alpha * c0;  // (-alpha) * c_bar, viscosity.rs:72
    const bool fast = kc.moderate && moderate_or_zero(nac);
    const double4 xk = s.pos[k];
    const double4 vk = s.vel[k];
    double ax = 0.0, ay = 0.0, az = 0.0;
    // neighbour state gathered one entry ahead (boundary samples need no velocity)
    auto load = [&](uint32_t e) {
        PosVel d;
        const uint32_t j = e & kEntrySlotMask;
        d.x = gather4(s.pos + j);
        d.v = gather4(s.vel + j);
        return d;
    };
    // fluid i < k, ascending original index
    for_each_loaded(list_ref(l, k, kListLower), load, [&](uint32_t, const PosVel& d) {
        double f[3] = {0.0, 0.0, 0.0};
        fluid_pair<CUBIC, BETA0>(kc, fast, nac, xk, vk, d.x, d.v, f);
        ax += f[0];
        ay += f[1];
        az += f[2];
    });
    // fluid j > k and boundary j, visiting order: the visit list without the
    // entries flagged lower (those came from the lower list, in index order).
    // The list is taken in chunks of kCompact entries whose kept entries are
    // first compacted into this thread's column of shared memory, so the pair
    // loop of a warp runs over kept entries only (the flagged ones are about
    // half and fall at different positions in each thread's list). Chunks stay
    // in step across the warp: a per-lane stream that refilled each lane's
    // buffer when it ran empty made the warp wait on every lane's list loads
    // in turn (forces 3.47 -> 4.75 ms at 1M, 19 of 32 lanes active).
    // The chunks are aligned to the list's end (the first one is the short
    // one): the kept entries cluster at the end of the visiting order (the
    // neighbour cells after the particle's own), so there every lane's chunk
    // is full and none waits on a fuller one.
    extern __shared__ uint32_t s_keep[];  // kCompact x blockDim.x, column per thread
    const uint32_t tid = threadIdx.x, bd = blockDim.x;
    const ListRef vr = list_ref(l, k, kListVisit);
    const uint32_t nv4 = (vr.n + 3u) & ~3u;  // chunk ends stay on 16-byte groups
    uint32_t t1 = nv4 ? nv4 - (nv4 - 1u) / kCompact * kCompact : 0u;
    for (uint32_t t0 = 0; t0 < vr.n; t0 = t1, t1 += kCompact) {
        const uint32_t te = min(vr.n, t1);
        uint32_t c = 0;
        for (uint32_t t = t0; t < te; t += 4) {
            const uint4 g4 = __ldg(reinterpret_cast<const uint4*>(vr.p + (size_t)(t >> 2) * vr.step));
            const uint32_t ge[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q)
                if (t + q < te && !(ge[q] & kEntryLower)) s_keep[(c++) * bd + tid] = ge[q];
        }
        if (c == 0) continue;
        uint32_t e = s_keep[tid];
        PosVel d = load(e);
        for (uint32_t u = 0; u < c; ++u) {
            const uint32_t ec = e;
            const PosVel dc = d;
            if (u + 1 < c) {
                e = s_keep[(u + 1) * bd + tid];
                d = load(e);
            }
            double f[3] = {0.0, 0.0, 0.0};
            if (ec & kEntryBoundary) {
                boundary_pair<CUBIC>(kc, xk, dc.x, (ec & kEntryOriented) != 0u, s.nout, ec & kEntrySlotMask, f);
            } else {
                fluid_pair<CUBIC, BETA0>(kc, fast, nac, xk, vk, dc.x, dc.v, f);
            }
            ax += f[0];
            ay += f[1];
            az += f[2];
        }
    }
    ax += kc.gx;
    ay += kc.gy;
    az += kc.gz;
    if (st_a) {  // wcsph.rs:273-277 a += surface-tension acceleration
        const double4 t = st_a[k];
        ax += t.x;
        ay += t.y;
        az += t.z;
    }
    s.acc[k] = make_double4(ax, ay, az, 0.0);
    if (INTEGRATE) {
        // wcsph.rs:336-341 symplectic Euler
        double vx = vk.x + ax * dt, vy = vk.y + ay * dt, vz = vk.z + az * dt;
        double px = xk.x + vx * dt, py = xk.y + vy * dt, pz = xk.z + vz * dt;
        if (DIM == 2) {
            pz = 0.0;
            vz = 0.0;
        }
        pos_next[k] = make_double4(px, py, pz, xk.w);
        vel_next[k] = make_double4(vx, vy, vz, vk.w);
    }
}

// boundary_force[j] (wcsph.rs:254): sum over fluid i in ascending index of
// f(i,j) * (-m) with f = gradW(x_j - x_i) * (-(rho0 psi_j) * p_i/rho_i^2).
template <bool CUBIC>
__global__ void __launch_bounds__(kThreads) k_boundary_force(uint32_t n, StepConst kc, StateBufs s,
                                                             ListBufs l) {
    uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n) return;
    if (!(s.flags[b] & kFlagBoundary)) return;
    const double4 xb = s.pos[b];
    const bool oriented = (s.flags[b] & kFlagOriented) != 0;
    const double4 nb = oriented ? s.nout[b] : make_double4(0, 0, 0, 0);
    const double mpsi = -(kc.rho0 * xb.w);
    const double mneg = -kc.mass;
    double fx = 0.0, fy = 0.0, fz = 0.0;
    for_each_entry(list_ref(l, b, kListLower), [&](uint32_t i) {
        double4 xi = s.pos[i];
        double rx = xb.x - xi.x, ry = xb.y - xi.y, rz = xb.z - xi.z;
        double sc;
        if (!grad_scale<CUBIC>(rx * rx + ry * ry + rz * rz, kc, &sc)) return;
        if (oriented && !sees_fluid(kc, xb, nb, xi.x, xi.y, xi.z)) return;
        double m = mpsi * xi.w;
        double ffx = (rx * sc) * m, ffy = (ry * sc) * m, ffz = (rz * sc) * m;
        fx += ffx * mneg;
        fy += ffy * mneg;
        fz += ffz * mneg;
    });
    s.bf[b] = make_double4(fx, fy, fz, 0.0);
}

// The XSPH sum of fluid slot i with velocity vi, each pair's W recomputed
// from the neighbour's position.
template <bool CUBIC>
__device__ __forceinline__ double3 xsph_dv(uint32_t i, const StepConst& kc, const StateBufs& s,
                                           const ListBufs& l, double4 vi) {
    const double4 xi = s.pos[i];
    double dvx = 0.0, dvy = 0.0, dvz = 0.0;
    for_each_loaded2(
        list_ref(l, i, kListVisit),
        [&](uint32_t e) {
            PosVel d{};
            if (!(e & kEntryBoundary)) {
                d.x = gather4(s.pos + (e & kEntrySlotMask));
                d.v = gather4(s.vel + (e & kEntrySlotMask));
            }
            return d;
        },
        [&](uint32_t e, const PosVel& d) {
        if (e & kEntryBoundary) return;
        const double4 xj = d.x;
        const double dx = xj.x - xi.x, dy = xj.y - xi.y, dz = xj.z - xi.z;
        const double wij = w_of_r2<CUBIC>(dx * dx + dy * dy + dz * dz, kc);
        const double4 vj = d.v;
        const double rho_bar = 0.5 * (vi.w + vj.w);
        const double f = mass_over(rho_bar, kc) * wij;
        dvx += (vj.x - vi.x) * f;
        dvy += (vj.y - vi.y) * f;
        dvz += (vj.z - vi.z) * f;
    });
    return make_double3(dvx, dvy, dvz);
}

// short_only: run only if the density pass met a list beyond the pair-weight
// buffer (the launch that follows k_xsph_w, which then did nothing).
template <bool CUBIC>
__global__ void __launch_bounds__(kMaxPassThreads) k_xsph(uint32_t n, StepConst kc, StateBufs s,
                                                   ListBufs l, double4* __restrict__ vel_out,
                                                   bool short_only) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (short_only && !__ldg(l.w_short)) return;
    const double4 vi = s.vel[i];
    if (s.flags[i] & kFlagBoundary) {
        vel_out[i] = vi;
        return;
    }
    const double3 dv = xsph_dv<CUBIC>(i, kc, s, l, vi);
    vel_out[i] = make_double4(vi.x + dv.x * kc.xsph_eps, vi.y + dv.y * kc.xsph_eps,
                              vi.z + dv.z * kc.xsph_eps, vi.w);
}

// k_xsph with each pair's W(r) read from the density pass of the same lists
// and positions (the bits the pair would compute) instead of recomputed from
// the neighbour's position: per fluid pair a quarter of one 32-byte read of a
// stream in place of a 32-byte gather, a square root and the kernel
// polynomial. Bound by the L1's data path like k_density; with rows of four
// entries and weights read in one access each, 32-byte gathers and the block
// form of m / rho_bar, 1412 -> 958 us at 1M (80 registers, one velocity ahead;
// 87 without the register limit 1016 us, two ahead 1270 us).
// When the density pass met a list beyond the buffer, it does nothing and
// the k_xsph launch after it recomputes W for every particle (a separate
// kernel, so that this one keeps its own, smaller register count).
__global__ void __launch_bounds__(kMaxPassThreads, 3) k_xsph_w(uint32_t n, StepConst kc, StateBufs s,
                                                     ListBufs l, double4* __restrict__ vel_out) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (__ldg(l.w_short)) return;
    const double4 vi = s.vel[i];
    if (s.flags[i] & kFlagBoundary) {
        vel_out[i] = vi;
        return;
    }
    double dvx = 0.0, dvy = 0.0, dvz = 0.0;
    const ListRef vr = list_ref(l, i, kListVisit);
    const double* wrow = l.wpair + (vr.p - l.pool);  // walks the rows as the loads advance
    // Both streams (entries, weights) come from DRAM; their rows four ahead
    // are prefetched into L1 (within the slot's own rows): 1.44 -> 1.40 ms at 1M.
    constexpr uint32_t kPfRows = 4;
    const uint32_t nrows = (vr.n + 3u) >> 2;
    const uint32_t* erow = vr.p;
    double w4[4];
    for_each_row<1>(
        vr, [&](uint32_t e) { return gather4(s.vel + (e & kEntrySlotMask)); },
        [&](uint32_t row) {
            load4(wrow, w4);
            if (row + kPfRows < nrows) {
                prefetch_l1(erow + (size_t)kPfRows * vr.step);
                prefetch_l1(wrow + (size_t)kPfRows * vr.step);
            }
            erow += vr.step;
            wrow += vr.step;
        },
        [&](uint32_t q, uint32_t e, const double4& vj) {
            if (e & kEntryBoundary) return;
            const double rho_bar = 0.5 * (vi.w + vj.w);
            const double f = mass_over(rho_bar, kc) * w4[q];
            dvx += (vj.x - vi.x) * f;
            dvy += (vj.y - vi.y) * f;
            dvz += (vj.z - vi.z) * f;
        },
        [](uint32_t) {});
    vel_out[i] = make_double4(vi.x + dvx * kc.xsph_eps, vi.y + dvy * kc.xsph_eps,
                              vi.z + dvz * kc.xsph_eps, vi.w);
}

// ---------------------------------------------------------------------------
// The same passes with G lanes on each slot (lane_group.cuh).
// ---------------------------------------------------------------------------
template <bool CUBIC, int G>
__global__ void __launch_bounds__(kMaxPassThreads) k_density_g(uint32_t n, StepConst k, StateBufs s, ListBufs l) {
    extern __shared__ __align__(16) double s_words[];
    const LaneGroup<G> g;
    const uint32_t i = g.slot;
    const bool fluid = i < n && !(s.flags[i] & kFlagBoundary);
    if (i < n && !fluid && g.sub == 0) s.vel[i].w = k.rho0;  // wcsph.rs:127
    if (!__any_sync(kFullWarp, fluid)) return;
    ListRef vr{l.pool, 0u, 0u};
    double4 xi = make_double4(0.0, 0.0, 0.0, 0.0);
    bool keep_w = false;
    if (fluid) {
        vr = list_ref(l, i, kListVisit);
        xi = s.pos[i];
        if (l.wpair) {
            keep_w = w_fits(l, vr);
            if (!keep_w && g.sub == 0) atomicOr(l.w_short, 1u);
        }
    }
    // W of entry t kept at the entry's pool index: the lanes of a row store 32
    // contiguous bytes
    OrderedSum<G, 1> rho(s_words + g.warp * OrderedSum<G, 1>::kDoubles, g, k.rho_self);  // 0.0 + mass * W(0)
    group_for_each<G>(
        vr, g, [&](uint32_t e, const uint32_t*) { return gather4(s.pos + (e & kEntrySlotMask)); },
        [&](bool has, uint32_t e, const double4& xj, const uint32_t* p) {
            double term[1] = {0.0};
            if (has) {
                const double dx = xj.x - xi.x, dy = xj.y - xi.y, dz = xj.z - xi.z;
                const double wij = w_of_r2<CUBIC>(dx * dx + dy * dy + dz * dz, k);
                if (keep_w) l.wpair[p - l.pool] = wij;
                if (!((e & kEntryOriented) && !sees_fluid(k, xj, s.nout[e & kEntrySlotMask], xi.x, xi.y, xi.z))) {
                    // fluid: mass * W; boundary: (rho0 * psi_j) * W (wcsph.rs:143-148)
                    const double f = (e & kEntryBoundary) ? k.rho0 * xj.w : k.mass;
                    term[0] = f * wij;
                }
            }
            rho.add(term);
        });
    if (fluid && g.sub == 0) {
        const double r = fmax(rho.acc, 1e-12);  // wcsph.rs:152 (f64::max)
        s.vel[i].w = r;
        s.pos[i].w = s.p[i] / (r * r);  // see k_density
    }
}

// Entries of one slot queued in shared memory for the force pass (per group;
// the padding spreads the groups of a warp over the banks).
template <int G>
struct ForceQueue {
    static constexpr uint32_t kFill = 4u * G;  // entries a fill step takes from a list
    static constexpr uint32_t kCap = G == 32 ? 256u : 128u;
    static constexpr uint32_t kPitch = kCap + (G == 4 ? 4u : G == 8 ? 8u : 0u);
    static constexpr uint32_t kWarpBytes = LaneGroup<G>::kPerWarp * kPitch * sizeof(uint32_t);
};

constexpr uint32_t kForceGroupThreads = 128;

template <int G>
constexpr size_t forces_smem(uint32_t threads) {
    return (size_t)(threads / 32u) * (OrderedSum<G, 3>::kDoubles * sizeof(double) + ForceQueue<G>::kWarpBytes);
}

__device__ __forceinline__ double comp(const double4* a, uint32_t i, uint32_t c) {
    return reinterpret_cast<const double*>(a + i)[c];
}

// The force pass with G lanes a slot. Five CTAs of 128 threads an SM (96
// registers; without the limit 110 registers, four CTAs and 2750 us at 1M
// against 2510). One stream of pairs per group: the lower list, then the visit entries not
// flagged lower, queued in order in shared memory and taken G at a time. A
// slot's two parts add up to its visit list, so the groups of a warp run
// equally long, where loops over the lower and the kept entries of 32 slots
// leave a quarter of the lanes idle.
template <bool CUBIC, bool BETA0, int G>
__global__ void __launch_bounds__(kForceGroupThreads, 5) k_forces_g(uint32_t n, StepConst kc, Tanks tk, StateBufs s,
                                                              ListBufs l, int integrate, double dt,
                                                              double4* __restrict__ pos_next,
                                                              double4* __restrict__ vel_next,
                                                              const double4* __restrict__ st_a) {
    extern __shared__ __align__(16) double s_words[];
    const LaneGroup<G> g;
    const uint32_t k = g.slot;
    const bool fluid = k < n && !(s.flags[k] & kFlagBoundary);
    if (!__any_sync(kFullWarp, fluid)) return;
    using Q = ForceQueue<G>;
    const uint32_t warps = blockDim.x >> 5;
    uint32_t* const queue = reinterpret_cast<uint32_t*>(s_words + warps * OrderedSum<G, 3>::kDoubles) +
                            (g.warp * LaneGroup<G>::kPerWarp + g.grp) * Q::kPitch;
    ListRef vr{l.pool, 0u, 0u}, lr{l.pool, 0u, 0u};
    double4 xk = make_double4(0.0, 0.0, 0.0, 0.0), vk = xk;
    double nac = 0.0;
    bool fast = false;
    if (fluid) {
        vr = list_ref(l, k, kListVisit);
        lr = list_ref(l, k, kListLower);
        xk = s.pos[k];
        vk = s.vel[k];
        nac = -kc.visc_alpha * tk.c[tk.slot_tank[k]];  // (-alpha) * c_bar, viscosity.rs:72
        fast = kc.moderate && moderate_or_zero(nac);
    }
    OrderedSum<G, 3> acc(s_words + g.warp * OrderedSum<G, 3>::kDoubles, g, 0.0);
    // fill step f takes rows f * G + sub of the lower list, then of the visit list
    const uint32_t lower_steps = warp_rounds(lr.n, Q::kFill), steps = lower_steps + warp_rounds(vr.n, Q::kFill);
    uint32_t step = 0, tail = 0;
    bool last;
    do {
        for (; step < steps && !__any_sync(kFullWarp, tail + Q::kFill > Q::kCap); ++step) {
            const bool low = step < lower_steps;
            const ListRef& r = low ? lr : vr;
            const uint32_t row = (low ? step : step - lower_steps) * G + g.sub;
            const uint32_t left = 4u * row < r.n ? r.n - 4u * row : 0u;  // entries from this row on
            uint4 e4 = make_uint4(0u, 0u, 0u, 0u);
            if (left) e4 = __ldg(reinterpret_cast<const uint4*>(r.p + (size_t)row * r.step));
            const uint32_t e[4] = {e4.x, e4.y, e4.z, e4.w};
            uint32_t keep = left >= 4u ? 15u : (1u << left) - 1u;
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q)
                if (!low && (e[q] & kEntryLower)) keep &= ~(1u << q);
            const uint32_t c = __popc(keep);
            uint32_t incl = c;  // over the group's lanes
#pragma unroll
            for (uint32_t o = 1; o < G; o <<= 1) {
                const uint32_t v = __shfl_up_sync(kFullWarp, incl, o, G);
                if (g.sub >= o) incl += v;
            }
            uint32_t at = tail + incl - c;
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q)
                if (keep & (1u << q)) queue[at++] = e[q];
            tail += __shfl_sync(kFullWarp, incl, G - 1, G);
        }
        __syncwarp();
        last = step >= steps;
        const uint32_t queued = last ? (tail + G - 1u) / G : tail / G;
        const uint32_t end = last ? tail : queued * G;
        const uint32_t rounds = __reduce_max_sync(kFullWarp, queued);
        uint32_t q = g.sub;
        auto entry = [&]() { return end ? queue[min(q, end - 1u)] : 0u; };  // a lane past the end repeats the last
        auto load = [&](uint32_t e) {
            const uint32_t j = e & kEntrySlotMask;
            return PosVel{gather4(s.pos + j), gather4(s.vel + j)};
        };
        uint32_t e0 = entry();
        bool h0 = q < end;
        PosVel d0 = load(e0);
        q += G;
        uint32_t e1 = entry();
        bool h1 = q < end;
        for (uint32_t u = 0; u < rounds; ++u) {
            const uint32_t e = e0;
            const bool h = h0;
            const PosVel d = d0;
            e0 = e1;
            h0 = h1;
            d0 = load(e0);
            q += G;
            e1 = entry();
            h1 = q < end;
            double f[3] = {0.0, 0.0, 0.0};
            if (h) {
                if (e & kEntryBoundary) {
                    boundary_pair<CUBIC>(kc, xk, d.x, (e & kEntryOriented) != 0u, s.nout, e & kEntrySlotMask, f);
                } else {
                    fluid_pair<CUBIC, BETA0>(kc, fast, nac, xk, vk, d.x, d.v, f);
                }
            }
            acc.add(f);
        }
        if (!last) {  // fewer than G queued entries carry over
            const uint32_t left = tail - queued * G;
            const uint32_t c = g.sub < left ? queue[queued * G + g.sub] : 0u;
            __syncwarp();
            if (g.sub < left) queue[g.sub] = c;
            tail = left;
            __syncwarp();
        }
    } while (!last);
    // Lane c < 4 finishes component c (w: the carried psi or p / rho^2, and rho).
    if (!fluid || g.sub >= 4u) return;
    double a = 0.0;
    if (g.sub < 3u) {
        a = acc.acc + (g.sub == 0 ? kc.gx : g.sub == 1 ? kc.gy : kc.gz);
        if (st_a) a += comp(st_a, k, g.sub);  // wcsph.rs:273-277 a += surface-tension acceleration
    }
    reinterpret_cast<double*>(s.acc + k)[g.sub] = a;
    if (integrate) {
        // wcsph.rs:336-341 symplectic Euler
        double v = comp(s.vel, k, g.sub), x = comp(s.pos, k, g.sub);
        if (g.sub < 3u) {
            v = v + a * dt;
            x = x + v * dt;
            if (kc.dim == 2 && g.sub == 2u) v = x = 0.0;
        }
        reinterpret_cast<double*>(pos_next + k)[g.sub] = x;
        reinterpret_cast<double*>(vel_next + k)[g.sub] = v;
    }
}

template <bool CUBIC, int G>
__global__ void __launch_bounds__(kMaxPassThreads) k_boundary_force_g(uint32_t n, StepConst kc, StateBufs s,
                                                                      ListBufs l) {
    extern __shared__ __align__(16) double s_words[];
    const LaneGroup<G> g;
    const uint32_t b = g.slot;
    const bool bound = b < n && (s.flags[b] & kFlagBoundary);
    if (!__any_sync(kFullWarp, bound)) return;
    ListRef lr{l.pool, 0u, 0u};
    double4 xb = make_double4(0.0, 0.0, 0.0, 0.0), nb = xb;
    bool oriented = false;
    if (bound) {
        lr = list_ref(l, b, kListLower);
        xb = s.pos[b];
        oriented = (s.flags[b] & kFlagOriented) != 0;
        if (oriented) nb = s.nout[b];
    }
    const double mpsi = -(kc.rho0 * xb.w);
    const double mneg = -kc.mass;
    OrderedSum<G, 3> acc(s_words + g.warp * OrderedSum<G, 3>::kDoubles, g, 0.0);
    group_for_each<G>(
        lr, g, [&](uint32_t i, const uint32_t*) { return gather4(s.pos + i); },
        [&](bool has, uint32_t, const double4& xi, const uint32_t*) {
            double f[3] = {0.0, 0.0, 0.0};
            const double rx = xb.x - xi.x, ry = xb.y - xi.y, rz = xb.z - xi.z;
            double sc;
            if (has && grad_scale<CUBIC>(rx * rx + ry * ry + rz * rz, kc, &sc) &&
                !(oriented && !sees_fluid(kc, xb, nb, xi.x, xi.y, xi.z))) {
                const double m = mpsi * xi.w;
                f[0] = ((rx * sc) * m) * mneg;
                f[1] = ((ry * sc) * m) * mneg;
                f[2] = ((rz * sc) * m) * mneg;
            }
            acc.add(f);
        });
    if (bound && g.sub < 4u) reinterpret_cast<double*>(s.bf + b)[g.sub] = g.sub < 3u ? acc.acc : 0.0;
}

// USE_W: each pair's W(r) read from the density pass of the same lists and
// positions (see k_xsph_w); otherwise recomputed. short_only as in k_xsph.
template <bool CUBIC, bool USE_W, int G>
__global__ void __launch_bounds__(kMaxPassThreads) k_xsph_g(uint32_t n, StepConst kc, StateBufs s, ListBufs l,
                                                            double4* __restrict__ vel_out, bool short_only) {
    extern __shared__ __align__(16) double s_words[];
    if (USE_W ? __ldg(l.w_short) != 0u : short_only && !__ldg(l.w_short)) return;
    const LaneGroup<G> g;
    const uint32_t i = g.slot;
    const bool fluid = i < n && !(s.flags[i] & kFlagBoundary);
    double4 vi = make_double4(0.0, 0.0, 0.0, 0.0), xi = vi;
    if (i < n && !fluid && g.sub == 0) vel_out[i] = s.vel[i];
    if (!__any_sync(kFullWarp, fluid)) return;
    ListRef vr{l.pool, 0u, 0u};
    if (fluid) {
        vr = list_ref(l, i, kListVisit);
        vi = s.vel[i];
        if (!USE_W) xi = s.pos[i];
    }
    struct VelW {
        double4 v, x;
        double w;
    };
    OrderedSum<G, 3> dv(s_words + g.warp * OrderedSum<G, 3>::kDoubles, g, 0.0);
    group_for_each<G>(
        vr, g,
        [&](uint32_t e, const uint32_t* p) {
            VelW d{};
            d.v = gather4(s.vel + (e & kEntrySlotMask));
            if (USE_W) d.w = __ldg(l.wpair + (p - l.pool));
            else d.x = gather4(s.pos + (e & kEntrySlotMask));
            return d;
        },
        [&](bool has, uint32_t e, const VelW& d, const uint32_t*) {
            double f[3] = {0.0, 0.0, 0.0};
            if (has && !(e & kEntryBoundary)) {
                double wij = d.w;
                if (!USE_W) {
                    const double dx = d.x.x - xi.x, dy = d.x.y - xi.y, dz = d.x.z - xi.z;
                    wij = w_of_r2<CUBIC>(dx * dx + dy * dy + dz * dz, kc);
                }
                const double rho_bar = 0.5 * (vi.w + d.v.w);
                const double m = mass_over(rho_bar, kc) * wij;
                f[0] = (d.v.x - vi.x) * m;
                f[1] = (d.v.y - vi.y) * m;
                f[2] = (d.v.z - vi.z) * m;
            }
            dv.add(f);
        });
    if (fluid && g.sub < 4u) {
        const double v = comp(s.vel, i, g.sub);
        reinterpret_cast<double*>(vel_out + i)[g.sub] = g.sub < 3u ? v + dv.acc * kc.xsph_eps : v;
    }
}

__global__ void k_in_support(uint32_t n, StepConst kc, StateBufs s, ListBufs l, uint32_t* out) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (s.flags[i] & kFlagBoundary) {
        out[i] = 0;
        return;
    }
    const double4 xi = s.pos[i];
    uint32_t c = 0;
    for_each_entry(list_ref(l, i, kListVisit), [&](uint32_t e) {
        const double4 xj = s.pos[e & kEntrySlotMask];
        const double dx = xj.x - xi.x, dy = xj.y - xi.y, dz = xj.z - xi.z;
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        c += in_support(r, kc);
    });
    out[i] = c;
}

template <bool I, int D, bool C, bool B>
void allow_compact_smem() {
    cudaFuncSetAttribute(k_forces<I, D, C, B>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(kCompact * kMaxPassThreads * sizeof(uint32_t)));
}

template <bool I, int D>
void allow_compact_smem_all() {
    allow_compact_smem<I, D, true, true>();
    allow_compact_smem<I, D, true, false>();
    allow_compact_smem<I, D, false, true>();
    allow_compact_smem<I, D, false, false>();
}

}  // namespace

// The force pass's compaction buffer exceeds the 48 KB a launch gets without
// opting in once a CTA has more than 192 threads.
template <int G>
void allow_forces_smem() {
    auto allow = [](auto* f) {
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)forces_smem<G>(kForceGroupThreads));
    };
    allow(k_forces_g<true, true, G>);
    allow(k_forces_g<true, false, G>);
    allow(k_forces_g<false, true, G>);
    allow(k_forces_g<false, false, G>);
}

void forces_prepare() {
    allow_compact_smem_all<true, 3>();
    allow_compact_smem_all<false, 3>();
    allow_compact_smem_all<true, 2>();
    allow_compact_smem_all<false, 2>();
    allow_forces_smem<4>();
    allow_forces_smem<8>();
    allow_forces_smem<16>();
    allow_forces_smem<32>();
}

// Calls f(integral_constant<int, G>) for the lanes per slot.
template <class F>
static void with_lanes(uint32_t lanes, F&& f) {
    switch (lanes) {
        case 4: f(std::integral_constant<int, 4>{}); break;
        case 8: f(std::integral_constant<int, 8>{}); break;
        case 16: f(std::integral_constant<int, 16>{}); break;
        default: f(std::integral_constant<int, 32>{}); break;
    }
}

template <int G, int K>
static size_t sum_smem(uint32_t threads) {
    return (size_t)(threads / 32u) * OrderedSum<G, K>::kDoubles * sizeof(double);
}

void launch_density(uint32_t n, uint32_t threads, uint32_t lanes, const StepConst& k, const StateBufs& s,
                    const ListBufs& l, cudaStream_t st) {
    if (!n) return;
    if (lanes == 1) {
        if (k.kernel == 0) k_density<true><<<blocks_for(n, threads), threads, 0, st>>>(n, k, s, l);
        else k_density<false><<<blocks_for(n, threads), threads, 0, st>>>(n, k, s, l);
        return;
    }
    with_lanes(lanes, [&](auto gc) {
        constexpr int G = decltype(gc)::value;
        const uint32_t b = blocks_for((uint64_t)n * G, threads);
        const size_t sm = sum_smem<G, 1>(threads);
        if (k.kernel == 0) k_density_g<true, G><<<b, threads, sm, st>>>(n, k, s, l);
        else k_density_g<false, G><<<b, threads, sm, st>>>(n, k, s, l);
    });
}

void launch_vmax(uint32_t n, const Tanks& tk, const StateBufs& s, cudaStream_t st) {
    if (n) k_vmax<<<blocks_for(n, 256), 256, 0, st>>>(n, tk, s);
}

void launch_pressure(uint32_t n, const StepConst& k, const Tanks& tk, const StateBufs& s,
                     cudaStream_t st) {
    if (n) k_pressure<<<blocks_for(n, 256), 256, 0, st>>>(n, k, tk, s);
}

void launch_forces(uint32_t n, uint32_t threads, uint32_t lanes, const StepConst& k, const Tanks& tk,
                   const StateBufs& s, const ListBufs& l, bool integrate, double dt,
                   double4* pos_next, double4* vel_next, const double4* st_a, cudaStream_t st) {
    if (!n) return;
    const bool cubic = k.kernel == 0;
    const bool beta0 = k.visc_beta == 0.0;
    if (lanes != 1) {
        with_lanes(lanes, [&](auto gc) {
            constexpr int G = decltype(gc)::value;
            const uint32_t t = std::min(threads, kForceGroupThreads), b = blocks_for((uint64_t)n * G, t);
            const size_t sm = forces_smem<G>(t);
            auto go = [&](auto* f) {
                f<<<b, t, sm, st>>>(n, k, tk, s, l, integrate ? 1 : 0, dt, pos_next, vel_next, st_a);
            };
            if (cubic) {
                if (beta0) go(k_forces_g<true, true, G>);
                else go(k_forces_g<true, false, G>);
            } else {
                if (beta0) go(k_forces_g<false, true, G>);
                else go(k_forces_g<false, false, G>);
            }
        });
        return;
    }
    const uint32_t b = blocks_for(n, threads);
    const size_t sm = (size_t)kCompact * threads * sizeof(uint32_t);
#define PE_FORCES(I, D, C, B) \
    k_forces<I, D, C, B><<<b, threads, sm, st>>>(n, k, tk, s, l, dt, pos_next, vel_next, st_a)
#define PE_FORCES_B(I, D, C)              \
    do {                                  \
        if (beta0) PE_FORCES(I, D, C, true); \
        else PE_FORCES(I, D, C, false);   \
    } while (0)
    if (k.dim == 3) {
        if (cubic) {
            if (integrate) PE_FORCES_B(true, 3, true);
            else PE_FORCES_B(false, 3, true);
        } else {
            if (integrate) PE_FORCES_B(true, 3, false);
            else PE_FORCES_B(false, 3, false);
        }
    } else {
        if (cubic) {
            if (integrate) PE_FORCES_B(true, 2, true);
            else PE_FORCES_B(false, 2, true);
        } else {
            if (integrate) PE_FORCES_B(true, 2, false);
            else PE_FORCES_B(false, 2, false);
        }
    }
#undef PE_FORCES_B
#undef PE_FORCES
}

void launch_boundary_force(uint32_t n, uint32_t lanes, const StepConst& k, const StateBufs& s, const ListBufs& l,
                           cudaStream_t st) {
    if (!n) return;
    if (lanes == 1) {
        if (k.kernel == 0) k_boundary_force<true><<<blocks_for(n, kThreads), kThreads, 0, st>>>(n, k, s, l);
        else k_boundary_force<false><<<blocks_for(n, kThreads), kThreads, 0, st>>>(n, k, s, l);
        return;
    }
    with_lanes(lanes, [&](auto gc) {
        constexpr int G = decltype(gc)::value;
        const uint32_t b = blocks_for((uint64_t)n * G, kThreads);
        const size_t sm = sum_smem<G, 3>(kThreads);
        if (k.kernel == 0) k_boundary_force_g<true, G><<<b, kThreads, sm, st>>>(n, k, s, l);
        else k_boundary_force_g<false, G><<<b, kThreads, sm, st>>>(n, k, s, l);
    });
}

void launch_xsph(uint32_t n, uint32_t threads, uint32_t lanes, const StepConst& k, const StateBufs& s,
                 const ListBufs& l, double4* vel_out, cudaStream_t st, bool use_w) {
    if (!n) return;
    const bool w = use_w && l.wpair;
    if (lanes == 1) {
        if (w) k_xsph_w<<<blocks_for(n, threads), threads, 0, st>>>(n, k, s, l, vel_out);
        if (k.kernel == 0) k_xsph<true><<<blocks_for(n, threads), threads, 0, st>>>(n, k, s, l, vel_out, w);
        else k_xsph<false><<<blocks_for(n, threads), threads, 0, st>>>(n, k, s, l, vel_out, w);
        return;
    }
    with_lanes(lanes, [&](auto gc) {
        constexpr int G = decltype(gc)::value;
        const uint32_t b = blocks_for((uint64_t)n * G, threads);
        const size_t sm = sum_smem<G, 3>(threads);
        if (w) k_xsph_g<true, true, G><<<b, threads, sm, st>>>(n, k, s, l, vel_out, false);
        if (k.kernel == 0) k_xsph_g<true, false, G><<<b, threads, sm, st>>>(n, k, s, l, vel_out, w);
        else k_xsph_g<false, false, G><<<b, threads, sm, st>>>(n, k, s, l, vel_out, w);
    });
}

void launch_in_support_counts(uint32_t n, const StepConst& k, const StateBufs& s,
                              const ListBufs& l, uint32_t* out, cudaStream_t st) {
    if (n) k_in_support<<<blocks_for(n, 256), 256, 0, st>>>(n, k, s, l, out);
}

}  // namespace pe

// Single-precision form of the SPH passes.
//
// The neighbour-loop state is float4: cell-local positions (offset from the
// corner of the particle's own grid cell, w = p/rho^2 for fluid or psi for
// boundary samples) and velocities (w = rho). The vector between two
// particles is (key_j - key_i) * cell + (local_j - local_i), so positions keep
// ~1e-9 m resolution at any distance from the origin. Pair arithmetic is
// single precision with fast reciprocals; the density, force and XSPH sums are
// Kahan-compensated. The grid, its sort and the global v_max reduction stay
// f64 (the f64 position of a particle is key * cell + local, exact in f64, and
// re-expressed against the new cell after each sort). This form does not
// reproduce the reference's bits; `bench.py --form f32` reports its error
// against the f64 path.
#include <type_traits>

#include "lane_group.cuh"
#include "list_iter.cuh"
#include "pe_math.cuh"
#include "wcsph_device.cuh"

namespace pe {

namespace {


inline uint32_t blocks_for(uint64_t n, uint32_t t) { return (uint32_t)((n + t - 1) / t); }

struct Kahan {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float y = x - c;
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
    // add(a b), the product fused with the compensation
    __device__ __forceinline__ void add_product(float a, float b) {
        const float y = fmaf(a, b, -c);
        const float t = s + y;
        c = (t - s) - y;
        s = t;
    }
};

__device__ __forceinline__ float w_f32(float r, const F32Const& k) {
    const float q = r * k.inv_h;
    if (q >= 2.f) return 0.f;
    if (q < 1.f) return k.alpha * (1.f - 1.5f * q * q + 0.75f * q * q * q);
    const float t = 2.f - q;
    return k.alpha * 0.25f * t * t * t;
}

// dW/dr / r, the scale of grad W (0 outside the support and at r = 0)
__device__ __forceinline__ float dwdr_over_r_f32(float r, float inv_r, const F32Const& k) {
    const float q = r * k.inv_h;
    if (q >= 2.f || q <= 0.f) return 0.f;
    float dwdq;
    if (q < 1.f) {
        dwdq = k.alpha * (-3.f * q + 2.25f * q * q);
    } else {
        const float t = 2.f - q;
        dwdq = k.alpha * (-0.75f * t * t);
    }
    return dwdq * k.inv_h * inv_r;
}

// The pair vector x_j - x_i of two particles in the same or adjacent cells:
// their keys differ by -1, 0 or 1 per axis, which the keys mod 4 (cm, two
// bits per axis) determine, so a neighbour's full key need not be read.
__device__ __forceinline__ float3 rel(uint32_t ci, const float4& pi, uint32_t cj, const float4& pj,
                                      float cell) {
    const int dx = (int)(((cj & 3u) - (ci & 3u) + 1u) & 3u) - 1;
    const int dy = (int)((((cj >> 2) & 3u) - ((ci >> 2) & 3u) + 1u) & 3u) - 1;
    const int dz = (int)((((cj >> 4) & 3u) - ((ci >> 4) & 3u) + 1u) & 3u) - 1;
    return make_float3((float)dx * cell + (pj.x - pi.x), (float)dy * cell + (pj.y - pi.y),
                       (float)dz * cell + (pj.z - pi.z));
}

// particles.rs:126 boundary_sees_fluid for an oriented sample b seen from a
// fluid particle at d = x_b - x_f
__device__ __forceinline__ bool sees_fluid_f32(const F32Const& k, const double4& nb, float3 d) {
    const float nx = (float)nb.x, ny = (float)nb.y, nz = (float)nb.z;
    const float n2 = nx * nx + ny * ny + nz * nz;
    if (n2 <= 0.f) return true;
    const float eps = k.boundary_eps_h * sqrtf(n2);
    return -(d.x * nx + d.y * ny + d.z * nz) > -eps;
}

// A neighbour's loop state, gathered one entry ahead of its use.
struct Nb32 {
    float4 p;
    uint32_t km;  // cell key mod 4 (F32Bufs.kmod)
    float4 v;
};

__global__ void __launch_bounds__(kMaxPassThreads) k_density_f32(uint32_t n, F32Const k, StateBufs s,
                                                          F32Bufs f, ListBufs l) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (s.flags[i] & kFlagBoundary) {
        f.vel[i].w = k.rho0;
        return;
    }
    const float4 pi = f.pos[i];
    const uint32_t ci = f.kmod[i];
    Kahan rho;
    rho.add(k.rho_self);
    const ListRef vr = list_ref(l, i, kListVisit);
    // W of each entry kept for the XSPH pass, one 16-byte store per group of
    // four entries at the group's pool index (wrow walks the slot's rows)
    bool keep_w = false;
    if (l.wpair32) {
        keep_w = w_fits(l, vr);
        if (!keep_w) atomicOr(l.w_short, 1u);
    }
    float* wrow = keep_w ? l.wpair32 + (vr.p - l.pool) : nullptr;
    float w4[4] = {0.f, 0.f, 0.f, 0.f};
    for_each_row<2>(
        vr,
        [&](uint32_t e) {
            Nb32 b;
            b.p = f.pos[e & kEntrySlotMask];
            b.km = f.kmod[e & kEntrySlotMask];
            return b;
        },
        [](uint32_t) {},
        [&](uint32_t q, uint32_t e, const Nb32& b) {
            const float4 pj = b.p;
            const float3 d = rel(ci, pi, b.km, pj, k.cell);
            const float r = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
            const float w = w_f32(r, k);
            w4[q] = w;
            if ((e & kEntryOriented) && !sees_fluid_f32(k, s.nout[e & kEntrySlotMask], d)) return;
            rho.add(((e & kEntryBoundary) ? k.rho0 * pj.w : k.mass) * w);
        },
        [&](uint32_t) {
            if (keep_w) {
                *reinterpret_cast<float4*>(wrow) = make_float4(w4[0], w4[1], w4[2], w4[3]);
                wrow += vr.step;
            }
        });
    const float r = fmaxf(rho.s, 1e-12f);
    f.vel[i].w = r;
    s.vel[i].w = (double)r;
}

__global__ void k_vmax_f32(uint32_t n, Tanks tk, StateBufs s, F32Bufs f) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    double m = 0.0;
    uint32_t t = 0xffffffffu;
    if (i < n) {
        t = tk.slot_tank[i];
        if (!(s.flags[i] & kFlagBoundary)) {
            const float4 v = f.vel[i];
            const double q = (double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z;
            if (q > m) m = q;
        }
    }
    unsigned long long b = __double_as_longlong(m);
    const uint32_t t0 = __shfl_sync(0xffffffffu, t, 0);
    if (i >= n) t = t0;
    if (__all_sync(0xffffffffu, t == t0)) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long x = __shfl_xor_sync(0xffffffffu, b, o);
            b = x > b ? x : b;
        }
        if ((threadIdx.x & 31u) == 0 && b != 0ull && t0 != 0xffffffffu) atomicMax(&tk.vmax2[t0], b);
    } else if (b != 0ull && i < n) {
        atomicMax(&tk.vmax2[t], b);
    }
}

__global__ void k_pressure_f32(uint32_t n, F32Const k, Tanks tk, StateBufs s, F32Bufs f) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // f64 control of each tank's sound speed (wcsph.rs:158-169)
    const uint32_t t = tk.slot_tank[i];
    double c = tk.c[t];
    if (k.adapt_sound_speed) {
        const double vmax = sqrt(__longlong_as_double((long long)tk.vmax2[t]));
        const double min_c = 10.0 * fmax(vmax, 0.0);
        c = c < min_c ? min_c : c;
    }
    if (i == tk.desc[t].slot_begin) tk.c[t] = c;
    if (s.flags[i] & kFlagBoundary) {
        s.p[i] = 0.0;
        return;
    }
    const float rho = f.vel[i].w;
    const float x = rho * k.inv_eos_rho0;
    float pw;
    if (k.gamma7) {
        const float x2 = x * x, x4 = x2 * x2;
        pw = x4 * x2 * x;
    } else {
        pw = powf(x, k.eos_gamma);
    }
    const float b = (float)(k.eos_rho0 * c * c / k.eos_gamma_d);
    const float p = b * (pw - 1.f);
    s.p[i] = (double)p;
    f.pos[i].w = p / (rho * rho);
}

// One pair of the force pass seen from fluid i: d = x_j - x_i and the factor of
// d (fluid neighbour) or of d grad (boundary sample) in the acceleration.
struct PairF32 {
    float grad, scale;
    bool counts;
};

__device__ __forceinline__ PairF32 force_pair_f32(const F32Const& k, const StateBufs& s, float nac, uint32_t ci,
                                                  const float4& pi, const float4& vi, uint32_t e, const Nb32& b,
                                                  float3* d_out) {
    PairF32 t{0.f, 0.f, false};
    const float4 pj = b.p;
    const float3 d = rel(ci, pi, b.km, pj, k.cell);  // x_j - x_i
    *d_out = d;
    const float r2 = d.x * d.x + d.y * d.y + d.z * d.z;
    if (r2 < 1e-30f) return t;
    const float inv_r = rsqrtf(r2);
    const float r = r2 * inv_r;
    t.grad = -dwdr_over_r_f32(r, inv_r, k);  // grad_i W = d * grad
    if (e & kEntryBoundary) {
        if ((e & kEntryOriented) && !sees_fluid_f32(k, s.nout[e & kEntrySlotMask], d)) return t;
        t.scale = -(k.rho0 * pj.w) * pi.w;
        t.counts = true;
        return t;
    }
    const float4 vj = b.v;
    const float press = pi.w + pj.w;
    const float vr = (vi.x - vj.x) * -d.x + (vi.y - vj.y) * -d.y + (vi.z - vj.z) * -d.z;
    float pic = 0.f;
    if (vr < 0.f) {
        const float mu = k.h * vr / (r2 + k.eps_h2);
        pic = (nac * mu + k.visc_beta * mu * mu) * (2.f / (vi.w + vj.w));
    }
    t.scale = t.grad * -k.mass * (press + pic);
    t.counts = true;
    return t;
}

// Kick and drift of fluid slot i (symplectic Euler in cell-local single
// precision) from its pair sums.
template <int DIM>
__device__ __forceinline__ void integrate_f32(const F32Const& k, const StateBufs& s, uint32_t i, const float4& pi,
                                              const float4& vi, float ax, float ay, float az, float dt,
                                              double4* __restrict__ pos_next, double4* __restrict__ vel_next) {
    const int4 ki = s.key[i];
    const float a_x = ax + k.gx, a_y = ay + k.gy, a_z = az + k.gz;
    s.acc[i] = make_double4(a_x, a_y, a_z, 0.0);
    float vx = vi.x + a_x * dt, vy = vi.y + a_y * dt, vz = vi.z + a_z * dt;
    float lx = pi.x + vx * dt, ly = pi.y + vy * dt, lz = pi.z + vz * dt;
    if (DIM == 2) {
        lz = 0.f;
        vz = 0.f;
    }
    // f64 position for the grid: key * cell + local, one f64 rounding
    pos_next[i] = make_double4((double)ki.x * k.cell_d + (double)lx, (double)ki.y * k.cell_d + (double)ly,
                               DIM == 2 ? 0.0 : (double)ki.z * k.cell_d + (double)lz, s.pos[i].w);
    vel_next[i] = make_double4(vx, vy, vz, vi.w);
}

template <int DIM>
__global__ void __launch_bounds__(kMaxPassThreads) k_forces_f32(uint32_t n, F32Const k, Tanks tk,
                                                                StateBufs s, F32Bufs f, ListBufs l,
                                                                float dt, double4* __restrict__ pos_next,
                                                                double4* __restrict__ vel_next,
                                                                float* __restrict__ bf) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || (s.flags[i] & kFlagBoundary)) return;
    const float c0 = (float)tk.c[tk.slot_tank[i]];
    const float nac = -k.visc_alpha * c0;
    const float4 pi = f.pos[i];
    const float4 vi = f.vel[i];
    const int4 ki = s.key[i];
    const uint32_t ci = f.kmod[i];
    Kahan ax, ay, az;
    auto load = [&](uint32_t e) {
        Nb32 b;
        b.p = f.pos[e & kEntrySlotMask];
        b.km = f.kmod[e & kEntrySlotMask];
        b.v = f.vel[e & kEntrySlotMask];
        return b;
    };
    for_each_loaded(list_ref(l, i, kListVisit), load, [&](uint32_t e, const Nb32& b) {
        const uint32_t j = e & kEntrySlotMask;
        const float4 pj = b.p;
        const float3 d = rel(ci, pi, b.km, pj, k.cell);  // x_j - x_i
        const float r2 = d.x * d.x + d.y * d.y + d.z * d.z;
        if (r2 < 1e-30f) return;
        const float inv_r = rsqrtf(r2);
        const float r = r2 * inv_r;
        const float sc_ = -dwdr_over_r_f32(r, inv_r, k);  // grad_i W = d * sc_
        if (e & kEntryBoundary) {
            if ((e & kEntryOriented) && !sees_fluid_f32(k, s.nout[j], d)) return;
            const float m = -(k.rho0 * pj.w) * pi.w;
            const float fx = d.x * sc_ * m, fy = d.y * sc_ * m, fz = d.z * sc_ * m;
            ax.add(fx);
            ay.add(fy);
            az.add(fz);
            if (bf) {
                atomicAdd(&bf[4 * (size_t)j], fx * -k.mass);
                atomicAdd(&bf[4 * (size_t)j + 1], fy * -k.mass);
                atomicAdd(&bf[4 * (size_t)j + 2], fz * -k.mass);
            }
            return;
        }
        const float4 vj = b.v;
        const float press = pi.w + pj.w;
        const float vr = (vi.x - vj.x) * -d.x + (vi.y - vj.y) * -d.y + (vi.z - vj.z) * -d.z;
        float pic = 0.f;
        if (vr < 0.f) {
            const float mu = k.h * vr / (r2 + k.eps_h2);
            pic = (nac * mu + k.visc_beta * mu * mu) * (2.f / (vi.w + vj.w));
        }
        const float s_ = sc_ * -k.mass * (press + pic);
        ax.add(d.x * s_);
        ay.add(d.y * s_);
        az.add(d.z * s_);
    });
    const float a_x = ax.s + k.gx, a_y = ay.s + k.gy, a_z = az.s + k.gz;
    s.acc[i] = make_double4(a_x, a_y, a_z, 0.0);
    // symplectic Euler in cell-local single precision
    float vx = vi.x + a_x * dt, vy = vi.y + a_y * dt, vz = vi.z + a_z * dt;
    float lx = pi.x + vx * dt, ly = pi.y + vy * dt, lz = pi.z + vz * dt;
    if (DIM == 2) {
        lz = 0.f;
        vz = 0.f;
    }
    // f64 position for the grid: key * cell + local, one f64 rounding
    pos_next[i] = make_double4((double)ki.x * k.cell_d + (double)lx, (double)ki.y * k.cell_d + (double)ly,
                               DIM == 2 ? 0.0 : (double)ki.z * k.cell_d + (double)lz, s.pos[i].w);
    vel_next[i] = make_double4(vx, vy, vz, vi.w);
}

// short_only: run only if the density pass met a list beyond the pair-weight
// buffer (the launch that follows k_xsph_f32_w, which then did nothing).
__global__ void __launch_bounds__(kMaxPassThreads) k_xsph_f32(uint32_t n, F32Const k, StateBufs s, F32Bufs f,
                                                       ListBufs l, float4* __restrict__ vel_out,
                                                       bool short_only) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (short_only && !__ldg(l.w_short)) return;
    const float4 vi = f.vel[i];
    if (s.flags[i] & kFlagBoundary) {
        vel_out[i] = vi;
        return;
    }
    const float4 pi = f.pos[i];
    const uint32_t ci = f.kmod[i];
    Kahan dx, dy, dz;
    auto load = [&](uint32_t e) {
        Nb32 b{};
        if (!(e & kEntryBoundary)) {
            b.p = f.pos[e & kEntrySlotMask];
            b.km = f.kmod[e & kEntrySlotMask];
            b.v = f.vel[e & kEntrySlotMask];
        }
        return b;
    };
    for_each_loaded(list_ref(l, i, kListVisit), load, [&](uint32_t e, const Nb32& b) {
        if (e & kEntryBoundary) return;
        const float4 pj = b.p;
        const float3 d = rel(ci, pi, b.km, pj, k.cell);
        const float r = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
        const float w = w_f32(r, k);
        const float4 vj = b.v;
        const float g = k.mass * 2.f / (vi.w + vj.w) * w;
        dx.add((vj.x - vi.x) * g);
        dy.add((vj.y - vi.y) * g);
        dz.add((vj.z - vi.z) * g);
    });
    const float4 vn = make_float4(vi.x + dx.s * k.xsph_eps, vi.y + dy.s * k.xsph_eps,
                                  vi.z + dz.s * k.xsph_eps, vi.w);
    vel_out[i] = vn;
    s.vel[i] = make_double4(vn.x, vn.y, vn.z, vn.w);
}

// k_xsph_f32 with each pair's W read from the density pass of the same lists
// and positions instead of recomputed: the neighbour's velocity is the only
// gather (16 bytes in place of 48).
__global__ void __launch_bounds__(kMaxPassThreads) k_xsph_f32_w(uint32_t n, F32Const k, StateBufs s, F32Bufs f,
                                                         ListBufs l, float4* __restrict__ vel_out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (__ldg(l.w_short)) return;  // k_xsph_f32 runs instead
    const float4 vi = f.vel[i];
    if (s.flags[i] & kFlagBoundary) {
        vel_out[i] = vi;
        return;
    }
    Kahan dx, dy, dz;
    const ListRef vr = list_ref(l, i, kListVisit);
    const float* wrow = l.wpair32 + (vr.p - l.pool);
    float4 w4 = make_float4(0.f, 0.f, 0.f, 0.f);
    for_each_row<1>(
        vr, [&](uint32_t e) { return f.vel[e & kEntrySlotMask]; },
        [&](uint32_t) {
            w4 = __ldg(reinterpret_cast<const float4*>(wrow));
            wrow += vr.step;
        },
        [&](uint32_t q, uint32_t e, const float4& vj) {
            if (e & kEntryBoundary) return;
            const float w = q == 0 ? w4.x : q == 1 ? w4.y : q == 2 ? w4.z : w4.w;
            const float g = k.mass * 2.f / (vi.w + vj.w) * w;
            dx.add((vj.x - vi.x) * g);
            dy.add((vj.y - vi.y) * g);
            dz.add((vj.z - vi.z) * g);
        },
        [](uint32_t) {});
    const float4 vn = make_float4(vi.x + dx.s * k.xsph_eps, vi.y + dy.s * k.xsph_eps,
                                  vi.z + dz.s * k.xsph_eps, vi.w);
    vel_out[i] = vn;
    s.vel[i] = make_double4(vn.x, vn.y, vn.z, vn.w);
}

// ---------------------------------------------------------------------------
// The passes with G lanes a slot (lane_group.cuh), while the slots do not fill
// the chip. A compensated sum is no sum of rounded terms: the product that makes
// a term is fused with the subtraction of the compensation, and a skipped entry
// is not an added zero (a zero added can move a tie). So the lanes exchange the
// two factors of each term and which entries count, and the sums come out bit
// for bit as one thread's.
// ---------------------------------------------------------------------------
template <int G, int K>
struct OrderedKahan {
    static constexpr uint32_t kPitch = G + 4u;  // floats between a group's components
    static constexpr uint32_t kBuf = (32u / G) * (K + 1) * kPitch;
    static constexpr uint32_t kFloats = 2u * kBuf;  // per warp
    Kahan sum;
    float *put, *get_a, *get_b;
    uint32_t flip;
    bool adds;
    __device__ __forceinline__ OrderedKahan(float* warp_words, const LaneGroup<G>& g, float start) : flip(0u) {
        float* const base = warp_words + g.grp * (K + 1) * kPitch;
        sum.s = start;
        put = base + g.sub;
        get_a = base + min(g.sub, (uint32_t)K - 1u) * kPitch;
        get_b = base + K * kPitch;
        adds = g.sub < (uint32_t)K;
    }
    // Adds a[k] b of this round's entries with `counts` to sum k, in lane order.
    __device__ __forceinline__ void add(const LaneGroup<G>& g, const float (&a)[K], float b, bool counts) {
#pragma unroll
        for (int k = 0; k < K; ++k) put[flip + k * kPitch] = a[k];
        put[flip + K * kPitch] = b;
        const uint32_t m = g.bits(__ballot_sync(kFullWarp, counts));
        __syncwarp();
        if (adds) {
#pragma unroll
            for (int j = 0; j < G / 4; ++j) {
                const float4 va = *reinterpret_cast<const float4*>(get_a + flip + 4 * j);
                const float4 vb = *reinterpret_cast<const float4*>(get_b + flip + 4 * j);
                const float x[4] = {va.x, va.y, va.z, va.w}, y[4] = {vb.x, vb.y, vb.z, vb.w};
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (m & (1u << (4 * j + q))) sum.add_product(x[q], y[q]);
            }
        }
        flip = kBuf - flip;
    }
    // Sum k, on each lane of the group. Every lane of the warp calls it.
    __device__ __forceinline__ float total(int k) const { return __shfl_sync(kFullWarp, sum.s, k, G); }
};

template <int G>
__global__ void __launch_bounds__(kMaxPassThreads) k_density_f32_g(uint32_t n, F32Const k, StateBufs s, F32Bufs f,
                                                                   ListBufs l) {
    extern __shared__ __align__(16) float s_floats[];
    const LaneGroup<G> g;
    const uint32_t i = g.slot;
    const bool fluid = i < n && !(s.flags[i] & kFlagBoundary);
    if (i < n && !fluid && g.sub == 0) f.vel[i].w = k.rho0;
    if (!__any_sync(kFullWarp, fluid)) return;
    ListRef vr{l.pool, 0u, 0u};
    float4 pi = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t ci = 0;
    bool keep_w = false;
    if (fluid) {
        vr = list_ref(l, i, kListVisit);
        pi = f.pos[i];
        ci = f.kmod[i];
        if (l.wpair32) {
            keep_w = w_fits(l, vr);
            if (!keep_w && g.sub == 0) atomicOr(l.w_short, 1u);
        }
    }
    OrderedKahan<G, 1> rho(s_floats + g.warp * OrderedKahan<G, 1>::kFloats, g, k.rho_self);
    group_for_each<G>(
        vr, g,
        [&](uint32_t e, const uint32_t*) {
            Nb32 b;
            b.p = f.pos[e & kEntrySlotMask];
            b.km = f.kmod[e & kEntrySlotMask];
            return b;
        },
        [&](bool has, uint32_t e, const Nb32& b, const uint32_t* p) {
            const float3 d = rel(ci, pi, b.km, b.p, k.cell);
            const float r = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
            const float w = w_f32(r, k);
            if (has && keep_w) l.wpair32[p - l.pool] = w;
            const bool counts =
                has && !((e & kEntryOriented) && !sees_fluid_f32(k, s.nout[e & kEntrySlotMask], d));
            const float m[1] = {(e & kEntryBoundary) ? k.rho0 * b.p.w : k.mass};
            rho.add(g, m, w, counts);
        });
    if (fluid && g.sub == 0) {
        const float r = fmaxf(rho.sum.s, 1e-12f);
        f.vel[i].w = r;
        s.vel[i].w = (double)r;
    }
}

template <int DIM, int G>
__global__ void __launch_bounds__(kMaxPassThreads) k_forces_f32_g(uint32_t n, F32Const k, Tanks tk, StateBufs s,
                                                                  F32Bufs f, ListBufs l, float dt,
                                                                  double4* __restrict__ pos_next,
                                                                  double4* __restrict__ vel_next,
                                                                  float* __restrict__ bf) {
    extern __shared__ __align__(16) float s_floats[];
    const LaneGroup<G> g;
    const uint32_t i = g.slot;
    const bool fluid = i < n && !(s.flags[i] & kFlagBoundary);
    if (!__any_sync(kFullWarp, fluid)) return;
    ListRef vr{l.pool, 0u, 0u};
    float4 pi = make_float4(0.f, 0.f, 0.f, 0.f), vi = make_float4(0.f, 0.f, 0.f, 1.f);
    uint32_t ci = 0;
    float nac = 0.f;
    if (fluid) {
        vr = list_ref(l, i, kListVisit);
        pi = f.pos[i];
        vi = f.vel[i];
        ci = f.kmod[i];
        const float c0 = (float)tk.c[tk.slot_tank[i]];
        nac = -k.visc_alpha * c0;
    }
    OrderedKahan<G, 3> acc(s_floats + g.warp * OrderedKahan<G, 3>::kFloats, g, 0.f);
    group_for_each<G>(
        vr, g,
        [&](uint32_t e, const uint32_t*) {
            Nb32 b;
            b.p = f.pos[e & kEntrySlotMask];
            b.km = f.kmod[e & kEntrySlotMask];
            b.v = f.vel[e & kEntrySlotMask];
            return b;
        },
        [&](bool has, uint32_t e, const Nb32& b, const uint32_t*) {
            float a[3] = {0.f, 0.f, 0.f}, m = 0.f;
            bool counts = false;
            if (has) {
                float3 d;
                const PairF32 t = force_pair_f32(k, s, nac, ci, pi, vi, e, b, &d);
                counts = t.counts;
                if (counts) {
                    a[0] = d.x;
                    a[1] = d.y;
                    a[2] = d.z;
                    m = t.scale;
                    if (e & kEntryBoundary) {  // the rounded force is the term
                        a[0] = d.x * t.grad * m;
                        a[1] = d.y * t.grad * m;
                        a[2] = d.z * t.grad * m;
                        m = 1.f;
                        if (bf) {
                            const size_t j = 4 * (size_t)(e & kEntrySlotMask);
                            atomicAdd(&bf[j], a[0] * -k.mass);
                            atomicAdd(&bf[j + 1], a[1] * -k.mass);
                            atomicAdd(&bf[j + 2], a[2] * -k.mass);
                        }
                    }
                }
            }
            acc.add(g, a, m, counts);
        });
    const float ax = acc.total(0), ay = acc.total(1), az = acc.total(2);
    if (fluid && g.sub == 0)
        integrate_f32<DIM>(k, s, i, pi, vi, ax, ay, az, dt, pos_next, vel_next);
}

// USE_W: each pair's W read from the density pass (k_xsph_f32_w), otherwise
// recomputed (k_xsph_f32, short_only as there).
template <bool USE_W, int G>
__global__ void __launch_bounds__(kMaxPassThreads) k_xsph_f32_g(uint32_t n, F32Const k, StateBufs s, F32Bufs f,
                                                                ListBufs l, float4* __restrict__ vel_out,
                                                                bool short_only) {
    extern __shared__ __align__(16) float s_floats[];
    if (USE_W ? __ldg(l.w_short) != 0u : short_only && !__ldg(l.w_short)) return;
    const LaneGroup<G> g;
    const uint32_t i = g.slot;
    const bool fluid = i < n && !(s.flags[i] & kFlagBoundary);
    if (i < n && !fluid && g.sub == 0) vel_out[i] = f.vel[i];
    if (!__any_sync(kFullWarp, fluid)) return;
    ListRef vr{l.pool, 0u, 0u};
    float4 vi = make_float4(0.f, 0.f, 0.f, 1.f), pi = vi;
    uint32_t ci = 0;
    if (fluid) {
        vr = list_ref(l, i, kListVisit);
        vi = f.vel[i];
        if (!USE_W) {
            pi = f.pos[i];
            ci = f.kmod[i];
        }
    }
    struct VelW {
        float4 v, p;
        uint32_t km;
        float w;
    };
    OrderedKahan<G, 3> dv(s_floats + g.warp * OrderedKahan<G, 3>::kFloats, g, 0.f);
    group_for_each<G>(
        vr, g,
        [&](uint32_t e, const uint32_t* p) {
            VelW b{};
            const uint32_t j = e & kEntrySlotMask;
            b.v = f.vel[j];
            if (USE_W) {
                b.w = __ldg(l.wpair32 + (p - l.pool));
            } else {
                b.p = f.pos[j];
                b.km = f.kmod[j];
            }
            return b;
        },
        [&](bool has, uint32_t e, const VelW& b, const uint32_t*) {
            float w = b.w;
            if (!USE_W) {
                const float3 d = rel(ci, pi, b.km, b.p, k.cell);
                w = w_f32(sqrtf(d.x * d.x + d.y * d.y + d.z * d.z), k);
            }
            const float m = k.mass * 2.f / (vi.w + b.v.w) * w;
            const float a[3] = {b.v.x - vi.x, b.v.y - vi.y, b.v.z - vi.z};
            dv.add(g, a, m, has && !(e & kEntryBoundary));
        });
    const float dx = dv.total(0), dy = dv.total(1), dz = dv.total(2);
    if (fluid && g.sub == 0) {
        const float4 vn = make_float4(vi.x + dx * k.xsph_eps, vi.y + dy * k.xsph_eps, vi.z + dz * k.xsph_eps, vi.w);
        vel_out[i] = vn;
        s.vel[i] = make_double4(vn.x, vn.y, vn.z, vn.w);
    }
}

// Cell-local single-precision state from the (sorted) f64 state.
__global__ void k_f32_from_f64(uint32_t n, double cell, StateBufs s, F32Bufs f) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double4 p = s.pos[i];
    const int4 kk = s.key[i];
    const bool fluid = !(s.flags[i] & kFlagBoundary);
    f.pos[i] = make_float4((float)(p.x - (double)kk.x * cell), (float)(p.y - (double)kk.y * cell),
                           (float)(p.z - (double)kk.z * cell), fluid ? 0.f : (float)p.w);
    f.kmod[i] = (uint8_t)(((uint32_t)kk.x & 3u) | (((uint32_t)kk.y & 3u) << 2) | (((uint32_t)kk.z & 3u) << 4));
    const double4 v = s.vel[i];
    f.vel[i] = make_float4((float)v.x, (float)v.y, (float)v.z, (float)v.w);
}

__global__ void k_bf_to_f64(uint32_t n, const float* __restrict__ bf, StateBufs s) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    s.bf[i] = make_double4(bf[4 * (size_t)i], bf[4 * (size_t)i + 1], bf[4 * (size_t)i + 2], 0.0);
}

}  // namespace

template <class F>
static void with_f32_lanes(uint32_t lanes, F&& f) {
    if (lanes == 8) f(std::integral_constant<int, 8>{});
    else f(std::integral_constant<int, 32>{});
}

template <int G, int K>
static size_t kahan_smem(uint32_t threads) {
    return (size_t)(threads / 32u) * OrderedKahan<G, K>::kFloats * sizeof(float);
}

void launch_f32_from_f64(uint32_t n, double cell, const StateBufs& s, const F32Bufs& f,
                         cudaStream_t st) {
    if (n) k_f32_from_f64<<<blocks_for(n, 256), 256, 0, st>>>(n, cell, s, f);
}

void launch_density_f32(uint32_t n, uint32_t threads, uint32_t lanes, const F32Const& k, const StateBufs& s,
                        const F32Bufs& f, const ListBufs& l, cudaStream_t st) {
    if (!n) return;
    if (lanes == 1) {
        k_density_f32<<<blocks_for(n, threads), threads, 0, st>>>(n, k, s, f, l);
        return;
    }
    with_f32_lanes(lanes, [&](auto gc) {
        constexpr int G = decltype(gc)::value;
        k_density_f32_g<G><<<blocks_for((uint64_t)n * G, threads), threads, kahan_smem<G, 1>(threads), st>>>(n, k, s, f, l);
    });
}

void launch_pressure_f32(uint32_t n, const F32Const& k, const Tanks& tk, const StateBufs& s,
                         const F32Bufs& f, cudaStream_t st) {
    if (!n) return;
    if (k.adapt_sound_speed) k_vmax_f32<<<blocks_for(n, 256), 256, 0, st>>>(n, tk, s, f);
    k_pressure_f32<<<blocks_for(n, 256), 256, 0, st>>>(n, k, tk, s, f);
}

void launch_forces_f32(uint32_t n, uint32_t threads, uint32_t lanes, const F32Const& k, const Tanks& tk,
                       const StateBufs& s, const F32Bufs& f, const ListBufs& l, float dt,
                       double4* pos_next, double4* vel_next, float* bf, cudaStream_t st) {
    if (!n) return;
    if (bf) cudaMemsetAsync(bf, 0, sizeof(float) * 4 * (size_t)n, st);
    const uint32_t b = blocks_for(n, threads);
    if (lanes != 1) {
        with_f32_lanes(lanes, [&](auto gc) {
            constexpr int G = decltype(gc)::value;
            const uint32_t bg = blocks_for((uint64_t)n * G, threads);
            const size_t sm = kahan_smem<G, 3>(threads);
            if (k.dim == 3) k_forces_f32_g<3, G><<<bg, threads, sm, st>>>(n, k, tk, s, f, l, dt, pos_next, vel_next, bf);
            else k_forces_f32_g<2, G><<<bg, threads, sm, st>>>(n, k, tk, s, f, l, dt, pos_next, vel_next, bf);
        });
    } else if (k.dim == 3)
        k_forces_f32<3><<<b, threads, 0, st>>>(n, k, tk, s, f, l, dt, pos_next, vel_next, bf);
    else
        k_forces_f32<2><<<b, threads, 0, st>>>(n, k, tk, s, f, l, dt, pos_next, vel_next, bf);
    if (bf) k_bf_to_f64<<<blocks_for(n, 256), 256, 0, st>>>(n, bf, s);
}

void launch_xsph_f32(uint32_t n, uint32_t threads, uint32_t lanes, const F32Const& k, const StateBufs& s,
                     const F32Bufs& f, const ListBufs& l, float4* vel_out, cudaStream_t st,
                     bool use_w) {
    if (!n) return;
    const bool w = use_w && l.wpair32;
    if (lanes != 1) {
        with_f32_lanes(lanes, [&](auto gc) {
            constexpr int G = decltype(gc)::value;
            const uint32_t b = blocks_for((uint64_t)n * G, threads);
            const size_t sm = kahan_smem<G, 3>(threads);
            if (w) k_xsph_f32_g<true, G><<<b, threads, sm, st>>>(n, k, s, f, l, vel_out, false);
            k_xsph_f32_g<false, G><<<b, threads, sm, st>>>(n, k, s, f, l, vel_out, w);
        });
        return;
    }
    if (w) k_xsph_f32_w<<<blocks_for(n, threads), threads, 0, st>>>(n, k, s, f, l, vel_out);
    k_xsph_f32<<<blocks_for(n, threads), threads, 0, st>>>(n, k, s, f, l, vel_out, w);
}

}  // namespace pe

// Neighbour-list build: CTAs per occupied cell.
//
// Replaces the per-particle `UniformGrid::neighbours` gathers
// (crates/pe-fluid/src/grid.rs:122-140) that the reference repeats six times
// per fluid particle per step. The 27 (3-D) or 9 (2-D) neighbour cells of a
// CTA's cell are visited in the reference's (dz, dy, dx) order; their
// particles (each cell's run already in ascending original index) are staged
// in shared memory as half-precision features, and every particle of the
// centre cell filters the staged union with a conservative squared-distance
// bound that exceeds the support's by far more than the features' rounding
// (see Features), so every pair with q = r/h < 2 is kept. Extra borderline
// candidates are harmless: the f64 passes evaluate q exactly and such pairs
// contribute an exact +-0.
//
// k_nlist_both writes, for fluid particles, the "visit" list (in-support
// candidates, self excluded, in visiting order, each flagged boundary /
// oriented / lower; the force pass reads its unflagged entries as the
// reference's j > i and boundary pairs) and the "lower" list: for fluid
// particles the fluid neighbours with a smaller original index, for boundary
// particles all fluid neighbours, both in ascending original index; the order
// comes from a shared-memory radix sort (9-bit digits) of the union's fluid
// entries per cell. k_nlist_visit writes the visit list alone (the passes that need no
// ascending-index order).
//
// The kernels work on chunks of up to 32 (or 64) centre particles with eight
// (or four) threads per particle; the fused kernel is compiled for three
// resident CTAs per SM (80 registers), which the 32-centre tile's shared
// memory allows. Each warp computes the in-support bit masks of 32 centres
// over its share of the union words on the tensor cores (word_masks); the
// chunk's longest list sizes one block of the list pool, reserved with one
// atomic add; then the entries are written, each thread an equal share of its
// particle's list (a share of the words would leave most of the kept
// candidates, which lie in the middle words, to two threads). While a thread
// walks its kept candidates it sets the bits of the lower ones in a second
// mask over the sorted positions, from which the lower list is written.
//
// A union with positions far from its cell is staged as f32 offsets there too.
//
// k_nlist_visit stages f32 offsets and tests them in packed f32 arithmetic: its
// lists feed the single-precision form, whose compensated sums notice a
// candidate more (a zero added moves a tie). k_nlist_near makes PBF's.
//
// k_nlist_both is bound by instruction issue and barriers (529M warp instructions for 262,144 fluid
// particles, IPC 2.4, with scalar distance tests and a lower mask read through
// every sorted position; 391M as it is). At 1M 3.51 -> 2.43 ms, by parts: the
// visit entries 0.75, radix sort 0.41, lower entries 0.28, staging 0.17, masks
// 0.14 ms, barriers and the rest 0.7.
#include <algorithm>
#include <climits>
#include <cmath>
#include <limits>

#include <cuda_fp16.h>

#include "list_iter.cuh"
#include "pe_math.cuh"
#include "wcsph_device.cuh"

namespace pe {

namespace {

constexpr int kNlThreads = 256;
// Centre particles per chunk (a launch shape the world's autotuner picks:
// 32, the world's default, or 64); kNlThreads / chunk threads work on each
// centre particle. kDefaultChunk is what an unknown value falls back to.
constexpr uint32_t kDefaultChunk = 64;
constexpr uint32_t kWarps = kNlThreads / 32;
// Largest stage: the fused kernel's dynamic bytes per staged entry at the
// 32-centre tile (features 16, slot 4, sort index 2, rank 2, masks 8) and
// ~2.4 KB of static shared memory must fit the 227 KB a CTA can opt in to on
// sm_100 (232,448 bytes). The 64-centre tile's masks take 16; a stage too large
// for it takes the 32-centre one.
constexpr uint32_t kMaxUnionStage = 5888;
constexpr size_t kMaxDynamicBytes = 232448u - 4096u;
static_assert(32u * kMaxUnionStage + kMaxUnionStage / 8u <= kMaxDynamicBytes,
              "list stage exceeds the shared-memory limit");
constexpr uint32_t kStageStep = 256;               // stage capacities are multiples of this

// Staged word w of a union entry: original index (29 bits) | kind flags.
constexpr uint32_t kStageBoundary = 1u << 31;
constexpr uint32_t kStageOriented = 1u << 30;
constexpr uint32_t kStageOrigMask = (1u << 29) - 1u;

template <int NC>
__device__ __forceinline__ uint32_t slot_of_union(const uint32_t* s_off, const uint32_t* s_cstart,
                                                  uint32_t u) {
    int lo = 0, hi = NC - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (s_off[mid] <= u) lo = mid;
        else hi = mid - 1;
    }
    return s_cstart[lo] + (u - s_off[lo]);
}

__device__ __forceinline__ uint32_t entry_flags(uint32_t w) {
    return ((w & kStageBoundary) ? kEntryBoundary : 0u) | ((w & kStageOriented) ? kEntryOriented : 0u);
}

// Block-wide exclusive scan (kNlThreads threads).
__device__ __forceinline__ void block_exclusive_scan(uint32_t v, uint32_t* ex, uint32_t* total) {
    __shared__ uint32_t warp_sums[kWarps];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)lane >= o) incl += x;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    uint32_t before = 0, tot = 0;
#pragma unroll
    for (uint32_t w = 0; w < kWarps; ++w) {
        if (w < warp) before += warp_sums[w];
        tot += warp_sums[w];
    }
    *ex = before + incl - v;
    *total = tot;
    __syncthreads();
}

__device__ __forceinline__ uint32_t warp_max(uint32_t v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

struct CellUnion {
    uint32_t U, cs, ncenter, center_off;
    double ox, oy, oz;
};

// Ranges of the NC neighbour cells of global dense cell c, in visiting order;
// neighbours are taken inside the box of c's tank.
template <int DIM>
__device__ __forceinline__ CellUnion cell_union(const GridDesc& g, const Tanks& tk, uint32_t c,
                                                const uint32_t* __restrict__ cell_start,
                                                uint32_t* s_cstart, uint32_t* s_off) {
    constexpr int NC = DIM == 3 ? 27 : 9;
    constexpr int CENTER = DIM == 3 ? 13 : 4;
    const uint32_t tid = threadIdx.x;
    const TankDesc td = tk.desc[tk.cell_tank[c]];
    const uint32_t lc = c - td.cell_base;
    const int cz = (int)(lc % (uint32_t)td.nz);
    const int cy = (int)((lc / (uint32_t)td.nz) % (uint32_t)td.ny);
    const int cx = (int)(lc / ((uint32_t)td.nz * (uint32_t)td.ny));
    if (tid < 32) {
        uint32_t st = 0, cnt = 0;
        if ((int)tid < NC) {
            int dz = DIM == 3 ? (int)tid / 9 - 1 : 0;
            int dy = DIM == 3 ? ((int)tid / 3) % 3 - 1 : (int)tid / 3 - 1;
            int dx = (int)tid % 3 - 1;
            int qx = cx + dx, qy = cy + dy, qz = cz + dz;
            if (qx >= 0 && qy >= 0 && qz >= 0 && qx < td.nx && qy < td.ny && qz < td.nz) {
                uint32_t nc = td.cell_base +
                              ((uint32_t)qx * (uint32_t)td.ny + (uint32_t)qy) * (uint32_t)td.nz + (uint32_t)qz;
                st = cell_start[nc];
                cnt = cell_start[nc + 1] - st;
            }
        }
        uint32_t incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)tid >= o) incl += x;
        }
        if ((int)tid < NC) {
            s_cstart[tid] = st;
            s_off[tid + 1] = incl;
        }
        if (tid == 0) s_off[0] = 0;
    }
    __syncthreads();
    CellUnion cu;
    cu.U = s_off[NC];
    cu.cs = s_cstart[CENTER];
    cu.ncenter = s_off[CENTER + 1] - s_off[CENTER];
    cu.center_off = s_off[CENTER];
    cu.ox = (double)(td.kx0 + cx) * g.cell_size;
    cu.oy = (double)(td.ky0 + cy) * g.cell_size;
    cu.oz = DIM == 3 ? (double)(td.kz0 + cz) * g.cell_size : 0.0;
    return cu;
}

template <int DIM>
__device__ __forceinline__ float4 stage_entry(const StateBufs& s, uint32_t slot, const CellUnion& cu,
                                              uint8_t* fl_out, uint32_t* orig_out) {
    const double4 p = s.pos[slot];
    const uint8_t fl = s.flags[slot];
    const uint32_t o = s.orig[slot];
    const uint32_t w = o | ((fl & kFlagBoundary) ? kStageBoundary : 0u) |
                       ((fl & kFlagOriented) ? kStageOriented : 0u);
    *fl_out = fl;
    *orig_out = o;
    return make_float4((float)(p.x - cu.ox), (float)(p.y - cu.oy),
                       DIM == 3 ? (float)(p.z - cu.oz) : 0.0f, __uint_as_float(w));
}

__device__ __forceinline__ bool within(const float4& q, const float4& me, float r2f) {
    const float dx = q.x - me.x, dy = q.y - me.y, dz = q.z - me.z;
    return dx * dx + dy * dy + dz * dz <= r2f;
}

// in-support, or a boundary candidate kept whatever its distance
__device__ __forceinline__ bool keep_entry(const float4& q, const float4& me, float r2f, int keep_boundary) {
    return within(q, me, r2f) || (keep_boundary && (__float_as_uint(q.w) & kStageBoundary));
}

// ---- the visit kernel's stage and test ----

// The staged union in shared memory as four float arrays (cell-local x, y, z
// and the staged word orig | kind flags), so that the candidates of a word can
// be read four at a time per coordinate.
struct Stage {
    float *x, *y, *z, *w;
    __device__ __forceinline__ Stage(float* base, uint32_t ucap)
        : x(base), y(base + ucap), z(base + 2 * ucap), w(base + 3 * ucap) {}
    __device__ __forceinline__ float4 get(uint32_t u) const { return make_float4(x[u], y[u], z[u], w[u]); }
    __device__ __forceinline__ void put(uint32_t u, const float4& p) {
        x[u] = p.x;
        y[u] = p.y;
        z[u] = p.z;
        w[u] = p.w;
    }
};

// Packed single-precision pairs (two f32 in one 64-bit register) and the
// sm_100 paired arithmetic on them, each half rounded to nearest like the
// scalar instruction.
__device__ __forceinline__ unsigned long long f2_pack(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(unsigned long long v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long f2_sub(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long f2_mul(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b,
                                                     unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Keep mask of the 32 staged entries from position base (keep_entry per bit):
// four candidates per 16-byte read of each coordinate, their squared
// distances in two packed pairs (dx dx + dy dy + dz dz, as the scalar test).
template <bool KEEP_BOUNDARY>
__device__ __forceinline__ uint32_t word_mask(const Stage& st, uint32_t base, const float4& me, float r2f) {
    const unsigned long long mx = f2_pack(me.x, me.x), my = f2_pack(me.y, me.y), mz = f2_pack(me.z, me.z);
    uint32_t m = 0;
#pragma unroll
    for (int g = 0; g < 8; ++g) {
        const float4 X = *reinterpret_cast<const float4*>(st.x + base + 4 * g);
        const float4 Y = *reinterpret_cast<const float4*>(st.y + base + 4 * g);
        const float4 Z = *reinterpret_cast<const float4*>(st.z + base + 4 * g);
        const unsigned long long dx0 = f2_sub(f2_pack(X.x, X.y), mx), dx1 = f2_sub(f2_pack(X.z, X.w), mx);
        const unsigned long long dy0 = f2_sub(f2_pack(Y.x, Y.y), my), dy1 = f2_sub(f2_pack(Y.z, Y.w), my);
        const unsigned long long dz0 = f2_sub(f2_pack(Z.x, Z.y), mz), dz1 = f2_sub(f2_pack(Z.z, Z.w), mz);
        const unsigned long long r0 = f2_fma(dz0, dz0, f2_fma(dy0, dy0, f2_mul(dx0, dx0)));
        const unsigned long long r1 = f2_fma(dz1, dz1, f2_fma(dy1, dy1, f2_mul(dx1, dx1)));
        float a, b, c, d;
        f2_unpack(r0, a, b);
        f2_unpack(r1, c, d);
        uint32_t k4 = (a <= r2f ? 1u : 0u) | (b <= r2f ? 2u : 0u) | (c <= r2f ? 4u : 0u) | (d <= r2f ? 8u : 0u);
        if (KEEP_BOUNDARY) {
            const float4 W = *reinterpret_cast<const float4*>(st.w + base + 4 * g);
            k4 |= ((__float_as_uint(W.x) >> 31) & 1u) | (((__float_as_uint(W.y) >> 31) & 1u) << 1) |
                  (((__float_as_uint(W.z) >> 31) & 1u) << 2) | (((__float_as_uint(W.w) >> 31) & 1u) << 3);
        }
        m |= k4 << (4 * g);
    }
    return m;
}

// ---- the fused kernel's stage and test ----

// Features of a staged candidate: eight halves (x, y, z, nh, nl, 1, 1, 0) with
// (x, y, z) its offset from the middle of the centre cell in units of the cell,
// rounded to half, and nh + nl the squared length of the rounded offset. With a
// centre's row (-2x, -2y, -2z, 1, 1, ah, al, 0),
// ah + al = its own squared length minus the bound, the product of the two is
// |xi - xj|^2 - bound, exact but for the splits (2^-20) and the f32 sum: the
// sign bit is the test, and one m16n8k8 tensor instruction makes 128 of them.
//
// The bound: the rounding error of an offset below kFeatureReach cells is at most
// 2^-11 a component, so a pair's distance is off by at most 2 sqrt(3) 2^-11 =
// 0.0017 cells, and a pair within the support (one cell) has a rounded squared
// distance of at most 1.0034. The filter keeps ~0.5 % more candidates than the
// support holds. Positions of the grid the cells were built from are within 1.5
// cells; those the host has set since, or of a particle outside the domain, may be
// any number away, and a union that holds one is staged as f32 offsets instead
// (wide_masks).
constexpr float kBound2 = 1.0036f;
constexpr float kFeatureReach = 2.0f;
constexpr float kLargestFloat = 3.402823466e38f;

struct Features {
    __half2 xy, zn, m1, one;
};
static_assert(sizeof(Features) == 16, "one 16-byte store a candidate");

// The largest magnitudes of the rounded offsets seen: (x, y) and (z, unused).
struct Reach {
    __half2 xy, z;
    __device__ __forceinline__ Reach() : xy(__float2half2_rn(0.0f)), z(__float2half2_rn(0.0f)) {}
    __device__ __forceinline__ void add(const Features& f) {
        xy = __hmax2(xy, __habs2(f.xy));
        z = __hmax2(z, __habs2(f.zn));
    }
    __device__ __forceinline__ bool beyond() const {
        return !(fmaxf(fmaxf(__low2float(xy), __high2float(xy)), __low2float(z)) < kFeatureReach);
    }
};

template <int DIM>
__device__ __forceinline__ Features features(double px, double py, double pz, const CellUnion& cu, float inv_cell) {
    Features f;
    f.xy = __floats2half2_rn((float)(px - cu.ox) * inv_cell - 0.5f, (float)(py - cu.oy) * inv_cell - 0.5f);
    const __half z = DIM == 3 ? __float2half_rn((float)(pz - cu.oz) * inv_cell - 0.5f) : __float2half_rn(0.0f);
    const float2 c = __half22float2(f.xy);
    const float cz = __half2float(z), n = c.x * c.x + c.y * c.y + cz * cz;
    const __half nh = __float2half_rn(n);
    f.zn = __halves2half2(z, nh);
    f.m1 = __halves2half2(__float2half_rn(n - __half2float(nh)), __float2half_rn(1.0f));
    f.one = __halves2half2(__float2half_rn(1.0f), __float2half_rn(0.0f));
    return f;
}

// Where candidate u's features are staged: within a word of 32, so that the
// two columns a lane receives of each of the word's four products are the
// candidates of one byte of the mask.
__device__ __forceinline__ uint32_t feature_pos(uint32_t u) {
    return (u & ~31u) | ((u & 6u) << 2) | ((u & 24u) >> 2) | (u & 1u);
}

// The pair `pair` of the row of the centre staged at pos.
__device__ __forceinline__ uint32_t centre_pair(const Features* st, uint32_t pos, uint32_t pair) {
    constexpr uint32_t kHalfOne = 0x3c00u;
    if (pair < 2u) {
        const __half2 v = __hmul2(pair ? st[pos].zn : st[pos].xy, __floats2half2_rn(-2.0f, -2.0f));
        const uint32_t r = *reinterpret_cast<const uint32_t*>(&v);
        return pair ? (r & 0xffffu) | kHalfOne << 16 : r;  // (-2x, -2y) or (-2z, 1)
    }
    const float a = (__high2float(st[pos].zn) + __low2float(st[pos].m1)) - kBound2;
    const __half ah = __float2half_rn(a);
    if (pair == 2u) return kHalfOne | (uint32_t)__half_as_ushort(ah) << 16;
    return __half_as_ushort(__float2half_rn(a - __half2float(ah)));
}

__device__ __forceinline__ void mma_m16n8k8(float (&d)[4], const uint32_t (&a)[2], uint32_t b) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(b), "f"(0.0f));
}

// In-support masks of 32 centres over the union words [wb, we): bit u of the
// word of centre c (masks[word * kChunk + c]) says that candidate 32 word + u
// passes the filter. A lane owns byte (lane & 3) of the words of the centres
// lane / 4 + 0, 8, 16, 24: it shifts the eight signs of a centre's products
// into the byte and stores it, 52 instructions a word for the warp's 1,024
// tests where packed f32 arithmetic and compares took over 200.
// With at most 16 centres the second half of the tile is left out.
template <uint32_t kChunk, bool HALF>
__device__ __forceinline__ void word_masks(const Features* st, uint32_t* masks, const uint32_t (&a0)[2],
                                           const uint32_t (&a1)[2], uint32_t wb, uint32_t we) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t* feat = reinterpret_cast<const uint32_t*>(st) + lane;
    unsigned char* out = reinterpret_cast<unsigned char*>(masks + (lane >> 2)) + (lane & 3u);
    for (uint32_t w = wb; w < we; ++w) {
        float d0[4][4], d1[4][4];
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const uint32_t b = feat[w * 128u + n * 32u];
            mma_m16n8k8(d0[n], a0, b);
            if (!HALF) mma_m16n8k8(d1[n], a1, b);
        }
        uint32_t m[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int n = 3; n >= 0; --n)
#pragma unroll
            for (int j = 1; j >= 0; --j) {
                m[0] = __funnelshift_l(__float_as_uint(d0[n][j]), m[0], 1);
                m[1] = __funnelshift_l(__float_as_uint(d0[n][2 + j]), m[1], 1);
                if (!HALF) {
                    m[2] = __funnelshift_l(__float_as_uint(d1[n][j]), m[2], 1);
                    m[3] = __funnelshift_l(__float_as_uint(d1[n][2 + j]), m[3], 1);
                }
            }
#pragma unroll
        for (int r = 0; r < (HALF ? 2 : 4); ++r) out[(w * kChunk + 8u * r) * 4u] = (unsigned char)m[r];
    }
}

__device__ __forceinline__ uint32_t rows_for(uint32_t n) { return (n + 3u) >> 2; }

// Reserved block of one chunk: `rows` rows of `stride` groups.
struct ChunkBlock {
    unsigned long long base;  // group index of row 0, lane 0
    bool ok;
};

// Cursor over the set bits of one centre's masks (word w at m[w * kChunk]),
// in ascending bit order: entry t of the list is the t-th set bit.
template <uint32_t kChunk>
struct MaskCursor {
    static constexpr uint32_t kWays = kNlThreads / kChunk;
    const uint32_t* m;
    uint32_t w, bits;
    // Positioned on entry t0, given this centre's per-way counts cnt[r] of the
    // way word ranges [W r / kWays, W (r + 1) / kWays); t0 < the total count.
    __device__ __forceinline__ MaskCursor(const uint32_t* masks, const uint32_t (*cnt)[kChunk], uint32_t lane,
                                          uint32_t W, uint32_t t0)
        : m(masks + lane) {
        uint32_t r = 0, acc = 0;
        while (r + 1u < kWays && acc + cnt[r][lane] <= t0) acc += cnt[r++][lane];
        w = W * r / kWays;
        bits = m[w * kChunk];
        while (acc + (uint32_t)__popc(bits) <= t0) {
            acc += __popc(bits);
            bits = m[++w * kChunk];
        }
        for (; acc < t0; ++acc) bits &= bits - 1u;
    }
    // Position of the next set bit; the caller takes no more than the count.
    __device__ __forceinline__ uint32_t next() {
        while (!bits) bits = m[++w * kChunk];
        const uint32_t u = (w << 5) + (__ffs(bits) - 1);
        bits &= bits - 1u;
        return u;
    }
};

// Every thread passes its list's length; thread 0 reserves the block for the
// chunk's longest one and all threads return it.
__device__ __forceinline__ ChunkBlock reserve_chunk(const ListBufs& l, DeviceScalars* sc, uint32_t stride, uint32_t n,
                                                    uint32_t* s_red, ChunkBlock* s_blk, bool* s_overflow) {
    n = __reduce_max_sync(0xffffffffu, n);
    if ((threadIdx.x & 31u) == 0) s_red[threadIdx.x >> 5] = n;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t m = 0;
#pragma unroll
        for (uint32_t w = 0; w < kWarps; ++w) m = max(m, s_red[w]);
        ChunkBlock blk;
        const unsigned long long groups = (unsigned long long)rows_for(m) * stride;
        blk.base = groups ? atomicAdd(&sc->list_used, groups) : 0ull;
        // counts and strides are stored in 16 bits
        blk.ok = m < 65536u && stride < 65536u && blk.base + groups <= l.pool_groups;
        if (!blk.ok) *s_overflow = true;
        *s_blk = blk;
    }
    __syncthreads();
    return *s_blk;
}

// LSD radix sort of a union's fluid positions (s_sorted[0..nf)) by original
// index, on 9-bit digits of (orig - omin) (two passes for spans below 2^18);
// keys are read through the staged words. Warp w ranks the w-th contiguous
// segment of the array, 32 entries at a time in order, grouping equal digits
// with a match, so every pass is stable; counter (digit, warp) is
// s_cnt[digit * kWarps + warp] and one exclusive scan over them in that order
// gives each group its start. The keys are unique, so the result does not
// depend on the staging order. Ends with a block barrier.
constexpr int kRadixBits = 9;
constexpr uint32_t kRadixDigits = 1u << kRadixBits;
static_assert(kRadixDigits * kWarps == 16 * kNlThreads, "radix counters fill the scan's 16 per thread");

__device__ __forceinline__ void radix_sort_by_orig(const uint32_t* s_w, uint16_t* s_sorted, uint16_t* s_tmp,
                                                   uint16_t* s_cnt, uint32_t nf, uint32_t omin, uint32_t omax) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t span = nf ? omax - omin : 0u;
    const int npass = span ? (32 - __clz(span) + kRadixBits - 1) / kRadixBits : 0;
    const uint32_t seg = ((nf + kWarps - 1) / kWarps + 31u) & ~31u;
    const uint32_t e0 = min(nf, warp * seg), e1 = min(nf, e0 + seg);
    uint16_t *src = s_sorted, *dst = s_tmp;
    for (int pass = 0; pass < npass; ++pass) {
        const int shift = kRadixBits * pass;
        {
            uint4* const cw = reinterpret_cast<uint4*>(s_cnt);  // 512 16-byte words
            cw[tid] = cw[tid + kNlThreads] = make_uint4(0u, 0u, 0u, 0u);
        }
        __syncthreads();
        for (uint32_t b = e0; b < e1; b += 32u) {
            const uint32_t e = b + lane;
            const bool valid = e < e1;
            uint32_t d = kRadixDigits;  // lanes past the segment: a digit of their own
            if (valid) d = (((s_w[src[e]] & kStageOrigMask) - omin) >> shift) & (kRadixDigits - 1u);
            const uint32_t peers = __match_any_sync(0xffffffffu, d);
            if (valid && lane == (uint32_t)(__ffs(peers) - 1)) s_cnt[d * kWarps + warp] += (uint16_t)__popc(peers);
            __syncwarp();
        }
        __syncthreads();
        {
            // this thread's 16 consecutive counters as two 16-byte words
            // (32-byte stride between lanes: two-way bank conflicts, not 8)
            uint4* cw = reinterpret_cast<uint4*>(s_cnt + tid * 16);
            const uint4 c0 = cw[0], c1 = cw[1];
            const uint32_t pk[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
            uint32_t sum = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) sum += (pk[j] & 0xffffu) + (pk[j] >> 16);
            uint32_t ex, tot;
            block_exclusive_scan(sum, &ex, &tot);
            uint32_t out[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t lo = ex;
                ex += pk[j] & 0xffffu;
                out[j] = lo | (ex << 16);
                ex += pk[j] >> 16;
            }
            cw[0] = make_uint4(out[0], out[1], out[2], out[3]);
            cw[1] = make_uint4(out[4], out[5], out[6], out[7]);
        }
        __syncthreads();
        for (uint32_t b = e0; b < e1; b += 32u) {
            const uint32_t e = b + lane;
            const bool valid = e < e1;
            uint32_t d = kRadixDigits;
            uint16_t pu = 0;
            if (valid) {
                pu = src[e];
                d = (((s_w[pu] & kStageOrigMask) - omin) >> shift) & (kRadixDigits - 1u);
            }
            const uint32_t peers = __match_any_sync(0xffffffffu, d);
            uint32_t base = 0;
            if (valid) {
                base = s_cnt[d * kWarps + warp];
                dst[base + __popc(peers & ((1u << lane) - 1u))] = pu;
            }
            __syncwarp();
            if (valid && lane == (uint32_t)(__ffs(peers) - 1)) s_cnt[d * kWarps + warp] = (uint16_t)(base + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        uint16_t* t = src;
        src = dst;
        dst = t;
    }
    if (src != s_sorted) {
        for (uint32_t i = tid; i < nf; i += blockDim.x) s_sorted[i] = src[i];
    }
    __syncthreads();
}

// Slow path of the visit list for a union larger than the stage.
template <int DIM, bool LOWER_FLAGS>
__device__ __forceinline__ void visit_slow(const StepConst& k, float r2f, const CellUnion& cu, uint32_t U,
                                           const StateBufs& s, const ListBufs& l, DeviceScalars* sc,
                                           const uint32_t* s_cstart, const uint32_t* s_off, uint32_t* s_red,
                                           ChunkBlock* s_blk, bool* s_overflow) {
    constexpr int NC = DIM == 3 ? 27 : 9;
    const uint32_t tid = threadIdx.x;
    // Slow path: a union larger than the stage, straight from global
    // memory, one thread per centre particle: count, reserve, write.
    if (tid == 0) atomicOr(&sc->status, kStatusSlowUnion);
    for (uint32_t c0 = 0; c0 < cu.ncenter; c0 += kNlThreads) {
        const uint32_t nc = min((uint32_t)kNlThreads, cu.ncenter - c0);
        const bool active = tid < nc;
        const uint32_t kslot = cu.cs + c0 + tid;
        uint8_t mfl = 0;
        uint32_t myo = 0;
        float4 me = make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t nv = 0;
        bool fluidc = false;
        if (active) {
            me = stage_entry<DIM>(s, kslot, cu, &mfl, &myo);
            fluidc = !(mfl & kFlagBoundary);
            if (fluidc) {
                for (int c = 0; c < NC; ++c) {
                    const uint32_t q0 = s_cstart[c], q1 = q0 + (s_off[c + 1] - s_off[c]);
                    for (uint32_t slot = q0; slot < q1; ++slot) {
                        if (slot == kslot) continue;
                        uint8_t fl;
                        uint32_t o;
                        if (keep_entry(stage_entry<DIM>(s, slot, cu, &fl, &o), me, r2f, k.keep_boundary))
                            ++nv;
                    }
                }
            }
        }
        const ChunkBlock blk = reserve_chunk(l, sc, nc, nv, s_red, s_blk, s_overflow);
        if (active) {
            const uint32_t gv = (uint32_t)blk.base + tid;
            l.desc[kslot] = blk.ok ? make_uint4(gv, nc, nv, 0u) : make_uint4(0u, 0u, 0u, 0u);
            l.ncand[kslot] = fluidc ? U : 0u;
            if (blk.ok && fluidc) {
                const size_t step = 4u * nc;
                uint32_t* pv = l.pool + 4 * (size_t)gv;
                uint32_t tv = 0;
                for (int c = 0; c < NC; ++c) {
                    const uint32_t q0 = s_cstart[c], q1 = q0 + (s_off[c + 1] - s_off[c]);
                    for (uint32_t slot = q0; slot < q1; ++slot) {
                        if (slot == kslot) continue;
                        uint8_t fl;
                        uint32_t o;
                        const float4 qp = stage_entry<DIM>(s, slot, cu, &fl, &o);
                        if (!keep_entry(qp, me, r2f, k.keep_boundary)) continue;
                        uint32_t e = slot | entry_flags(__float_as_uint(qp.w));
                        if (LOWER_FLAGS && !(fl & kFlagBoundary) && o < myo) e |= kEntryLower;
                        if (tv < nv) pv[(tv >> 2) * step + (tv & 3u)] = e;
                        ++tv;
                    }
                }
            }
        }
        __syncthreads();
    }
}

// Slow path of the lower list for a union larger than the stage.
template <int DIM>
__device__ __forceinline__ void lower_slow(const StepConst& k, float r2f, const CellUnion& cu, const StateBufs& s,
                                           const ListBufs& l, DeviceScalars* sc, const uint32_t* s_cstart,
                                           const uint32_t* s_off, uint32_t* s_red, ChunkBlock* s_blk,
                                           bool* s_overflow) {
    constexpr int NC = DIM == 3 ? 27 : 9;
    const uint32_t tid = threadIdx.x;
    // Slow path: ascending original index by repeated selection, one
    // thread per centre particle: count, reserve, write.
    if (tid == 0) atomicOr(&sc->status, kStatusSlowUnion);
    for (uint32_t c0 = 0; c0 < cu.ncenter; c0 += kNlThreads) {
        const uint32_t nc = min((uint32_t)kNlThreads, cu.ncenter - c0);
        const bool active = tid < nc;
        const uint32_t kslot = cu.cs + c0 + tid;
        uint8_t mfl = 0;
        uint32_t myo = 0;
        float4 me = make_float4(0.f, 0.f, 0.f, 0.f);
        bool fluidc = false;
        uint32_t nl = 0;
        float r2c = r2f;
        if (active) {
            me = stage_entry<DIM>(s, kslot, cu, &mfl, &myo);
            fluidc = !(mfl & kFlagBoundary);
            if (!fluidc && k.keep_boundary) r2c = __int_as_float(0x7f800000);
            if (!(fluidc && k.lower_boundary_only)) {
                for (int c = 0; c < NC; ++c) {
                    const uint32_t q0 = s_cstart[c], q1 = q0 + (s_off[c + 1] - s_off[c]);
                    for (uint32_t slot = q0; slot < q1; ++slot) {
                        uint8_t fl;
                        uint32_t o;
                        const float4 qp = stage_entry<DIM>(s, slot, cu, &fl, &o);
                        if ((fl & kFlagBoundary) || (fluidc && o >= myo)) continue;
                        if (within(qp, me, r2c)) ++nl;
                    }
                }
            }
        }
        const ChunkBlock blk = reserve_chunk(l, sc, nc, nl, s_red, s_blk, s_overflow);
        if (active) {
            const uint32_t gl = (uint32_t)blk.base + tid;
            l.ldesc[kslot] = blk.ok ? make_uint2(gl, nl | (nc << 16)) : make_uint2(0u, 0u);
            if (blk.ok) {
                const size_t step = 4u * nc;
                uint32_t* pl = l.pool + 4 * (size_t)gl;
                uint32_t tl = 0;
                long long last = -1;
                while (tl < nl) {
                    unsigned long long best = ULLONG_MAX;
                    uint32_t best_slot = 0;
                    for (int c = 0; c < NC; ++c) {
                        const uint32_t q0 = s_cstart[c], q1 = q0 + (s_off[c + 1] - s_off[c]);
                        for (uint32_t slot = q0; slot < q1; ++slot) {
                            if (s.flags[slot] & kFlagBoundary) continue;
                            const uint32_t o = s.orig[slot];
                            if ((long long)o <= last || (fluidc && o >= myo) ||
                                (unsigned long long)o >= best)
                                continue;
                            uint8_t fl;
                            uint32_t oo;
                            if (within(stage_entry<DIM>(s, slot, cu, &fl, &oo), me, r2c)) {
                                best = o;
                                best_slot = slot;
                            }
                        }
                    }
                    if (best == ULLONG_MAX) break;
                    pl[(tl >> 2) * step + (tl & 3u)] = best_slot;
                    ++tl;
                    last = (long long)best;
                }
            }
        }
        __syncthreads();
    }
}

// The threads of a CTA shared out over a chunk's nc centres for the writing of
// their entries: way `way` of `ways` of centre `lane`, so that a cell's last,
// shorter chunk costs its share. ways = 0 for a thread left over.
struct Share {
    uint32_t lane, way, ways;
    __device__ __forceinline__ explicit Share(uint32_t nc) : ways(kNlThreads / nc) {
        way = threadIdx.x / nc;
        lane = threadIdx.x - way * nc;
        if (way >= ways) way = ways = 0;
    }
    // this way's entries [first, last) of n
    __device__ __forceinline__ uint32_t first(uint32_t n) const { return ways ? n * way / ways : 0u; }
    __device__ __forceinline__ uint32_t last(uint32_t n) const { return ways ? n * (way + 1u) / ways : 0u; }
};

// Where entry t of a list is written, and the next one's place after it.
struct EntryOut {
    uint32_t* p;
    uint32_t t, row;  // row: from a row's last entry to the next row's first
    __device__ __forceinline__ EntryOut(uint32_t* list, uint32_t step, uint32_t t0)
        : p(list + (size_t)(t0 >> 2) * step + (t0 & 3u)), t(t0), row(step - 3u) {}
    __device__ __forceinline__ void put(uint32_t e) const { *p = e; }
    __device__ __forceinline__ void next() {
        p += (t & 3u) == 3u ? row : 1u;
        ++t;
    }
};

// CTAs a cell: its chunks are shared out over several (each stages the union
// again) while the occupied cells leave most of the grid's 2,368 CTAs idle. us a
// build with 1 / 2 / 4 / 8 of them, f64 and f32: 48 cells -/28/22/23, 22/17/15/15;
// 118 cells 50/35/33/35, 31/21/21/22; 237 56/41/39/46, 37/27/24/25; 406 63/48/48/65,
// 41/31/29/34; 663 67/55/66/112, 45/35/35/53; 1,050 75/77/108/186, 51/42/54/79. A 2-D
// cell is one chunk: 113 cells 15/17/18/17, 10/11/12/13.
template <int DIM>
__device__ __forceinline__ uint32_t cell_parts(uint32_t nocc) {
    if (DIM == 2) return 1u;
    return 16u * nocc <= gridDim.x ? 4u : 3u * nocc <= gridDim.x ? 2u : 1u;
}

// ----------------------------------------------------------------- visit
// Dynamic shared memory (ucap a multiple of kStageStep): float x, y, z, w[ucap] (Stage);
// uint32 s_ent[ucap]; uint32 s_mask[(ucap / 32) * kChunk] (word w of chunk
// lane c at s_mask[w * kChunk + c]).
template <int DIM, uint32_t kChunk>
__global__ void __launch_bounds__(kNlThreads, 4) k_nlist_visit(GridDesc g, Tanks tk, StepConst k, uint32_t ucap,
                                                            const uint32_t* __restrict__ occ,
                                                            const uint32_t* __restrict__ cell_start,
                                                            StateBufs s, ListBufs l,
                                                            DeviceScalars* sc) {
    constexpr int NC = DIM == 3 ? 27 : 9;
    constexpr uint32_t kWays = kNlThreads / kChunk;
    extern __shared__ __align__(16) unsigned char smem[];
    Stage st(reinterpret_cast<float*>(smem), ucap);
    uint32_t* s_ent = reinterpret_cast<uint32_t*>(smem) + 4 * (size_t)ucap;
    uint32_t* s_mask = s_ent + ucap;
    __shared__ uint32_t s_cstart[NC];
    __shared__ uint32_t s_off[NC + 1];
    __shared__ uint32_t s_cv[kWays][kChunk];
    __shared__ uint32_t s_red[kWarps];
    __shared__ ChunkBlock s_blk;
    __shared__ bool s_overflow;

    const float r2f = k.r2_filter;
    const uint32_t nocc = sc->nocc;
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid % kChunk, q = tid / kChunk;
    uint32_t max_union = 0;
    if (tid == 0) s_overflow = false;

    const uint32_t parts = cell_parts<DIM>(nocc);
    for (uint32_t item = blockIdx.x; item < nocc * parts; item += gridDim.x) {
        const uint32_t it = item / parts, part = item - it * parts;
        const CellUnion cu = cell_union<DIM>(g, tk, occ[it], cell_start, s_cstart, s_off);
        const uint32_t U = cu.U;
        max_union = max(max_union, U);
        if (U <= ucap) {
            for (uint32_t u = tid; u < U; u += blockDim.x) {
                const uint32_t slot = slot_of_union<NC>(s_off, s_cstart, u);
                uint8_t fl;
                uint32_t o;
                const float4 p = stage_entry<DIM>(s, slot, cu, &fl, &o);
                st.put(u, p);
                s_ent[u] = slot | entry_flags(__float_as_uint(p.w));
            }
            __syncthreads();
            const uint32_t W = (U + 31u) >> 5;
            const uint32_t wb = W * q / kWays, we = W * (q + 1) / kWays;
            for (uint32_t c0 = part * kChunk; c0 < cu.ncenter; c0 += parts * kChunk) {
                const uint32_t nc = min(kChunk, cu.ncenter - c0);
                const bool active = lane < nc;
                const uint32_t myu = cu.center_off + c0 + lane;
                bool fluidc = false;
                // ---- pass 1: in-support masks of this quarter's words, counts
                if (active) {
                    const float4 me = st.get(myu);
                    const uint32_t mw = __float_as_uint(me.w);
                    fluidc = !(mw & kStageBoundary);
                    uint32_t cv = 0;
                    if (fluidc) {
                        for (uint32_t w = wb; w < we; ++w) {
                            uint32_t m = k.keep_boundary ? word_mask<true>(st, w << 5, me, r2f)
                                                         : word_mask<false>(st, w << 5, me, r2f);
                            if (w == W - 1u && (U & 31u)) m &= (1u << (U & 31u)) - 1u;
                            if (w == (myu >> 5)) m &= ~(1u << (myu & 31u));
                            s_mask[w * kChunk + lane] = m;
                            cv += __popc(m);
                        }
                    }
                    s_cv[q][lane] = cv;
                }
                __syncthreads();
                // ---- list lengths and the chunk's block
                uint32_t nv = 0;
                if (active) {
#pragma unroll
                    for (uint32_t r = 0; r < kWays; ++r) nv += s_cv[r][lane];
                }
                const ChunkBlock blk = reserve_chunk(l, sc, nc, nv, s_red, &s_blk, &s_overflow);
                // ---- pass 2: descriptors and entries
                if (active && q == 0) {
                    const uint32_t kslot = cu.cs + c0 + lane;
                    const uint32_t gv = (uint32_t)blk.base + lane;  // < pool_groups < 2^32 when ok
                    l.desc[kslot] = blk.ok ? make_uint4(gv, nc, nv, 0u) : make_uint4(0u, 0u, 0u, 0u);
                    l.ncand[kslot] = fluidc ? U : 0u;
                }
                if (blk.ok) {
                    const Share sh(nc);
                    uint32_t n = 0;
#pragma unroll
                    for (uint32_t r = 0; r < kWays; ++r) n += s_cv[r][sh.lane];
                    const uint32_t v0 = sh.first(n), v1 = sh.last(n);
                    if (v0 < v1) {
                        EntryOut out(l.pool + 4 * (size_t)(blk.base + sh.lane), 4u * nc, v0);
                        MaskCursor<kChunk> cur(s_mask, s_cv, sh.lane, W, v0);
                        for (; out.t < v1; out.next()) out.put(s_ent[cur.next()]);
                    }
                }
                __syncthreads();  // masks and counts are reused by the next chunk
            }
        } else if (part == 0) {
            visit_slow<DIM, false>(k, r2f, cu, U, s, l, sc, s_cstart, s_off, s_red, &s_blk, &s_overflow);
        }
        __syncthreads();  // shared memory is reused by the next cell
    }
    if (tid == 0 && s_overflow) atomicOr(&sc->status, kStatusListOverflow);
    if (tid == 0 && max_union) atomicMax(&sc->max_union, max_union);
}

// ----------------------------------------------------------------- near
// Visit lists of the fluid slots' candidates within the support radius of their
// present positions, the candidates taken from the cells of the last grid: what
// PBF's constraint iterations need, whose predictions move between two grids.
// A warp a cell, for cells of a few particles (PBF's support is one cell, ~8 of
// them, ~216 candidates): the CTA a cell of the kernels above leaves three
// quarters of its threads idle there. Positions are staged as f32 offsets from
// the cell; as they may be any number of cells away from it, the test's margin
// follows the largest staged offset (a candidate more adds +-0 to PBF's sums).
// 64,000 fluid particles and 43,000 samples: 51 us, bound by its own chain of
// loads and instruction issue (24M warp instructions, 30% of the ALU); lists of
// every candidate took 126 us once a step, but then each of the twelve passes
// over them 86 to 122 us instead of 28 to 32.
constexpr uint32_t kNearWarps = 4;    // warps a CTA
constexpr uint32_t kNearTile = 320;   // candidates staged at once
constexpr uint32_t kNearWords = kNearTile / 32u;

struct NearStage {
    float4 at[kNearTile];               // offset from the cell's corner, list entry
    uint32_t mask[32][kNearWords + 1];  // word w of centre c; the odd pitch spreads the words of 32 centres
    uint32_t head[kNearWords];          // union positions of the tile where a non-empty cell begins
    uint32_t shift[32];                 // non-empty cell k of the union: its slots minus its union positions
};

template <int DIM>
__global__ void __launch_bounds__(32 * kNearWarps, 8) k_nlist_near(GridDesc g, Tanks tk, float support,
                                                                  const uint32_t* __restrict__ occ,
                                                                  const uint32_t* __restrict__ cell_start,
                                                                  StateBufs s, ListBufs l, DeviceScalars* sc) {
    constexpr int NC = DIM == 3 ? 27 : 9;
    constexpr int CENTER = DIM == 3 ? 13 : 4;
    constexpr uint32_t kAll = 0xffffffffu;
    __shared__ NearStage s_stage[kNearWarps];
    NearStage& sm = s_stage[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nocc = sc->nocc, warps = gridDim.x * kNearWarps;
    const uint32_t parts = min(max(warps / max(nocc, 1u), 1u), 8u);  // warps a cell while there are more than cells
    uint32_t max_union = 0;
    bool overflow = false;

    for (uint32_t item = blockIdx.x * kNearWarps + (threadIdx.x >> 5); item < nocc * parts; item += warps) {
        const uint32_t it = parts == 1u ? item : item / parts, part = item - it * parts;
        const uint32_t c = occ[it];
        const TankDesc td = tk.desc[tk.cell_tank[c]];
        const uint32_t lc = c - td.cell_base;
        // ---- lane r: range of neighbour cell r, in visiting order
        const int cz = (int)(lc % (uint32_t)td.nz), cxy = (int)(lc / (uint32_t)td.nz);
        const int cx = (int)((uint32_t)cxy / (uint32_t)td.ny), cy = cxy - cx * td.ny;
        uint32_t st = 0, cnt = 0;
        if (lane < (uint32_t)NC) {
            const int qz = cz + (DIM == 3 ? (int)lane / 9 - 1 : 0);
            const int qy = cy + (DIM == 3 ? ((int)lane / 3) % 3 - 1 : (int)lane / 3 - 1);
            const int qx = cx + (int)lane % 3 - 1;
            if (qx >= 0 && qy >= 0 && qz >= 0 && qx < td.nx && qy < td.ny && qz < td.nz) {
                const uint32_t nc = td.cell_base + ((uint32_t)qx * (uint32_t)td.ny + (uint32_t)qy) * (uint32_t)td.nz +
                                    (uint32_t)qz;
                st = cell_start[nc];
                cnt = cell_start[nc + 1] - st;
            }
        }
        uint32_t off = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(kAll, off, o);
            if ((int)lane >= o) off += x;
        }
        const uint32_t U = __shfl_sync(kAll, off, 31);
        off -= cnt;
        const uint32_t cs = __shfl_sync(kAll, st, CENTER), coff = __shfl_sync(kAll, off, CENTER);
        const uint32_t ncenter = __shfl_sync(kAll, cnt, CENTER);
        max_union = max(max_union, U);
        const uint32_t tiles = (U + kNearTile - 1u) / kNearTile;
        const double ox = (double)(td.kx0 + cx) * g.cell_size, oy = (double)(td.ky0 + cy) * g.cell_size;
        const double oz = DIM == 3 ? (double)(td.kz0 + cz) * g.cell_size : 0.0;
        const uint32_t filled = __ballot_sync(kAll, cnt != 0u);
        uint32_t staged = kAll;  // tile in the stage
        float limit = 0.f;       // squared distance a candidate of it is kept within

        auto offset = [&](const double4& p) {
            return make_float4((float)(p.x - ox), (float)(p.y - oy), DIM == 3 ? (float)(p.z - oz) : 0.f, 0.f);
        };
        auto stage_tile = [&](uint32_t tile) {
            if (staged == tile) return;
            staged = tile;
            const uint32_t t0 = tile * kNearTile, m = min(kNearTile, U - t0);
            __syncwarp();
            // Union position u lies in the non-empty cell whose beginning is the
            // last at or below it; the tile's first position counts as one.
            if (lane < kNearWords) sm.head[lane] = 0u;
            __syncwarp();
            if (cnt) {
                sm.shift[__popc(filled & ((1u << lane) - 1u))] = st - off;
                if (off > t0 && off - t0 < kNearTile) atomicOr(&sm.head[(off - t0) >> 5], 1u << ((off - t0) & 31u));
            }
            uint32_t cell = __popc(__ballot_sync(kAll, cnt && off <= t0)) - 1u;  // of the tile's first position
            __syncwarp();
            float far = 0.f;
#pragma unroll 4
            for (uint32_t w = 0; w < (m + 31u) >> 5; ++w) {
                const uint32_t u = 32u * w + lane, h = sm.head[w];
                const uint32_t k = cell + __popc(h & (kAll >> (31u - lane)));
                cell += __popc(h);
                const uint32_t slot = sm.shift[k] + min(t0 + u, U - 1u);
                float4 p = offset(gather4(s.pos + slot));
                const uint8_t fl = s.flags[slot];
                far = fmaxf(far, fmaxf(fabsf(p.x), fmaxf(fabsf(p.y), fabsf(p.z))));
                p.w = __uint_as_float(slot | ((fl & kFlagBoundary) ? kEntryBoundary : 0u) |
                                      ((fl & kFlagOriented) ? kEntryOriented : 0u));
                sm.at[u] = p;
            }
            // The centres' offsets count too, where another tile stages them.
            for (uint32_t j = lane; tiles > 1u && j < ncenter; j += 32u) {
                const float4 p = offset(gather4(s.pos + cs + j));
                far = fmaxf(far, fmaxf(fabsf(p.x), fmaxf(fabsf(p.y), fabsf(p.z))));
            }
            // An offset is rounded by at most far / 2^24, a difference of two by
            // twice that and its own rounding (far / 2^23): 3.5 far / 2^23 in
            // distance, and the squares and their sum by 2^-22 of themselves.
            const float r = support + __uint_as_float(__reduce_max_sync(kAll, __float_as_uint(far))) * 0x1p-21f;
            limit = r * r * (1.f + 0x1p-20f);
            __syncwarp();
        };

        // ---- the part's centres, 32 at a time
        const uint32_t b0 = (uint32_t)((unsigned long long)ncenter * part / parts);
        const uint32_t b1 = (uint32_t)((unsigned long long)ncenter * (part + 1u) / parts);
        for (uint32_t c0 = b0; c0 < b1; c0 += 32u) {
            const uint32_t nc = min(32u, b1 - c0), kslot = cs + c0 + min(lane, nc - 1u);
            const bool fluid = lane < nc && !(s.flags[kslot] & kFlagBoundary);
            const uint32_t fluids = __ballot_sync(kAll, fluid);
            // masks of a tile's words, two centres at a time: their tests share a candidate's loads
            auto tile_masks = [&](uint32_t tile) {
                const uint32_t t0 = tile * kNearTile, m = min(kNearTile, U - t0), words = (m + 31u) >> 5;
                stage_tile(tile);
                for (uint32_t left = fluids; left; left &= left - 1u) {
                    const uint32_t q0 = (uint32_t)__ffs(left) - 1u;
                    left &= left - 1u;
                    const uint32_t q1 = left ? (uint32_t)__ffs(left) - 1u : q0;
                    if (!left) left = 1u;  // the last round
                    const uint32_t self0 = coff + c0 + q0 - t0, self1 = coff + c0 + q1 - t0;
                    const float4 a = tiles == 1u ? sm.at[self0] : offset(gather4(s.pos + cs + c0 + q0));
                    const float4 b = tiles == 1u ? sm.at[self1] : offset(gather4(s.pos + cs + c0 + q1));
                    uint32_t keep0 = 0, keep1 = 0;
#pragma unroll 2
                    for (uint32_t w = 0; w < words; ++w) {
                        const float4 p = sm.at[32u * w + lane];
                        const float ax = p.x - a.x, ay = p.y - a.y, az = p.z - a.z;
                        const float bx = p.x - b.x, by = p.y - b.y, bz = p.z - b.z;
                        // (unlike the other builds' tests, this one keeps a position that is no
                        // number: PBF's passes then carry it on as those of all candidates did)
                        const uint32_t ma = __ballot_sync(kAll, !(ax * ax + ay * ay + az * az > limit));
                        const uint32_t mb = __ballot_sync(kAll, !(bx * bx + by * by + bz * bz > limit));
                        if (lane == w) {
                            keep0 = ma;
                            keep1 = mb;
                        }
                    }
                    if (lane < words) {  // candidates past the union and the centre itself out
                        if (lane == words - 1u && (m & 31u)) {
                            keep0 &= (1u << (m & 31u)) - 1u;
                            keep1 &= (1u << (m & 31u)) - 1u;
                        }
                        if (lane == (self0 >> 5)) keep0 &= ~(1u << (self0 & 31u));
                        if (lane == (self1 >> 5)) keep1 &= ~(1u << (self1 & 31u));
                        sm.mask[q0][lane] = keep0;
                        sm.mask[q1][lane] = keep1;
                    }
                }
                __syncwarp();
            };
            // The lanes share out the centres' words: lane r * nc + q takes the
            // r-th of `ways` shares of centre q's (a lane past them none).
            const uint32_t ways = 32u / nc, q = lane % nc, r = lane / nc;
            const bool mine = r < ways && ((fluids >> q) & 1u);
            auto share = [&](uint32_t tile, uint32_t* wb, uint32_t* we) {
                const uint32_t words = (min(kNearTile, U - tile * kNearTile) + 31u) >> 5;
                *wb = mine ? words * r / ways : 0u;
                *we = mine ? words * (r + 1u) / ways : 0u;
                uint32_t n = 0;
                for (uint32_t w = *wb; w < *we; ++w) n += __popc(sm.mask[q][w]);
                return n;
            };
            // sum over centre q's lanes of v, and over its lanes before this one
            auto centre_sum = [&](uint32_t v, uint32_t* before) {
                uint32_t tot = 0, pre = 0;
                for (uint32_t w = 0; w < ways; ++w) {
                    const uint32_t x = __shfl_sync(kAll, v, w * nc + q);
                    if (w < r) pre += x;
                    tot += x;
                }
                *before = pre;
                return tot;
            };
            uint32_t nv = 0, wb = 0, we = 0, before = 0, n = 0;  // the centre's entries, this lane's share of them
            if (fluids) {
                for (uint32_t tile = 0; tile < tiles; ++tile) {
                    tile_masks(tile);
                    n = share(tile, &wb, &we);
                    nv += centre_sum(n, &before);
                }
            }
            // ---- the chunk's block
            const uint32_t longest = __reduce_max_sync(kAll, nv);
            const unsigned long long groups = (unsigned long long)rows_for(longest) * nc;
            unsigned long long base = 0;
            if (lane == 0 && groups) base = atomicAdd(&sc->list_used, groups);
            base = __shfl_sync(kAll, base, 0);
            const bool ok = longest < 65536u && base + groups <= l.pool_groups;  // counts are stored in 16 bits
            overflow |= !ok;
            if (lane < nc) {
                l.desc[kslot] = ok ? make_uint4((uint32_t)base + lane, nc, nv, 0u) : make_uint4(0u, 0u, 0u, 0u);
                l.ncand[kslot] = fluid ? U : 0u;
            }
            if (!ok || !longest) continue;
            // ---- the entries: a lane writes those of its words
            uint32_t* const out = l.pool + 4 * (size_t)(base + q);
            uint32_t done = 0;  // entries of the centre written from earlier tiles
            for (uint32_t tile = 0; tile < tiles; ++tile) {
                uint32_t all = nv;
                if (tiles > 1u) {
                    tile_masks(tile);
                    n = share(tile, &wb, &we);
                    all = centre_sum(n, &before);
                }
                if (n) {
                    uint32_t t = done + before, w = wb, b = sm.mask[q][w];
                    for (const uint32_t end = t + n; t < end; ++t) {
                        while (!b) b = sm.mask[q][++w];
                        out[(size_t)(t >> 2) * (4u * nc) + (t & 3u)] = __float_as_uint(sm.at[32u * w + (uint32_t)__ffs(b) - 1u].w);
                        b &= b - 1u;
                    }
                }
                done += all;
                __syncwarp();
            }
        }
        __syncwarp();
    }
    if (lane == 0 && overflow) atomicOr(&sc->status, kStatusListOverflow);
    if (lane == 0 && max_union) atomicMax(&sc->max_union, max_union);
}

// ----------------------------------------------------------------- both
// Stages candidate u of a union: features, list entry and staged word.
template <int DIM>
__device__ __forceinline__ uint32_t stage_candidate(const StateBufs& s, const CellUnion& cu, float inv_cell,
                                                    uint32_t slot, uint32_t u, Features* st, uint32_t* s_ent,
                                                    Reach& reach) {
    const double4 p = s.pos[slot];
    const uint8_t fl = s.flags[slot];
    const uint32_t w = s.orig[slot] | ((fl & kFlagBoundary) ? kStageBoundary : 0u) |
                       ((fl & kFlagOriented) ? kStageOriented : 0u);
    const Features f = features<DIM>(p.x, p.y, p.z, cu, inv_cell);
    st[feature_pos(u)] = f;
    reach.add(f);
    s_ent[u] = slot | entry_flags(w);
    return w;
}

// In-support masks of the nc (1 to 32) centres from union position u0 over
// the words [wb, we). Rows past nc repeat the last centre.
template <uint32_t kChunk>
__device__ __forceinline__ void centre_masks(const Features* st, uint32_t* masks, uint32_t u0, uint32_t nc,
                                             uint32_t wb, uint32_t we) {
    const uint32_t row = (threadIdx.x & 31u) >> 2, pair = threadIdx.x & 3u;
    auto at = [&](uint32_t r) { return centre_pair(st, feature_pos(u0 + min(r, nc - 1u)), pair); };
    const uint32_t a0[2] = {at(row), at(row + 8u)};
    if (nc <= 16u) {
        word_masks<kChunk, true>(st, masks, a0, a0, wb, we);
    } else {
        const uint32_t a1[2] = {at(row + 16u), at(row + 24u)};
        word_masks<kChunk, false>(st, masks, a0, a1, wb, we);
    }
}

// The union staged anew as f32 offsets, in place of the features; raises *far to the
// bits of the largest one (a position that is no number has no neighbours).
template <int DIM>
__device__ __forceinline__ void stage_wide(const double4* __restrict__ pos, double ox, double oy, double oz, uint32_t U,
                                           const uint32_t* s_ent, Features* st, uint32_t* far) {
    float4* const at = reinterpret_cast<float4*>(st);
    for (uint32_t u = threadIdx.x; u < U; u += blockDim.x) {
        const double4 p = pos[s_ent[u] & kEntrySlotMask];
        const float4 o = make_float4((float)(p.x - ox), (float)(p.y - oy), DIM == 3 ? (float)(p.z - oz) : 0.0f, 0.0f);
        at[u] = o;
        const float m = fmaxf(fmaxf(fabsf(o.x), fabsf(o.y)), fabsf(o.z));
        if (m <= kLargestFloat) atomicMax(far, __float_as_uint(m));
    }
}

// centre_masks from f32 offsets, for the thread's own centre (union position me).
// In line: as calls, these two cost the unions that never come here 4 % (list build
// at 1M 2.73 ms; 2.65 so, 2.63 without them).
// The margin follows the union's largest offset `far`: an offset is rounded by at
// most far / 2^24 a component and a difference of two by far / 2^23, below far /
// 2^21 in distance. (A difference that overflows is no neighbour's.) A candidate
// more adds +-0 to the sums.
template <uint32_t kChunk>
__device__ __forceinline__ void wide_masks(const Features* st, uint32_t* mask, uint32_t me, float far, float r2f,
                                           uint32_t wb, uint32_t we) {
    const float4* const at = reinterpret_cast<const float4*>(st);
    const float4 a = at[me];
    const float r = sqrtf(r2f) + far * 0x1p-21f;
    const float limit = fminf(r * r * (1.f + 0x1p-20f), kLargestFloat);
    for (uint32_t w = wb; w < we; ++w) {
        uint32_t m = 0;
#pragma unroll 4
        for (uint32_t b = 0; b < 32u; ++b) m |= within(at[32u * w + b], a, limit) ? 1u << b : 0u;
        mask[w * kChunk] = m;
    }
}

// A fluid centre's share [wb, we) of the mask words m[w * kChunk] made whole:
// candidates past the union and the centre itself (union position myu) out,
// every candidate in (all) or every boundary candidate (keep_boundary).
// Returns their count.
template <uint32_t kChunk>
__device__ __forceinline__ uint32_t finish_masks(uint32_t* m, const uint32_t* s_fluid, uint32_t U, uint32_t myu,
                                                 uint32_t wb, uint32_t we, bool all, int keep_boundary) {
    if (all || keep_boundary)
        for (uint32_t w = wb; w < we; ++w) m[w * kChunk] = all ? 0xffffffffu : m[w * kChunk] | ~s_fluid[w];
    const uint32_t tail = U >> 5, own = myu >> 5;
    if ((U & 31u) && tail >= wb && tail < we) m[tail * kChunk] &= (1u << (U & 31u)) - 1u;
    if (own >= wb && own < we) m[own * kChunk] &= ~(1u << (myu & 31u));
    uint32_t n = 0;
    for (uint32_t w = wb; w < we; ++w) n += __popc(m[w * kChunk]);
    return n;
}

// One pass per occupied cell for both lists: the union is staged once, the
// in-support masks of a chunk's centres are computed once, and a centre's lower
// list comes out of its own mask: each kept candidate below the centre's rank
// sets its bit in a mask over the radix-sorted fluid positions. Visit rows and
// lower rows are reserved one after the other. Dynamic shared memory:
// Features[ucap]; uint32 s_ent[ucap] (slot | flags); uint32
// s_vmask[(ucap / 32) * kChunk], which holds the staged words until the sort is
// done; uint32 s_fluid[ucap / 32]; uint16 s_sorted[ucap]; uint16 s_rank[ucap],
// until then the sort's scratch; then the sort's counters, whose place the
// lower masks take. At 2,304 entries 74 KB, so three CTAs fit an SM.
template <int DIM, uint32_t kChunk>
__global__ void __launch_bounds__(kNlThreads, 3) k_nlist_both(GridDesc g, Tanks tk, StepConst k, uint32_t ucap,
                                                           const uint32_t* __restrict__ occ,
                                                           const uint32_t* __restrict__ cell_start,
                                                           StateBufs s, ListBufs l, DeviceScalars* sc) {
    constexpr int NC = DIM == 3 ? 27 : 9;
    constexpr uint32_t kWays = kNlThreads / kChunk;
    extern __shared__ __align__(16) unsigned char smem[];
    Features* st = reinterpret_cast<Features*>(smem);
    uint32_t* s_ent = reinterpret_cast<uint32_t*>(st + ucap);
    uint32_t* s_vmask = s_ent + ucap;
    uint32_t* s_fluid = s_vmask + (ucap / 32) * kChunk;
    uint16_t* s_sorted = reinterpret_cast<uint16_t*>(s_fluid + ucap / 32);
    uint16_t* s_rank = s_sorted + ucap;
    uint32_t* s_lmask = reinterpret_cast<uint32_t*>(s_rank + ucap);
    uint32_t* s_w = s_vmask;
    uint16_t* s_tmp = s_rank;
    uint16_t* s_cnt = reinterpret_cast<uint16_t*>(s_lmask);
    __shared__ uint32_t s_cstart[NC];
    __shared__ uint32_t s_off[NC + 1];
    __shared__ uint32_t s_nf, s_omin, s_omax, s_far;
    __shared__ bool s_wide;
    __shared__ uint32_t s_cv[kWays][kChunk], s_cl[kWays][kChunk];
    __shared__ uint32_t s_red[kWarps];
    __shared__ ChunkBlock s_blk;
    __shared__ bool s_overflow;

    constexpr uint32_t kNoRank = 0xffffu;  // of a boundary candidate (a stage holds fewer)
    const float r2f = k.r2_filter;
    const bool all = isinf(r2f);
    const float inv_cell = (float)g.inv_cell;
    const uint32_t nocc = sc->nocc;
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid % kChunk, q = tid / kChunk, cb = lane & ~31u;
    uint32_t max_union = 0;
    if (tid == 0) s_overflow = false;

    const uint32_t parts = cell_parts<DIM>(nocc);
    for (uint32_t item = blockIdx.x; item < nocc * parts; item += gridDim.x) {
        const uint32_t it = item / parts, part = item - it * parts;
        if (tid == 0) {
            s_nf = 0;
            s_omin = 0xffffffffu;
            s_omax = 0u;
            s_far = 0u;
            s_wide = false;
        }
        const CellUnion cu = cell_union<DIM>(g, tk, occ[it], cell_start, s_cstart, s_off);
        const uint32_t U = cu.U;
        max_union = max(max_union, U);
        if (U <= ucap) {
            // Stage the union; fluid entries are appended to s_sorted with one
            // shared atomic per warp, their index range reduced per warp.
            uint32_t tmin = 0xffffffffu, tmax = 0u;
            Reach reach;
            for (uint32_t u0 = 0; u0 < U; u0 += blockDim.x) {
                const uint32_t u = u0 + tid;
                bool fluid = false;
                if (u < U) {
                    const uint32_t w = stage_candidate<DIM>(s, cu, inv_cell, slot_of_union<NC>(s_off, s_cstart, u), u,
                                                            st, s_ent, reach);
                    s_w[u] = w;
                    fluid = !(w & kStageBoundary);
                    if (fluid) {
                        tmin = min(tmin, w & kStageOrigMask);
                        tmax = max(tmax, w & kStageOrigMask);
                    }
                }
                const uint32_t fm = __ballot_sync(0xffffffffu, fluid);
                uint32_t base = 0;
                if ((tid & 31u) == 0) {
                    if (fm) base = atomicAdd(&s_nf, (uint32_t)__popc(fm));
                    if (u < U) s_fluid[u >> 5] = fm;
                }
                base = __shfl_sync(0xffffffffu, base, 0);
                if (fluid) s_sorted[base + __popc(fm & ((1u << (tid & 31u)) - 1u))] = (uint16_t)u;
            }
            tmin = __reduce_min_sync(0xffffffffu, tmin);
            tmax = __reduce_max_sync(0xffffffffu, tmax);
            if ((tid & 31u) == 0 && tmin <= tmax) {
                atomicMin(&s_omin, tmin);
                atomicMax(&s_omax, tmax);
            }
            if (reach.beyond()) s_wide = true;
            __syncthreads();
            const uint32_t nf = s_nf;
            const bool wide = s_wide && !all;
            if (wide) stage_wide<DIM>(s.pos, cu.ox, cu.oy, cu.oz, U, s_ent, st, &s_far);
            radix_sort_by_orig(s_w, s_sorted, s_tmp, s_cnt, nf, s_omin, s_omax);
            for (uint32_t u = 2u * tid; u < U; u += 2u * blockDim.x)
                *reinterpret_cast<uint32_t*>(s_rank + u) = kNoRank | kNoRank << 16;
            __syncthreads();
            for (uint32_t i = tid; i < nf; i += blockDim.x) s_rank[s_sorted[i]] = (uint16_t)i;
            __syncthreads();
            const uint32_t W = (U + 31u) >> 5;
            const uint32_t wb = W * q / kWays, we = W * (q + 1) / kWays;
            for (uint32_t c0 = part * kChunk; c0 < cu.ncenter; c0 += parts * kChunk) {
                const uint32_t nc = min(kChunk, cu.ncenter - c0);
                const bool active = lane < nc;
                const uint32_t myu = cu.center_off + c0 + lane;
                // ---- pass 1: in-support masks of this share of the union words
                // (no fluid in reach: no list to build)
                if (!all && nf) {
                    if (wide) {
                        if (active) wide_masks<kChunk>(st, s_vmask + lane, myu, __uint_as_float(s_far), r2f, wb, we);
                    } else if (cb < nc) {
                        centre_masks<kChunk>(st, s_vmask + cb, cu.center_off + c0 + cb, min(nc - cb, 32u), wb, we);
                    }
                }
                __syncwarp();
                // R: the centre's lower list holds the kept fluid candidates of
                // rank below R (all of them for a boundary centre)
                bool fluidc = false;
                uint32_t R = 0, cv = 0;
                if (active) {
                    const uint32_t rank = s_rank[myu];
                    fluidc = rank != kNoRank;
                    R = fluidc ? rank : nf;
                    if (fluidc) {
                        cv = finish_masks<kChunk>(s_vmask + lane, s_fluid, U, myu, wb, we, all, k.keep_boundary);
                    } else if (nf) {  // a boundary centre: the fluid candidates in reach, or all of them
                        for (uint32_t w = wb; w < we; ++w) {
                            uint32_t m = s_fluid[w];
                            if (!all && !k.keep_boundary) m &= s_vmask[w * kChunk + lane];
                            s_vmask[w * kChunk + lane] = m;
                            cv += __popc(m);
                        }
                    }
                    s_cv[q][lane] = cv;
                }
                // this share of the lower mask's words, cleared
                const bool lowers = !(fluidc && k.lower_boundary_only);
                const uint32_t WR = lowers ? (R + 31u) >> 5 : 0u;
                const uint32_t lb = WR * q / kWays, le = WR * (q + 1) / kWays;
                if (active)
                    for (uint32_t w = lb; w < le; ++w) s_lmask[w * kChunk + lane] = 0u;
                __syncthreads();
                // ---- the visit list: length, block, entries; lower bits
                uint32_t nv = 0;
                if (active && fluidc) {
#pragma unroll
                    for (uint32_t r = 0; r < kWays; ++r) nv += s_cv[r][lane];
                }
                const ChunkBlock blk = reserve_chunk(l, sc, nc, nv, s_red, &s_blk, &s_overflow);
                const uint32_t kslot = cu.cs + c0 + lane;
                if (active && q == 0) {
                    const uint32_t gv = (uint32_t)blk.base + lane;  // < pool_groups < 2^32 when ok
                    l.desc[kslot] = blk.ok ? make_uint4(gv, nc, nv, 0u) : make_uint4(0u, 0u, 0u, 0u);
                    l.ncand[kslot] = fluidc ? U : 0u;
                }
                // Entries are split evenly over the threads (split by words, a
                // few would hold most of the kept candidates).
                const Share sh(nc);
                {
                    uint32_t n = 0;  // kept candidates
#pragma unroll
                    for (uint32_t r = 0; r < kWays; ++r) n += s_cv[r][sh.lane];
                    const uint32_t v0 = sh.first(n), v1 = sh.last(n);
                    if (v0 < v1) {
                        const uint32_t rank = s_rank[cu.center_off + c0 + sh.lane];
                        const bool fl = rank != kNoRank, put = blk.ok && fl;
                        const uint32_t below = fl ? rank : nf, lower_below = fl && k.lower_boundary_only ? 0u : below;
                        EntryOut out(l.pool + 4 * (size_t)(blk.base + sh.lane), 4u * nc, v0);
                        uint32_t* const lm = s_lmask + sh.lane;
                        MaskCursor<kChunk> cur(s_vmask, s_cv, sh.lane, W, v0);
                        for (; out.t < v1; out.next()) {
                            const uint32_t u = cur.next();
                            const uint32_t r = s_rank[u];
                            if (put) out.put(s_ent[u] | (r < below ? kEntryLower : 0u));
                            if (r < lower_below) atomicOr(lm + (r >> 5) * kChunk, 1u << (r & 31u));
                        }
                    }
                }
                __syncthreads();  // every share's lower bits are in place
                // ---- the lower list
                if (active) {
                    uint32_t cl = 0;
                    for (uint32_t w = lb; w < le; ++w) cl += __popc(s_lmask[w * kChunk + lane]);
                    s_cl[q][lane] = cl;
                }
                __syncthreads();
                uint32_t nl = 0;
                if (active) {
#pragma unroll
                    for (uint32_t r = 0; r < kWays; ++r) nl += s_cl[r][lane];
                }
                const ChunkBlock lblk = reserve_chunk(l, sc, nc, nl, s_red, &s_blk, &s_overflow);
                const bool ok = blk.ok && lblk.ok;
                if (active && q == 0)
                    l.ldesc[kslot] = ok ? make_uint2((uint32_t)lblk.base + lane, nl | (nc << 16)) : make_uint2(0u, 0u);
                if (ok) {
                    uint32_t n = 0;
#pragma unroll
                    for (uint32_t r = 0; r < kWays; ++r) n += s_cl[r][sh.lane];
                    const uint32_t l0 = sh.first(n), l1 = sh.last(n);
                    if (l0 < l1) {
                        const uint32_t rank = s_rank[cu.center_off + c0 + sh.lane];
                        EntryOut out(l.pool + 4 * (size_t)(lblk.base + sh.lane), 4u * nc, l0);
                        MaskCursor<kChunk> cur(s_lmask, s_cl, sh.lane, ((rank != kNoRank ? rank : nf) + 31u) >> 5, l0);
                        for (; out.t < l1; out.next()) out.put(s_ent[s_sorted[cur.next()]] & kEntrySlotMask);
                    }
                }
                __syncthreads();  // masks and counts are reused by the next chunk
            }
        } else if (part == 0) {
            visit_slow<DIM, true>(k, r2f, cu, U, s, l, sc, s_cstart, s_off, s_red, &s_blk, &s_overflow);
            lower_slow<DIM>(k, r2f, cu, s, l, sc, s_cstart, s_off, s_red, &s_blk, &s_overflow);
        }
        __syncthreads();  // shared memory is reused by the next cell
    }
    if (tid == 0 && s_overflow) atomicOr(&sc->status, kStatusListOverflow);
    if (tid == 0 && max_union) atomicMax(&sc->max_union, max_union);
}

// Largest neighbour-cell union of the current grid (a thread per occupied cell;
// the cells of a z column are adjacent in the dense order).
template <int DIM>
__global__ void k_union_max(Tanks tk, const uint32_t* __restrict__ occ, const uint32_t* __restrict__ cell_start,
                            DeviceScalars* sc) {
    const uint32_t it = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t u = 0;
    if (it < sc->nocc) {
        const uint32_t c = occ[it];
        const TankDesc td = tk.desc[tk.cell_tank[c]];
        const uint32_t lc = c - td.cell_base;
        const int cz = (int)(lc % (uint32_t)td.nz);
        const int cy = (int)((lc / (uint32_t)td.nz) % (uint32_t)td.ny);
        const int cx = (int)(lc / ((uint32_t)td.nz * (uint32_t)td.ny));
        const int z0 = max(cz - 1, 0), z1 = min(cz + 1, td.nz - 1);
        for (int qx = max(cx - 1, 0); qx <= min(cx + 1, td.nx - 1); ++qx)
            for (int qy = max(cy - 1, 0); qy <= min(cy + 1, td.ny - 1); ++qy) {
                const uint32_t base = td.cell_base + ((uint32_t)qx * (uint32_t)td.ny + (uint32_t)qy) * (uint32_t)td.nz;
                u += cell_start[base + (uint32_t)z1 + 1u] - cell_start[base + (uint32_t)z0];
            }
    }
    u = warp_max(u);
    if ((threadIdx.x & 31u) == 0 && u) atomicMax(&sc->max_union, u);
}

size_t both_smem_bytes(uint32_t ucap, uint32_t chunk) {
    const size_t cnt = 16 * kNlThreads * sizeof(uint16_t), mask = (size_t)(ucap / 32) * chunk * sizeof(uint32_t);
    return (size_t)ucap * (sizeof(Features) + sizeof(uint32_t) + 2 * sizeof(uint16_t)) + mask +
           (ucap / 32) * sizeof(uint32_t) + (cnt > mask ? cnt : mask);
}

size_t visit_smem_bytes(uint32_t ucap, uint32_t chunk) {
    return (size_t)ucap * (sizeof(float4) + sizeof(uint32_t)) + (size_t)(ucap / 32) * chunk * sizeof(uint32_t);
}

// the tile a stage of ucap entries is built with
uint32_t valid_chunk(uint32_t ucap, uint32_t chunk) {
    if (chunk != 32u) chunk = kDefaultChunk;
    return both_smem_bytes(ucap, chunk) > kMaxDynamicBytes ? 32u : chunk;
}

}  // namespace

uint32_t nlist_union_capacity(uint32_t max_union) {
    // The largest union seen plus an eighth, in steps of kStageStep, within
    // the shared-memory limit; larger unions take the slow path. The margin
    // is kept small so that three CTAs of the fused kernel fit an SM at the
    // 32-centre tile (at 1M: a 2,304-entry stage, 75 KB per CTA; with a
    // quarter's margin the stage was 2,560 entries and two CTAs fit).
    uint64_t want = (uint64_t)max_union + max_union / 8u;
    want = (want + kStageStep - 1) / kStageStep * kStageStep;
    if (want < kStageStep) want = kStageStep;
    if (want > kMaxUnionStage) want = kMaxUnionStage;
    return (uint32_t)want;
}

namespace {
template <int DIM, uint32_t C>
uint32_t prepare_for(uint32_t ucap) {
    // the attribute is the kernel's, not the world's: the largest stage's bytes,
    // so that no world's setting falls below another's launch
    const int sv = (int)visit_smem_bytes(ucap, C), sb = (int)both_smem_bytes(ucap, C);
    int bv = 0, bb = 0;
    cudaFuncSetAttribute(k_nlist_visit<DIM, C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)std::min(visit_smem_bytes(kMaxUnionStage, C), kMaxDynamicBytes));
    cudaFuncSetAttribute(k_nlist_both<DIM, C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)std::min(both_smem_bytes(kMaxUnionStage, C), kMaxDynamicBytes));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bv, k_nlist_visit<DIM, C>, kNlThreads, sv);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bb, k_nlist_both<DIM, C>, kNlThreads, sb);
    const int b = bv > bb ? bv : bb;
    return b > 0 ? (uint32_t)b : 1u;
}

template <int DIM, uint32_t C>
void launch_for(const GridDesc& g, const Tanks& tk, const StepConst& k, uint32_t ucap, uint32_t nblocks,
                const uint32_t* occ, const uint32_t* cell_start, const StateBufs& s, const ListBufs& l,
                DeviceScalars* sc, cudaStream_t st, bool visit_only) {
    if (visit_only)
        k_nlist_visit<DIM, C><<<nblocks, kNlThreads, visit_smem_bytes(ucap, C), st>>>(
            g, tk, k, ucap, occ, cell_start, s, l, sc);
    else
        k_nlist_both<DIM, C><<<nblocks, kNlThreads, both_smem_bytes(ucap, C), st>>>(g, tk, k, ucap, occ,
                                                                                  cell_start, s, l, sc);
}
}  // namespace

uint32_t nlist_prepare(int dim, uint32_t ucap, uint32_t chunk) {
    chunk = valid_chunk(ucap, chunk);
    if (dim == 3) return chunk == 32u ? prepare_for<3, 32>(ucap) : prepare_for<3, 64>(ucap);
    return chunk == 32u ? prepare_for<2, 32>(ucap) : prepare_for<2, 64>(ucap);
}

void launch_union_max(const GridDesc& g, const Tanks& tk, uint32_t ncell_max, const uint32_t* occ,
                      const uint32_t* cell_start, DeviceScalars* sc, cudaStream_t st) {
    const uint32_t b = (ncell_max + 255u) / 256u;
    if (g.dim == 3) k_union_max<3><<<b, 256, 0, st>>>(tk, occ, cell_start, sc);
    else k_union_max<2><<<b, 256, 0, st>>>(tk, occ, cell_start, sc);
}

void launch_nlist_near(const GridDesc& g, const Tanks& tk, double support, uint32_t ncell_max, uint32_t sms,
                       const uint32_t* occ, const uint32_t* cell_start, const StateBufs& s, const ListBufs& l,
                       DeviceScalars* sc, cudaStream_t st) {
    // several CTAs a resident one: cells of boundary samples alone are done at once
    const uint32_t b = std::min((ncell_max + kNearWarps - 1u) / kNearWarps * 8u, 40u * sms);
    const float r = std::nextafter((float)support, std::numeric_limits<float>::infinity());
    if (g.dim == 3) k_nlist_near<3><<<b, 32 * kNearWarps, 0, st>>>(g, tk, r, occ, cell_start, s, l, sc);
    else k_nlist_near<2><<<b, 32 * kNearWarps, 0, st>>>(g, tk, r, occ, cell_start, s, l, sc);
}

void launch_nlist(const GridDesc& g, const Tanks& tk, const StepConst& k, uint32_t ucap,
                  uint32_t nblocks, const uint32_t* occ, const uint32_t* cell_start,
                  const StateBufs& s, const ListBufs& l, DeviceScalars* sc, cudaStream_t st,
                  bool visit_only, uint32_t chunk) {
    chunk = valid_chunk(ucap, chunk);
    if (g.dim == 3) {
        if (chunk == 32u) launch_for<3, 32>(g, tk, k, ucap, nblocks, occ, cell_start, s, l, sc, st, visit_only);
        else launch_for<3, 64>(g, tk, k, ucap, nblocks, occ, cell_start, s, l, sc, st, visit_only);
    } else {
        if (chunk == 32u) launch_for<2, 32>(g, tk, k, ucap, nblocks, occ, cell_start, s, l, sc, st, visit_only);
        else launch_for<2, 64>(g, tk, k, ucap, nblocks, occ, cell_start, s, l, sc, st, visit_only);
    }
}

}  // namespace pe

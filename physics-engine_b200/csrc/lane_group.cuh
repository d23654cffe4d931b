// Several lanes of a warp on one slot's neighbour list, with the sums still in
// list order.
//
// One thread per slot walks ~250 pairs one after another, each a chain of
// square root, divisions and dependent multiplies: with 32,768 fluid particles
// an SM holds seven warps and the passes wait on that chain (the force pass
// took 310 us where its share of the 1M-particle pass is 100 us). A group of G
// lanes computes the terms of G consecutive entries at once, and the lane of
// each component adds the G terms in entry order, so every sum is the same
// sequence of roundings as one thread's; an idle lane's term is +0, which
// leaves a sum that started at +0 (or above) unchanged.
//
// The terms cross lanes through shared memory, not shuffles: K 8-byte stores
// and G / 2 16-byte loads a round, against 2 shuffles a value and component
// and the selects of a transpose. The words of one warp are double-buffered,
// so a round needs one warp barrier.
#pragma once

#include "lane_rules.cuh"
#include "wcsph_device.cuh"

namespace pe {

constexpr uint32_t kFullWarp = 0xffffffffu;

template <int G>
struct LaneGroup {
    static constexpr uint32_t kPerWarp = 32u / G;
    uint32_t sub, grp, warp, slot;  // lane in group, group in warp, warp in CTA, the group's slot
    __device__ __forceinline__ LaneGroup()
        : sub(threadIdx.x % G), grp((threadIdx.x & 31u) / G), warp(threadIdx.x >> 5),
          slot(lane_slot<G>(blockIdx.x, blockDim.x, threadIdx.x)) {}
    // this group's bits of a warp ballot
    __device__ __forceinline__ uint32_t bits(uint32_t ballot) const {
        return G == 32 ? ballot : (ballot >> (grp * G)) & ((1u << (G % 32)) - 1u);
    }
    // sum over the group's lanes, on each of them
    __device__ __forceinline__ uint32_t sum(uint32_t v) const {
#pragma unroll
        for (uint32_t o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(kFullWarp, v, o);
        return v;
    }
};

// K ordered sums per group (K <= G); lane k < K of the group holds sum k.
template <int G, int K>
struct OrderedSum {
    static_assert(K <= G, "a lane a sum");
    // Terms t and t + 1 of a component form one 16-byte word; the words of one
    // pair index (a plane) are adjacent over groups and components, and planes
    // are padded so that a half warp's stores fall into different banks.
    static constexpr uint32_t kRow = 2u * (32u / G) * K;
    static constexpr uint32_t kPlane = kRow + (G == 4 ? 8u : G == 8 ? (K == 1 || K == 3 ? 12u : 4u) : 0u);
    static constexpr uint32_t kBuf = (G / 2) * kPlane;
    static constexpr uint32_t kDoubles = 2u * kBuf;  // per warp
    double acc;
    double *put, *get;
    uint32_t flip;
    bool adds;
    __device__ __forceinline__ OrderedSum(double* warp_words, const LaneGroup<G>& g, double start)
        : acc(start),
          put(warp_words + (g.sub >> 1) * kPlane + 2u * (g.grp * K) + (g.sub & 1u)),
          get(warp_words + 2u * (g.grp * K + min(g.sub, (uint32_t)K - 1u))), flip(0u), adds(g.sub < (uint32_t)K) {}
    __device__ __forceinline__ OrderedSum(double* warp_words, const LaneGroup<G>& g, const double (&start)[K])
        : OrderedSum(warp_words, g, 0.0) {
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (g.sub == (uint32_t)k) acc = start[k];
    }
    // Adds this round's G terms to each sum in lane order. Every lane of the
    // warp calls it.
    __device__ __forceinline__ void add(const double (&t)[K]) {
        double* const p = put + flip;
#pragma unroll
        for (int k = 0; k < K; ++k) p[2 * k] = t[k];
        __syncwarp();
        if (adds) {
            const double* const q = get + flip;
#pragma unroll
            for (int j = 0; j < G / 2; ++j) {
                const double2 v = *reinterpret_cast<const double2*>(q + j * kPlane);
                acc += v.x;
                acc += v.y;
            }
        }
        flip = kBuf - flip;
    }
    // Every sum, on each lane of the group. Every lane of the warp calls it.
    __device__ __forceinline__ void totals(double (&r)[K]) const {
#pragma unroll
        for (int k = 0; k < K; ++k) r[k] = __shfl_sync(kFullWarp, acc, k, G);
    }
};

// One lane a slot: the sums are its own.
template <int K>
struct OrderedSum<1, K> {
    static constexpr uint32_t kDoubles = 0u;
    double acc[K];
    __device__ __forceinline__ OrderedSum(double*, const LaneGroup<1>&, double start) {
#pragma unroll
        for (int k = 0; k < K; ++k) acc[k] = start;
    }
    __device__ __forceinline__ OrderedSum(double*, const LaneGroup<1>&, const double (&start)[K]) {
#pragma unroll
        for (int k = 0; k < K; ++k) acc[k] = start[k];
    }
    __device__ __forceinline__ void add(const double (&t)[K]) {
#pragma unroll
        for (int k = 0; k < K; ++k) acc[k] += t[k];
    }
    __device__ __forceinline__ void totals(double (&r)[K]) const {
#pragma unroll
        for (int k = 0; k < K; ++k) r[k] = acc[k];
    }
};

__device__ __forceinline__ uint32_t warp_rounds(uint32_t n, uint32_t lanes) {
    return __reduce_max_sync(kFullWarp, (n + lanes - 1u) / lanes);
}

// A group's lanes walk a list together: round r hands lane `sub` entry
// r * G + sub. A lane past the list's end keeps reading its last valid entry
// (slot 0 for an empty list), so that no load sits behind a branch: waiting for
// loads at the branches' joins made the walk wait on every gather in turn.
template <int G>
struct GroupWalk {
    const uint32_t* p;
    uint32_t step;  // between rounds (u32 units; one lane: from a row's end to the next row)
    uint32_t t, n;
    __device__ __forceinline__ GroupWalk(const ListRef& r, uint32_t sub)
        : p(r.p + (sub < r.n ? (size_t)(sub >> 2) * r.step + (sub & 3u) : 0u)),
          step(G == 1 ? r.step - 3u : (G / 4) * r.step), t(sub), n(r.n) {}
    __device__ __forceinline__ bool has() const { return t < n; }
    __device__ __forceinline__ uint32_t peek() const {
        const uint32_t e = __ldg(p);
        return n ? e : 0u;
    }
    __device__ __forceinline__ void advance() {
        t += G;
        if (t < n) p += G > 1 || (t & 3u) == 0u ? step : 1u;  // one lane: along the row, then to the next
    }
};

// Calls f(has, entry, data) once a round on every lane of the warp, over the
// longest list of its groups: has says whether the lane holds an entry of its
// own, data = load(entry, pointer to the entry) was issued a round ahead.
template <int G, class Load, class F>
__device__ __forceinline__ void group_for_each(const ListRef& r, const LaneGroup<G>& g, Load&& load, F&& f) {
    const uint32_t rounds = warp_rounds(r.n, G);
    if (!rounds) return;
    GroupWalk<G> w(r, g.sub);
    bool h0 = w.has();
    uint32_t e0 = w.peek();
    const uint32_t* p0 = w.p;
    auto d0 = load(e0, p0);
    w.advance();
    bool h1 = w.has();
    uint32_t e1 = w.peek();
    for (uint32_t u = 0; u < rounds; ++u) {
        const uint32_t e = e0;
        const uint32_t* const p = p0;
        const bool h = h0;
        const auto d = d0;
        e0 = e1;
        h0 = h1;
        p0 = w.p;
        d0 = load(e0, p0);
        w.advance();
        h1 = w.has();
        e1 = w.peek();
        f(h, e, d, p);
    }
}

}  // namespace pe

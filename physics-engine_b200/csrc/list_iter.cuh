// Walking a slot's neighbour list in order (see ListRef), shared by the SPH
// passes of every solver.
#pragma once

#include "wcsph_device.cuh"

namespace pe {

// One 32-byte load of a neighbour's state (double4 arrays are 32-byte aligned:
// each is an allocation of its own), where the compiler makes two of 16.
__device__ __forceinline__ double4 gather4(const double4* p) {
    double4 v;
    asm("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
    return v;
}

// Four doubles at a 32-byte boundary in one access.
__device__ __forceinline__ void load4(const double* p, double (&v)[4]) {
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}
__device__ __forceinline__ void store4(double* p, const double (&v)[4]) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3])
                 : "memory");
}

// Walks a slot's list a row (four entries, one 16-byte read) at a time: calls
// begin(row), then pair(q, entry, data) for the row's entries q = 0..3 in
// order (fewer in the last row), then end(row). data = load(entry) is issued
// DEPTH (1 or 2) entries ahead; the four steps are written out, so that
// neither entries nor data move between registers. Rows are read two ahead.
template <int DEPTH, class Load, class Begin, class Pair, class End>
__device__ __forceinline__ void for_each_row(const ListRef r, Load&& load, Begin&& begin, Pair&& pair, End&& end) {
    const uint32_t rows = (r.n + 3u) >> 2;
    if (rows == 0) return;
    const uint4* p = reinterpret_cast<const uint4*>(r.p);
    const uint32_t step = r.step >> 2;
    uint4 cur = __ldg(p), nxt = cur;
    if (rows > 1) {
        p += step;
        nxt = __ldg(p);
    }
    // entries past the list's end repeat its first one
    const uint32_t first = cur.x;
    auto trim = [&](uint4& e, uint32_t row) {
        const uint32_t left = r.n - 4u * row;
        if (left < 4u) {
            e.w = first;
            if (left < 3u) e.z = first;
            if (left < 2u) e.y = first;
        }
    };
    trim(cur, 0u);
    auto d0 = load(cur.x);
    auto d1 = d0;
    if (DEPTH == 2) d1 = load(cur.y);
    for (uint32_t row = 0; row < rows; ++row) {
        const uint32_t left = r.n - 4u * row;
        const uint4 e = cur;
        if (row + 1u < rows) {
            cur = nxt;
            trim(cur, row + 1u);
        }
        if (row + 2u < rows) {
            p += step;
            nxt = __ldg(p);
        }
        begin(row);
        if (DEPTH == 2) {
            auto d2 = load(e.z);
            pair(0u, e.x, d0);
            auto d3 = load(e.w);
            if (left > 1u) pair(1u, e.y, d1);
            d0 = load(cur.x);
            if (left > 2u) pair(2u, e.z, d2);
            d1 = load(cur.y);
            if (left > 3u) pair(3u, e.w, d3);
        } else {
            d1 = load(e.y);
            pair(0u, e.x, d0);
            d0 = load(e.z);
            if (left > 1u) pair(1u, e.y, d1);
            d1 = load(e.w);
            if (left > 2u) pair(2u, e.z, d0);
            d0 = load(cur.x);
            if (left > 3u) pair(3u, e.w, d1);
        }
        end(row);
    }
}

// Calls f(entry) over a slot's list in order, with the loads of the next two
// entries issued before the current one is processed.
template <class F>
__device__ __forceinline__ void for_each_entry(const ListRef r, F&& f) {
    const uint32_t n = r.n;
    if (n == 0) return;
    auto at = [&](uint32_t t) { return __ldg(r.p + (size_t)(t >> 2) * r.step + (t & 3u)); };
    uint32_t e0 = at(0), e1 = n > 1 ? at(1) : 0u;
    for (uint32_t t = 0; t < n; ++t) {
        const uint32_t e = e0;
        e0 = e1;
        if (t + 2 < n) e1 = at(t + 2);
        f(e);
    }
}

// Calls f(t, entry, data) over a slot's list in order (t the entry's
// position), where data = load(t, entry) is issued one entry ahead: the
// gather of the next neighbour's state is in flight while the current pair
// is computed. load sees t = 0, 1, 2, ... in order.
template <class Load, class F>
__device__ __forceinline__ void for_each_loaded_t(const ListRef r, Load&& load, F&& f) {
    const uint32_t n = r.n;
    if (n == 0) return;
    auto at = [&](uint32_t t) { return __ldg(r.p + (size_t)(t >> 2) * r.step + (t & 3u)); };
    uint32_t e0 = at(0), e1 = n > 1 ? at(1) : 0u;
    auto d0 = load(0u, e0);
    for (uint32_t t = 0; t < n; ++t) {
        const uint32_t e = e0;
        const auto d = d0;
        if (t + 1 < n) {
            e0 = e1;
            d0 = load(t + 1, e1);
            if (t + 2 < n) e1 = at(t + 2);
        }
        f(t, e, d);
    }
}

// for_each_loaded_t without the positions.
template <class Load, class F>
__device__ __forceinline__ void for_each_loaded(const ListRef r, Load&& load, F&& f) {
    for_each_loaded_t(
        r, [&](uint32_t, uint32_t e) { return load(e); },
        [&](uint32_t, uint32_t e, const auto& d) { f(e, d); });
}

// Calls f(t, entry, data) over a slot's list in order (t the entry's
// position), data = load(t, entry), with the data of the next two entries in
// flight.
template <class Load, class F>
__device__ __forceinline__ void for_each_loaded2_t(const ListRef r, Load&& load, F&& f) {
    const uint32_t n = r.n;
    if (n == 0) return;
    auto at = [&](uint32_t t) { return __ldg(r.p + (size_t)(t >> 2) * r.step + (t & 3u)); };
    uint32_t e0 = at(0), e1 = n > 1 ? at(1) : 0u, e2 = n > 2 ? at(2) : 0u;
    auto d0 = load(0u, e0);
    auto d1 = n > 1 ? load(1u, e1) : d0;
    for (uint32_t t = 0; t < n; ++t) {
        const uint32_t e = e0;
        const auto d = d0;
        e0 = e1;
        d0 = d1;
        if (t + 2 < n) {
            e1 = e2;
            d1 = load(t + 2, e2);
            if (t + 3 < n) e2 = at(t + 3);
        }
        f(t, e, d);
    }
}

// for_each_loaded with the data of the next two entries in flight.
template <class Load, class F>
__device__ __forceinline__ void for_each_loaded2(const ListRef r, Load&& load, F&& f) {
    for_each_loaded2_t(
        r, [&](uint32_t, uint32_t e) { return load(e); },
        [&](uint32_t, uint32_t e, const auto& d) { f(e, d); });
}

}  // namespace pe

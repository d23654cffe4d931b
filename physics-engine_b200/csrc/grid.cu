// Deterministic uniform-grid build (replaces `UniformGrid::rebuild`,
// crates/pe-fluid/src/grid.rs:76-107, and `key_of`, grid.rs:62).
//
// The reference sorts particle indices by (CellKey, index) with a comparison
// sort. Here the same total order is produced by a counting sort over a dense
// key box: cell ids are computed with the reference's exact floor_i32 rule,
// counted with warp-aggregated atomics, scanned, placed with warp-aggregated
// atomics, and each cell's run is then ranked by original index so that the
// within-cell order is ascending original index, exactly as the reference's
// tie-break. The dense linearisation is ix-major, so ascending linear cell id
// equals ascending CellKey (the derived Ord on {ix, iy, iz}).
//
// Four launches, no memset: small worlds wait on launches and on nothing else
// (930 particles: with seven launches and two memsets a step took 116 us, now 92;
// 16,000 in 2-D 146 and 127; 57,570 487 and 457).
// The counting pass keeps each slot's rank in its cell, so that placing needs no
// second round of atomics, and adds up the scan's tiles, so that the scan is one
// pass (two beyond kFlatTiles tiles); the scan clears the counts and the placing
// pass the tiles for the next build; a slot's thread finds its place in its cell
// and moves the state there.
#include "pe_math.cuh"
#include "wcsph_device.cuh"

namespace pe {

namespace {

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr uint32_t kScanTile = kScanThreads * kScanItems;
// Up to this many tiles each adds up the ones before it; beyond, where that sum
// would be quadratic in the cells, one block scans the tiles' sums first. us a
// build of 8,000 particles, flat / scanned first: 2.0M cells 32 / 35, 3.9M 40 / 41,
// 8.2M 58 / 56, 33M 160 / 145, 130M 628 / 462, 267M 1534 / 900 (a batch of tanks
// may have 2^31).
constexpr uint32_t kFlatTiles = 1536;

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

// count and tiles are zero on entry. tiles[t] holds the particles (low word) and
// occupied cells (high word) of the scan's tile t.
__global__ void k_cell_ids(GridDesc g, Tanks tk, uint32_t n, const double4* __restrict__ pos_cur,
                           const double4* __restrict__ pos_next, const uint8_t* __restrict__ flags,
                           uint32_t* __restrict__ cellid, int4* __restrict__ key_tmp,
                           uint32_t* __restrict__ count, uint32_t* __restrict__ rank,
                           unsigned long long* __restrict__ tiles, DeviceScalars* sc) {
    uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    bool active = s < n;
    uint32_t c = 0;
    if (active) {
        bool boundary = flags[s] & kFlagBoundary;
        double4 p = (pos_next != nullptr && !boundary) ? pos_next[s] : pos_cur[s];
        // grid.rs:63-70: inv = 1.0 / cell_size; key = floor_i32(p * inv)
        int32_t ix = floor_i32(p.x * g.inv_cell);
        int32_t iy = floor_i32(p.y * g.inv_cell);
        int32_t iz = g.dim == 2 ? 0 : floor_i32(p.z * g.inv_cell);
        if (!isfinite(p.x) || !isfinite(p.y) || (g.dim == 3 && !isfinite(p.z)))
            atomicOr(&sc->status, kStatusNonFinite);
        key_tmp[s] = make_int4(ix, iy, iz, 0);
        // the box of this slot's tank (slots keep their tank across re-sorts)
        TankDesc td;
        if (tk.desc) {
            td = tk.desc[tk.slot_tank[s]];
        } else {
            td.kx0 = g.kx0;
            td.ky0 = g.ky0;
            td.kz0 = g.kz0;
            td.nx = g.nx;
            td.ny = g.ny;
            td.nz = g.nz;
            td.cell_base = 0;
        }
        long long dx = (long long)ix - td.kx0, dy = (long long)iy - td.ky0, dz = (long long)iz - td.kz0;
        if (dx < 0 || dy < 0 || dz < 0 || dx >= td.nx || dy >= td.ny || dz >= td.nz) {
            atomicOr(&sc->status, kStatusDomain);
            dx = dx < 0 ? 0 : (dx >= td.nx ? td.nx - 1 : dx);
            dy = dy < 0 ? 0 : (dy >= td.ny ? td.ny - 1 : dy);
            dz = dz < 0 ? 0 : (dz >= td.nz ? td.nz - 1 : dz);
        }
        c = td.cell_base + (uint32_t)((dx * td.ny + dy) * td.nz + dz);
        cellid[s] = c;
    }
    unsigned mask = __ballot_sync(0xffffffffu, active);
    if (!active) return;
    const unsigned peers = __match_any_sync(mask, c);
    const int leader = __ffs(peers) - 1;
    const bool leads = (int)lane_id() == leader;
    uint32_t base = 0;
    if (leads) base = atomicAdd(&count[c], (uint32_t)__popc(peers));
    const unsigned opened = __ballot_sync(mask, leads && base == 0u);  // cells that were empty
    base = __shfl_sync(mask, base, leader);
    rank[s] = base + __popc(peers & ((1u << lane_id()) - 1u));
    const uint32_t t = c / kScanTile;
    const unsigned same = __match_any_sync(mask, t);
    if ((int)lane_id() == __ffs(same) - 1)
        atomicAdd(&tiles[t], (unsigned long long)__popc(same) | ((unsigned long long)__popc(same & opened) << 32));
}

// Block-wide exclusive scan of (a, b) pairs with warp shuffles.
__device__ __forceinline__ void block_scan2(uint32_t a, uint32_t b, uint32_t* ea, uint32_t* eb,
                                            uint32_t* ta, uint32_t* tb) {
    __shared__ uint32_t wa[32], wb[32];
    uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    uint32_t ia = a, ib = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t xa = __shfl_up_sync(0xffffffffu, ia, o);
        uint32_t xb = __shfl_up_sync(0xffffffffu, ib, o);
        if ((int)lane >= o) { ia += xa; ib += xb; }
    }
    if (lane == 31) { wa[warp] = ia; wb[warp] = ib; }
    __syncthreads();
    if (warp == 0) {
        uint32_t nw = blockDim.x >> 5;
        uint32_t va = lane < nw ? wa[lane] : 0u, vb = lane < nw ? wb[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t xa = __shfl_up_sync(0xffffffffu, va, o);
            uint32_t xb = __shfl_up_sync(0xffffffffu, vb, o);
            if ((int)lane >= o) { va += xa; vb += xb; }
        }
        wa[lane] = va;
        wb[lane] = vb;
    }
    __syncthreads();
    uint32_t pa = warp ? wa[warp - 1] : 0u, pb = warp ? wb[warp - 1] : 0u;
    *ea = pa + ia - a;
    *eb = pb + ib - b;
    *ta = wa[(blockDim.x >> 5) - 1];
    *tb = wb[(blockDim.x >> 5) - 1];
    __syncthreads();
}

// Each tile's sum becomes that of the tiles before it (one block).
__global__ void k_scan_tiles(uint32_t ntiles, unsigned long long* __restrict__ tiles) {
    uint32_t carry_a = 0, carry_b = 0;
    for (uint32_t off = 0; off < ntiles; off += kScanTile) {
        const uint32_t first = off + threadIdx.x * kScanItems;
        unsigned long long v[kScanItems];
        uint32_t a = 0, b = 0;
#pragma unroll
        for (int i = 0; i < kScanItems; ++i) {
            v[i] = first + i < ntiles ? tiles[first + i] : 0ull;
            a += (uint32_t)v[i];
            b += (uint32_t)(v[i] >> 32);
        }
        uint32_t ea, eb, ta, tb;
        block_scan2(a, b, &ea, &eb, &ta, &tb);
        ea += carry_a;
        eb += carry_b;
#pragma unroll
        for (int i = 0; i < kScanItems; ++i) {
            if (first + i < ntiles) tiles[first + i] = (unsigned long long)ea | ((unsigned long long)eb << 32);
            ea += (uint32_t)v[i];
            eb += (uint32_t)(v[i] >> 32);
        }
        carry_a += ta;
        carry_b += tb;
    }
}

// cell_start (exclusive) and the list of occupied cells in linear order; each
// tile adds up the ones before it, or with `summed` reads their sum. Clears count.
// clear_lists: a list build and its density pass follow, their counters are
// cleared too.
__global__ void k_scan(uint32_t ncell, uint32_t* __restrict__ count, const unsigned long long* __restrict__ tiles,
                       bool summed, uint32_t* __restrict__ cell_start, uint32_t* __restrict__ occ, DeviceScalars* sc,
                       int clear_lists) {
    uint32_t before_a, before_b;
    if (summed) {
        const unsigned long long v = tiles[blockIdx.x];
        before_a = (uint32_t)v;
        before_b = (uint32_t)(v >> 32);
    } else {
        uint32_t pa = 0, pb = 0, ea, eb;
        for (uint32_t t = threadIdx.x; t < blockIdx.x; t += kScanThreads) {
            const unsigned long long v = tiles[t];
            pa += (uint32_t)v;
            pb += (uint32_t)(v >> 32);
        }
        block_scan2(pa, pb, &ea, &eb, &before_a, &before_b);
    }
    uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    uint32_t a = 0, b = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        uint32_t c = base + i;
        v[i] = c < ncell ? count[c] : 0u;
        if (v[i]) count[c] = 0u;
        a += v[i];
        b += v[i] != 0u;
    }
    uint32_t ea, eb, ta, tb;
    block_scan2(a, b, &ea, &eb, &ta, &tb);
    uint32_t ra = before_a + ea, rb = before_b + eb;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        uint32_t c = base + i;
        if (c < ncell) {
            cell_start[c] = ra;
            if (v[i]) occ[rb++] = c;
            ra += v[i];
        }
    }
    // The thread that owns the last cell writes the end sentinel.
    if (ncell > 0 && base <= ncell - 1 && ncell - 1 < base + kScanItems) {
        cell_start[ncell] = ra;
        sc->nocc = rb;
        if (clear_lists) {
            sc->list_used = 0ull;
            sc->w_short = 0u;
        }
    }
}

// Slots by cell, in any order within it. Clears tiles.
__global__ void k_place(uint32_t n, const uint32_t* __restrict__ cellid, const uint32_t* __restrict__ rank,
                        const uint32_t* __restrict__ cell_start, const uint32_t* __restrict__ orig,
                        uint2* __restrict__ placed, unsigned long long* __restrict__ tiles, uint32_t ntiles) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t t = s; t < ntiles; t += gridDim.x * blockDim.x) tiles[t] = 0ull;
    if (s >= n) return;
    placed[cell_start[cellid[s]] + rank[s]] = make_uint2(orig[s], s);
}

// The place of the k-th placed slot: its cell's run is ordered by original index
// (unique; grid.rs:86-87 tie-break).
__device__ __forceinline__ uint32_t sorted_place(uint32_t k, const uint2* __restrict__ placed,
                                                 const uint32_t* __restrict__ cellid,
                                                 const uint32_t* __restrict__ cell_start, uint32_t* old) {
    const uint2 me = placed[k];
    const uint32_t c = cellid[me.y];
    const uint32_t b = cell_start[c], e = cell_start[c + 1];
    uint32_t at = b;
#pragma unroll 4
    for (uint32_t j = b; j < e; ++j) at += placed[j].x < me.x;
    *old = me.y;
    return at;
}

__global__ void k_order(uint32_t n, const uint2* __restrict__ placed, const uint32_t* __restrict__ cellid,
                        const uint32_t* __restrict__ cell_start, uint32_t* __restrict__ perm) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    uint32_t old;
    const uint32_t s = sorted_place(k, placed, cellid, cell_start, &old);
    perm[s] = old;
}

__global__ void k_move(uint32_t n, const uint2* __restrict__ placed, const uint32_t* __restrict__ cellid,
                       const uint32_t* __restrict__ cell_start, StateBufs src, const double4* __restrict__ pos_next,
                       const double4* __restrict__ vel_next, const int4* __restrict__ key_tmp, StateBufs dst,
                       uint32_t* __restrict__ slot_of_orig) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    uint32_t old;
    const uint32_t s = sorted_place(k, placed, cellid, cell_start, &old);
    uint8_t fl = src.flags[old];
    bool moved = !(fl & kFlagBoundary);
    dst.pos[s] = (moved && pos_next) ? pos_next[old] : src.pos[old];
    dst.vel[s] = (moved && vel_next) ? vel_next[old] : src.vel[old];
    dst.acc[s] = src.acc[old];
    dst.bf[s] = src.bf[old];
    dst.p[s] = src.p[old];
    dst.flags[s] = fl;
    uint32_t o = src.orig[old];
    dst.orig[s] = o;
    dst.nout[s] = src.nout[old];
    dst.key[s] = key_tmp[old];
    slot_of_orig[o] = s;
}

__global__ void k_occupied_export(const uint32_t* __restrict__ occ, const DeviceScalars* sc,
                                  const uint32_t* __restrict__ cell_start,
                                  const int4* __restrict__ key, int32_t* __restrict__ occ_keys,
                                  uint64_t* __restrict__ ranges) {
    uint32_t nocc = sc->nocc;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nocc; i += gridDim.x * blockDim.x) {
        uint32_t c = occ[i];
        uint32_t a = cell_start[c], b = cell_start[c + 1];
        int4 k = key[a];
        occ_keys[3 * (size_t)i] = k.x;
        occ_keys[3 * (size_t)i + 1] = k.y;
        occ_keys[3 * (size_t)i + 2] = k.z;
        ranges[2 * (size_t)i] = a;
        ranges[2 * (size_t)i + 1] = b;
    }
}

inline uint32_t blocks_for(uint64_t n, uint32_t t) { return (uint32_t)((n + t - 1) / t); }

}  // namespace

size_t scan_tiles_bytes(uint32_t ncell) {
    return sizeof(unsigned long long) * (size_t)((ncell + kScanTile - 1) / kScanTile + 1);
}

uint32_t launch_cell_sort(const GridDesc& g, const Tanks& tk, uint32_t n, const double4* pos_cur,
                          const double4* pos_next, const uint8_t* flags, const uint32_t* orig, const GridBufs& b,
                          DeviceScalars* sc, bool clear_lists, cudaStream_t st) {
    const uint32_t ntiles = (g.ncell + kScanTile - 1) / kScanTile, nb = blocks_for(n, 256);
    if (n)
        k_cell_ids<<<nb, 256, 0, st>>>(g, tk, n, pos_cur, pos_next, flags, b.cellid, b.key_tmp, b.count, b.rank,
                                       b.tiles, sc);
    const bool summed = ntiles > kFlatTiles;
    if (summed) k_scan_tiles<<<1, kScanThreads, 0, st>>>(ntiles, b.tiles);
    k_scan<<<ntiles, kScanThreads, 0, st>>>(g.ncell, b.count, b.tiles, summed, b.cell_start, b.occ, sc,
                                            clear_lists ? 1 : 0);
    if (n) k_place<<<nb, 256, 0, st>>>(n, b.cellid, b.rank, b.cell_start, orig, b.placed, b.tiles, ntiles);
    return summed ? 4u : 3u;
}

void launch_order(uint32_t n, const GridBufs& b, uint32_t* perm, cudaStream_t st) {
    if (n) k_order<<<blocks_for(n, 256), 256, 0, st>>>(n, b.placed, b.cellid, b.cell_start, perm);
}

void launch_move(uint32_t n, const GridBufs& b, const StateBufs& src, const double4* pos_next,
                 const double4* vel_next, const StateBufs& dst, uint32_t* slot_of_orig, cudaStream_t st) {
    if (n)
        k_move<<<blocks_for(n, 256), 256, 0, st>>>(n, b.placed, b.cellid, b.cell_start, src, pos_next, vel_next,
                                                  b.key_tmp, dst, slot_of_orig);
}

void launch_occupied_export(const GridDesc& g, const uint32_t* occ, const DeviceScalars* sc,
                            const uint32_t* cell_start, const int4* key, int32_t* occ_keys,
                            uint64_t* ranges, cudaStream_t st) {
    uint32_t blocks = blocks_for(g.ncell, 256);
    if (blocks > 148u * 8u) blocks = 148u * 8u;
    if (blocks == 0) blocks = 1;
    k_occupied_export<<<blocks, 256, 0, st>>>(occ, sc, cell_start, key, occ_keys, ranges);
}

}  // namespace pe

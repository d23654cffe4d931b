// Fused edge MLP of one message-passing hop, for inference (the learned
// step): for every edge e = (i <- j) of the message graph (edges sorted by
// destination)
//
//   z1  = relu(x_e Wc + b1 + P[i] + Q[j])      P = h Wa, Q = h Wb (per node)
//   z2  = relu(z1 W2 + b2)
//   m_e = z2 W3 + b3
//   out[i] += m_e
//
// which the unfused path computes as three GEMM launches writing E x 128
// activations to memory (~60 GB of traffic per hop at 3.3e7 edges) and a
// segment sum. Here one persistent CTA per SM keeps Wc, W2 and W3 in shared
// memory; its four warpgroups walk their own tiles of 128 edges, each with its
// own 128 tensor-memory columns, buffers and barriers, so one group's MMA
// waits and gathers overlap the others' epilogues.
//
// The layers are computed transposed: the weights are the MMAs' A operand (128
// features), the tile's edges the N dimension, so that a thread holds one
// feature of all its edges. Then a warp reads 128 contiguous bytes of Q[j] for
// each edge, P[i] once a run of equal destinations, biases stay in registers,
// and the messages of a run are summed in registers, one atomic add per run,
// block of 32 edges and column. Per tile, Wc^T x_e^T is one K = 16 MMA; the
// epilogue adds b1, P[i] and Q[j] in the unfused epilogue's order (the next
// sixteen edges' Q, the next four runs' P and the next tile's endpoints and
// features are already loading), applies ReLU and writes bf16 into a swizzled
// tile, a row of edges for each feature, that is the N-major B operand of the
// next 8 MMAs (K = 128), and so on. Activations are rounded to bf16 at the
// same points as in the unfused path; only the message sum's order differs.
//
// A tile is one long chain (copy, MMA, epilogue, MMA, ...), so what counts is how
// many run on an SM. 2.56M edges, a hop: 1.72 ms with two groups and a thread an
// edge (each reading its own rows of P and Q); 0.74 with four, the shared-memory
// and L1 path 78% busy; 0.49 with a thread a feature, that path 35%, the ALU 47%
// (loops over the blocks unrolled, the instruction cache missed: 0.65).
//
// Every mbarrier wait is bounded; a wait that runs out sets bit 0 of *err and
// ends the tile loop of the whole CTA (at the tile's end, by a block-wide
// vote), and the CTA still waits (bounded) for its committed MMAs before
// freeing its tensor memory.
#include <cuda_bf16.h>
#include <cstdint>

#include "mlp.cuh"
#include "umma_tile.cuh"

namespace pe {

namespace {

using namespace umma;

constexpr int kGroups = 4;             // warpgroups per CTA, each on its own tiles
constexpr int kEdgeThreads = kGroups * kGroupThreads;
constexpr uint32_t kOffW2 = 0;                    // W2^T [128 x 128]: two slices
constexpr uint32_t kOffW3 = kOffW2 + 2 * kSlice;  // W3^T: two slices
// Matrices of 16 columns (two 16-byte chunks a row) share slices, four to one:
// matrix m in chunks 2 (m % 4) and 2 (m % 4) + 1 of slice m / 4. Matrix 0 is
// Wc^T [128 x 16], matrix 1 + g group g's edge features [128 x 16].
constexpr uint32_t kOffNarrow = kOffW3 + 2 * kSlice;
constexpr uint32_t kNarrowSlices = (1 + kGroups + 3) / 4;
// per group the activation tile: a slice for 64 edges, 128 bytes of them for each feature
constexpr uint32_t kOffGroup = kOffNarrow + kNarrowSlices * kSlice;
constexpr uint32_t kGroupBytes = 2 * kSlice;
constexpr uint32_t kSmemBytes = kOffGroup + kGroups * kGroupBytes + 1024u;  // + alignment slack
static_assert(kSmemBytes + 2048u <= 232448u, "one CTA's shared memory, with its barriers");

// 128 edges' activations (MN-major: a row of 128 edges for each feature) times W
__device__ __forceinline__ void issue_edges(uint32_t tmem, const uint8_t* sW, const uint8_t* sZ) {
    const uint32_t a0 = smem_addr(sW), b0 = smem_addr(sZ);
#pragma unroll
    for (int kk = 0; kk < 8; ++kk)
        umma_bf16<kTileN, true>(tmem, sw128_desc(a0 + (uint32_t)(kk >> 2) * kSlice + (kk & 3) * 32),
                                sw128_mn_desc(b0 + kk * 2048u, kSlice), kk ? 1u : 0u);
}

// N values of feature `row` for the edges from e0 on, as bf16
template <int N>
__device__ __forceinline__ void put_edges(uint8_t* sZ, int row, int e0, const float (&x)[N]) {
#pragma unroll
    for (int q = 0; q < N / 8; ++q) {
        uint32_t w[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const __nv_bfloat162 b = __floats2bfloat162_rn(x[q * 8 + 2 * h], x[q * 8 + 2 * h + 1]);
            w[h] = *reinterpret_cast<const uint32_t*>(&b);
        }
        const int c = e0 / 8 + q;  // 16-byte chunk of the feature's edges
        *reinterpret_cast<uint4*>(sZ + (uint32_t)(c >> 3) * kSlice + sw_off(row, c & 7)) =
            make_uint4(w[0], w[1], w[2], w[3]);
    }
}

__global__ void __launch_bounds__(kEdgeThreads, 1) k_edge_hop(EdgeHopArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t mbar[kGroups];
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = tid / kGroupThreads, gt = tid % kGroupThreads, gw = gt >> 5;
    uint8_t* sWc = smem + kOffNarrow;
    uint8_t* sW2 = smem + kOffW2;
    uint8_t* sW3 = smem + kOffW3;
    uint8_t* sX = smem + kOffNarrow + (uint32_t)((g + 1) / 4) * kSlice;
    const int xc = 2 * ((g + 1) % 4);  // first chunk of the group's edge features in it
    uint8_t* sZ = smem + kOffGroup + (uint32_t)g * kGroupBytes;
    // endpoints of the tile's edges: sources 4 q .. 4 q + 3 in chunk 2 of row
    // 32 g + q of the second narrow slice, destinations in chunk 3
    uint8_t* const sEnd = smem + kOffNarrow + kSlice;
    auto ends = [&](int q, int which) { return sEnd + sw_off(32 * g + q, 2 + which); };

    if (tid == 0) {
        for (int i = 0; i < kGroups; ++i) mbar_init(smem_addr(&mbar[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)),
                     "r"(128u * kGroups)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // the weights stay in shared memory for every tile of the CTA
    stage_rows(sWc, a.Wc, 16, 2);
    stage_rows(sW2, a.W2, 128, 16);
    stage_rows(sW3, a.W3, 128, 16);
    const float b1 = __ldg(a.b1 + gt), b2 = __ldg(a.b2 + gt), b3 = __ldg(a.b3 + gt);  // this thread's feature
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem + 128u * (uint32_t)g;         // this group's 128 columns
    const uint32_t trow = tmem + ((uint32_t)(gw * 32) << 16);  // this warp's lanes (features)
    const uint32_t bar = smem_addr(&mbar[g]);

    bool ok = true;
    uint32_t phase = 0u;
    auto mma_wait = [&]() {
        const bool done = mbar_wait(bar, phase);
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        return done;
    };
    auto to_tensor = [&]() {  // generic-proxy shared writes visible to the MMAs, TMEM reads done
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        group_sync(g);
        if (gt == 0) asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    };
    const int ntiles = (a.E + kGroupThreads - 1) / kGroupThreads;
    const int stride = (int)gridDim.x * kGroups;
    // Edge gt of a tile: endpoints and its two 16-byte chunks of edge features, loaded one tile ahead.
    auto fetch_edge = [&](int tile, int& d, int& sj, uint4& x0, uint4& x1) {
        const int e = tile * kGroupThreads + gt;
        d = -1;
        sj = 0;
        x0 = x1 = make_uint4(0u, 0u, 0u, 0u);
        if (tile < ntiles && e < a.E) {
            d = __ldg(a.dst + e);
            sj = __ldg(a.src + e);
            x0 = __ldg(reinterpret_cast<const uint4*>(a.xe + (size_t)e * 16));
            x1 = __ldg(reinterpret_cast<const uint4*>(a.xe + (size_t)e * 16 + 8));
        }
    };
    // this feature of the Q rows of the sixteen edges from e0 on
    const float* const Qc = a.Q + gt;
    const float* const Pc = a.P + gt;
    auto fetch_q = [&](int e0, float (&q)[16]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int4 j = *reinterpret_cast<const int4*>(ends(e0 / 4 + i, 0));
            q[4 * i] = __ldg(Qc + (size_t)j.x * 128);
            q[4 * i + 1] = __ldg(Qc + (size_t)j.y * 128);
            q[4 * i + 2] = __ldg(Qc + (size_t)j.z * 128);
            q[4 * i + 3] = __ldg(Qc + (size_t)j.w * 128);
        }
    };
    // Destinations of a block of 32 edges, a lane an edge, and where a new one begins
    auto block_runs = [&](int b, int& dest) {
        dest = *reinterpret_cast<const int*>(ends(8 * b + (lane >> 2), 1) + 4 * (lane & 3));
        const int above = __shfl_up_sync(0xffffffffu, dest, 1);
        return __ballot_sync(0xffffffffu, lane == 0 || above != dest);
    };
    int d, sj;
    uint4 x0, x1;
    const int first = (int)blockIdx.x * kGroups + g;
    fetch_edge(first, d, sj, x0, x1);
    for (int tile = first; tile < ntiles; tile += stride) {
        // ---- edge features and endpoints of the tile (fetched a tile ahead)
        *reinterpret_cast<uint4*>(sX + sw_off(gt, xc)) = x0;
        *reinterpret_cast<uint4*>(sX + sw_off(gt, xc + 1)) = x1;
        *reinterpret_cast<int*>(ends(gt >> 2, 0) + 4 * (gt & 3)) = sj;
        *reinterpret_cast<int*>(ends(gt >> 2, 1) + 4 * (gt & 3)) = d;
        to_tensor();
        // ---- layer 1: x_e Wc (one K = 16 MMA), then + b1 + P[dst] + Q[src], ReLU
        if (gt == 0) {
            umma_bf16(tmem, sw128_desc(smem_addr(sWc)), sw128_desc(smem_addr(sX) + 16u * (uint32_t)xc), 0u);
            umma_commit(bar);
        }
        // the next tile's edge and the first edges' Q load while the MMA runs
        fetch_edge(tile + stride, d, sj, x0, x1);
        float qa[16], qb[16];
        fetch_q(0, qa);
        ok = mma_wait() && ok;
        float p = 0.f;  // P of the edge's destination
#pragma unroll 1
        for (int b = 0; b < 4; ++b) {
            int dest;
            uint32_t ahead = block_runs(b, dest);
            uint32_t heads = ahead;
            // P of the block's runs, the next four ahead
            auto next_p = [&]() {
                float v = 0.f;
                if (ahead) {
                    const int to = __shfl_sync(0xffffffffu, dest, __ffs(ahead) - 1);
                    ahead &= ahead - 1u;
                    v = __ldg(Pc + (size_t)max(to, 0) * 128);
                }
                return v;
            };
            float p0 = next_p(), p1 = next_p(), p2 = next_p(), p3 = next_p();
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int e0 = 32 * b + 16 * half;
                if (half == 0) fetch_q(e0 + 16, qb);
                else if (b < 3) fetch_q(e0 + 16, qa);
                float pv[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) pv[j] = p;
                for (uint32_t left = (heads >> (16 * half)) & 0xffffu; left; left &= left - 1u) {
                    const int k = __ffs(left) - 1;  // a run begins: its P from there on
                    p = p0;
                    p0 = p1;
                    p1 = p2;
                    p2 = p3;
                    p3 = next_p();
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (j >= k) pv[j] = p;
                }
                uint32_t v[16];
                tmem_ld16(trow + (uint32_t)e0, v);
                float x[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    float t = __uint_as_float(v[j]) + b1;  // the unfused epilogue's order
                    t += pv[j];
                    t += half ? qb[j] : qa[j];
                    x[j] = fmaxf(t, 0.f);
                }
                put_edges(sZ, gt, e0, x);
            }
        }
        to_tensor();
        // ---- layer 2: relu(z1 W2 + b2)
        if (gt == 0) {
            issue_edges(tmem, sW2, sZ);
            umma_commit(bar);
        }
        ok = mma_wait() && ok;
#pragma unroll 1
        for (int b = 0; b < 4; ++b) {
            uint32_t v[32];
            tmem_ld32(trow + (uint32_t)(b * 32), v);
            float x[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) x[j] = fmaxf(__uint_as_float(v[j]) + b2, 0.f);
            put_edges(sZ, gt, 32 * b, x);  // the MMAs that read sZ have completed
        }
        to_tensor();
        // ---- layer 3: m_e = z2 W3 + b3, summed per destination
        if (gt == 0) {
            issue_edges(tmem, sW3, sZ);
            umma_commit(bar);
        }
        ok = mma_wait() && ok;
#pragma unroll 1
        for (int b = 0; b < 4; ++b) {
            int dest;
            const uint32_t heads = block_runs(b, dest);
            uint32_t v[32];
            tmem_ld32(trow + (uint32_t)(b * 32), v);
            int to = -1;
            float acc = 0.f;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                if ((heads >> j) & 1u) {
                    if (j && to >= 0) atomicAdd(a.out + (size_t)to * 128 + gt, acc);
                    to = __shfl_sync(0xffffffffu, dest, j);  // -1 past the last edge
                    acc = 0.f;
                }
                acc += __uint_as_float(v[j]) + b3;
            }
            if (to >= 0) atomicAdd(a.out + (size_t)to * 128 + gt, acc);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        // the tile's TMEM reads and shared-memory use end before the group's
        // next tile; a run-out wait on any thread of the group stops the whole
        // group (a decision its threads share, so none is left at a barrier)
        ok = group_all(g, ok);
        if (!ok) break;
    }
    // every committed MMA completes before the tensor memory is freed
    if (gt == 0) umma_commit(bar);
    ok = mma_wait() && ok;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "r"(128u * kGroups)
                     : "memory");
    }
    if (!ok && gt == 0) atomicOr(a.err, 1u);
}

}  // namespace

bool edge_hop_prepare() {
    return cudaFuncSetAttribute(k_edge_hop, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes) ==
           cudaSuccess;
}

void launch_edge_hop(const EdgeHopArgs& a, int sms, cudaStream_t st) {
    if (a.E <= 0) return;
    const int ntiles = (a.E + kGroupThreads - 1) / kGroupThreads;
    const int ctas = (ntiles + kGroups - 1) / kGroups;
    const int grid = ctas < sms ? ctas : sms;
    k_edge_hop<<<grid, kEdgeThreads, kSmemBytes, st>>>(a);
}

}  // namespace pe

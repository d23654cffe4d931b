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
// waits and gathers overlap the others' epilogues. Per tile, x_e Wc is one
// K=16 tcgen05 MMA into the group's accumulator; the epilogue (thread r =
// edge r = TMEM lane r) adds b1, P[i] and Q[j] in the unfused epilogue's
// order (the next tile's endpoints and features, and the next 16-column block
// of P[i] and Q[j], are already loading), applies ReLU and
// writes bf16 into a swizzled shared-memory tile that is the A operand of
// the next 8 MMAs (K = 128), and so on; the last epilogue stages the
// messages in shared memory and sums each run of equal destinations before
// one atomic add per run and column. Activations are rounded to bf16 at the
// same points as in the unfused path; only the message sum's order differs.
//
// A tile is one long chain (copy, MMA, epilogue, MMA, ...), so what counts is how
// many run on an SM: with two groups, a third buffer and 32-column blocks in
// flight (16 KB more a group, twice the registers) 2.56M edges took 1.72 ms, with
// four 0.74. The shared-memory and L1 data path is 78% busy then, half of it the
// gathers of Q[j] and the messages' staging.
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
// per group the activation tile [128 x 128]; the last epilogue reuses it for
// fp32 messages, a warp's 32 rows x 32 columns in its own rows of a slice
constexpr uint32_t kOffGroup = kOffNarrow + kNarrowSlices * kSlice;
constexpr uint32_t kGroupBytes = 2 * kSlice;
constexpr uint32_t kSmemBytes = kOffGroup + kGroups * kGroupBytes + 1024u;  // + alignment slack
static_assert(kSmemBytes + 2048u <= 232448u, "one CTA's shared memory, with its biases and barriers");

__global__ void __launch_bounds__(kEdgeThreads, 1) k_edge_hop(EdgeHopArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t mbar[kGroups];
    __shared__ uint32_t s_tmem;
    __shared__ __align__(16) float s_bias[3][128];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = tid / kGroupThreads, gt = tid % kGroupThreads, gw = gt >> 5;
    uint8_t* sWc = smem + kOffNarrow;
    uint8_t* sW2 = smem + kOffW2;
    uint8_t* sW3 = smem + kOffW3;
    uint8_t* sX = smem + kOffNarrow + (uint32_t)((g + 1) / 4) * kSlice;
    const int xc = 2 * ((g + 1) % 4);  // first chunk of the group's edge features in it
    uint8_t* sA = smem + kOffGroup + (uint32_t)g * kGroupBytes;

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
    if (tid < 3 * 128) s_bias[tid >> 7][tid & 127] = __ldg((tid < 128 ? a.b1 : tid < 256 ? a.b2 : a.b3) + (tid & 127));
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem + 128u * (uint32_t)g;            // this group's 128 columns
    const uint32_t trow = tmem + ((uint32_t)(gw * 32) << 16);      // this warp's lanes (warp % 4)
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
    };
    const int ntiles = (a.E + kGroupThreads - 1) / kGroupThreads;
    const int stride = (int)gridDim.x * kGroups;
    // This thread's edge (row gt) of a tile: endpoints and its two 16-byte
    // chunks of edge features, loaded one tile ahead.
    auto fetch_edge = [&](int tile, int& d, int& sj, uint4& x0, uint4& x1) {
        const int e = tile * kGroupThreads + gt;
        d = -1;
        sj = -1;
        x0 = x1 = make_uint4(0u, 0u, 0u, 0u);
        if (tile < ntiles && e < a.E) {
            d = __ldg(a.dst + e);
            sj = __ldg(a.src + e);
            x0 = __ldg(reinterpret_cast<const uint4*>(a.xe + (size_t)e * 16));
            x1 = __ldg(reinterpret_cast<const uint4*>(a.xe + (size_t)e * 16 + 8));
        }
    };
    // 16 columns (block cb) of this edge's P[dst] and Q[src] rows
    auto fetch_pq = [&](int d, int sj, int cb, float4 (&p)[4], float4 (&q)[4]) {
        const float4* P4 = reinterpret_cast<const float4*>(a.P + (size_t)(d < 0 ? 0 : d) * 128 + cb * 16);
        const float4* Q4 = reinterpret_cast<const float4*>(a.Q + (size_t)(sj < 0 ? 0 : sj) * 128 + cb * 16);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            p[i] = __ldg(P4 + i);
            q[i] = __ldg(Q4 + i);
        }
    };
    int d, sj;
    uint4 x0, x1;
    const int first = (int)blockIdx.x * kGroups + g;
    fetch_edge(first, d, sj, x0, x1);
    for (int tile = first; tile < ntiles; tile += stride) {
        // ---- edge features and endpoints of the tile (fetched a tile ahead)
        *reinterpret_cast<uint4*>(sX + sw_off(gt, xc)) = x0;
        *reinterpret_cast<uint4*>(sX + sw_off(gt, xc + 1)) = x1;
        const int dc = d, sc = sj;
        to_tensor();
        // ---- layer 1: x_e Wc (one K = 16 MMA), then + b1 + P[dst] + Q[src], ReLU
        if (gt == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            umma_bf16(tmem, sw128_desc(smem_addr(sX) + 16u * (uint32_t)xc), sw128_desc(smem_addr(sWc)), 0u);
            umma_commit(bar);
        }
        // the next tile's edge and this edge's first P/Q block load while the MMA runs
        fetch_edge(tile + stride, d, sj, x0, x1);
        float4 pq[2][2][4];
        fetch_pq(dc, sc, 0, pq[0][0], pq[0][1]);
        ok = mma_wait() && ok;
#pragma unroll
        for (int cb = 0; cb < 8; ++cb) {
            const int now = cb & 1;
            if (cb < 7) fetch_pq(dc, sc, cb + 1, pq[now ^ 1][0], pq[now ^ 1][1]);  // one block ahead
            uint32_t v[16];
            tmem_ld16(trow + (uint32_t)(cb * 16), v);
            float x[16], bias[16];
            get_bias(s_bias[0] + cb * 16, bias);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 p4 = pq[now][0][i], q4 = pq[now][1][i];
                const float pv[4] = {p4.x, p4.y, p4.z, p4.w}, qv[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const int j = i * 4 + h;
                    float t = __uint_as_float(v[j]) + bias[j];  // the unfused epilogue's order
                    t += pv[h];
                    t += qv[h];
                    x[j] = fmaxf(t, 0.f);
                }
            }
            put_bf16_row(sA, gt, cb * 16, x);
        }
        to_tensor();
        // ---- layer 2: relu(z1 W2 + b2)
        if (gt == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            issue_k128(tmem, sA, sW2);
            umma_commit(bar);
        }
        ok = mma_wait() && ok;
#pragma unroll 1
        for (int cb = 0; cb < 4; ++cb) {
            uint32_t v[32];
            tmem_ld32(trow + (uint32_t)(cb * 32), v);
            float x[32], bias[32];
            get_bias(s_bias[1] + cb * 32, bias);
#pragma unroll
            for (int j = 0; j < 32; ++j) x[j] = fmaxf(__uint_as_float(v[j]) + bias[j], 0.f);
            put_bf16_row(sA, gt, cb * 32, x);  // the MMAs that read sA have completed
        }
        to_tensor();
        // ---- layer 3: m_e = z2 W3 + b3, summed per destination
        if (gt == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            issue_k128(tmem, sA, sW3);
            umma_commit(bar);
        }
        ok = mma_wait() && ok;
        // A warp sums its own 32 rows (rows past the last edge close the tile):
        // lane j column j, row by row, one atomic per run of a destination.
        const int rows = __popc(__ballot_sync(0xffffffffu, dc >= 0));
        const int above = __shfl_up_sync(0xffffffffu, dc, 1);
        const uint32_t heads = __ballot_sync(0xffffffffu, dc >= 0 && (lane == 0 || above != dc));
#pragma unroll 1
        for (int cb = 0; cb < 4; ++cb) {
            uint32_t v[32];
            tmem_ld32(trow + (uint32_t)(cb * 32), v);
            float bias[32];
            get_bias(s_bias[2] + cb * 32, bias);
            // column j of row r at j ^ r; blocks alternate between the slices, so
            // that one is read while the next is written
            float* const st = reinterpret_cast<float*>(sA + (uint32_t)(cb & 1) * kSlice + (uint32_t)gw * 4096u);
#pragma unroll
            for (int j = 0; j < 32; ++j) st[lane * 32 + (j ^ lane)] = __uint_as_float(v[j]) + bias[j];
            __syncwarp();
            for (uint32_t left = heads; left; left &= left - 1u) {
                const int r0 = __ffs(left) - 1, r1 = (left & (left - 1u)) ? __ffs(left & (left - 1u)) - 1 : rows;
                const int to = __shfl_sync(0xffffffffu, dc, r0);
                float acc = 0.f;
#pragma unroll 8
                for (int r = r0; r < r1; ++r) acc += st[r * 32 + (lane ^ r)];
                atomicAdd(a.out + (size_t)to * 128 + cb * 32 + lane, acc);
            }
        }
        __syncwarp();  // the next tile's activations go where the messages were
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

// The three layers of a node MLP in one kernel, for inference (the learned step):
//
//   z1 = relu(x W1 + b1)    x = node features, h, or (h, scale * messages)
//   z2 = relu(z1 W2 + b2)
//   y  = z2 W3 + b3         h = y, h += y on fluid nodes, or the outputs
//
// As three GEMMs with a concatenation before and a residual after them, 101,376
// nodes take 230 us: each launch reads and writes 26 to 78 MB of activations, 35 us
// where memory alone would take 8 to 12. Here a persistent CTA per SM keeps the
// weights in shared memory and its three warpgroups walk tiles of 128 nodes (see
// edge_fused.cu), so that only x and h cross memory: 69 us for a hop's update (208
// MB, 32 us of them), 36 for the encoder (138 before), 26 for the decoder (105),
// bound by each tile's chain: two rounds of tiles for 444 groups. Rounding to bf16 happens where the GEMMs round, and every sum is in
// their order: the same bits.
//
// Waits are bounded as in edge_fused.cu: one that runs out sets bit 0 of *err and
// ends its group's tiles.
#include <cuda_bf16.h>
#include <cstdint>

#include "mlp.cuh"
#include "umma_tile.cuh"

namespace pe {

namespace {

using namespace umma;

constexpr int kGroups = 3;
constexpr int kNodeThreads = kGroups * kGroupThreads;
constexpr uint32_t kOffW1 = 0;                    // W1^T [128 x up to 256]: four slices
constexpr uint32_t kOffW2 = kOffW1 + 4 * kSlice;  // W2^T, W3^T: two slices each
constexpr uint32_t kOffW3 = kOffW2 + 2 * kSlice;
constexpr uint32_t kOffGroup = kOffW3 + 2 * kSlice;
constexpr uint32_t kSmemBytes = kOffGroup + kGroups * 2 * kSlice + 1024u;  // + alignment slack
static_assert(kSmemBytes + 2048u <= 232448u, "one CTA's shared memory, with its biases and barriers");

__global__ void __launch_bounds__(kNodeThreads, 1) k_node_mlp(NodeMlpArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t mbar[kGroups];
    __shared__ uint32_t s_tmem;
    __shared__ __align__(16) float s_bias[3][128];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = tid / kGroupThreads, gt = tid % kGroupThreads, gw = gt >> 5;
    uint8_t* sW1 = smem + kOffW1;
    uint8_t* sW2 = smem + kOffW2;
    uint8_t* sW3 = smem + kOffW3;
    uint8_t* sA = smem + kOffGroup + (uint32_t)g * 2 * kSlice;

    if (tid == 0) {
        for (int i = 0; i < kGroups; ++i) mbar_init(smem_addr(&mbar[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    stage_rows(sW1, a.W1, a.k1, a.k1 / 8);
    if (a.k1 == 8 && tid < 128) *reinterpret_cast<uint4*>(sW1 + sw_off(tid, 1)) = zero;
    stage_rows(sW2, a.W2, 128, 16);
    stage_rows(sW3, a.W3, 128, 16, a.n3);
    if (a.n3 == 8)
        for (int i = tid; i < 8 * 16; i += kNodeThreads)  // rows 8 .. 15 of the narrowest MMA
            *reinterpret_cast<uint4*>(sW3 + (uint32_t)((i & 15) >> 3) * kSlice + sw_off(8 + (i >> 4), i & 7)) = zero;
    if (tid < 128) {
        s_bias[0][tid] = __ldg(a.b1 + tid);
        s_bias[1][tid] = __ldg(a.b2 + tid);
        s_bias[2][tid] = tid < a.n3 ? __ldg(a.b3 + tid) : 0.f;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem + 128u * (uint32_t)g;         // this group's 128 columns
    const uint32_t trow = tmem + ((uint32_t)(gw * 32) << 16);  // this warp's lanes
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
    // relu(accumulator + bias) into the activation tile, once its MMAs have completed
    auto activate = [&](const float* b) {
#pragma unroll 1
        for (int cb = 0; cb < 4; ++cb) {
            uint32_t v[32];
            tmem_ld32(trow + (uint32_t)(cb * 32), v);
            float x[32], bias[32];
            get_bias(b + cb * 32, bias);
#pragma unroll
            for (int j = 0; j < 32; ++j) x[j] = fmaxf(__uint_as_float(v[j]) + bias[j], 0.f);
            put_bf16_row(sA, gt, cb * 32, x);
        }
    };
    const int ntiles = (a.n + kGroupThreads - 1) / kGroupThreads;
    for (int tile = (int)blockIdx.x + g * (int)gridDim.x; tile < ntiles; tile += (int)gridDim.x * kGroups) {
        const int row0 = tile * kGroupThreads, mine = row0 + gw * 32;  // the warp copies its own 32 rows
        // ---- layer 1
        if (a.k1 == 8) {
            *reinterpret_cast<uint4*>(sA + sw_off(gt, 0)) =
                row0 + gt < a.n ? __ldg(reinterpret_cast<const uint4*>(a.x + (size_t)(row0 + gt) * 8)) : zero;
            *reinterpret_cast<uint4*>(sA + sw_off(gt, 1)) = zero;
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int r = 2 * i + (lane >> 4), c = lane & 15;
                const uint4 v = mine + r < a.n
                                    ? __ldg(reinterpret_cast<const uint4*>(a.x + (size_t)(mine + r) * 128 + c * 8))
                                    : zero;
                *reinterpret_cast<uint4*>(sA + (uint32_t)(c >> 3) * kSlice + sw_off(gw * 32 + r, c & 7)) = v;
            }
        }
        to_tensor();
        if (gt == 0) {
            if (a.k1 == 8) umma_bf16(tmem, sw128_desc(smem_addr(sA)), sw128_desc(smem_addr(sW1)), 0u);
            else issue_k128(tmem, sA, sW1);
            umma_commit(bar);
        }
        if (a.k1 == 256) {  // the messages: columns 128 .. 255
            float4 m[32];
#pragma unroll
            for (int r = 0; r < 32; ++r)
                m[r] = mine + r < a.n ? __ldg(reinterpret_cast<const float4*>(a.msg + (size_t)(mine + r) * 128) + lane)
                                      : make_float4(0.f, 0.f, 0.f, 0.f);
            ok = mma_wait() && ok;
#pragma unroll
            for (int r = 0; r < 32; ++r) {
                const __nv_bfloat162 lo = __floats2bfloat162_rn(m[r].x * a.scale, m[r].y * a.scale),
                                     hi = __floats2bfloat162_rn(m[r].z * a.scale, m[r].w * a.scale);
                const int c = lane >> 1;
                *reinterpret_cast<uint2*>(sA + (uint32_t)(c >> 3) * kSlice + sw_off(gw * 32 + r, c & 7) +
                                          8u * (lane & 1)) =
                    make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
            }
            to_tensor();
            if (gt == 0) {
                issue_k128(tmem, sA, sW1 + 2 * kSlice, true);
                umma_commit(bar);
            }
        }
        ok = mma_wait() && ok;
        activate(s_bias[0]);
        to_tensor();
        // ---- layer 2
        if (gt == 0) {
            issue_k128(tmem, sA, sW2);
            umma_commit(bar);
        }
        ok = mma_wait() && ok;
        activate(s_bias[1]);
        to_tensor();
        // ---- layer 3
        if (gt == 0) {
            if (a.n3 == 8) issue_k128<16>(tmem, sA, sW3);
            else issue_k128(tmem, sA, sW3);
            umma_commit(bar);
        }
        ok = mma_wait() && ok;
        if (a.n3 == 8) {
            uint32_t v[16];
            tmem_ld16(trow, v);
            float y[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) y[j] = __uint_as_float(v[j]) + s_bias[2][j];
            if (row0 + gt < a.n) {
                float4* const out = reinterpret_cast<float4*>(a.y + (size_t)(row0 + gt) * 8);
                out[0] = make_float4(y[0], y[1], y[2], y[3]);
                out[1] = make_float4(y[4], y[5], y[6], y[7]);
            }
        } else {
            const bool add = a.fluid != nullptr;
            const uint32_t adds = __ballot_sync(0xffffffffu, add && mine + lane < a.n && a.fluid[mine + lane]);
#pragma unroll 1
            for (int cb = 0; cb < 4; ++cb) {
                uint32_t v[32];
                tmem_ld32(trow + (uint32_t)(cb * 32), v);
                float bias[32];
                get_bias(s_bias[2] + cb * 32, bias);
                // column j of row r at j ^ r, in the warp's own rows of a slice
                float* const st = reinterpret_cast<float*>(sA + (uint32_t)(cb & 1) * kSlice + (uint32_t)gw * 4096u);
#pragma unroll
                for (int j = 0; j < 32; ++j) st[lane * 32 + (j ^ lane)] = __uint_as_float(v[j]) + bias[j];
                __syncwarp();
                const int rows = min(32, a.n - mine);  // may be negative: past the last node
                float* const h = a.h + (size_t)mine * 128 + cb * 32 + lane;
                __nv_bfloat16* const hb = a.hb + (size_t)mine * 128 + cb * 32 + lane;
                // h is read 16 rows ahead of its stores (one row at a time, each load waited for the last store's)
#pragma unroll
                for (int r0 = 0; r0 < 32; r0 += 16) {
                    float old[16];
                    if (add) {
#pragma unroll
                        for (int q = 0; q < 16; ++q) old[q] = r0 + q < rows ? h[(r0 + q) * 128] : 0.f;
                    }
#pragma unroll
                    for (int q = 0; q < 16; ++q) {
                        const int r = r0 + q;
                        if (r >= rows) break;
                        float y = st[r * 32 + (lane ^ r)];
                        if (add) y = ((adds >> r) & 1u) ? old[q] + y : old[q];
                        h[r * 128] = y;
                        hb[r * 128] = __float2bfloat16_rn(y);
                    }
                }
            }
            __syncwarp();  // the next tile's input goes where the outputs were
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        // the tile's TMEM reads and shared-memory use end before the group's next
        // tile; a run-out wait on any thread of the group stops the whole group
        ok = group_all(g, ok);
        if (!ok) break;
    }
    // every committed MMA completes before the tensor memory is freed
    if (gt == 0) umma_commit(bar);
    ok = mma_wait() && ok;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "r"(512u) : "memory");
    if (!ok && gt == 0) atomicOr(a.err, 1u);
}

}  // namespace

bool node_mlp_prepare() {
    return cudaFuncSetAttribute(k_node_mlp, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes) ==
           cudaSuccess;
}

void launch_node_mlp(const NodeMlpArgs& a, int sms, cudaStream_t st) {
    if (a.n <= 0) return;
    const int ntiles = (a.n + kGroupThreads - 1) / kGroupThreads;
    k_node_mlp<<<ntiles < sms ? ntiles : sms, kNodeThreads, kSmemBytes, st>>>(a);
}

}  // namespace pe

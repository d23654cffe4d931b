// Learned surrogate: parameters, forward and backward passes of the two-hop
// message-passing network (see surrogate.cuh), Adam, and the graph built from
// a world's state. Training materialises the activations of a tank-sized
// graph; every matrix product runs on the tcgen05 GEMM (mlp_gemm.cu).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <stdexcept>

#include "surrogate.cuh"

namespace pe {

namespace {

constexpr float kAggScale = 1.0f / 16.0f;

inline unsigned blocks(size_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }
inline int round8(int v) { return (v + 7) & ~7; }

void cu(cudaError_t e, const char* what) {
    if (e != cudaSuccess) throw std::runtime_error(std::string("surrogate ") + what + ": " + cudaGetErrorString(e));
}

__global__ void k_to_bf16(size_t n, const float* __restrict__ src, __nv_bfloat16* __restrict__ dst) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = __float2bfloat16_rn(src[i]);
}

// out_i = scale * sum of rows [row_i, row_{i+1}) of in (a warp per node)
__global__ void k_segsum(int n, const int* __restrict__ row, const float* __restrict__ in, float scale,
                         float* __restrict__ out) {
    const int node = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (node >= n) return;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int e = row[node]; e < row[node + 1]; ++e) {
        const float4 v = reinterpret_cast<const float4*>(in + (size_t)e * kWidth)[lane];
        s.x += v.x;
        s.y += v.y;
        s.z += v.z;
        s.w += v.w;
    }
    s.x *= scale;
    s.y *= scale;
    s.z *= scale;
    s.w *= scale;
    reinterpret_cast<float4*>(out + (size_t)node * kWidth)[lane] = s;
}

// [h | scale * a] as the node MLP's bf16 input
__global__ void k_concat(int n, const __nv_bfloat16* __restrict__ hb, const float* __restrict__ a, float scale,
                         __nv_bfloat16* __restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)n * 2 * kWidth) return;
    const size_t node = i / (2 * kWidth);
    const int c = (int)(i % (2 * kWidth));
    out[i] = c < kWidth ? hb[node * kWidth + c] : __float2bfloat16_rn(a[node * kWidth + c - kWidth] * scale);
}

// h += u on fluid nodes; hb_next = bf16(h)
__global__ void k_residual(int n, const float* __restrict__ u, const uint8_t* __restrict__ fluid,
                           float* __restrict__ h, __nv_bfloat16* __restrict__ hb_next) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)n * kWidth) return;
    float v = h[i];
    if (fluid[i / kWidth]) v += u[i];
    h[i] = v;
    hb_next[i] = __float2bfloat16_rn(v);
}

// The outputs without the padding columns: what crosses to the host is what the
// caller asked for (101,376 nodes: 0.1 ms of copy, where 3.2 MB and a loop over
// them on the host took 0.7).
__global__ void k_pack_outputs(int n, const float* __restrict__ Y, float4* __restrict__ out) {
    static_assert(kOut == 4 && kOutPad == 8, "a row is the first of two float4");
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = reinterpret_cast<const float4*>(Y)[2 * (size_t)i];
}

// loss = sum over fluid nodes of |y - t|^2 / nf; dY = 2 (y - t) / nf (padding columns 0)
__global__ void k_loss(int n, const float* __restrict__ Y, const float* __restrict__ T,
                       const uint8_t* __restrict__ fluid, float inv_nf, float* __restrict__ dY,
                       float* __restrict__ loss) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    float l = 0.f;
    if (i < n) {
#pragma unroll
        for (int c = 0; c < kOutPad; ++c) {
            float d = 0.f;
            if (c < kOut && fluid[i]) d = Y[(size_t)i * kOutPad + c] - T[(size_t)i * kOut + c];
            dY[(size_t)i * kOutPad + c] = 2.f * d * inv_nf;
            l += d * d;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((threadIdx.x & 31) == 0 && l != 0.f) atomicAdd(loss, l * inv_nf);
}

// Whether this block is the last of `blocks` to arrive here, whose writes before
// are then visible to it (ticket is zero before the first arrives and after the last).
__device__ __forceinline__ bool last_block(unsigned* ticket, unsigned blocks) {
    __shared__ bool s_last;
    const bool first = threadIdx.x == 0 && threadIdx.y == 0;
    __threadfence();
    __syncthreads();
    if (first) {
        s_last = atomicAdd(ticket, 1u) == blocks - 1u;
        if (s_last) *ticket = 0u;
    }
    __syncthreads();
    if (s_last) __threadfence();
    return s_last;
}

// dZ (fp32 [R x N]) masked in place by mask > 0; bf16 copies dZ [R8 x N] and
// dZ^T [N x R8] (zero-padded rows / columns); column sums into gbias. A block
// takes `tiles` tiles of 32 rows and leaves their sums in part [blocks x N]; the
// last block adds these up in block order, so that a gradient's bits do not
// depend on which block came first. (One atomic a tile and row group put 306,000
// edges' sums on 128 addresses 9,556 x 8 times over: 802 us of a pass that moves
// 470 MB.) Unmasked, dZ stays as it is and is not written back.
__global__ void k_grad_prep(int R, int R8, int N, int tiles, float* __restrict__ dZ,
                            const __nv_bfloat16* __restrict__ mask, __nv_bfloat16* __restrict__ g16,
                            __nv_bfloat16* __restrict__ gT, float* __restrict__ gbias, float* __restrict__ part,
                            unsigned* ticket) {
    __shared__ float tile[32][33];
    __shared__ float sums[8][32];
    const int c0 = blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
    float csum = 0.f;
    for (int t = 0; t < tiles; ++t) {
        const int r0 = (blockIdx.x * tiles + t) * 32;
        if (r0 >= R8) break;
        for (int k = ty; k < 32; k += 8) {
            const int r = r0 + k, c = c0 + tx;
            float v = 0.f;
            if (r < R && c < N) {
                v = dZ[(size_t)r * N + c];
                if (mask) {
                    if (!(__bfloat162float(mask[(size_t)r * N + c]) > 0.f)) v = 0.f;
                    dZ[(size_t)r * N + c] = v;
                }
            }
            if (r < R8 && c < N) g16[(size_t)r * N + c] = __float2bfloat16_rn(v);
            tile[k][tx] = v;
            csum += v;
        }
        __syncthreads();
        for (int k = ty; k < 32; k += 8) {
            const int c = c0 + k, r = r0 + tx;
            if (c < N && r < R8) gT[(size_t)c * R8 + r] = __float2bfloat16_rn(tile[tx][k]);
        }
        __syncthreads();
    }
    if (!gbias) return;
    auto block_sum = [&]() {  // over the eight rows of threads, in order
        sums[ty][tx] = csum;
        __syncthreads();
        float v = sums[0][tx];
#pragma unroll
        for (int k = 1; k < 8; ++k) v += sums[k][tx];
        return v;
    };
    const float mine = block_sum();
    if (ty == 0 && c0 + tx < N) part[(size_t)blockIdx.x * N + c0 + tx] = mine;
    if (!last_block(ticket + blockIdx.y, gridDim.x)) return;
    csum = 0.f;
    if (c0 + tx < N)
#pragma unroll 8
        for (unsigned b = ty; b < gridDim.x; b += 8) csum += __ldcg(part + (size_t)b * N + c0 + tx);
    const float all = block_sum();
    if (ty == 0 && c0 + tx < N) gbias[c0 + tx] = all;
}

// k_grad_prep for 128 columns, and with idx (rows gathered: dZ's row r is in's
// row idx[r]; nothing is written back): a warp reads whole 512-byte rows, and
// the transposed copy leaves through shared memory in 16-byte pieces. 64 rows a
// tile. Bound by HBM: 306,000 rows move 400 to 550 MB in 101 us (202 us with
// k_grad_prep, 802 before its sums were a block's, and 142 more for the gathered
// copy it needed).
constexpr int kPrepRows = 64;
__global__ void __launch_bounds__(256) k_grad_prep128(int R, int R8, int tiles, float* __restrict__ dZ,
                                                      const int* __restrict__ idx,
                                                      const __nv_bfloat16* __restrict__ mask,
                                                      __nv_bfloat16* __restrict__ g16, __nv_bfloat16* __restrict__ gT,
                                                      float* __restrict__ gbias, float* __restrict__ part,
                                                      unsigned* ticket) {
    // element (c, r) of the transposed tile; 16-byte piece p of column c at p ^ ((c / 4) & 7)
    __shared__ __align__(16) __nv_bfloat16 tile[kWidth][kPrepRows];
    __shared__ float4 sums[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c0 = lane * 4;
    float4 csum = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int t = 0; t < tiles; ++t) {
        const int r0 = (blockIdx.x * tiles + t) * kPrepRows;
        if (r0 >= R8) break;
#pragma unroll
        for (int k = 0; k < kPrepRows / 8; ++k) {
            const int lr = k * 8 + warp, r = r0 + lr;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < R) {
                const size_t at = (size_t)r * kWidth + c0;
                v = *reinterpret_cast<const float4*>(idx ? dZ + (size_t)idx[r] * kWidth + c0 : dZ + at);
                if (mask) {
                    const uint2 mb = *reinterpret_cast<const uint2*>(mask + at);
                    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&mb.x));
                    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&mb.y));
                    if (!(a.x > 0.f)) v.x = 0.f;
                    if (!(a.y > 0.f)) v.y = 0.f;
                    if (!(b.x > 0.f)) v.z = 0.f;
                    if (!(b.y > 0.f)) v.w = 0.f;
                    *reinterpret_cast<float4*>(dZ + at) = v;
                }
            }
            const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
            if (r < R8)
                *reinterpret_cast<uint2*>(g16 + (size_t)r * kWidth + c0) =
                    make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
            const int at = (((lr >> 3) ^ (lane & 7)) << 3) | (lr & 7);
            tile[c0][at] = lo.x;
            tile[c0 + 1][at] = lo.y;
            tile[c0 + 2][at] = hi.x;
            tile[c0 + 3][at] = hi.y;
            csum.x += v.x;
            csum.y += v.y;
            csum.z += v.z;
            csum.w += v.w;
        }
        __syncthreads();
        // eight lanes a column: its 64 rows are 128 contiguous bytes
        for (int c = threadIdx.x >> 3; c < kWidth; c += 32) {
            const int p = threadIdx.x & 7, r = r0 + p * 8;
            if (r < R8)
                *reinterpret_cast<uint4*>(gT + (size_t)c * R8 + r) =
                    *reinterpret_cast<const uint4*>(&tile[c][(p ^ ((c >> 2) & 7)) << 3]);
        }
        __syncthreads();
    }
    if (!gbias) return;
    auto block_sum = [&](float4* out) {  // over the warps, in order
        sums[warp][lane] = csum;
        __syncthreads();
        if (warp != 0) return;
#pragma unroll
        for (int k = 1; k < 8; ++k) {
            const float4 v = sums[k][lane];
            csum.x += v.x;
            csum.y += v.y;
            csum.z += v.z;
            csum.w += v.w;
        }
        out[lane] = csum;
    };
    float4* const rows = reinterpret_cast<float4*>(part);
    block_sum(rows + (size_t)blockIdx.x * 32);
    if (!last_block(ticket, gridDim.x)) return;
    csum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (unsigned b = warp; b < gridDim.x; b += 8) {
        const float4 v = __ldcg(rows + (size_t)b * 32 + lane);
        csum.x += v.x;
        csum.y += v.y;
        csum.z += v.z;
        csum.w += v.w;
    }
    block_sum(reinterpret_cast<float4*>(gbias));
}

// k_transpose for K a multiple of 16: a tile of 64 rows x 16 columns a warp,
// 16-byte reads and writes through shared memory (306,000 x 128: 24 us, 76 with
// 2-byte accesses; 157 MB at the copy rate take 24).
__global__ void __launch_bounds__(256) k_transpose16(int R, int R8, int K, const __nv_bfloat16* __restrict__ X,
                                                     __nv_bfloat16* __restrict__ XT) {
    __shared__ __align__(16) __nv_bfloat16 tile[8][16][kPrepRows];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = blockIdx.x * kPrepRows, c0 = (blockIdx.y * 8 + warp) * 16;
    if (c0 >= K) return;  // a whole warp; warps do not meet below
    __nv_bfloat16(*t)[kPrepRows] = tile[warp];
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // 16 rows a pass, two 16-byte halves a row
        const int lr = k * 16 + (lane >> 1), h = lane & 1, r = r0 + lr;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (r < R) v = *reinterpret_cast<const uint4*>(X + (size_t)r * K + c0 + h * 8);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int c = h * 8 + j;
            const uint16_t b = (uint16_t)(w[j >> 1] >> ((j & 1) * 16));
            *reinterpret_cast<uint16_t*>(&t[c][(((lr >> 3) ^ (c & 7)) << 3) | (lr & 7)]) = b;
        }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // eight lanes a column, four columns a pass
        const int c = k * 4 + (lane >> 3), p = lane & 7, r = r0 + p * 8;
        if (r < R8)
            *reinterpret_cast<uint4*>(XT + (size_t)(c0 + c) * R8 + r) =
                *reinterpret_cast<const uint4*>(&t[c][(p ^ (c & 7)) << 3]);
    }
}

// X (bf16 [R x K]) -> X^T (bf16 [K x R8]), zero columns R..R8
__global__ void k_transpose(int R, int R8, int K, const __nv_bfloat16* __restrict__ X,
                            __nv_bfloat16* __restrict__ XT) {
    __shared__ __nv_bfloat16 tile[32][34];
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int k = ty; k < 32; k += 8) {
        const int r = r0 + k, c = c0 + tx;
        tile[k][tx] = (r < R && c < K) ? X[(size_t)r * K + c] : __float2bfloat16_rn(0.f);
    }
    __syncthreads();
    for (int k = ty; k < 32; k += 8) {
        const int c = c0 + k, r = r0 + tx;
        if (c < K && r < R8) XT[(size_t)c * R8 + r] = tile[tx][k];
    }
}

__global__ void k_mask_rows(int n, const float* __restrict__ in, const uint8_t* __restrict__ fluid,
                            float* __restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < (size_t)n * kWidth) out[i] = fluid[i / kWidth] ? in[i] : 0.f;
}

// dHp = dH + dXN[:, :128]; da = scale * dXN[:, 128:]
__global__ void k_split_dxn(int n, const float* __restrict__ dH, const float* __restrict__ dXN, float scale,
                            float* __restrict__ dHp, float* __restrict__ da) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)n * kWidth) return;
    const size_t node = i / kWidth, c = i % kWidth;
    dHp[i] = dH[i] + dXN[node * 2 * kWidth + c];
    da[i] = scale * dXN[node * 2 * kWidth + kWidth + c];
}

// The edges by source, each source's in ascending order: a count that keeps every
// edge's arrival number, then (after the scan of the counts) the edges in their
// source's run in order of arrival, then each edge at its rank within the run.
__global__ void k_source_count(int E, const int* __restrict__ src, int* __restrict__ cnt, int* __restrict__ arrival) {
    const int e = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (e < E) arrival[e] = atomicAdd(&cnt[src[e]], 1);
}

__global__ void k_source_place(int E, const int* __restrict__ src, const int* __restrict__ srow,
                               const int* __restrict__ arrival, int* __restrict__ placed) {
    const int e = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (e < E) placed[srow[src[e]] + arrival[e]] = e;
}

__global__ void k_source_order(int E, const int* __restrict__ src, const int* __restrict__ srow,
                               const int* __restrict__ placed, int* __restrict__ by_src) {
    const int k = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (k >= E) return;
    const int e = placed[k], s = src[e], b = srow[s], end = srow[s + 1];
    int at = b;
#pragma unroll 4
    for (int j = b; j < end; ++j) at += placed[j] < e;
    by_src[at] = e;
}

// out_j = sum of the rows of in that node j sends, in edge order (a warp per node).
// The sums are rounded to bf16 next, where one that lies at a boundary costs every
// gradient behind it 2^-9 of that element: fp32 atomics in order of arrival left two
// runs on the same inputs up to 5e-5 apart. Edge order is also about the order they
// arrived in, so the gradients stay where most of those runs had them (sums in
// fp64 do not: 2.5e-5 off on a graph whose runs agreed to 4e-6).
__global__ void k_source_sum(int n, const int* __restrict__ srow, const int* __restrict__ by_src,
                             const float* __restrict__ in, float* __restrict__ out) {
    const int node = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (node >= n) return;
    float x = 0.f, y = 0.f, z = 0.f, w = 0.f;
    const int end = srow[node + 1];
#pragma unroll 4
    for (int k = srow[node]; k < end; ++k) {
        const float4 v = reinterpret_cast<const float4*>(in + (size_t)by_src[k] * kWidth)[lane];
        x += v.x;
        y += v.y;
        z += v.z;
        w += v.w;
    }
    reinterpret_cast<float4*>(out + (size_t)node * kWidth)[lane] = make_float4(x, y, z, w);
}

__global__ void k_add(size_t n, float* __restrict__ a, const float* __restrict__ b) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] += b[i];
}

__global__ void k_adam(size_t n, float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, float lr, float c1, float c2) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = 0.9f * m[i] + 0.1f * gi;
    const float vi = 0.999f * v[i] + 0.001f * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + 1e-8f);
}

// bf16 copies of a master Wt [Np x K]: Wt16 (same layout) and W16 [K x Np]
__global__ void k_refresh(int Np, int K, const float* __restrict__ Wt, __nv_bfloat16* __restrict__ Wt16,
                          __nv_bfloat16* __restrict__ W16) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Np * K) return;
    const int n = i / K, k = i % K;
    const __nv_bfloat16 b = __float2bfloat16_rn(Wt[i]);
    Wt16[i] = b;
    W16[(size_t)k * Np + n] = b;
}

// host-side seeded normal numbers (xoshiro256** + Box-Muller)
struct HostRng {
    uint64_t s[4];
    explicit HostRng(uint64_t seed) {
        uint64_t z = seed;
        for (auto& v : s) {
            z += 0x9e3779b97f4a7c15ULL;
            uint64_t x = z;
            x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
            x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
            v = x ^ (x >> 31);
        }
    }
    static uint64_t rotl(uint64_t x, int k) { return (x << k) | (x >> (64 - k)); }
    uint64_t next() {
        const uint64_t r = rotl(s[1] * 5, 7) * 9, t = s[1] << 17;
        s[2] ^= s[0];
        s[3] ^= s[1];
        s[1] ^= s[2];
        s[0] ^= s[3];
        s[2] ^= t;
        s[3] = rotl(s[3], 45);
        return r;
    }
    double uniform() { return ((next() >> 11) + 0.5) * (1.0 / 9007199254740992.0); }
    double normal() { return std::sqrt(-2.0 * std::log(uniform())) * std::cos(6.283185307179586 * uniform()); }
};

}  // namespace

template <typename T>
T* Surrogate::dalloc(size_t n) {
    void* p = nullptr;
    cu(cudaMalloc(&p, std::max<size_t>(n * sizeof(T), 256)), "cudaMalloc");
    cu(cudaMemsetAsync(p, 0, std::max<size_t>(n * sizeof(T), 256), st_), "memset");
    return static_cast<T*>(p);
}

Surrogate::Surrogate(uint64_t seed, double r_msg_over_h) : r_msg_over_h_(r_msg_over_h) {
    cu(cudaStreamCreateWithFlags(&st_, cudaStreamNonBlocking), "stream");
    own_stream_ = true;
    if (!gemm_prepare()) throw std::runtime_error("surrogate: GEMM shared-memory limit");
    if (!edge_hop_prepare() || !node_mlp_prepare())
        throw std::runtime_error("surrogate: fused kernels' shared-memory limit");
    {
        int dev = 0;
        if (cudaGetDevice(&dev) == cudaSuccess)
            cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, dev);
    }
    err_ = dalloc<uint32_t>(1);
    allocs_.push_back(err_);
    loss_ = dalloc<float>(1);
    allocs_.push_back(loss_);
    tickets_ = dalloc<unsigned>(kTickets);
    allocs_.push_back(tickets_);
    for (int c = 0; c < kOut; ++c) {
        stats_.mean[c] = 0.f;
        stats_.std[c] = 1.f;
    }
    alloc_params(seed);
}

Surrogate::~Surrogate() {
    if (st_) cudaStreamSynchronize(st_);
    for (void* p : allocs_) cudaFree(p);
    for (void* p : graph_allocs_) cudaFree(p);
    for (void* p : act_allocs_) cudaFree(p);
    if (part_) cudaFree(part_);
    if (scan_tmp_) cudaFree(scan_tmp_);
    if (own_stream_ && st_) cudaStreamDestroy(st_);
}

void Surrogate::alloc_params(uint64_t seed) {
    auto add = [&](const std::string& name, int K, int N, bool bias) {
        Linear L;
        L.name = name;
        L.K = K;
        L.N = N;
        L.Np = round8(N);
        L.has_bias = bias;
        layers_.push_back(L);
    };
    auto mlp = [&](const std::string& name, int K, int N) {
        add(name + ".0", K, kWidth, true);
        add(name + ".1", kWidth, kWidth, true);
        add(name + ".2", kWidth, N, true);
    };
    mlp("enc", kNodeFeat, kWidth);
    for (int l = 1; l <= 2; ++l) {
        const std::string h = "hop" + std::to_string(l);
        add(h + ".edge.a", kWidth, kWidth, false);
        add(h + ".edge.b", kWidth, kWidth, false);
        add(h + ".edge.0", kEdgeFeat, kWidth, true);
        add(h + ".edge.1", kWidth, kWidth, true);
        add(h + ".edge.2", kWidth, kWidth, true);
        mlp(h + ".node", 2 * kWidth, kWidth);
    }
    mlp("dec", kWidth, kOut);
    HostRng rng(seed);
    for (Linear& L : layers_) {
        const size_t nw = (size_t)L.Np * L.K;
        L.Wt = dalloc<float>(nw);
        L.gWt = dalloc<float>(nw);
        L.mW = dalloc<float>(nw);
        L.vW = dalloc<float>(nw);
        L.b = dalloc<float>(L.Np);
        L.gb = dalloc<float>(L.Np);
        L.mb = dalloc<float>(L.Np);
        L.vb = dalloc<float>(L.Np);
        L.Wt16 = dalloc<__nv_bfloat16>(nw);
        L.W16 = dalloc<__nv_bfloat16>(nw);
        for (void* p : {(void*)L.Wt, (void*)L.gWt, (void*)L.mW, (void*)L.vW, (void*)L.b, (void*)L.gb, (void*)L.mb,
                        (void*)L.vb, (void*)L.Wt16, (void*)L.W16})
            allocs_.push_back(p);
        // He initialisation for the ReLU layers; the decoder's output layer starts small
        const bool out_layer = L.name == "dec.2";
        const double sd = std::sqrt(2.0 / L.K) * (out_layer ? 0.1 : 1.0);
        std::vector<float> w(nw, 0.f);
        for (int n = 0; n < L.N; ++n)
            for (int k = 0; k < L.K; ++k) w[(size_t)n * L.K + k] = (float)(sd * rng.normal());
        cu(cudaMemcpyAsync(L.Wt, w.data(), nw * sizeof(float), cudaMemcpyHostToDevice, st_), "init");
        cu(cudaStreamSynchronize(st_), "init");
        refresh_bf16(L);
    }
}

void Surrogate::refresh_bf16(Linear& L) {
    const int n = L.Np * L.K;
    k_refresh<<<blocks(n, 256), 256, 0, st_>>>(L.Np, L.K, L.Wt, L.Wt16, L.W16);
}

void Surrogate::get_param(int i, float* W, float* b, bool grad) {
    const Linear& L = layers_.at(i);
    std::vector<float> wt((size_t)L.Np * L.K), bb(L.Np);
    cu(cudaMemcpyAsync(wt.data(), grad ? L.gWt : L.Wt, wt.size() * 4, cudaMemcpyDeviceToHost, st_), "get");
    cu(cudaMemcpyAsync(bb.data(), grad ? L.gb : L.b, bb.size() * 4, cudaMemcpyDeviceToHost, st_), "get");
    cu(cudaStreamSynchronize(st_), "get");
    if (W)
        for (int k = 0; k < L.K; ++k)
            for (int n = 0; n < L.N; ++n) W[(size_t)k * L.N + n] = wt[(size_t)n * L.K + k];
    if (b)
        for (int n = 0; n < L.N; ++n) b[n] = L.has_bias ? bb[n] : 0.f;
}

void Surrogate::set_param(int i, const float* W, const float* b) {
    Linear& L = layers_.at(i);
    std::vector<float> wt((size_t)L.Np * L.K, 0.f), bb(L.Np, 0.f);
    cu(cudaMemcpyAsync(wt.data(), L.Wt, wt.size() * 4, cudaMemcpyDeviceToHost, st_), "set");
    cu(cudaStreamSynchronize(st_), "set");
    if (W)
        for (int k = 0; k < L.K; ++k)
            for (int n = 0; n < L.N; ++n) wt[(size_t)n * L.K + k] = W[(size_t)k * L.N + n];
    if (b && L.has_bias)
        for (int n = 0; n < L.N; ++n) bb[n] = b[n];
    cu(cudaMemcpyAsync(L.Wt, wt.data(), wt.size() * 4, cudaMemcpyHostToDevice, st_), "set");
    if (b && L.has_bias) cu(cudaMemcpyAsync(L.b, bb.data(), bb.size() * 4, cudaMemcpyHostToDevice, st_), "set");
    cu(cudaStreamSynchronize(st_), "set");
    refresh_bf16(L);
}

void Surrogate::ensure_graph(int n, int E) {
    g_.by_source = false;
    if (n <= g_.cap_n && E <= g_.cap_e) {
        g_.n = n;
        g_.E = E;
        return;
    }
    cu(cudaStreamSynchronize(st_), "graph");
    for (void* p : graph_allocs_) cudaFree(p);
    graph_allocs_.clear();
    if (scan_tmp_) cudaFree(scan_tmp_);
    scan_tmp_ = nullptr;
    scan_bytes_ = 0;
    // grow with a quarter of headroom: the edge count creeps up step by step as
    // the fluid compresses, and every growth reallocates
    const int cn = std::max(n + n / 4, g_.cap_n), ce = std::max(E + E / 4, g_.cap_e);
    g_.cap_n = g_.cap_e = 0;  // until all of them are there
    auto ga = [&](size_t bytes) {
        void* p = nullptr;
        cu(cudaMalloc(&p, std::max<size_t>(bytes, 256)), "cudaMalloc graph");
        graph_allocs_.push_back(p);
        return p;
    };
    g_.row = static_cast<int*>(ga((size_t)(cn + 1) * 4));
    g_.src = static_cast<int*>(ga((size_t)ce * 4));
    g_.dst = static_cast<int*>(ga((size_t)ce * 4));
    g_.srow = static_cast<int*>(ga((size_t)(cn + 1) * 4));
    g_.by_src = static_cast<int*>(ga((size_t)ce * 4));
    g_.xe = static_cast<__nv_bfloat16*>(ga((size_t)ce * kEdgeFeat * 2));
    g_.f = static_cast<__nv_bfloat16*>(ga((size_t)cn * kNodeFeat * 2));
    g_.fluid = static_cast<uint8_t*>(ga((size_t)cn));
    node_orig_ = static_cast<uint32_t*>(ga((size_t)cn * 4));
    node_v_ = static_cast<double*>(ga((size_t)cn * 4 * 8));
    target_ = static_cast<float*>(ga((size_t)cn * kOut * 4));
    raw_t_ = static_cast<float*>(ga((size_t)cn * kOut * 4));
    cnt_ = static_cast<int*>(ga((size_t)(cn + 1) * 4));
    g_.cap_n = cn;
    g_.cap_e = ce;
    g_.n = n;
    g_.E = E;
}

// Buffers of a forward pass: what the fused kernels of inference touch (kActsFused:
// nodes only), the layers' activations beside them (kActsLayers: ~1.5 KB an edge,
// one hop's), or those of both hops and the backward pass's (kActsTrain: ~4.6 KB).
// At 101,376 nodes and 2.56M edges a new network's first forward pass allocated
// 4.6 GB for the 0.36 it uses: 12.5 ms, 5.6 now.
void Surrogate::ensure_acts(int level) {
    const int n = g_.n, E = g_.E;
    if (act_level_ >= level && n <= act_n_ && (level == kActsFused || E <= act_e_)) return;
    cu(cudaStreamSynchronize(st_), "acts");
    for (void* p : act_allocs_) cudaFree(p);
    act_allocs_.clear();
    // grow with a quarter of headroom; a switch to training sizes for the
    // current graph only (training buffers cost ~3x per edge)
    const bool keep = act_level_ >= level, layers = level >= kActsLayers, train = level >= kActsTrain;
    const int cn = round8(std::max(n + n / 4, keep ? act_n_ : 0));
    const int ce = layers ? round8(std::max(E + E / 4, keep ? act_e_ : 0)) : 0;
    act_n_ = act_e_ = 0;  // until all of them are there
    act_level_ = -1;
    auto take = [&](bool wanted, size_t bytes) -> void* {
        if (!wanted) return nullptr;
        void* p = nullptr;
        cu(cudaMalloc(&p, std::max<size_t>(bytes, 256)), "cudaMalloc acts");
        act_allocs_.push_back(p);
        return p;
    };
    auto fa = [&](size_t count, bool wanted) { return static_cast<float*>(take(wanted, count * 4)); };
    auto ba = [&](size_t count, bool wanted) { return static_cast<__nv_bfloat16*>(take(wanted, count * 2)); };
    const size_t W = kWidth, N = (size_t)cn * W, NE = (size_t)ce * W;
    h_ = fa(N, true);
    for (auto& p : hb_) p = ba(N, true);
    P_ = fa(N, true);
    Q_ = fa(N, true);
    A_ = fa(N, true);
    Y_ = fa((size_t)cn * kOutPad, true);
    dY_ = fa((size_t)cn * kOutPad, true);  // inference packs its outputs there
    enc_a1_ = ba(N, layers);
    enc_a2_ = ba(N, layers);
    for (int l = 0; l < 2; ++l) {
        eh1_[l] = (l == 0 || train) ? ba(NE, layers) : eh1_[0];
        eh2_[l] = (l == 0 || train) ? ba(NE, layers) : eh2_[0];
        xn_[l] = ba(2 * N, layers);
        na1_[l] = ba(N, layers);
        na2_[l] = ba(N, layers);
    }
    M_ = fa(NE, layers);
    U_ = fa(N, layers);
    da1_ = ba(N, layers);
    da2_ = ba(N, layers);
    dH_ = fa(N, train);
    dHp_ = fa(N, train);
    dXN_ = fa(2 * N, train);
    dE_ = fa(NE, train);
    dE2_ = fa(NE, train);
    dP_ = fa(N, train);
    dQ_ = fa(N, train);
    dT1_ = fa(N, train);
    dT2_ = fa(N, train);
    const size_t rows = (size_t)std::max(cn, ce);
    gb16_ = ba(rows * 2 * W, train);
    gbT_ = ba(rows * 2 * W, train);
    xT_ = ba(rows * 2 * W, train);
    act_n_ = cn;
    act_e_ = ce;
    act_level_ = level;
}

// Room for `need` partial sums of the launch that follows.
float* Surrogate::partials(size_t need) {
    if (need > part_floats_) {
        cu(cudaStreamSynchronize(st_), "part");
        if (part_) cudaFree(part_);
        part_ = nullptr;
        part_floats_ = 0;
        cu(cudaMalloc(&part_, need * 4), "cudaMalloc part");
        part_floats_ = need;
    }
    return part_;
}

void Surrogate::gemm(const __nv_bfloat16* A, int lda, const __nv_bfloat16* Bt, int ldb, int M, int N, int K,
                     float* Cf, __nv_bfloat16* Cb, int ldc, const float* bias, bool relu, int splits) {
    if (M <= 0 || N <= 0) return;
    if (splits > 1) {
        partials((size_t)splits * M * ldc);
        GemmArgs g{A, Bt, part_, nullptr, nullptr, M, N, K, lda, ldb, ldc, 0, err_};
        launch_gemm(g, splits, st_);
        launch_gemm_reduce(M, N, ldc, splits, part_, bias, relu ? 1 : 0, Cf, Cb, st_);
    } else {
        GemmArgs g{A, Bt, Cf, Cb, bias, M, N, K, lda, ldb, ldc, relu ? 1 : 0, err_};
        launch_gemm(g, 1, st_);
    }
}

void Surrogate::linear_fwd(const Linear& L, const __nv_bfloat16* X, int R, float* Yf, __nv_bfloat16* Yb,
                           bool relu) {
    gemm(X, L.K, L.Wt16, L.K, R, L.Np, L.K, Yf, Yb, L.Np, L.has_bias ? L.b : nullptr, relu);
}

void Surrogate::mlp_fwd(int first, const __nv_bfloat16* X, int R, __nv_bfloat16* A1, __nv_bfloat16* A2,
                        float* Yf) {
    linear_fwd(layers_[first], X, R, nullptr, A1, true);
    linear_fwd(layers_[first + 1], A1, R, nullptr, A2, true);
    linear_fwd(layers_[first + 2], A2, R, Yf, nullptr, false);
}

void Surrogate::forward(bool keep_for_backward) {
    const bool fused = fused_edges_ && !keep_for_backward;
    ensure_acts(keep_for_backward ? kActsTrain : fused ? kActsFused : kActsLayers);
    const int n = g_.n, E = g_.E;
    const size_t nW = (size_t)n * kWidth;
    // one fused node MLP: layers first .. first + 2 on x (and the messages)
    auto node_mlp = [&](int first, const __nv_bfloat16* x, const float* msg, const uint8_t* fluid,
                        __nv_bfloat16* hb) {
        const Linear &L0 = layers_[first], &L1 = layers_[first + 1], &L2 = layers_[first + 2];
        NodeMlpArgs na{n, L0.K, L2.Np, x, msg, kAggScale, L0.Wt16, L0.b, L1.Wt16, L1.b, L2.Wt16, L2.b, Y_, h_, hb,
                       fluid, err_};
        launch_node_mlp(na, sms_, st_);
    };
    if (fused) {
        node_mlp(0, g_.f, nullptr, nullptr, hb_[0]);
    } else {
        mlp_fwd(0, g_.f, n, enc_a1_, enc_a2_, h_);
        k_to_bf16<<<blocks(nW, 256), 256, 0, st_>>>(nW, h_, hb_[0]);
    }
    for (int l = 0; l < 2; ++l) {
        const int base = 3 + 8 * l;
        linear_fwd(layers_[base + 0], hb_[l], n, P_, nullptr, false);
        linear_fwd(layers_[base + 1], hb_[l], n, Q_, nullptr, false);
        if (E > 0 && fused) {
            // the whole edge MLP and the sum per destination in one kernel
            const Linear &L0 = layers_[base + 2], &L1 = layers_[base + 3], &L2 = layers_[base + 4];
            cu(cudaMemsetAsync(A_, 0, sizeof(float) * nW, st_), "memset");
            EdgeHopArgs ea{E, g_.src, g_.dst, g_.xe, P_, Q_, L0.Wt16, L0.b, L1.Wt16, L1.b, L2.Wt16, L2.b, A_, err_};
            launch_edge_hop(ea, sms_, st_);
        } else if (E > 0) {
            // layer 1: relu(x_e Wc + b1 + P[dst] + Q[src]), the gathers fused into the GEMM's epilogue
            const Linear& L0 = layers_[base + 2];
            GemmArgs ga{g_.xe, L0.Wt16, nullptr, eh1_[l], L0.b, E, L0.Np, L0.K, L0.K, L0.K, L0.Np, 1, err_};
            ga.add0 = P_;
            ga.idx0 = g_.dst;
            ga.add1 = Q_;
            ga.idx1 = g_.src;
            ga.ld_add = kWidth;
            launch_gemm(ga, 1, st_);
            linear_fwd(layers_[base + 3], eh1_[l], E, nullptr, eh2_[l], true);
            linear_fwd(layers_[base + 4], eh2_[l], E, M_, nullptr, false);
        }
        if (!(E > 0 && fused)) k_segsum<<<blocks((size_t)n * 32, 256), 256, 0, st_>>>(n, g_.row, M_, 1.f, A_);
        if (fused) {
            node_mlp(base + 5, hb_[l], A_, g_.fluid, hb_[l + 1]);
            continue;
        }
        k_concat<<<blocks(2 * nW, 256), 256, 0, st_>>>(n, hb_[l], A_, kAggScale, xn_[l]);
        mlp_fwd(base + 5, xn_[l], n, na1_[l], na2_[l], U_);
        k_residual<<<blocks(nW, 256), 256, 0, st_>>>(n, U_, g_.fluid, h_, hb_[l + 1]);
    }
    if (fused) node_mlp(19, hb_[2], nullptr, nullptr, nullptr);
    else mlp_fwd(19, hb_[2], n, da1_, da2_, Y_);
    cu(cudaGetLastError(), "forward");
}

void Surrogate::get_outputs(float* y) {
    const int n = g_.n;
    if (n <= 0) return;
    // dY_ is the backward pass's, which writes it before it reads it
    k_pack_outputs<<<blocks(n, 256), 256, 0, st_>>>(n, Y_, reinterpret_cast<float4*>(dY_));
    cu(cudaMemcpyAsync(y, dY_, sizeof(float) * kOut * (size_t)n, cudaMemcpyDeviceToHost, st_), "outputs");
    cu(cudaStreamSynchronize(st_), "outputs");
}

void Surrogate::linear_bwd(Linear& L, const __nv_bfloat16* X, int R, float* dZ, const __nv_bfloat16* mask,
                           float* dX, const int* rows) {
    if (R <= 0) return;
    const int R8 = round8(R);
    dim3 tb(32, 8);
    // eight resident blocks an SM, up to 32 tiles each
    float* const gb = L.has_bias ? L.gb : nullptr;
    if (L.Np == kWidth) {
        const int row_tiles = (int)blocks(R8, kPrepRows);
        const int tiles = std::max(1, std::min(32, row_tiles / (8 * sms_)));
        const unsigned nb = blocks(row_tiles, tiles);
        k_grad_prep128<<<nb, 256, 0, st_>>>(R, R8, tiles, dZ, rows, mask, gb16_, gbT_, gb,
                                            partials((size_t)nb * kWidth), tickets_);
    } else {
        const int row_tiles = (int)blocks(R8, 32), col_tiles = (int)blocks(L.Np, 32);
        const int tiles = std::max(1, std::min(32, row_tiles * col_tiles / (8 * sms_)));
        dim3 gz(blocks(row_tiles, tiles), col_tiles);
        if (col_tiles > kTickets) throw std::length_error("surrogate: layer width");
        k_grad_prep<<<gz, tb, 0, st_>>>(R, R8, L.Np, tiles, dZ, mask, gb16_, gbT_, gb,
                                        partials((size_t)gz.x * L.Np), tickets_);
    }
    if (L.K % 16 == 0) {
        k_transpose16<<<dim3(blocks(R8, kPrepRows), blocks(L.K, 128)), 256, 0, st_>>>(R, R8, L.K, X, xT_);
    } else {
        dim3 gx(blocks(R8, 32), blocks(L.K, 32));
        k_transpose<<<gx, tb, 0, st_>>>(R, R8, L.K, X, xT_);
    }
    // dW^T [Np x K] = dZ^T [Np x R] * X [R x K]
    const int splits = std::max(1, std::min(64, R8 / 8192));
    gemm(gbT_, R8, xT_, R8, L.Np, L.K, R8, L.gWt, nullptr, L.K, nullptr, false, splits);
    // dX [R x K] = dZ [R x Np] * W^T
    if (dX) gemm(gb16_, L.Np, L.W16, L.Np, R, L.K, L.Np, dX, nullptr, L.K, nullptr, false);
}

void Surrogate::mlp_bwd(int first, const __nv_bfloat16* X, int R, const __nv_bfloat16* A1,
                        const __nv_bfloat16* A2, float* dY, float* dX) {
    // dY [R x Np2] -> dA2 (dT1) -> masked by A2 -> dA1 (dT2) -> masked by A1 -> dX
    float* t1 = R <= g_.n ? dT1_ : dE2_;
    float* t2 = R <= g_.n ? dT2_ : dE_;
    linear_bwd(layers_[first + 2], A2, R, dY, nullptr, t1);
    linear_bwd(layers_[first + 1], A1, R, t1, A2, t2);
    linear_bwd(layers_[first + 0], X, R, t2, A1, dX);
}

void Surrogate::adam(Linear& L, float lr) {
    const float c1 = 1.f / (1.f - std::pow(0.9f, (float)adam_t_));
    const float c2 = 1.f / (1.f - std::pow(0.999f, (float)adam_t_));
    const size_t nw = (size_t)L.Np * L.K;
    k_adam<<<blocks(nw, 256), 256, 0, st_>>>(nw, L.Wt, L.gWt, L.mW, L.vW, lr, c1, c2);
    if (L.has_bias) k_adam<<<blocks(L.Np, 256), 256, 0, st_>>>(L.Np, L.b, L.gb, L.mb, L.vb, lr, c1, c2);
    refresh_bf16(L);
}

// The graph's edges by source, for the backward pass: laid out once a graph.
void Surrogate::order_by_source() {
    const int n = g_.n, E = g_.E;
    if (g_.by_source || E <= 0) return;
    int* const placed = reinterpret_cast<int*>(M_);  // free between the forward pass and the next: 128 words an edge
    int* const arrival = placed + E;
    cu(cudaMemsetAsync(cnt_, 0, (size_t)(n + 1) * 4, st_), "memset");
    k_source_count<<<blocks(E, 256), 256, 0, st_>>>(E, g_.src, cnt_, arrival);
    scan_counts(n, g_.srow);
    k_source_place<<<blocks(E, 256), 256, 0, st_>>>(E, g_.src, g_.srow, arrival, placed);
    k_source_order<<<blocks(E, 256), 256, 0, st_>>>(E, g_.src, g_.srow, placed, g_.by_src);
    cu(cudaGetLastError(), "edges by source");
    g_.by_source = true;
}

float Surrogate::train_step(float lr) {
    forward(true);
    order_by_source();
    const int n = g_.n, E = g_.E;
    const size_t nW = (size_t)n * kWidth;
    std::vector<uint8_t> fl(n);
    cu(cudaMemcpyAsync(fl.data(), g_.fluid, n, cudaMemcpyDeviceToHost, st_), "fluid");
    cu(cudaMemsetAsync(loss_, 0, 4, st_), "memset");
    for (Linear& L : layers_) cu(cudaMemsetAsync(L.gb, 0, (size_t)L.Np * 4, st_), "memset");
    cu(cudaStreamSynchronize(st_), "fluid");
    int nf = 0;
    for (uint8_t v : fl) nf += v ? 1 : 0;
    k_loss<<<blocks(n, 256), 256, 0, st_>>>(n, Y_, target_, g_.fluid, 1.f / (float)std::max(nf, 1), dY_, loss_);
    mlp_bwd(19, hb_[2], n, da1_, da2_, dY_, dH_);
    for (int l = 1; l >= 0; --l) {
        const int base = 3 + 8 * l;
        k_mask_rows<<<blocks(nW, 256), 256, 0, st_>>>(n, dH_, g_.fluid, U_);
        mlp_bwd(base + 5, xn_[l], n, na1_[l], na2_[l], U_, dXN_);
        k_split_dxn<<<blocks(nW, 256), 256, 0, st_>>>(n, dH_, dXN_, kAggScale, dHp_, A_);
        if (E > 0) {
            linear_bwd(layers_[base + 4], eh2_[l], E, A_, nullptr, dE2_, g_.dst);  // the messages' rows of A_
            linear_bwd(layers_[base + 3], eh1_[l], E, dE2_, eh2_[l], dE_);
            linear_bwd(layers_[base + 2], g_.xe, E, dE_, eh1_[l], nullptr);  // masks dE_ to dZ1
            k_segsum<<<blocks((size_t)n * 32, 256), 256, 0, st_>>>(n, g_.row, dE_, 1.f, dP_);
            k_source_sum<<<blocks((size_t)n * 32, 256), 256, 0, st_>>>(n, g_.srow, g_.by_src, dE_, dQ_);
            linear_bwd(layers_[base + 0], hb_[l], n, dP_, nullptr, dT1_);
            k_add<<<blocks(nW, 256), 256, 0, st_>>>(nW, dHp_, dT1_);
            linear_bwd(layers_[base + 1], hb_[l], n, dQ_, nullptr, dT1_);
            k_add<<<blocks(nW, 256), 256, 0, st_>>>(nW, dHp_, dT1_);
        } else {
            for (int k = 0; k < 5; ++k) {
                Linear& L = layers_[base + k];
                cu(cudaMemsetAsync(L.gWt, 0, (size_t)L.Np * L.K * 4, st_), "memset");
            }
        }
        std::swap(dH_, dHp_);
    }
    mlp_bwd(0, g_.f, n, enc_a1_, enc_a2_, dH_, nullptr);
    if (lr > 0.f) {
        ++adam_t_;
        for (Linear& L : layers_) adam(L, lr);
    }
    float loss = 0.f;
    cu(cudaMemcpyAsync(&loss, loss_, 4, cudaMemcpyDeviceToHost, st_), "loss");
    cu(cudaStreamSynchronize(st_), "train");
    cu(cudaGetLastError(), "train");
    return loss;
}

void Surrogate::set_graph(int n, int E, const int* row, const int* src, const float* f, const float* xe,
                          const uint8_t* fluid) {
    ensure_graph(n, E);
    std::vector<int> dst(E);
    for (int i = 0; i < n; ++i)
        for (int e = row[i]; e < row[i + 1]; ++e) dst[e] = i;
    std::vector<__nv_bfloat16> fb((size_t)n * kNodeFeat), xb((size_t)E * kEdgeFeat);
    for (size_t i = 0; i < fb.size(); ++i) fb[i] = __float2bfloat16_rn(f[i]);
    for (size_t i = 0; i < xb.size(); ++i) xb[i] = __float2bfloat16_rn(xe[i]);
    cu(cudaMemcpyAsync(g_.row, row, (size_t)(n + 1) * 4, cudaMemcpyHostToDevice, st_), "graph");
    if (E) {
        cu(cudaMemcpyAsync(g_.src, src, (size_t)E * 4, cudaMemcpyHostToDevice, st_), "graph");
        cu(cudaMemcpyAsync(g_.dst, dst.data(), (size_t)E * 4, cudaMemcpyHostToDevice, st_), "graph");
        cu(cudaMemcpyAsync(g_.xe, xb.data(), xb.size() * 2, cudaMemcpyHostToDevice, st_), "graph");
    }
    cu(cudaMemcpyAsync(g_.f, fb.data(), fb.size() * 2, cudaMemcpyHostToDevice, st_), "graph");
    cu(cudaMemcpyAsync(g_.fluid, fluid, (size_t)n, cudaMemcpyHostToDevice, st_), "graph");
    cu(cudaStreamSynchronize(st_), "graph");
}

void Surrogate::set_targets(const float* t) {
    cu(cudaMemcpyAsync(target_, t, (size_t)g_.n * kOut * 4, cudaMemcpyHostToDevice, st_), "targets");
    cu(cudaStreamSynchronize(st_), "targets");
}

uint32_t Surrogate::device_error() {
    uint32_t e = 0;
    cu(cudaMemcpyAsync(&e, err_, 4, cudaMemcpyDeviceToHost, st_), "err");
    cu(cudaStreamSynchronize(st_), "err");
    return e;
}

}  // namespace pe

// The end of a post-norm layer with a token input, for steps of few tokens, in one kernel:
//
//   s = alpha x + delta;              x1 = keep x + s / rms(s) * w1                (the layer's last post-norm)
//   z = Wg x1;  g = gelu_tanh(z) * table[token, column0 ..];  y = Wp g             (the token's own input)
//   x <- x1 + y / rms(y) * w2,  and a copy of x in bfloat16
//
// In a decode step these are five launches (norm, product, gate, product, norm) of 2.3 to 3 us each that hardly move any
// bytes: what they cost is handing over.  Here a cluster of 8 CTAs holds the rows of TB tokens, an eighth of the columns
// each.  Both weights' parts of a CTA (Wg: D rows of its columns; Wp: the rows of its columns) and the table's rows are
// fetched while the kernel before this one still runs, into REGISTERS: that kernel is a product whose two CTAs leave an SM
// 7 KB of shared memory, and a CTA that needs more cannot start before they are gone (with the weights in shared memory
// a launch took 11.5 us of the step instead of 7.6).  The three sums that need whole rows (two norms, z) cross the
// cluster through distributed shared memory, every CTA adding the eight parts in rank order.
// (One CTA per token walked 1 MB of weights at its loads' latency: 47 us.)
//
// Precision is that of the five kernels: float32 sums, x1 and g rounded to bfloat16 where they enter a product.
#include "common.cuh"
#include "mma_helpers.cuh"

using namespace mhb;

MHB_EXPORT const char* mhb_last_error() { return error_buffer(); }

namespace {
constexpr int CLUSTER = 8;
constexpr int THREADS = 256;
constexpr int WARPS = THREADS / 32;

struct SideArgs {
    float* x;                      // [T, W]
    const float* delta;            // nsplit parts [T, W], split_stride elements apart
    int nsplit;
    size_t split_stride;
    const float* w1;
    float eps1, alpha, keep;
    const __nv_bfloat16* gate;     // [D, W]
    const __nv_bfloat16* proj;     // [W, D]
    const __nv_bfloat16* table;    // [vocab, table_width]
    int table_width, column0, vocab;
    const int* tokens;
    const float* w2;
    float eps2;
    __nv_bfloat16* copy;           // [T, W]
    int* status;
    int T, W, D;
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// a float into the shared memory of CTA `rank` of the cluster, at the place that `p` has in this CTA's
__device__ __forceinline__ void st_peer(float* p, uint32_t rank, float v) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ float rounded(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ float gelu_tanhf(float z) {
    const float c = 0.7978845608028654f;      // sqrt(2 / pi)
    return 0.5f * z * (1.f + tanhf(c * (z + 0.044715f * z * z * z)));
}
// as the norms of postnorm.cu write it
__device__ __forceinline__ float normed(float s, float rstd, float weight, float keep, float x) {
    const float n = __fmul_rn(s, rstd);
    return keep != 0.f ? fmaf(n, weight, __fmul_rn(keep, x)) : __fmul_rn(n, weight);
}
__device__ __forceinline__ float4 normed(const float4& s, float rstd, const float4& w, float keep, const float4& x) {
    return make_float4(normed(s.x, rstd, w.x, keep, x.x), normed(s.y, rstd, w.y, keep, x.y), normed(s.z, rstd, w.z, keep, x.z),
                       normed(s.w, rstd, w.w, keep, x.w));
}
__device__ __forceinline__ float squares(const float4& s) {
    return fmaf(s.w, s.w, fmaf(s.z, s.z, fmaf(s.x, s.x, __fmul_rn(s.y, s.y))));
}
// eight values a lane -> value (lane >> 2) of the warp's sums, on four lanes each
__device__ __forceinline__ float warp_sum8(float (&v)[8], int lane) {
#pragma unroll
    for (int half = 4, bit = 16; half >= 1; half >>= 1, bit >>= 1) {
        const bool up = lane & bit;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float other = __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + half], bit);
            v[i] = (up ? v[i + half] : v[i]) + other;
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// Shared memory, floats: [rows TB x S][second TB x S][e TB x D][g TB x D][z parts CLUSTER x TB x D][two sums CLUSTER x TB]
// [warp sums TB x 32]
size_t smem_bytes(int TB, int S, int D) {
    return 4 * ((size_t)2 * TB * S + 2 * TB * D + CLUSTER * TB * D + 2 * CLUSTER * TB + 32 * TB);
}
__device__ __forceinline__ float low(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float high(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }

// CH: a CTA's columns are CH runs of 128
template <int TB, int CH>
__global__ void __launch_bounds__(THREADS)
side_branch_kernel(const SideArgs a) {
    extern __shared__ __align__(16) float rows[];      // alpha x + delta, then x1
    constexpr int S = CH * 128, CP = (S + THREADS - 1) / THREADS;
    const int W = a.W, D = a.D;
    const int rank = (int)cluster_rank(), t0 = ((int)blockIdx.x / CLUSTER) * TB, col0 = rank * S;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* second = rows + TB * S;                // x1 rounded, then y
    float* es = second + TB * S;
    float* gs = es + TB * D;
    float* zp = gs + TB * D;
    float* sum1 = zp + CLUSTER * TB * D;
    float* sum2 = sum1 + CLUSTER * TB;
    float* wsum = sum2 + CLUSTER * TB;            // [TB][32]

    pdl_launch_dependents();
    // constant: this warp's eight rows of the gate weight (four columns a lane and run), this thread's rows of the projection
    uint2 wg[8][CH];
    uint4 wp[CP][8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int k = 0; k < CH; ++k)
            wg[j][k] = 8 * warp < D ? __ldg((const uint2*)(a.gate + (size_t)(8 * warp + j) * W + col0 + k * 128 + 4 * lane)) : make_uint2(0, 0);
#pragma unroll
    for (int i = 0; i < CP; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j)
            wp[i][j] = 8 * j < D && tid + i * THREADS < S ? __ldg((const uint4*)(a.proj + (size_t)(col0 + tid + i * THREADS) * D + 8 * j))
                                                           : make_uint4(0, 0, 0, 0);
    bool outside = false;
    for (int i = tid; i < TB * D; i += THREADS) {
        const int tb = i / D, j = i - tb * D;
        float e = 0.f;
        if (t0 + tb < a.T) {
            const int tok = a.tokens[t0 + tb];
            if (tok >= 0 && tok < a.vocab) e = __bfloat162float(a.table[(size_t)tok * a.table_width + a.column0 + j]);
            else outside = true;
        }
        es[i] = e;
    }
    cluster_sync();            // all eight run: their shared memory may be written
    pdl_wait();
    if (outside && rank == 0 && a.status) atomicOr(a.status, 1);

    // ---- s and its squares: a warp takes 128 columns of one token at a time
    constexpr int chunks = CH;
    for (int u = warp; u < TB * chunks; u += WARPS) {
        const int tb = u / chunks, c = (u - tb * chunks) * 128 + 4 * lane;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t0 + tb < a.T) {
            const size_t at = (size_t)(t0 + tb) * W + col0 + c;
            s = sum_parts4<8>(a.delta + at, a.nsplit, a.split_stride);
            if (a.alpha != 0.f) {
                const float4 v = vec4(a.x + at);
                s.x = fmaf(a.alpha, v.x, s.x); s.y = fmaf(a.alpha, v.y, s.y); s.z = fmaf(a.alpha, v.z, s.z); s.w = fmaf(a.alpha, v.w, s.w);
            }
        }
        *(float4*)(rows + tb * S + c) = s;
        const float ss = warp_sum(squares(s));
        if (lane == 0) wsum[tb * 32 + u - tb * chunks] = ss;
    }
    __syncthreads();
    if (tid < TB * CLUSTER) {
        const int tb = tid / CLUSTER, peer = tid - tb * CLUSTER;
        float ss = 0.f;
        for (int i = 0; i < chunks; ++i) ss += wsum[tb * 32 + i];
        st_peer(sum1 + rank * TB + tb, peer, ss);
    }
    cluster_sync();
    for (int u = warp; u < TB * chunks; u += WARPS) {
        const int tb = u / chunks, c = (u - tb * chunks) * 128 + 4 * lane;
        float total = 0.f;
#pragma unroll
        for (int r = 0; r < CLUSTER; ++r) total += sum1[r * TB + tb];
        const float rstd = 1.f / sqrtf(total / (float)W + a.eps1);
        float4 n = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t0 + tb < a.T) {
            const float4 v = a.keep != 0.f ? vec4(a.x + (size_t)(t0 + tb) * W + col0 + c) : n;
            n = normed(vec4(rows + tb * S + c), rstd, vec4(a.w1 + col0 + c), a.keep, v);
        }
        *(float4*)(rows + tb * S + c) = n;
        *(float4*)(second + tb * S + c) = make_float4(rounded(n.x), rounded(n.y), rounded(n.z), rounded(n.w));
    }
    __syncthreads();

    // ---- this CTA's part of z: a warp takes eight rows of the gate weight
    if (8 * warp < D) {
        float acc[TB][8];
#pragma unroll
        for (int tb = 0; tb < TB; ++tb)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[tb][j] = 0.f;
#pragma unroll
        for (int k = 0; k < CH; ++k) {
            float4 h[TB];
#pragma unroll
            for (int tb = 0; tb < TB; ++tb) h[tb] = vec4(second + tb * S + k * 128 + 4 * lane);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint2 w = wg[j][k];
#pragma unroll
                for (int tb = 0; tb < TB; ++tb)
                    acc[tb][j] = fmaf(h[tb].w, high(w.y), fmaf(h[tb].z, low(w.y), fmaf(h[tb].y, high(w.x), fmaf(h[tb].x, low(w.x), acc[tb][j]))));
            }
        }
#pragma unroll
        for (int tb = 0; tb < TB; ++tb) {
            const float z = warp_sum8(acc[tb], lane);
            float* slot = zp + (rank * TB + tb) * D + warp * 8 + (lane >> 2);
            st_peer(slot, 2 * (lane & 3), z);
            st_peer(slot, 2 * (lane & 3) + 1, z);
        }
    }
    cluster_sync();
    for (int i = tid; i < TB * D; i += THREADS) {
        float z = 0.f;
#pragma unroll
        for (int r = 0; r < CLUSTER; ++r) z += zp[r * TB * D + i];
        gs[i] = rounded(gelu_tanhf(z) * es[i]);
    }
    __syncthreads();

    // ---- y of this CTA's columns, a column a thread, and its squares
    float ss[TB];
#pragma unroll
    for (int tb = 0; tb < TB; ++tb) ss[tb] = 0.f;
#pragma unroll
    for (int i = 0; i < CP; ++i) {
        const int c = tid + i * THREADS;
        if (c >= S) break;
        float y[TB];
#pragma unroll
        for (int tb = 0; tb < TB; ++tb) y[tb] = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (8 * j >= D) break;
            const uint4 w = wp[i][j];
#pragma unroll
            for (int tb = 0; tb < TB; ++tb) {
                const float4 g0 = vec4(gs + tb * D + 8 * j), g1 = vec4(gs + tb * D + 8 * j + 4);
                y[tb] = fmaf(high(w.y), g0.w, fmaf(low(w.y), g0.z, fmaf(high(w.x), g0.y, fmaf(low(w.x), g0.x, y[tb]))));
                y[tb] = fmaf(high(w.w), g1.w, fmaf(low(w.w), g1.z, fmaf(high(w.z), g1.y, fmaf(low(w.z), g1.x, y[tb]))));
            }
        }
#pragma unroll
        for (int tb = 0; tb < TB; ++tb) {
            second[tb * S + c] = y[tb];
            ss[tb] = fmaf(y[tb], y[tb], ss[tb]);
        }
    }
#pragma unroll
    for (int tb = 0; tb < TB; ++tb) {
        const float s = warp_sum(ss[tb]);
        if (lane == 0) wsum[tb * 32 + warp] = s;
    }
    __syncthreads();
    if (tid < TB * CLUSTER) {
        const int tb = tid / CLUSTER, peer = tid - tb * CLUSTER;
        float s = 0.f;
        for (int i = 0; i < WARPS; ++i) s += wsum[tb * 32 + i];
        st_peer(sum2 + rank * TB + tb, peer, s);
    }
    cluster_sync();            // nobody writes another CTA's shared memory behind it
    for (int u = warp; u < TB * chunks; u += WARPS) {
        const int tb = u / chunks, c = (u - tb * chunks) * 128 + 4 * lane;
        if (t0 + tb >= a.T) continue;
        float total = 0.f;
#pragma unroll
        for (int r = 0; r < CLUSTER; ++r) total += sum2[r * TB + tb];
        const float rstd = 1.f / sqrtf(total / (float)W + a.eps2);
        const float4 n = normed(vec4(second + tb * S + c), rstd, vec4(a.w2 + col0 + c), 1.f, vec4(rows + tb * S + c));
        const size_t at = (size_t)(t0 + tb) * W + col0 + c;
        *(float4*)(a.x + at) = n;
        *(uint2*)(a.copy + at) = make_uint2(pack_bf16(n.x, n.y), pack_bf16(n.z, n.w));
    }
}

// Tokens a cluster: one while 16 clusters (128 CTAs) take them all, up to four.  Beyond 2,048 columns an SM's registers hold
// one CTA and 8 clusters are what runs at once (16 tokens of 4,096: 13.8 us with 16 clusters, 8.3 with 8).
int most_clusters(int W) { return W > 2048 ? 8 : 16; }
int tokens_per_cluster(int T, int W) { return T <= most_clusters(W) ? 1 : T <= 2 * most_clusters(W) ? 2 : 4; }

template <int TB, int CH>
int launch(const SideArgs& a, cudaStream_t stream) {
    auto kern = side_branch_kernel<TB, CH>;
    const size_t smem = smem_bytes(TB, a.W / CLUSTER, a.D);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CLUSTER * ((a.T + TB - 1) / TB));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CLUSTER;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a);
    if (e != cudaSuccess) return fail("side_branch: %s", cudaGetErrorString(e));
    return check_launch("side_branch");
}
}  // namespace

// Widths of 1024 to 4096 in steps of 1024 (an eighth is whole warps' 128 columns), up to 64 tokens (32 beyond 2,048), D in steps of 8 up to 64
// (eight warps' eight rows): what a CTA's registers hold.
MHB_EXPORT int mhb_side_branch_supports(int T, int W, int D) {
    return T >= 1 && W >= 1024 && W <= 4096 && T <= 4 * most_clusters(W) && W % 1024 == 0 && D >= 8 && D <= 64 && D % 8 == 0;
}

template <int CH>
static int by_tokens(const SideArgs& a, cudaStream_t stream) {
    switch (tokens_per_cluster(a.T, a.W)) {
        case 1: return launch<1, CH>(a, stream);
        case 2: return launch<2, CH>(a, stream);
        default: return launch<4, CH>(a, stream);
    }
}

MHB_EXPORT int mhb_side_branch(float* x, const float* delta, int nsplit, long long split_stride, const float* w1, float eps1,
                               float alpha, float keep, const void* gate, const void* proj, const void* table,
                               int table_width, int column0, int vocab, const int* tokens, const float* w2, float eps2,
                               void* copy, int T, int W, int D, int* status, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (!mhb_side_branch_supports(T, W, D)) return fail("side_branch: %d tokens of %d with a branch of %d is not built", T, W, D);
    if (column0 < 0 || column0 + D > table_width) return fail("side_branch: columns %d..%d outside a table %d wide", column0, column0 + D, table_width);
    if (nsplit < 1 || split_stride % 4 || (((uintptr_t)x | (uintptr_t)delta | (uintptr_t)w1 | (uintptr_t)w2 | (uintptr_t)gate | (uintptr_t)proj | (uintptr_t)copy) & 15))
        return fail("side_branch: rows and weights must lie on 16 bytes");
    SideArgs a;
    a.x = x; a.delta = delta; a.nsplit = nsplit; a.split_stride = (size_t)split_stride; a.w1 = w1; a.eps1 = eps1;
    a.alpha = alpha; a.keep = keep; a.gate = (const __nv_bfloat16*)gate; a.proj = (const __nv_bfloat16*)proj;
    a.table = (const __nv_bfloat16*)table; a.table_width = table_width; a.column0 = column0; a.vocab = vocab;
    a.tokens = tokens; a.w2 = w2; a.eps2 = eps2; a.copy = (__nv_bfloat16*)copy; a.status = status; a.T = T; a.W = W; a.D = D;
    switch (W / 1024) {
        case 1: return by_tokens<1>(a, stream);
        case 2: return by_tokens<2>(a, stream);
        case 3: return by_tokens<3>(a, stream);
        default: return by_tokens<4>(a, stream);
    }
}

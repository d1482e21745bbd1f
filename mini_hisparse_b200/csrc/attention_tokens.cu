// Causal grouped-query attention of single decoded tokens over the paged KV cache on the CUDA cores: float32 scores,
// softmax and sums, keys and values in float32 or bfloat16.  (Math: mini_hisparse/attention.py:26-35.)
//
// attention_simt.cu deals a tile's query ROWS to its warps, which suits prompts: a decoded token has 1 to 8 rows per KV
// head, so most warps had nothing to do and the others walked every key in turn, some 900 instructions of a lone warp
// per 32 keys.  Here a CTA of 16 warps holds one token (or one of its key splits) and one KV head, and the KEYS are dealt:
// a warp takes every sixteenth run of 32 keys with all rows, keys and values straight from the cache (a lane a key, then
// lanes along a value row), and the warps' (maximum, sum, accumulator) meet once at the end.
// Four requests of up to 281 keys, 3 heads of 32, float32, inside a step: 19.0 us and a merge of 2.7 in attention_simt.cu (cut
// in four); here with 8 warps 5.4 and the merge (cut in four) or 8.2 uncut, so 16 warps: one round of 512 keys, uncut.
// Items are those of attention_simt.cu with one token and all heads of the group; splits leave un-normalised partials.
#include "common.cuh"

using namespace mhb;

MHB_EXPORT const char* mhb_last_error() { return error_buffer(); }

namespace {
constexpr int WARPS = 16;
constexpr int RUN = 32;          // keys of a warp at a time: one per lane
constexpr int ITEM_INTS = 8;

struct TokenArgs {
    const void* q;             // [T, nq, d]
    const void* cache;         // [pages, 2, nkv, P, d] of one layer
    void* out;                 // [T, nq, d]
    float* part_acc;           // [rows, nq, d]
    float* part_ml;            // [rows, nq, 2]
    const int* items;
    const int* block_table;    // [S, width]
    const int* tok_part_row;   // [T]
    int width, nq, nkv, d, P, num_pages;
    float scale;
};

// G: heads of a KV head (at most); DPL: elements of a row per lane
template <typename CT, int G, int DPL>
__global__ void __launch_bounds__(WARPS * 32, 1)
attention_tokens_kernel(const TokenArgs a) {
    extern __shared__ __align__(16) float sh[];        // [G][d] queries, [WARPS][G][d + 2] the warps' parts
    pdl_launch_dependents();
    const int* it = a.items + (size_t)blockIdx.x * ITEM_INTS;
    const int t = it[1], kv_begin = it[5], kv_end = it[6], split = it[7], kvh = blockIdx.y;
    const int* table = a.block_table + (size_t)it[0] * a.width;
    const int d = a.d, groups = a.nq / a.nkv, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const CT* cache = (const CT*)a.cache;
    float* parts = sh + G * d;
    // the cache row of this lane's key in run u (-1: no key)
    auto row_of = [&](int u) {
        const int kp = kv_begin + u * RUN + lane;
        if (kp >= kv_end) return -1;
        const int slot = kp / a.P, page = table[slot];
        return page < 0 || page >= a.num_pages ? -1 : (page * 2 * a.nkv + kvh) * a.P + (kp - slot * a.P);
    };
    const int runs = (kv_end - kv_begin + RUN - 1) / RUN;
    int row = warp < runs ? row_of(warp) : -1;          // index arrays do not change during a step
    pdl_wait();
    const CT* q = (const CT*)a.q + ((size_t)t * a.nq + (size_t)kvh * groups) * d;
    for (int i = threadIdx.x; i < G * d; i += WARPS * 32) sh[i] = i < groups * d ? to_float(q[i]) : 0.f;
    __syncthreads();

    float m[G], l[G], acc[G][DPL];
#pragma unroll
    for (int r = 0; r < G; ++r) {
        m[r] = -INFINITY;
        l[r] = 0.f;
#pragma unroll
        for (int i = 0; i < DPL; ++i) acc[r][i] = 0.f;
    }
    for (int u = warp; u < runs; u += WARPS) {
        const int keys = min(RUN, kv_end - kv_begin - u * RUN);
        float s[G];
#pragma unroll
        for (int r = 0; r < G; ++r) s[r] = 0.f;
        const CT* k = cache + (size_t)max(row, 0) * d;
#pragma unroll 4
        for (int e = 0; e < d; e += 4) {
            const float4 k4 = vec4(k + e);
#pragma unroll
            for (int r = 0; r < G; ++r) {
                const float4 q4 = *(const float4*)(sh + r * d + e);
                s[r] = fmaf(q4.w, k4.w, fmaf(q4.z, k4.z, fmaf(q4.y, k4.y, fmaf(q4.x, k4.x, s[r]))));
            }
        }
        float p[G];
#pragma unroll
        for (int r = 0; r < G; ++r) {
            const float x = lane < keys ? (row >= 0 ? s[r] * a.scale : 0.f) : -INFINITY;
            const float m_new = fmaxf(m[r], warp_max(x)), m_use = m_new == -INFINITY ? 0.f : m_new;
            const float alpha = expf(m[r] - m_use);
            p[r] = expf(x - m_use);
            m[r] = m_new;
            l[r] = l[r] * alpha + p[r];                            // this lane's keys; the lanes' sums meet at the end
#pragma unroll
            for (int i = 0; i < DPL; ++i) acc[r][i] *= alpha;
        }
#pragma unroll 8
        for (int j = 0; j < keys; ++j) {
            const int rj = __shfl_sync(0xffffffffu, row, j);
            const CT* v = cache + ((size_t)max(rj, 0) + (size_t)a.nkv * a.P) * d;
            float x[DPL];
#pragma unroll
            for (int i = 0; i < DPL; ++i) x[i] = rj >= 0 && lane + 32 * i < d ? to_float(v[lane + 32 * i]) : 0.f;
#pragma unroll
            for (int r = 0; r < G; ++r) {
                const float pj = __shfl_sync(0xffffffffu, p[r], j);
#pragma unroll
                for (int i = 0; i < DPL; ++i) acc[r][i] = fmaf(pj, x[i], acc[r][i]);
            }
        }
        if (u + WARPS < runs) row = row_of(u + WARPS);
    }
#pragma unroll
    for (int r = 0; r < G; ++r) {
        if (r >= groups) break;
        float* dst = parts + (warp * G + r) * (d + 2);
        const float sum = warp_sum(l[r]);
#pragma unroll
        for (int i = 0; i < DPL; ++i)
            if (lane + 32 * i < d) dst[lane + 32 * i] = acc[r][i];
        if (lane == 0) { dst[d] = m[r]; dst[d + 1] = sum; }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < groups * d; i += WARPS * 32) {
        const int r = i / d, e = i - r * d;
        const float* src = parts + r * (d + 2);
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) M = fmaxf(M, src[w * G * (d + 2) + d]);
        float o = 0.f, sum = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float* part = src + w * G * (d + 2);
            const float f = part[d] == -INFINITY ? 0.f : expf(part[d] - M);
            o = fmaf(f, part[e], o);
            sum = fmaf(f, part[d + 1], sum);
        }
        const size_t h = (size_t)kvh * groups + r;
        if (split < 0) {
            ((CT*)a.out)[((size_t)t * a.nq + h) * d + e] = from_float<CT>(sum > 0.f ? o / sum : 0.f);
        } else {
            const size_t prow = ((size_t)a.tok_part_row[t] + split) * a.nq + h;
            a.part_acc[prow * d + e] = o;
            if (e == 0) { a.part_ml[2 * prow] = M; a.part_ml[2 * prow + 1] = sum; }
        }
    }
}

template <typename CT, int G, int DPL>
int launch(const TokenArgs& a, int num_items, cudaStream_t stream) {
    auto kern = attention_tokens_kernel<CT, G, DPL>;
    const size_t smem = sizeof(float) * ((size_t)G * a.d + (size_t)WARPS * G * (a.d + 2));
    if (smem > 47 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return fail("attention_tokens: shared memory %zu: %s", smem, cudaGetErrorString(e));
    }
    launch_kernel(kern, dim3(num_items, a.nkv), dim3(WARPS * 32), smem, stream, a);
    return check_launch("attention_tokens");
}

template <typename CT, int G>
int by_width(const TokenArgs& a, int num_items, cudaStream_t stream) {
    return a.d <= 32 ? launch<CT, G, 1>(a, num_items, stream) : a.d <= 64 ? launch<CT, G, 2>(a, num_items, stream)
                                                                          : launch<CT, G, 4>(a, num_items, stream);
}
}  // namespace

// Head sizes in steps of 4 up to 128, up to 8 heads per KV head, a pool of fewer than 2^31 rows.
MHB_EXPORT int mhb_attention_tokens_supports(int nq, int nkv, int d, int P, long long num_pages) {
    return nkv > 0 && nkv <= 65535 && nq % nkv == 0 && nq / nkv <= 8 && d >= 4 && d <= 128 && d % 4 == 0 && P >= 1 &&
           num_pages * 2 * nkv * P <= 0x7fffffffLL;
}

MHB_EXPORT int mhb_attention_tokens(const void* q, const void* cache, void* out, int dtype, float* part_acc, float* part_ml,
                                    const int* items, int num_items, const int* block_table, int width,
                                    const int* tok_part_row, int nq, int nkv, int d, int P, int num_pages, float scale,
                                    cudaStream_t stream) {
    if (num_items <= 0) return 0;
    if (!mhb_attention_tokens_supports(nq, nkv, d, P, num_pages) || ((uintptr_t)cache & 15))
        return fail("attention_tokens: %d query heads over %d KV heads of %d is not built", nq, nkv, d);
    const TokenArgs a = {q, cache, out, part_acc, part_ml, items, block_table, tok_part_row, width, nq, nkv, d, P, num_pages, scale};
    const int groups = nq / nkv;
    MHB_DISPATCH_DTYPE(dtype, CT, {
        return groups == 1   ? by_width<CT, 1>(a, num_items, stream)
               : groups == 2 ? by_width<CT, 2>(a, num_items, stream)
               : groups <= 4 ? by_width<CT, 4>(a, num_items, stream)
                             : by_width<CT, 8>(a, num_items, stream);
    });
}

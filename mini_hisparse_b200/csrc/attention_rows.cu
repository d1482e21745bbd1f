// Causal grouped-query attention of prompt portions over the paged KV cache on the CUDA cores: float32 scores, softmax and
// sums, keys and values in float32 or bfloat16.  (Math: mini_hisparse/model.py:173-179.)
//
// attention_simt.cu gives a CTA 16 query rows and a lane a key: every key and value is read from shared memory once per one
// to four rows of a warp, and a tile's chain of reductions and shuffles sets the pace (three prompts of 250, 187 and 125
// tokens, 28 heads of 128: 172 us a layer).  Here a CTA of 256 threads holds 64 query rows and walks tiles of 32 keys like
// two small matrix products: a thread has 4 rows x 2 keys of the scores and 4 rows x 4 (or 8) columns of the output, so an
// operand read from shared memory is used eight to sixteen times; the next tile waits in registers meanwhile: 84 us.
// Items are those of attention_simt.cu (unsplit ones), planned for tiles of 64 rows.
#include "common.cuh"

using namespace mhb;

MHB_EXPORT const char* mhb_last_error() { return error_buffer(); }

namespace {
constexpr int ROWS = 64;         // query rows of a CTA: 16 groups of 4
constexpr int KT = 32;           // keys of a tile: 2 per thread
constexpr int THREADS = 256;
constexpr int ITEM_INTS = 8;
constexpr int P_LD = KT + 4;

struct RowArgs {
    const void* q;             // [T, nq, d]
    const void* cache;         // [pages, 2, nkv, P, d] of one layer
    void* out;                 // [T, nq, d]
    const int* items;
    const int* positions;      // [T]
    const int* block_table;    // [S, width]
    int width, nq, nkv, d, P, num_pages, window;
    float scale;
};

__device__ __forceinline__ float dot4(const float4& a, const float4& b, float s) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
}
__device__ __forceinline__ void add_scaled(float4& o, float p, const float4& v) {
    o.x = fmaf(p, v.x, o.x); o.y = fmaf(p, v.y, o.y); o.z = fmaf(p, v.z, o.z); o.w = fmaf(p, v.w, o.w);
}
__device__ __forceinline__ void store_row4(float* p, float4 v) { *(float4*)p = v; }
__device__ __forceinline__ void store_row4(__nv_bfloat16* p, float4 v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    *(uint2*)p = make_uint2(*(const uint32_t*)&a, *(const uint32_t*)&b);
}

size_t smem_bytes(int d) { return sizeof(float) * ((size_t)(ROWS + KT) * (d + 4) + (size_t)KT * d + ROWS * P_LD); }

// C: runs of 64 columns of a head
template <typename CT, int C>
__global__ void __launch_bounds__(THREADS, 2)
attention_rows_kernel(const RowArgs a) {
    extern __shared__ __align__(16) float sh[];
    const int d = a.d, ld = d + 4, quads = d >> 2;
    float* qs = sh;                          // [ROWS][ld]
    float* ks = qs + ROWS * ld;              // [KT][ld]
    float* vs = ks + KT * ld;                // [KT][d]
    float* ps = vs + KT * d;                 // [ROWS][P_LD]
    __shared__ int row_pos[ROWS];
    pdl_launch_dependents();
    const int* it = a.items + (size_t)blockIdx.x * ITEM_INTS;
    const int seg = it[0], tok0 = it[1], ntok = it[2], head0 = it[3], nheads = it[4], kv_begin = it[5], kv_end = it[6];
    const int kvh = blockIdx.y, groups = a.nq / a.nkv, nrows = ntok * nheads;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int* table = a.block_table + (size_t)seg * a.width;
    const CT* q = (const CT*)a.q;
    const CT* cache = (const CT*)a.cache;
    if (tid < ROWS) row_pos[tid] = tid < nrows ? a.positions[tok0 + tid / nheads] : -1;
    pdl_wait();
    for (int i = tid; i < ROWS * quads; i += THREADS) {
        const int r = i / quads, e = (i - r * quads) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < nrows) v = vec4(q + ((size_t)(tok0 + r / nheads) * a.nq + kvh * groups + head0 + r % nheads) * d + e);
        *(float4*)(qs + r * ld + e) = v;
    }
    // this thread's part of a tile: quads `tx`, tx + 16 of the keys and values ty, ty + 16
    float4 kn[2][C], vn[2][C];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int kp = k0 + ty + 16 * h;
            int page = -1;
            if (kp < kv_end) page = table[kp / a.P];
            const bool in = page >= 0 && page < a.num_pages;
            const size_t row = in ? ((size_t)page * 2 * a.nkv + kvh) * a.P + kp % a.P : 0;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int e = 4 * (tx + 16 * c);
                const bool live = in && e < d;
                kn[h][c] = live ? vec4(cache + row * d + e) : make_float4(0.f, 0.f, 0.f, 0.f);
                vn[h][c] = live ? vec4(cache + (row + (size_t)a.nkv * a.P) * d + e) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    };
    float m[4], l[4];
    float4 o[4][C];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < C; ++c) o[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (kv_begin < kv_end) fetch(kv_begin);
    for (int k0 = kv_begin; k0 < kv_end; k0 += KT) {
        __syncthreads();          // the tile before has been read (and, the first time, the queries are there)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int e = 4 * (tx + 16 * c), r = ty + 16 * h;
                if (e < d) {
                    *(float4*)(ks + r * ld + e) = kn[h][c];
                    *(float4*)(vs + r * d + e) = vn[h][c];
                }
            }
        __syncthreads();
        if (k0 + KT < kv_end) fetch(k0 + KT);
        float s[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i][0] = s[i][1] = 0.f;
#pragma unroll 4
        for (int e = 0; e < d; e += 4) {
            const float4 k1 = vec4(ks + tx * ld + e), k2 = vec4(ks + (tx + 16) * ld + e);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 q4 = vec4(qs + (4 * ty + i) * ld + e);
                s[i][0] = dot4(q4, k1, s[i][0]);
                s[i][1] = dot4(q4, k2, s[i][1]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int qp = row_pos[4 * ty + i];
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int kp = k0 + tx + 16 * j;
                const bool valid = kp < kv_end && kp <= qp && (a.window <= 0 || kp > qp - a.window);
                s[i][j] = valid ? s[i][j] * a.scale : -INFINITY;
                mx = fmaxf(mx, s[i][j]);
            }
#pragma unroll
            for (int b = 8; b > 0; b >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, b));
            const float m_new = fmaxf(m[i], mx), m_use = m_new == -INFINITY ? 0.f : m_new;
            const float alpha = expf(m[i] - m_use), p0 = expf(s[i][0] - m_use), p1 = expf(s[i][1] - m_use);
            m[i] = m_new;
            l[i] = l[i] * alpha + (p0 + p1);          // this thread's keys; the 16 threads of a row meet at the end
            ps[(4 * ty + i) * P_LD + tx] = p0;
            ps[(4 * ty + i) * P_LD + tx + 16] = p1;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                o[i][c].x *= alpha; o[i][c].y *= alpha; o[i][c].z *= alpha; o[i][c].w *= alpha;
            }
        }
        __syncwarp();             // a row's weights are written and read by the same half of a warp
#pragma unroll 2
        for (int j = 0; j < KT; j += 4) {
            float4 p[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) p[i] = vec4(ps + (4 * ty + i) * P_LD + j);
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int e = 4 * (tx + 16 * c);
                if (e >= d) continue;
                const float4 v0 = vec4(vs + j * d + e), v1 = vec4(vs + (j + 1) * d + e), v2 = vec4(vs + (j + 2) * d + e),
                             v3 = vec4(vs + (j + 3) * d + e);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    add_scaled(o[i][c], p[i].x, v0);
                    add_scaled(o[i][c], p[i].y, v1);
                    add_scaled(o[i][c], p[i].z, v2);
                    add_scaled(o[i][c], p[i].w, v3);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int b = 8; b > 0; b >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], b);
        const int r = 4 * ty + i;
        if (r >= nrows) continue;
        CT* dst = (CT*)a.out + ((size_t)(tok0 + r / nheads) * a.nq + kvh * groups + head0 + r % nheads) * d;
        const float sum = l[i];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const int e = 4 * (tx + 16 * c);
            if (e >= d) continue;
            const float4 v = o[i][c];
            store_row4(dst + e, sum > 0.f ? make_float4(v.x / sum, v.y / sum, v.z / sum, v.w / sum) : make_float4(0.f, 0.f, 0.f, 0.f));
        }
    }
}

template <typename CT, int C>
int launch(const RowArgs& a, int num_items, cudaStream_t stream) {
    auto kern = attention_rows_kernel<CT, C>;
    const size_t smem = smem_bytes(a.d);
    if (smem > 47 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return fail("attention_rows: shared memory %zu: %s", smem, cudaGetErrorString(e));
    }
    launch_kernel(kern, dim3(num_items, a.nkv), dim3(THREADS), smem, stream, a);
    return check_launch("attention_rows");
}
}  // namespace

// Unsplit items of tiles of up to 64 query rows; head sizes in steps of 4 up to 128.
MHB_EXPORT int mhb_attention_rows(const void* q, const void* cache, void* out, int dtype, const int* items, int num_items,
                                  const int* positions, const int* block_table, int width, int nq, int nkv, int d, int P,
                                  int num_pages, int window, float scale, cudaStream_t stream) {
    if (num_items <= 0) return 0;
    if (nkv <= 0 || nkv > 65535 || nq % nkv) return fail("attention_rows: %d query heads over %d KV heads", nq, nkv);
    if (d < 4 || d > 128 || d % 4 || P < 1) return fail("attention_rows: heads of %d, pages of %d keys are not built", d, P);
    if (((uintptr_t)q | (uintptr_t)cache | (uintptr_t)out) & 15) return fail("attention_rows: q, the pool and the output must lie on 16 bytes");
    const RowArgs a = {q, cache, out, items, positions, block_table, width, nq, nkv, d, P, num_pages, window, scale};
    MHB_DISPATCH_DTYPE(dtype, CT, { return d <= 64 ? launch<CT, 1>(a, num_items, stream) : launch<CT, 2>(a, num_items, stream); });
}

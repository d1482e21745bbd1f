// Memory-bound kernels of blocks that normalise AFTER the residual sum, and of mixers that
// normalise or gate their own vectors:
//
//   norm_mix        x <- keep * x + rms(alpha * x + delta) * w, and a copy of x in the compute dtype
//                   (post-norm: keep = 0; a normalised branch added to the stream: alpha = 0, keep = 1)
//   act_rows        relu(z)^2 (and other activations by code, or a plain conversion) of a product that may
//                   come in split-K parts
//   table_gate      gelu_tanh(z[t, j]) * table[token[t], column0 + j]
//   gated_rmsnorm   rms(o) * w * sigmoid(g)
//   qknorm_rope_append   RMS norm over the WHOLE q projection and over the whole k projection (all
//                   heads at once), rotation of the first rdim elements of every head, q to a
//                   matrix, k and v into the pages of the cache
//
// Everything is computed in float32; inputs from a split-K product arrive as `nsplit` float32
// partial matrices `split_stride` elements apart and are summed in index order.
#include "common.cuh"

using namespace mhb;

MHB_EXPORT const char* mhb_last_error() { return error_buffer(); }

namespace {

__device__ __forceinline__ float load_parts(const float* p, size_t idx, int nsplit, size_t split_stride) {
    return sum_parts(p + idx, nsplit, split_stride);
}
template <typename T>
__device__ __forceinline__ float load_parts_t(const T* p, size_t idx, int nsplit, size_t split_stride) {
    return sum_parts(p + idx, nsplit, split_stride);
}

__device__ __forceinline__ float sigmoidf(float z) { return 1.f / (1.f + expf(-z)); }
__device__ __forceinline__ float geluf(float z) { return 0.5f * z * (1.f + erff(z * 0.7071067811865476f)); }
__device__ __forceinline__ float gelu_tanhf(float z) {
    const float c = 0.7978845608028654f;      // sqrt(2 / pi)
    return 0.5f * z * (1.f + tanhf(c * (z + 0.044715f * z * z * z)));
}

template <typename T> __device__ __forceinline__ void store4(T* p, float4 v);
template <> __device__ __forceinline__ void store4<float>(float* p, float4 v) { *(float4*)p = v; }
template <> __device__ __forceinline__ void store4<__nv_bfloat16>(__nv_bfloat16* p, float4 v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    uint2 u;
    u.x = *(const uint32_t*)&a;
    u.y = *(const uint32_t*)&b;
    *(uint2*)p = u;
}
// ---- x <- keep x + rms(alpha x + delta) w ---------------------------------------------------------
template <typename DT, typename OT>
__global__ void norm_mix_kernel(float* __restrict__ x, const DT* __restrict__ delta, int nsplit,
                                size_t split_stride, const float* __restrict__ weight, float eps,
                                float alpha, float keep, OT* __restrict__ copy, int H) {
    extern __shared__ float row[];           // alpha x + delta of this row
    __shared__ float scratch[33];
    pdl_launch_dependents();
    pdl_wait();
    const size_t r = blockIdx.x;
    float* xr = x + r * H;
    float ss = 0.f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        float s = alpha != 0.f ? alpha * xr[i] : 0.f;
        if (delta) s += load_parts_t(delta, r * H + i, nsplit, split_stride);
        row[i] = s;
        ss += s * s;
    }
    const float total = block_sum(ss, scratch);
    const float rstd = 1.f / sqrtf(total / (float)H + eps);
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        float n = row[i] * rstd * weight[i];
        if (keep != 0.f) n += keep * xr[i];
        xr[i] = n;
        if (copy) copy[r * H + i] = from_float<OT>(n);
    }
}

// What the four-element forms below do to a vector.  Every product that is added to something is fused as written here, not
// as a compiler may choose in each kernel, so that all forms round alike.
__device__ __forceinline__ void add_scaled(float4& s, float alpha, const float4& v) {
    s.x = fmaf(alpha, v.x, s.x); s.y = fmaf(alpha, v.y, s.y); s.z = fmaf(alpha, v.z, s.z); s.w = fmaf(alpha, v.w, s.w);
}
__device__ __forceinline__ float squares(const float4& s) {
    return fmaf(s.w, s.w, fmaf(s.z, s.z, fmaf(s.x, s.x, __fmul_rn(s.y, s.y))));
}
__device__ __forceinline__ float normed(float s, float rstd, float weight, float keep, float x) {
    const float n = __fmul_rn(s, rstd);
    return keep != 0.f ? fmaf(n, weight, __fmul_rn(keep, x)) : __fmul_rn(n, weight);
}
__device__ __forceinline__ float4 normed(const float4& s, float rstd, const float4& weight, float keep, const float4& x) {
    return make_float4(normed(s.x, rstd, weight.x, keep, x.x), normed(s.y, rstd, weight.y, keep, x.y),
                       normed(s.z, rstd, weight.z, keep, x.z), normed(s.w, rstd, weight.w, keep, x.w));
}

// The same with the row in registers (H % 4 == 0, every row 16-byte aligned).  The sum of squares is `sums` partial sums in the
// order of norm_mix_wide_kernel below, so that a row's result does not depend on the form: partial sum j takes the vectors j,
// j + sums, ..., M of them.  A thread holds Q partial sums: one where rows are few and a thread's chain of loads is the
// kernel's time (8 rows of 2048 with 18 parts: 6.0 us in the wide form, 4.9 here), up to four where rows are many.
template <typename DT, typename OT, int Q, int M>
__global__ void __launch_bounds__(512 / Q)
norm_mix_vec_kernel(float* __restrict__ x, const DT* __restrict__ delta, int nsplit,
                                    size_t split_stride, const float* __restrict__ weight, float eps,
                                    float alpha, float keep, OT* __restrict__ copy, int H, int sums) {
    __shared__ float scratch[16];
    pdl_launch_dependents();
    const int nvec = H >> 2, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    // vector c = q M + m of this thread; past the end: none
    auto at = [&](int c) {
        const int j = ((c / M) * nwarps + warp) * 32 + lane;
        return j < sums ? j + (c % M) * sums : nvec;
    };
    float4 w = make_float4(0.f, 0.f, 0.f, 0.f);         // constant: fetched while the kernel before this one still runs
    if (Q * M == 1 && at(0) < nvec) w = vec4(weight + 4 * at(0));
    pdl_wait();
    const size_t r = blockIdx.x;
    float* xr = x + r * H;
    float4 v[Q * M], s[Q * M];
#pragma unroll
    for (int c = 0; c < Q * M; ++c) {
        const int i = at(c);
        if (i >= nvec) continue;
        v[c] = s[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (alpha != 0.f || keep != 0.f) v[c] = vec4(xr + 4 * i);
        if (delta) s[c] = sum_parts4<Q == 1 && M <= 2 ? 8 : 2>(delta + r * H + 4 * i, nsplit, split_stride);
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        float ss = 0.f;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int c = q * M + m;
            if (at(c) >= nvec) continue;
            if (alpha != 0.f) add_scaled(s[c], alpha, v[c]);
            ss = __fadd_rn(ss, squares(s[c]));
        }
        ss = warp_sum(ss);
        if (lane == 0 && q * nwarps + warp < sums / 32) scratch[q * nwarps + warp] = ss;
    }
    __syncthreads();
    const float total = warp_sum(lane < sums / 32 ? scratch[lane] : 0.f);
    const float rstd = 1.f / sqrtf(total / (float)H + eps);
#pragma unroll
    for (int c = 0; c < Q * M; ++c) {
        const int i = at(c);
        if (i >= nvec) continue;
        const float4 n = normed(s[c], rstd, Q * M == 1 ? w : vec4(weight + 4 * i), keep, v[c]);
        *(float4*)(xr + 4 * i) = n;
        if (copy) store4<OT>(copy + r * H + 4 * i, n);
    }
}

// Rows of more vectors than 512 threads hold in registers (H > 16384): the row waits in shared memory.
template <typename DT, typename OT>
__global__ void __launch_bounds__(512)
norm_mix_wide_kernel(float* __restrict__ x, const DT* __restrict__ delta, int nsplit,
                                    size_t split_stride, const float* __restrict__ weight, float eps,
                                    float alpha, float keep, OT* __restrict__ copy, int H) {
    extern __shared__ __align__(16) float row[];
    __shared__ float scratch[32];
    pdl_launch_dependents();
    pdl_wait();
    const size_t r = blockIdx.x;
    float* xr = x + r * H;
    float ss = 0.f;
    for (int i = 4 * threadIdx.x; i < H; i += 4 * blockDim.x) {
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        if (delta) s = sum_parts4<8>(delta + r * H + i, nsplit, split_stride);
        if (alpha != 0.f) add_scaled(s, alpha, vec4(xr + i));
        *(float4*)(row + i) = s;
        ss = __fadd_rn(ss, squares(s));
    }
    const float total = block_sum_once(ss, scratch);
    const float rstd = 1.f / sqrtf(total / (float)H + eps);
    for (int i = 4 * threadIdx.x; i < H; i += 4 * blockDim.x) {
        const float4 s = vec4(row + i), n = normed(s, rstd, vec4(weight + i), keep, keep != 0.f ? vec4(xr + i) : s);
        *(float4*)(xr + i) = n;
        if (copy) store4<OT>(copy + r * H + i, n);
    }
}

// ---- activations of a product ----------------------------------------------------------------------
enum { ACT_RELU2 = 0, ACT_SILU = 1, ACT_GELU_TANH = 2, ACT_COPY = 3, ACT_GELU = 4 };

__device__ __forceinline__ float act_of(float v, int act) {
    if (act == ACT_RELU2) { const float a = fmaxf(v, 0.f); return a * a; }
    if (act == ACT_SILU) return v * sigmoidf(v);
    if (act == ACT_GELU_TANH) return gelu_tanhf(v);
    if (act == ACT_GELU) return geluf(v);
    return v;
}

template <typename IT, typename OT>
__global__ void act_rows_kernel(const IT* __restrict__ z, int nsplit, size_t split_stride, OT* __restrict__ out,
                                size_t n, int act) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v = load_parts_t(z, i, nsplit, split_stride);
    out[i] = from_float<OT>(act_of(v, act));
}

// four elements per thread (n % 4 == 0, 16-byte aligned, parts a multiple of four elements apart)
template <typename IT, typename OT, int B>
__global__ void act_rows_vec_kernel(const IT* __restrict__ z, int nsplit, size_t split_stride, OT* __restrict__ out,
                                    size_t n, int act) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t i = 4 * ((size_t)blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= n) return;
    const float4 v = sum_parts4<B>(z + i, nsplit, split_stride);
    store4<OT>(out + i, make_float4(act_of(v.x, act), act_of(v.y, act), act_of(v.z, act), act_of(v.w, act)));
}

// ---- gelu_tanh(z) * table[token, column0 + j] -------------------------------------------------------
template <typename IT, typename WT, typename OT>
__global__ void table_gate_kernel(const IT* __restrict__ z, int nsplit, size_t split_stride,
                                  const WT* __restrict__ table, int table_width, int column0, int vocab,
                                  const int* __restrict__ tokens, OT* __restrict__ out, int T, int D,
                                  int* __restrict__ status) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)T * D) return;
    const int t = (int)(i / D), j = (int)(i - (size_t)t * D);
    const int tok = tokens[t];
    float e = 0.f;
    if (tok >= 0 && tok < vocab) e = to_float(table[(size_t)tok * table_width + column0 + j]);
    else if (status) atomicOr(status, 1);
    out[i] = from_float<OT>(gelu_tanhf(load_parts_t(z, i, nsplit, split_stride)) * e);
}

// ---- rms(o) * w * sigmoid(g) -------------------------------------------------------------------------
template <typename OT>
__global__ void gated_rmsnorm_kernel(const float* __restrict__ o, const float* __restrict__ gate, int gate_nsplit,
                                     size_t gate_split_stride, int gate_ld, const float* __restrict__ weight,
                                     float eps, OT* __restrict__ out, int N) {
    __shared__ float scratch[33];
    pdl_launch_dependents();
    pdl_wait();
    const size_t r = blockIdx.x;
    const float* orow = o + r * N;
    float ss = 0.f;
    for (int i = threadIdx.x; i < N; i += blockDim.x) { const float v = orow[i]; ss += v * v; }
    const float total = block_sum(ss, scratch);
    const float rstd = 1.f / sqrtf(total / (float)N + eps);
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        float n = orow[i] * rstd * weight[i];
        if (gate) n *= sigmoidf(load_parts(gate, r * gate_ld + i, gate_nsplit, gate_split_stride));
        out[r * N + i] = from_float<OT>(n);
    }
}

// The same with the row and its gate in registers, VC vectors of four elements a thread (N, strides and addresses in 16-byte
// steps).  The sum of squares is that of the kernel above, element by element in its order (`sums`: its threads): a thread reads
// the elements of its partial sums once more, from L1, at the same time as its vectors.
template <typename OT, int VC>
__global__ void __launch_bounds__(512)
gated_rmsnorm_vec_kernel(const float* __restrict__ o, const float* __restrict__ gate, int gate_nsplit,
                                         size_t gate_split_stride, int gate_ld, const float* __restrict__ weight,
                                         float eps, OT* __restrict__ out, int N, int sums) {
    __shared__ float scratch[16];
    pdl_launch_dependents();
    pdl_wait();
    const size_t r = blockIdx.x;
    const int nvec = N >> 2, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const float* row = o + r * N;
    float4 v[VC], g[VC];
#pragma unroll
    for (int c = 0; c < VC; ++c) {
        const int i = threadIdx.x + c * blockDim.x;
        if (i >= nvec) continue;
        v[c] = vec4(row + 4 * i);
        if (gate) g[c] = sum_parts4<VC <= 2 ? 8 : 2>(gate + r * gate_ld + 4 * i, gate_nsplit, gate_split_stride);
    }
    for (int u = warp; u < sums / 32; u += nwarps) {
        float ss = 0.f;
#pragma unroll 8
        for (int i = u * 32 + lane; i < N; i += sums) { const float e = row[i]; ss = fmaf(e, e, ss); }
        ss = warp_sum(ss);
        if (lane == 0) scratch[u] = ss;
    }
    __syncthreads();
    const float total = warp_sum(lane < sums / 32 ? scratch[lane] : 0.f);
    const float rstd = 1.f / sqrtf(total / (float)N + eps);
#pragma unroll
    for (int c = 0; c < VC; ++c) {
        const int i = threadIdx.x + c * blockDim.x;
        if (i >= nvec) continue;
        const float4 w = vec4(weight + 4 * i);
        float4 n = make_float4(v[c].x * rstd * w.x, v[c].y * rstd * w.y, v[c].z * rstd * w.z, v[c].w * rstd * w.w);
        if (gate) { n.x *= sigmoidf(g[c].x); n.y *= sigmoidf(g[c].y); n.z *= sigmoidf(g[c].z); n.w *= sigmoidf(g[c].w); }
        store4<OT>(out + r * N + 4 * i, n);
    }
}

// A rotated pair, fused the same way wherever it is computed
__device__ __forceinline__ float turned_first(float a, float b, float c, float s) { return fmaf(a, c, -__fmul_rn(b, s)); }
__device__ __forceinline__ float turned_second(float a, float b, float c, float s) { return fmaf(a, s, __fmul_rn(b, c)); }

// ---- q/k norm over the whole projection, rotation, append ------------------------------------------
// A row of the product holds [q: nq * dk | k: nkv * dk | v: nkv * dv | anything else]; a layer that
// reads another layer's cache has [q | anything else] and has_kv = 0.  With v_from_k the row holds [q | k | anything
// else] and the values are the keys as projected (with their bias, before norm and rotation; dv = dk).  One page of the
// cache holds [keys: nkv][P][dk] followed by [values: nkv][P][dv].
template <typename QT, typename CT>
__global__ void qknorm_rope_append_kernel(const float* __restrict__ qkv, int nsplit, size_t split_stride, int ld,
                                          const float* __restrict__ q_weight, const float* __restrict__ k_weight,
                                          float eps, const int* __restrict__ positions,
                                          const int* __restrict__ tok_seg, const int* __restrict__ block_table,
                                          int table_width, const float* __restrict__ inv_freq, int rdim,
                                          QT* __restrict__ q_out, CT* __restrict__ cache, int nq, int nkv, int dk,
                                          int dv, int P, int num_pages, int has_kv, int* __restrict__ status,
                                          int per_head, float v_eps, size_t page_extra, float temp_coef,
                                          double temp_every, float v_scale, const float* __restrict__ bias,
                                          int v_from_k) {
    extern __shared__ float sh[];            // q row, k row, cos, sin (and the v row, if it is normalised)
    __shared__ float scratch[33];
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x;
    const int pos = positions[t];
    const int qw = nq * dk, kw = has_kv ? nkv * dk : 0, vw = has_kv ? nkv * dv : 0;
    const int rhalf = rdim >> 1;
    float* qs = sh;
    float* ks = qs + qw;
    float* cs = ks + kw;
    float* sn = cs + rhalf;
    const size_t base = (size_t)t * ld;
    float* vs = sn + rhalf;                  // [vw], only with v_eps > 0 or v_from_k
    float ssq = 0.f, ssk = 0.f;
    for (int i = threadIdx.x; i < qw + kw; i += blockDim.x) {
        const float v = load_parts(qkv, base + i, nsplit, split_stride) + (bias ? bias[i] : 0.f);
        sh[i] = v;
        if (i < qw) ssq += v * v;
        else {
            ssk += v * v;
            if (v_from_k) vs[i - qw] = v;
        }
    }
    for (int i = threadIdx.x; i < rhalf; i += blockDim.x) {
        float s, c;
        sincosf((float)pos * inv_freq[i], &s, &c);
        cs[i] = c;
        sn[i] = s;
    }
    if (v_eps > 0.f && !v_from_k)
        for (int i = threadIdx.x; i < vw; i += blockDim.x) vs[i] = load_parts(qkv, base + qw + kw + i, nsplit, split_stride);
    if (per_head) {
        // one norm per head over its dk elements, the weight [dk] shared by the heads: a warp per head; and a temperature
        // that grows with the position, on q alone: 1 + coef ln(floor((pos + 1) / every) + 1)
        const float temp = temp_coef != 0.f ? 1.f + temp_coef * log1pf((float)floor((double)(pos + 1) / temp_every)) : 1.f;
        __syncthreads();
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
        for (int head = warp; head < (qw + kw) / dk; head += nwarps) {
            float* row = sh + head * dk;
            const float* w = head < nq ? q_weight : k_weight;
            float ss = 0.f;
            for (int e = lane; e < dk; e += 32) ss += row[e] * row[e];
            const float r = 1.f / sqrtf(warp_sum(ss) / (float)dk + eps);
            const float f = head < nq ? temp : 1.f;
            for (int e = lane; e < dk; e += 32) row[e] = row[e] * r * (w ? w[e] : 1.f) * f;
        }
    } else {
        const float tq = block_sum(ssq, scratch);
        const float tk = block_sum(ssk, scratch);
        const float rq = 1.f / sqrtf(tq / (float)qw + eps);
        const float rk = kw ? 1.f / sqrtf(tk / (float)kw + eps) : 0.f;
        for (int i = threadIdx.x; i < qw + kw; i += blockDim.x)
            sh[i] = i < qw ? sh[i] * rq * q_weight[i] : sh[i] * rk * k_weight[i - qw];
    }
    __syncthreads();
    if (v_eps > 0.f) {
        // every head's value divided by its own root mean square (no weight): a warp per head
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
        for (int head = warp; head < (has_kv ? nkv : 0); head += nwarps) {
            float* row = vs + head * dv;
            float ss = 0.f;
            for (int e = lane; e < dv; e += 32) ss += row[e] * row[e];
            const float r = 1.f / sqrtf(warp_sum(ss) / (float)dv + v_eps);
            for (int e = lane; e < dv; e += 32) row[e] *= r;
        }
        __syncthreads();
    }
    CT* page_k = nullptr;
    CT* page_v = nullptr;
    const int within = pos % P;
    if (has_kv) {
        const int page = block_table[(size_t)tok_seg[t] * table_width + pos / P];
        if (page < 0 || page >= num_pages) {          // never write outside the pool
            if (threadIdx.x == 0 && status) atomicOr(status, 2);
        } else {
            page_k = cache + (size_t)page * ((size_t)nkv * P * (dk + dv) + page_extra);
            page_v = page_k + (size_t)nkv * P * dk;
        }
    }
    // one thread per unit: rdim/2 rotated pairs and dk - rdim plain elements per head
    const int units = rhalf + (dk - rdim);
    const int heads = nq + (has_kv ? nkv : 0);
    for (int idx = threadIdx.x; idx < heads * units; idx += blockDim.x) {
        const int head = idx / units, u = idx - head * units;
        const float* src = sh + head * dk;       // k heads follow the q heads in shared memory
        QT* qdst = head < nq ? q_out + (size_t)t * qw + head * dk : nullptr;
        CT* kdst = (head >= nq && page_k) ? page_k + ((size_t)(head - nq) * P + within) * dk : nullptr;
        if (u < rhalf) {
            const float a = src[u], b = src[u + rhalf];
            const float oa = turned_first(a, b, cs[u], sn[u]);
            const float ob = turned_second(a, b, cs[u], sn[u]);
            if (qdst) { qdst[u] = from_float<QT>(oa); qdst[u + rhalf] = from_float<QT>(ob); }
            else if (kdst) { kdst[u] = from_float<CT>(oa); kdst[u + rhalf] = from_float<CT>(ob); }
        } else {
            const int e = rdim + (u - rhalf);
            if (qdst) qdst[e] = from_float<QT>(src[e]);
            else if (kdst) kdst[e] = from_float<CT>(src[e]);
        }
    }
    if (page_v) {
        for (int i = threadIdx.x; i < vw; i += blockDim.x) {
            const int g = i / dv, e = i - g * dv;
            page_v[((size_t)g * P + within) * dv + e] =
                from_float<CT>(v_scale * (v_eps > 0.f || v_from_k ? vs[i] : load_parts(qkv, base + qw + kw + i, nsplit, split_stride)));
        }
    }
}

// The same four elements at a time (head sizes and the rotated width in steps of 4 and 8, rows and strides on 16 bytes): a
// thread asks for all its loads at once, both norms' sums cross the CTA at one barrier, and angles, pages and the
// destination are worked out before the kernel waits for the product.  One element a thread and step, with two block-wide
// sums in turn and the values loaded after them, took 18.4 us for 8 tokens of 16 heads and 67 us for 2,048 of 32; this form
// 12.3 and 45 (caches cold, launch included).  The norms' sums are those of the general kernel, `nsums` partial sums in its order,
// read back from shared memory.
template <typename CT, int B, int MOST>
__global__ void __launch_bounds__(MOST)
qknorm_rope_append_vec_kernel(const float* __restrict__ qkv, int nsplit, size_t split_stride, int ld,
                                              const float* __restrict__ q_weight, const float* __restrict__ k_weight,
                                              float eps, const int* __restrict__ positions,
                                              const int* __restrict__ tok_seg, const int* __restrict__ block_table,
                                              int table_width, const float* __restrict__ inv_freq, int rdim,
                                              CT* __restrict__ q_out, CT* __restrict__ cache, int nq, int nkv, int dk,
                                              int dv, int P, int num_pages, int has_kv, int* __restrict__ status,
                                              int per_head, float v_eps, size_t page_extra, float temp_coef,
                                              double temp_every, float v_scale, const float* __restrict__ bias,
                                              int v_from_k, int nsums) {
    extern __shared__ __align__(16) float sh[];            // q and k rows, cos, sin, the v row if it is kept
    __shared__ float sums[2][32];
    pdl_launch_dependents();
    const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int qw = nq * dk, kw = has_kv ? nkv * dk : 0, vw = has_kv ? nkv * dv : 0, rhalf = rdim >> 1;
    float* cs = sh + qw + kw;
    float* sn = cs + rhalf;
    float* vs = sn + rhalf;
    // positions and block tables do not change during a step
    const int pos = positions[t], within = pos % P;
    for (int i = threadIdx.x; i < rhalf; i += blockDim.x) {
        float sine, cosine;
        sincosf((float)pos * inv_freq[i], &sine, &cosine);
        cs[i] = cosine;
        sn[i] = sine;
    }
    CT* page_k = nullptr;
    CT* page_v = nullptr;
    bool outside = false;
    if (has_kv) {
        const int page = block_table[(size_t)tok_seg[t] * table_width + pos / P];
        outside = page < 0 || page >= num_pages;          // never write outside the pool
        if (!outside) {
            page_k = cache + (size_t)page * ((size_t)nkv * P * (dk + dv) + page_extra);
            page_v = page_k + (size_t)nkv * P * dk;
        }
    }
    pdl_wait();
    if (outside && threadIdx.x == 0 && status) atomicOr(status, 2);
    const float* row = qkv + (size_t)t * ld;
    const bool keep_v = v_eps > 0.f || v_from_k;
    const int loads = (qw + kw + (v_from_k ? 0 : vw)) >> 2;
#pragma unroll (B == 1 ? 4 : 1)
    for (int u = threadIdx.x; u < loads; u += blockDim.x) {
        const int i = 4 * u;
        float4 v = sum_parts4<B>(row + i, nsplit, split_stride);
        if (i < qw + kw) {
            const float4 b = bias ? vec4(bias + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
            *(float4*)(sh + i) = v;
            if (v_from_k && i >= qw) *(float4*)(vs + i - qw) = v;
        } else if (keep_v) {
            *(float4*)(vs + i - qw - kw) = v;
        } else if (page_v) {
            const int e = i - qw - kw, g = e / dv;
            store4<CT>(page_v + ((size_t)g * P + within) * dv + (e - g * dv),
                       make_float4(v_scale * v.x, v_scale * v.y, v_scale * v.z, v_scale * v.w));
        }
    }
    float rq = 1.f, rk = 1.f;
    __syncthreads();
    if (per_head) {
        const float temp = temp_coef != 0.f ? 1.f + temp_coef * log1pf((float)floor((double)(pos + 1) / temp_every)) : 1.f;
        for (int head = warp; head < (qw + kw) / dk; head += nwarps) {
            float* hr = sh + head * dk;
            const float* w = head < nq ? q_weight : k_weight;
            float ss = 0.f;
            for (int e = lane; e < dk; e += 32) ss = fmaf(hr[e], hr[e], ss);
            const float r = 1.f / sqrtf(warp_sum(ss) / (float)dk + eps);
            const float f = head < nq ? temp : 1.f;
            __syncwarp();
            for (int e = 4 * lane; e < dk; e += 128) {
                float4 v = vec4(hr + e);
                const float4 m = w ? vec4(w + e) : make_float4(1.f, 1.f, 1.f, 1.f);
                v.x = v.x * r * m.x * f; v.y = v.y * r * m.y * f; v.z = v.z * r * m.z * f; v.w = v.w * r * m.w * f;
                *(float4*)(hr + e) = v;
            }
        }
    } else {
        // both sums cross the CTA at one barrier; partial sum j takes the elements j, j + nsums, ...
        for (int u = warp; u < nsums / 32; u += nwarps) {
            float ssq = 0.f, ssk = 0.f;
            for (int i = u * 32 + lane; i < qw + kw; i += nsums) {
                const float v = sh[i];
                if (i < qw) ssq = fmaf(v, v, ssq);
                else ssk = fmaf(v, v, ssk);
            }
            ssq = warp_sum(ssq);
            ssk = warp_sum(ssk);
            if (lane == 0) { sums[0][u] = ssq; sums[1][u] = ssk; }
        }
        __syncthreads();
        const float tq = warp_sum(lane < nsums / 32 ? sums[0][lane] : 0.f), tk = warp_sum(lane < nsums / 32 ? sums[1][lane] : 0.f);
        rq = 1.f / sqrtf(tq / (float)qw + eps);
        rk = kw ? 1.f / sqrtf(tk / (float)kw + eps) : 0.f;
    }
    if (v_eps > 0.f) {
        for (int head = warp; head < (has_kv ? nkv : 0); head += nwarps) {
            float* hr = vs + head * dv;
            float ss = 0.f;
            for (int e = lane; e < dv; e += 32) ss = fmaf(hr[e], hr[e], ss);
            const float r = 1.f / sqrtf(warp_sum(ss) / (float)dv + v_eps);
            for (int e = lane; e < dv; e += 32) hr[e] *= r;
        }
    }
    if (per_head || v_eps > 0.f) __syncthreads();
    // a thread per four rotated pairs, or four elements that are not rotated
    auto scaled = [&](int head, int e) {
        float4 v = vec4(sh + head * dk + e);
        if (!per_head) {
            const float r = head < nq ? rq : rk;
            const float4 w = head < nq ? vec4(q_weight + head * dk + e) : vec4(k_weight + (head - nq) * dk + e);
            v.x = v.x * r * w.x; v.y = v.y * r * w.y; v.z = v.z * r * w.z; v.w = v.w * r * w.w;
        }
        return v;
    };
    const int pairs4 = rhalf >> 2, units = pairs4 + ((dk - rdim) >> 2), heads = nq + (has_kv ? nkv : 0);
    for (int idx = threadIdx.x; idx < heads * units; idx += blockDim.x) {
        const int head = idx / units, u = idx - head * units;
        CT* dst = head < nq ? q_out + (size_t)t * qw + head * dk
                  : page_k  ? page_k + ((size_t)(head - nq) * P + within) * dk : nullptr;
        if (!dst) continue;
        if (u < pairs4) {
            const float4 a = scaled(head, 4 * u), b = scaled(head, 4 * u + rhalf), c = vec4(cs + 4 * u), n = vec4(sn + 4 * u);
            store4<CT>(dst + 4 * u, make_float4(turned_first(a.x, b.x, c.x, n.x), turned_first(a.y, b.y, c.y, n.y),
                                                turned_first(a.z, b.z, c.z, n.z), turned_first(a.w, b.w, c.w, n.w)));
            store4<CT>(dst + 4 * u + rhalf, make_float4(turned_second(a.x, b.x, c.x, n.x), turned_second(a.y, b.y, c.y, n.y),
                                                        turned_second(a.z, b.z, c.z, n.z), turned_second(a.w, b.w, c.w, n.w)));
        } else {
            const int e = rdim + 4 * (u - pairs4);
            store4<CT>(dst + e, scaled(head, e));
        }
    }
    if (page_v && keep_v) {
        for (int i = 4 * threadIdx.x; i < vw; i += 4 * blockDim.x) {
            const int g = i / dv;
            const float4 v = vec4(vs + i);
            store4<CT>(page_v + ((size_t)g * P + within) * dv + (i - g * dv),
                       make_float4(v_scale * v.x, v_scale * v.y, v_scale * v.z, v_scale * v.w));
        }
    }
}

int row_threads(int H) {
    int t = (H + 31) / 32 * 32;
    if (t > 512) t = 512;
    if (t < 64) t = 64;
    return t;
}

template <typename Kern>
int allow_smem(Kern kern, size_t smem, const char* what) {
    if (smem > 47 * 1024) {                  // 48 KB without being asked, the static part included
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return fail("%s: shared memory %zu: %s", what, smem, cudaGetErrorString(e));
    }
    return 0;
}
}  // namespace

MHB_EXPORT int mhb_norm_mix(float* x, const void* delta, int delta_dtype, int nsplit, long long split_stride,
                            const float* weight, float eps, float alpha, float keep, void* copy, int copy_dtype,
                            int R, int H, cudaStream_t stream) {
    if (R <= 0) return 0;
    if (nsplit > 1 && delta_dtype != MHB_F32) return fail("norm_mix: split partials must be float32");
    const size_t smem = sizeof(float) * (size_t)H;
    const bool vec = H % 4 == 0 && !((uintptr_t)x & 15) && !((uintptr_t)delta & 15) && !((uintptr_t)weight & 15) &&
                     !((uintptr_t)copy & 15) && split_stride % 4 == 0;
    if (vec) {
        // up to 512 partial sums of M vectors each; a thread takes one of them for up to 128 rows, four vectors beyond
        const int sums = row_threads(H / 4), m = (H / 4 + sums - 1) / sums;
        const bool few = R <= 128;
        MHB_DISPATCH_DTYPE(delta_dtype, DT, MHB_DISPATCH_DTYPE(copy_dtype, OT, {
            if (m > 8) {
                auto kern = norm_mix_wide_kernel<DT, OT>;
                if (allow_smem(kern, smem, "norm_mix")) return -1;
                launch_kernel(kern, dim3(R), dim3(sums), smem, stream, x, (const DT*)delta, nsplit, (size_t)split_stride, weight,
                              eps, alpha, keep, (OT*)copy, H);
            } else {
                const int q = few || m > 2 ? 1 : m == 2 ? 2 : 4;
                auto kern = m > 4 ? norm_mix_vec_kernel<DT, OT, 1, 8> : m > 2 ? norm_mix_vec_kernel<DT, OT, 1, 4>
                            : m == 2 ? (few ? norm_mix_vec_kernel<DT, OT, 1, 2> : norm_mix_vec_kernel<DT, OT, 2, 2>)
                                     : (few ? norm_mix_vec_kernel<DT, OT, 1, 1> : norm_mix_vec_kernel<DT, OT, 4, 1>);
                launch_kernel(kern, dim3(R), dim3((sums / 32 + q - 1) / q * 32), 0, stream, x, (const DT*)delta, nsplit,
                              (size_t)split_stride, weight, eps, alpha, keep, (OT*)copy, H, sums);
            }
        }));
        return check_launch("norm_mix");
    }
    MHB_DISPATCH_DTYPE(delta_dtype, DT, MHB_DISPATCH_DTYPE(copy_dtype, OT, {
        auto kern = norm_mix_kernel<DT, OT>;
        if (allow_smem(kern, smem, "norm_mix")) return -1;
        launch_kernel(kern, dim3(R), dim3(row_threads(H)), smem, stream, x, (const DT*)delta, nsplit,
                      (size_t)split_stride, weight, eps, alpha, keep, (OT*)copy, H);
    }));
    return check_launch("norm_mix");
}

MHB_EXPORT int mhb_act_rows(const void* z, int in_dtype, int nsplit, long long split_stride, void* out,
                            int out_dtype, long long n, int act, cudaStream_t stream) {
    if (n <= 0) return 0;
    if (act < 0 || act > ACT_GELU) return fail("act_rows: unknown activation %d", act);
    if (nsplit > 1 && in_dtype != MHB_F32) return fail("act_rows: split partials must be float32");
    const int threads = 256;
    if (n % 4 == 0 && !((uintptr_t)z & 15) && !((uintptr_t)out & 15) && split_stride % 4 == 0) {
        const unsigned vblocks = (unsigned)((n / 4 + threads - 1) / threads);
        MHB_DISPATCH_DTYPE(in_dtype, IT, MHB_DISPATCH_DTYPE(out_dtype, OT,
            launch_kernel((nsplit == 1 ? act_rows_vec_kernel<IT, OT, 1> : act_rows_vec_kernel<IT, OT, 8>), dim3(vblocks), dim3(threads), 0, stream, (const IT*)z, nsplit,
                          (size_t)split_stride, (OT*)out, (size_t)n, act)));
        return check_launch("act_rows");
    }
    const unsigned blocks = (unsigned)((n + threads - 1) / threads);
    MHB_DISPATCH_DTYPE(in_dtype, IT, MHB_DISPATCH_DTYPE(out_dtype, OT,
        launch_kernel((act_rows_kernel<IT, OT>), dim3(blocks), dim3(threads), 0, stream, (const IT*)z, nsplit,
                      (size_t)split_stride, (OT*)out, (size_t)n, act)));
    return check_launch("act_rows");
}

MHB_EXPORT int mhb_table_gate(const void* z, int in_dtype, int nsplit, long long split_stride, const void* table,
                              int table_dtype, int table_width, int column0, int vocab, const int* tokens,
                              void* out, int out_dtype, int T, int D, int* status, cudaStream_t stream) {
    if (T <= 0 || D <= 0) return 0;
    if (column0 < 0 || column0 + D > table_width) return fail("table_gate: columns %d..%d outside a table %d wide", column0, column0 + D, table_width);
    if (nsplit > 1 && in_dtype != MHB_F32) return fail("table_gate: split partials must be float32");
    const int threads = 256;
    const unsigned blocks = (unsigned)(((size_t)T * D + threads - 1) / threads);
    MHB_DISPATCH_DTYPE(in_dtype, IT, MHB_DISPATCH_DTYPE(table_dtype, WT, MHB_DISPATCH_DTYPE(out_dtype, OT,
        launch_kernel((table_gate_kernel<IT, WT, OT>), dim3(blocks), dim3(threads), 0, stream, (const IT*)z, nsplit,
                      (size_t)split_stride, (const WT*)table, table_width, column0, vocab, tokens, (OT*)out, T, D,
                      status))));
    return check_launch("table_gate");
}

MHB_EXPORT int mhb_gated_rmsnorm(const float* o, const float* gate, int gate_nsplit, long long gate_split_stride,
                                 int gate_ld, const float* weight, float eps, void* out, int out_dtype, int R, int N,
                                 cudaStream_t stream) {
    if (R <= 0) return 0;
    const bool vec = N % 4 == 0 && gate_ld % 4 == 0 && gate_split_stride % 4 == 0 &&
                     !(((uintptr_t)o | (uintptr_t)gate | (uintptr_t)weight | (uintptr_t)out) & 15);
    // a thread for every four elements of up to 128 rows, a quarter as many beyond; 512 at most
    const int sums = row_threads(N), want = R <= 128 ? N / 4 : (N / 4 + 3) / 4;
    const int threads = row_threads(want), vc = (N / 4 + threads - 1) / threads;
    if (vec && vc <= 8) {
        MHB_DISPATCH_DTYPE(out_dtype, OT, {
            auto kern = vc == 1 ? gated_rmsnorm_vec_kernel<OT, 1> : vc == 2 ? gated_rmsnorm_vec_kernel<OT, 2>
                        : vc <= 4 ? gated_rmsnorm_vec_kernel<OT, 4> : gated_rmsnorm_vec_kernel<OT, 8>;
            launch_kernel(kern, dim3(R), dim3(threads), 0, stream, o, gate, gate_nsplit, (size_t)gate_split_stride, gate_ld,
                          weight, eps, (OT*)out, N, sums);
        });
        return check_launch("gated_rmsnorm");
    }
    MHB_DISPATCH_DTYPE(out_dtype, OT,
        launch_kernel(gated_rmsnorm_kernel<OT>, dim3(R), dim3(row_threads(N)), 0, stream, o, gate, gate_nsplit,
                      (size_t)gate_split_stride, gate_ld, weight, eps, (OT*)out, N));
    return check_launch("gated_rmsnorm");
}

// per_head: the two norms run over each head alone, with weights [dk] that the heads share, instead of over the whole
// projections.  v_eps > 0: every head's value is divided by its root mean square (with that eps) before it is stored.
// page_extra: elements of a page behind its keys and values (left alone here).  temp_coef != 0 (with per_head): q is
// multiplied by 1 + temp_coef ln(floor((position + 1) / temp_every) + 1).  v_scale: a factor on the stored values.
// With per_head the weights may be null (norms without a weight).  bias (or null): [nq dk + nkv dk], added to q and k
// before anything else.  v_from_k: the row has no v columns, the values are the keys as projected.
MHB_EXPORT int mhb_qknorm_rope_append_opts(const float* qkv, int nsplit, long long split_stride, int ld,
                                      const float* q_weight, const float* k_weight, float eps, const int* positions,
                                      const int* tok_seg, const int* block_table, int table_width,
                                      const float* inv_freq, int rdim, void* q_out, void* cache, int dtype, int T,
                                      int nq, int nkv, int dk, int dv, int P, int num_pages, int has_kv, int* status,
                                      int per_head, float v_eps, long long page_extra, float temp_coef,
                                      double temp_every, float v_scale, const float* bias, int v_from_k,
                                      cudaStream_t stream) {
    if (T <= 0) return 0;
    if (v_from_k && (dv != dk || !has_kv)) return fail("qknorm_rope_append: keys that serve as values are as wide as these");
    if (!per_head && (!q_weight || (has_kv && !k_weight) || temp_coef != 0.f))
        return fail("qknorm_rope_append: norms over whole projections have weights and no temperature");
    if (temp_coef != 0.f && !(temp_every > 0.)) return fail("qknorm_rope_append: a temperature needs a positive step");
    if (rdim < 0 || rdim > dk || (rdim & 1)) return fail("qknorm_rope_append: %d rotated elements of a head of %d", rdim, dk);
    const int qw = nq * dk, kw = has_kv ? nkv * dk : 0;
    const size_t smem = sizeof(float) * ((size_t)qw + kw + rdim + ((v_eps > 0.f || v_from_k) && has_kv ? (size_t)nkv * dv : 0));
    // how many partial sums the norms over whole projections have, whichever form sums them
    const int nsums = T <= 64 && qw + kw > 512 ? 1024 : row_threads(qw + kw);
    const uintptr_t addresses = (uintptr_t)qkv | (uintptr_t)q_weight | (uintptr_t)k_weight | (uintptr_t)q_out |
                                (uintptr_t)cache | (uintptr_t)bias;
    if (dk % 4 == 0 && dv % 4 == 0 && rdim % 8 == 0 && ld % 4 == 0 && split_stride % 4 == 0 && page_extra % 4 == 0 &&
        !(addresses & 15)) {
        // few tokens: a thread for every four elements; many: a quarter as many, with four loads of its own in flight, so
        // that several tokens share an SM
        const int quads = (qw + kw + (has_kv && !v_from_k ? nkv * dv : 0)) / 4, want = T <= 64 ? quads : (quads + 3) / 4;
        const int most = T <= 64 ? 1024 : 256;
        int threads = (want + 31) / 32 * 32;
        threads = threads < 64 ? 64 : threads > most ? most : threads;
        MHB_DISPATCH_DTYPE(dtype, CT, {
            auto kern = T <= 64       ? qknorm_rope_append_vec_kernel<CT, 8, 1024>
                        : nsplit > 1 ? qknorm_rope_append_vec_kernel<CT, 8, 256>
                                     : qknorm_rope_append_vec_kernel<CT, 1, 256>;
            if (allow_smem(kern, smem, "qknorm_rope_append")) return -1;
            launch_kernel(kern, dim3(T), dim3(threads), smem, stream, qkv, nsplit, (size_t)split_stride, ld, q_weight,
                          k_weight, eps, positions, tok_seg, block_table, table_width, inv_freq, rdim, (CT*)q_out,
                          (CT*)cache, nq, nkv, dk, dv, P, num_pages, has_kv, status, per_head, v_eps, (size_t)page_extra,
                          temp_coef, temp_every, v_scale, bias, v_from_k, nsums);
        });
        return check_launch("qknorm_rope_append");
    }
    MHB_DISPATCH_DTYPE(dtype, CT, {
        auto kern = qknorm_rope_append_kernel<CT, CT>;
        if (allow_smem(kern, smem, "qknorm_rope_append")) return -1;
        launch_kernel(kern, dim3(T), dim3(nsums), smem, stream, qkv, nsplit, (size_t)split_stride, ld,
                      q_weight, k_weight, eps, positions, tok_seg, block_table, table_width, inv_freq, rdim,
                      (CT*)q_out, (CT*)cache, nq, nkv, dk, dv, P, num_pages, has_kv, status, per_head, v_eps,
                      (size_t)page_extra, temp_coef, temp_every, v_scale, bias, v_from_k);
    });
    return check_launch("qknorm_rope_append");
}

MHB_EXPORT int mhb_qknorm_rope_append(const float* qkv, int nsplit, long long split_stride, int ld,
                                      const float* q_weight, const float* k_weight, float eps, const int* positions,
                                      const int* tok_seg, const int* block_table, int table_width,
                                      const float* inv_freq, int rdim, void* q_out, void* cache, int dtype, int T,
                                      int nq, int nkv, int dk, int dv, int P, int num_pages, int has_kv, int* status,
                                      cudaStream_t stream) {
    return mhb_qknorm_rope_append_opts(qkv, nsplit, split_stride, ld, q_weight, k_weight, eps, positions, tok_seg,
                                       block_table, table_width, inv_freq, rdim, q_out, cache, dtype, T, nq, nkv, dk, dv,
                                       P, num_pages, has_kv, status, 0, 0.f, 0, 0.f, 1., 1.f, nullptr, 0, stream);
}

// Causal grouped-query attention over the paged KV cache with TMA-fed key/value tiles, for decode
// tokens and short portions (long portions go to attention_tc.cu).
//
// The math, the work items and the tile shape are those of attention_mma.cu
// (mini_hisparse/model.py:173-179, mini_hisparse/attention.py:26-35): 16 query rows per CTA, the
// keys of a tile split over the four compute warps, key splits across CTAs merged by the last CTA
// of a token.  What differs is how keys and values reach shared memory: a fifth warp walks the block table and issues one
// cp.async.bulk.tensor (TMA) per page, plane and 64-column half, with the 128-byte swizzle, into a
// ring of stages guarded by full/empty mbarriers.  The compute warps never issue a load, so the
// ring stays full while they work, which is what a decode step needs: it is bound by how many
// bytes are in flight.  ldmatrix reads the swizzled tiles without bank conflicts.
//
// A step of decoded tokens alone can have the splits of a token and KV head merged in a thread-block cluster instead
// (AttnArgs::cluster): every CTA sends its rows to the CTA that owns them (CTA r the rows r, r + cluster, ...) through
// distributed shared memory, and each owner merges in split order.  A merge through global memory (partials, a fence, a
// counter, the last CTA's loads) costs as much as 200 keys, so shares were 256 keys long at least and 8 requests of 300
// keys ran on 32 of 148 SMs; the cluster's merge pays for shares of 64.
//
// Needs head_dim 64 or 128 and a page size that divides 64; other shapes use attention_mma.cu or
// attention_simt.cu.  Every mbarrier wait is bounded (status bit 8 when one runs out).
#include "mma_helpers.cuh"
#include "tma_helpers.cuh"

using namespace mhb;

MHB_EXPORT const char* mhb_last_error() { return error_buffer(); }

namespace {
constexpr int KT = 64;
constexpr int ROWS = 16;                     // query rows of a tile: two blocks of 8
constexpr int CWARPS = 4;                    // compute warps
constexpr int THREADS = (CWARPS + 1) * 32;   // + the TMA warp
constexpr int ITEM_INTS = 8;
constexpr int MAX_MERGE_SPLITS = 64;

struct AttnArgs {
    const __nv_bfloat16* q;
    __nv_bfloat16* out;
    float* part_acc;
    float* part_ml;
    const int* items;
    const int* positions;
    const int* block_table;
    const int* tok_part_row;
    const int* tok_nsplit;
    int* counters;
    int* status;
    int num_items, width, nq, nkv, P, num_pages, window;
    int fresh;      // keys at positions > positions[tok0] - fresh may have been written by the kernel
                    // before this one (the append of this step); 0: any key may
    float scale;
    // the options of a mixer that brings them (EXT instances only): a sink per query head in the softmax's
    // denominator and a gate (columns of a float32 product, split-K parts summed in order) on the output
    const float* sink;
    const float* gate;
    int gate_nsplit, gate_ld;
    size_t gate_split_stride;
    int gate_per_head;          // the gate has one column per head instead of one per output element
    int shared_kv;              // a latent cache: the pool is [pages][P][d] rows (one KV head), a row is key AND value
    float softcap;              // s <- softcap * tanh(s / softcap) on the scaled score (0: none)
    int out_f32;                // `out` is float32 (a sum of the outputs is still to be taken in 32 bits)
    int cluster;                // > 1: blockIdx.x = token * cluster + split, and a cluster of that many CTAs merges them
    int gate_vec;               // the gate's columns can be read four at a time
    int out_vec, part_vec;      // the outputs and the partial buffers lie where four elements can be stored at a time
    const float* slopes;        // [nq] or null: slope_h * (query position - key position) is taken off the scaled score
};

__device__ __forceinline__ float gate_of(const AttnArgs& a, int t, int col) {
    if (!a.gate) return 1.f;
    const size_t idx = (size_t)t * a.gate_ld + col;
    return 1.f / (1.f + expf(-sum_parts(a.gate + idx, a.gate_nsplit, a.gate_split_stride)));
}

// four neighbouring columns of a gate (or one head's, four times)
__device__ __forceinline__ float4 gate4_of(const AttnArgs& a, int t, int hq, int D, int e) {
    if (!a.gate) return make_float4(1.f, 1.f, 1.f, 1.f);
    if (a.gate_per_head) {
        const float g = gate_of(a, t, hq);
        return make_float4(g, g, g, g);
    }
    const int col = hq * D + e;
    if (!a.gate_vec) {
        float g[4];
#pragma unroll 1
        for (int i = 0; i < 4; ++i) g[i] = gate_of(a, t, col + i);
        return make_float4(g[0], g[1], g[2], g[3]);
    }
    float4 z = sum_parts4<8>(a.gate + (size_t)t * a.gate_ld + col, a.gate_nsplit, a.gate_split_stride);
    z.x = 1.f / (1.f + expf(-z.x)); z.y = 1.f / (1.f + expf(-z.y)); z.z = 1.f / (1.f + expf(-z.z)); z.w = 1.f / (1.f + expf(-z.w));
    return z;
}
__device__ __forceinline__ void store4_out(const AttnArgs& a, size_t idx, float4 v) {
    if (!a.out_vec) {
        const float f[4] = {v.x, v.y, v.z, v.w};
        for (int i = 0; i < 4; ++i) {
            if (a.out_f32) ((float*)a.out)[idx + i] = f[i];
            else a.out[idx + i] = __float2bfloat16_rn(f[i]);
        }
    } else if (a.out_f32) {
        *(float4*)((float*)a.out + idx) = v;
    } else {
        *(uint2*)(a.out + idx) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
    }
}
__device__ __forceinline__ float4 times(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float4 over(float4 acc, float lsum) {
    return lsum > 0.f ? make_float4(acc.x / lsum, acc.y / lsum, acc.z / lsum, acc.w / lsum) : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ uint32_t peer_addr(const void* p, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

template <int D>
struct Layout {
    static constexpr int HALVES = D / 64;
    static constexpr int STAGES = 3;
    static constexpr int Q_BYTES = ROWS * D * 2;            // [HALVES][ROWS][128 B], swizzled
    static constexpr int KV_BYTES = KT * D * 2;             // K or V of one stage: [HALVES][64][128 B]
    static constexpr int STAGE_BYTES = 2 * KV_BYTES;
    static constexpr int BAR_OFFSET = Q_BYTES + STAGES * STAGE_BYTES;
    static constexpr int LOOP_BYTES = BAR_OFFSET + 2 * STAGES * 8;
    static constexpr int MS = D + 4;                        // a partial row: accumulator, maximum, sum (16-byte rows)
    static constexpr int MERGE_BYTES = CWARPS * 16 * MS * 4;
    static constexpr int RECV_ROWS = 17;                    // splits x rows a cluster's CTA owns, and the gates of these
    static constexpr int RECV_OFFSET = ((LOOP_BYTES > MERGE_BYTES ? LOOP_BYTES : MERGE_BYTES) + 15) / 16 * 16;
    static constexpr int TOTAL = RECV_OFFSET + RECV_ROWS * MS * 4 + 1024;
};

// Address of element (row r, column e) of a tile stored as halves of 64 columns, rows of 128 bytes,
// 16-byte chunks XOR-ed with the row's low three bits (what TMA's 128-byte swizzle writes).
__device__ __forceinline__ uint32_t swz(uint32_t base, int rows_per_half, int r, int e) {
    return base + (e >> 6) * rows_per_half * 128 + r * 128 + ((((e & 63) >> 3) ^ (r & 7)) << 4);
}
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, %0;" ::"n"(CWARPS * 32) : "memory"); }

// EXT: the options.  The sink starts ONE thread's running (max, sum) of a row at (sink / scale, 1), in the
// unsplit item or in split 0 only; the softmax's weights enter the value product as two bfloat16 numbers (the
// weight and what rounding it lost: 16 bits instead of 8); the output is multiplied by sigmoid(gate).
template <int D, bool EXT>
__global__ void __launch_bounds__(THREADS, 2)
attention_tma_kernel(const __grid_constant__ CUtensorMap kv_map, const AttnArgs a) {
    using L = Layout<D>;
    constexpr int STAGES = L::STAGES;
    constexpr int KSTEPS = D / 16;
    extern __shared__ uint8_t smem_raw[];
    __shared__ int row_pos[ROWS];
    __shared__ int cta_failed;      // a bounded wait ran out somewhere in this CTA: it merges and stores nothing
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);

    // Programmatic dependent launch: this kernel may start while the append of this step's keys
    // still runs.  Work items, positions and the block table were copied in before the step's first
    // kernel, and all keys but the step's own are older still, so everything up to the first tile
    // that may hold a fresh key (and the queries) is done before waiting for the append.
    pdl_launch_dependents();
    if ((int)blockIdx.x >= a.num_items) return;
    const int* it = a.items + (size_t)blockIdx.x * ITEM_INTS;
    const int seg = it[0], tok0 = it[1], ntok = it[2], head0 = it[3], nheads = it[4];
    const int kv_begin = it[5], kv_end = it[6], split = it[7];
    const int kvh = blockIdx.y;
    const int groups = a.nq / a.nkv;
    const int nrows = ntok * nheads;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t q_s = smem_addr(smem);
    const uint32_t kv_s = q_s + L::Q_BYTES;
    const uint32_t bar0 = q_s + L::BAR_OFFSET;
    auto full_bar = [&](int s) { return bar0 + 8 * s; };
    auto empty_bar = [&](int s) { return bar0 + 8 * (STAGES + s); };
    const int* table = a.block_table + (size_t)seg * a.width;
    // tiles start on a multiple of 64 keys (so on a page edge); keys before kv_begin are masked
    const int tile_begin = (kv_begin / KT) * KT;
    const int ntiles = kv_end > kv_begin ? (kv_end - tile_begin + KT - 1) / KT : 0;

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), CWARPS); }
        mbar_fence_init();
        cta_failed = 0;
    }
    __syncthreads();
    const bool clustered = EXT && a.cluster > 1;
    if (clustered) cluster_arrive();        // this CTA runs: its shared memory may be written

    if (warp == CWARPS) {
        // ---- TMA warp: one lane per page of the tile ----------------------------------------------
        const int pages_per_tile = KT / a.P;
        bool ok = true, waited = false;
        int armed = 0;
        const int first_fresh = a.fresh > 0 ? a.positions[tok0] - (a.fresh - 1) : -0x7fffffff;
        for (int itile = 0; itile < ntiles && ok; ++itile) {
            const int stage = itile % STAGES;
            const uint32_t phase = (itile / STAGES) & 1;
            if (!waited && tile_begin + (itile + 1) * KT > first_fresh) {
                pdl_wait();
                waited = true;
            }
            if (lane == 0) ok = mbar_wait(empty_bar(stage), phase ^ 1);
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;
            // Every page slot of the stage is filled: a slot past the last key (or before the first,
            // inside a page that a window has given back) gets the page of key kv_begin again, so
            // that the masked positions hold finite numbers (0 * NaN would poison the output).
            const int kp0 = tile_begin + itile * KT + lane * a.P;
            int page = -1;
            if (lane < pages_per_tile) {
                if (kp0 < kv_end) page = table[kp0 / a.P];
                if (page < 0 || page >= a.num_pages) page = table[kv_begin / a.P];
                if (page >= a.num_pages) page = -1;
            }
            const unsigned have = __ballot_sync(0xffffffffu, page >= 0);
            if (lane == 0) mbar_expect_tx(full_bar(stage), __popc(have) * 2 * a.P * D * 2);
            __syncwarp();
            if (page >= 0) {
                const bool shared = EXT && a.shared_kv;
                const int row0 = shared ? page * a.P : ((page * 2) * a.nkv + kvh) * a.P;
                const int vrow0 = shared ? row0 : row0 + a.nkv * a.P;
                const uint32_t dst = kv_s + stage * L::STAGE_BYTES + lane * a.P * 128;
#pragma unroll
                for (int h = 0; h < L::HALVES; ++h) {
                    tma_load_2d(dst + h * KT * 128, &kv_map, h * 64, row0, full_bar(stage));
                    tma_load_2d(dst + L::KV_BYTES + h * KT * 128, &kv_map, h * 64, vrow0, full_bar(stage));
                }
            }
            armed = itile + 1;
        }
        if (!ok && lane == 0) {
            // Nothing of ours may still be in flight when the CTA leaves (the copies would land in shared
            // memory that belongs to the next CTA on this SM): wait, bounded again, for the armed stages.
            cta_failed = 1;
            for (int i = max(0, armed - STAGES); i < armed; ++i) mbar_wait(full_bar(i % STAGES), (i / STAGES) & 1);
            if (a.status) atomicOr(a.status, 8);
        }
        if (clustered) {                // the two meetings of the compute warps' merge
            __syncwarp();
            cluster_wait();
            cluster_arrive();
            cluster_wait();
        }
        return;
    }

    // ---- compute warps ---------------------------------------------------------------------------------
    if (tid < ROWS) row_pos[tid] = tid < nrows ? a.positions[tok0 + tid / nheads] : -1;
    pdl_wait();         // the queries come from the kernel before this one
    for (int c = tid; c < ROWS * (D / 8); c += CWARPS * 32) {
        const int r = c / (D / 8), ch = c % (D / 8);
        const bool live = r < nrows;
        const int t = tok0 + (live ? r / nheads : 0), h = kvh * groups + head0 + (live ? r % nheads : 0);
        const __nv_bfloat16* src = a.q + ((size_t)t * a.nq + h) * D + ch * 8;
        cp_async16(swz(q_s, ROWS, r, ch * 8), src, live ? 16 : 0);
    }
    cp_async_commit();
    // The rows that this CTA will write, four columns a thread and turn, and their gates: asked for while the queries come
    // (at the end, each of these was a round trip to the L2 that the whole launch waited for).
    const int rank = clustered ? split : 0, nranks = clustered ? a.cluster : 1;
    const int own_rows = nrows > rank ? (nrows - rank + nranks - 1) / nranks : 0;
    const int owned = (nrows + nranks - 1) / nranks;
    float* recv = (float*)(smem + L::RECV_OFFSET);          // [split][row this CTA owns][MS], then the gates of these rows
    float* gates = recv + (clustered ? nranks * owned * L::MS : 0);
    if constexpr (EXT) {
        if (a.gate && (split < 0 || clustered)) {
#pragma unroll 1
            for (int idx = tid; idx < own_rows * (D / 4); idx += CWARPS * 32) {
                const int l = idx / (D / 4), e = (idx - l * (D / 4)) * 4, row = rank + l * nranks;
                *(float4*)(gates + l * L::MS + e) = gate4_of(a, tok0 + row / nheads, kvh * groups + head0 + row % nheads, D, e);
            }
        }
    }
    cp_async_wait<0>();
    compute_sync();

    // The products have the KEYS (or the head's elements) along the 16 rows of an mma and the tile's query rows along its 8
    // columns: S^T = K Q^T, O^T = V^T P^T, in two blocks of 8 query rows.  A decoded token has 4 to 8 heads per KV head in
    // most models: the second block is left out, which halves the mmas of a launch of decoded tokens.
    const bool both = nrows > 8;
    // sums of the outputs, transposed: tile i of block b holds elements 16 i + (lane >> 2) (+ 8: [2], [3]) of the query rows
    // 8 b + 2 (lane & 3) ([0], [2]) and the one after it ([1], [3])
    float o[2][KSTEPS][4];
    float m_run[2][2], l_run[2][2];
    float slope[2][2];          // in the raw products' units
    int qp[2][2];               // the rows' positions
    uint32_t qf[2][KSTEPS][2];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
#pragma unroll
        for (int i = 0; i < KSTEPS; ++i) o[b][i][0] = o[b][i][1] = o[b][i][2] = o[b][i][3] = 0.f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = 8 * b + 2 * (lane & 3) + h;
            m_run[b][h] = -INFINITY;
            l_run[b][h] = slope[b][h] = 0.f;
            qp[b][h] = row_pos[row];
            if constexpr (EXT) {
                const int hq = kvh * groups + head0 + row % nheads;
                if (a.slopes && row < nrows) slope[b][h] = a.slopes[hq] / a.scale;
                if (a.sink && split <= 0 && warp == 0 && row < nrows) {
                    m_run[b][h] = a.sink[hq] / a.scale;
                    l_run[b][h] = lane < 4 ? 1.f : 0.f;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < KSTEPS; k += 2)
            ldmatrix_x4(swz(q_s, ROWS, 8 * b + (lane & 7), k * 16 + 8 * (lane >> 3)), qf[b][k][0], qf[b][k][1], qf[b][k + 1][0], qf[b][k + 1][1]);
    }
    const float scale_log2 = a.scale * 1.4426950408889634f;
    bool ok = true;

    for (int itile = 0; itile < ntiles; ++itile) {
        const int stage = itile % STAGES;
        ok = mbar_wait(full_bar(stage), (itile / STAGES) & 1);
        if (!ok) break;
        const uint32_t k_s = kv_s + stage * L::STAGE_BYTES;
        const uint32_t v_s = k_s + L::KV_BYTES;
        const int key0 = warp * 16, kr = key0 + (lane & 7);
        const int kp0 = tile_begin + itile * KT + key0 + (lane >> 2);      // this lane's keys: kp0 and kp0 + 8

        float s[2][4];
#pragma unroll
        for (int b = 0; b < 2; ++b) s[b][0] = s[b][1] = s[b][2] = s[b][3] = 0.f;
#pragma unroll
        for (int k = 0; k < KSTEPS; ++k) {
            uint32_t ka[4];
            ldmatrix_x4(swz(k_s, KT, kr + 8 * ((lane >> 3) & 1), k * 16 + 8 * (lane >> 4)), ka[0], ka[1], ka[2], ka[3]);
            mma_bf16(s[0], ka, qf[0][k][0], qf[0][k][1]);
            if (both) mma_bf16(s[1], ka, qf[1][k][0], qf[1][k][1]);
        }
        uint32_t pf[2][2], pl[EXT ? 2 : 1][2];
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            if (b == 1 && !both) break;
            if constexpr (EXT) {
                if (a.softcap > 0.f) {      // the cap works on the scaled score; the tile stays in the raw products' units
                    const float to_cap = a.scale / a.softcap, from_cap = a.softcap / a.scale;
#pragma unroll
                    for (int x = 0; x < 4; ++x) s[b][x] = from_cap * tanhf(s[b][x] * to_cap);
                }
            }
            float alpha[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int x = h; x < 4; x += 2) {
                    const int kp = kp0 + 4 * (x & 2);
                    const bool valid = kp >= kv_begin && kp < kv_end && kp <= qp[b][h] && (a.window <= 0 || kp > qp[b][h] - a.window);
                    if (EXT && a.slopes) s[b][x] = fmaf(-slope[b][h], (float)(qp[b][h] - kp), s[b][x]);
                    s[b][x] = valid ? s[b][x] : -INFINITY;
                }
                float mx = fmaxf(s[b][h], s[b][2 + h]);
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                const float m_new = fmaxf(m_run[b][h], mx);
                const float m_use = m_new == -INFINITY ? 0.f : m_new;
                alpha[h] = exp2f((m_run[b][h] - m_use) * scale_log2);
                m_run[b][h] = m_new;
                s[b][h] = exp2f((s[b][h] - m_use) * scale_log2);
                s[b][2 + h] = exp2f((s[b][2 + h] - m_use) * scale_log2);
                l_run[b][h] = l_run[b][h] * alpha[h] + (s[b][h] + s[b][2 + h]);
            }
            pf[b][0] = transposed(pack_bf16(s[b][0], s[b][1]));
            pf[b][1] = transposed(pack_bf16(s[b][2], s[b][3]));
            if constexpr (EXT) {
                float r[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) r[x] = s[b][x] - __bfloat162float(__float2bfloat16_rn(s[b][x]));
                pl[b][0] = transposed(pack_bf16(r[0], r[1]));
                pl[b][1] = transposed(pack_bf16(r[2], r[3]));
            }
#pragma unroll
            for (int i = 0; i < KSTEPS; ++i) {
                o[b][i][0] *= alpha[0]; o[b][i][1] *= alpha[1];
                o[b][i][2] *= alpha[0]; o[b][i][3] *= alpha[1];
            }
        }
#pragma unroll
        for (int i = 0; i < KSTEPS; ++i) {
            uint32_t va[4];
            ldmatrix_x4_trans(swz(v_s, KT, kr + 8 * (lane >> 4), i * 16 + 8 * ((lane >> 3) & 1)), va[0], va[1], va[2], va[3]);
            mma_bf16(o[0][i], va, pf[0][0], pf[0][1]);
            if constexpr (EXT) mma_bf16(o[0][i], va, pl[0][0], pl[0][1]);
            if (both) {
                mma_bf16(o[1][i], va, pf[1][0], pf[1][1]);
                if constexpr (EXT) mma_bf16(o[1][i], va, pl[1][0], pl[1][1]);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty_bar(stage));     // this warp is done with the stage
    }
    // A wait that ran out is reported; the warp still walks through the barriers below so that
    // the others are not left waiting for it, but the CTA then merges and stores nothing: the ring
    // may still receive copies (the TMA warp waits for them before it leaves).
    if (!ok && lane == 0) {
        cta_failed = 1;
        if (a.status) atomicOr(a.status, 8);
    }

#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            l_run[b][h] += __shfl_xor_sync(0xffffffffu, l_run[b][h], 4);
            l_run[b][h] += __shfl_xor_sync(0xffffffffu, l_run[b][h], 8);
            l_run[b][h] += __shfl_xor_sync(0xffffffffu, l_run[b][h], 16);
        }
    {
        compute_sync();     // all warps are past their last tile: the ring can become merge scratch
        ok = cta_failed == 0;
        if (!ok && !clustered) return;
        float* mg = (float*)smem;
        constexpr int MS = L::MS;
        if (ok) {
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float* dst = mg + (warp * 16 + 8 * b + 2 * (lane & 3) + h) * MS;
#pragma unroll
                    for (int i = 0; i < KSTEPS; ++i) {
                        dst[16 * i + (lane >> 2)] = o[b][i][h];
                        dst[16 * i + (lane >> 2) + 8] = o[b][i][2 + h];
                    }
                    if (lane < 4) *(float2*)(dst + D) = make_float2(m_run[b][h], l_run[b][h]);
                }
        }
        compute_sync();
        if (clustered) cluster_wait();      // the peers run (each has arrived when it started)
#pragma unroll 1
        for (int idx = tid; idx < nrows * (D / 4); idx += CWARPS * 32) {
            const int row = idx / (D / 4), e = (idx - row * (D / 4)) * 4;
            float2 ml[CWARPS];
            float M = -INFINITY;
#pragma unroll
            for (int w = 0; w < CWARPS; ++w) {
                ml[w] = *(const float2*)(mg + (w * 16 + row) * MS + D);
                M = fmaxf(M, ml[w].x);
            }
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            float lsum = 0.f;
#pragma unroll
            for (int w = 0; w < CWARPS; ++w) {
                const float wgt = ml[w].x == -INFINITY ? 0.f : exp2f((ml[w].x - M) * scale_log2);
                const float4 v = vec4(mg + (w * 16 + row) * MS + e);
                acc.x += wgt * v.x; acc.y += wgt * v.y; acc.z += wgt * v.z; acc.w += wgt * v.w;
                lsum += wgt * ml[w].y;
            }
            const int t = tok0 + row / nheads, hq = kvh * groups + head0 + row % nheads;
            if (clustered) {
                if (!ok) { M = -INFINITY; acc = make_float4(0.f, 0.f, 0.f, 0.f); lsum = 0.f; }
                const uint32_t dst = peer_addr(recv + (split * owned + row / nranks) * MS, row % nranks);
                asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(dst + e * 4), "f"(acc.x), "f"(acc.y), "f"(acc.z), "f"(acc.w) : "memory");
                if (e == 0) asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(dst + D * 4), "f"(M), "f"(lsum) : "memory");
            } else if (split < 0) {
                float4 res = over(acc, lsum);
                if (EXT && a.gate) res = times(res, vec4(gates + row * MS + e));
                store4_out(a, ((size_t)t * a.nq + hq) * D + e, res);
            } else {
                const size_t prow = (size_t)a.tok_part_row[t] + split;
                float* part = a.part_acc + (prow * a.nq + hq) * D + e;
                if (a.part_vec) {
                    *(float4*)part = acc;
                } else {
                    part[0] = acc.x; part[1] = acc.y; part[2] = acc.z; part[3] = acc.w;
                }
                if (e == 0) {
                    a.part_ml[(prow * a.nq + hq) * 2] = M == -INFINITY ? -INFINITY : M * a.scale;
                    a.part_ml[(prow * a.nq + hq) * 2 + 1] = lsum;
                }
            }
        }
        if constexpr (EXT) {
            if (clustered) {
                __syncwarp();
                cluster_arrive();
                cluster_wait();         // every part has been sent; nobody writes another CTA's shared memory behind it
                if (!ok) return;
#pragma unroll 1
                for (int idx = tid; idx < own_rows * (D / 4); idx += CWARPS * 32) {
                    const int l = idx / (D / 4), e = (idx - l * (D / 4)) * 4;
                    const int row = rank + l * nranks;
                    float M = -INFINITY;
                    for (int p = 0; p < nranks; ++p) M = fmaxf(M, recv[(p * owned + l) * MS + D]);
                    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                    float lsum = 0.f;
                    for (int p = 0; p < nranks; ++p) {          // in split order
                        const float* src = recv + (p * owned + l) * MS;
                        const float w = src[D] == -INFINITY ? 0.f : exp2f((src[D] - M) * scale_log2);
                        const float4 v = vec4(src + e);
                        acc.x += w * v.x; acc.y += w * v.y; acc.z += w * v.z; acc.w += w * v.w;
                        lsum += w * src[D + 1];
                    }
                    float4 res = over(acc, lsum);
                    if (a.gate) res = times(res, vec4(gates + l * MS + e));
                    const int t = tok0 + row / nheads, hq = kvh * groups + head0 + row % nheads;
                    store4_out(a, ((size_t)t * a.nq + hq) * D + e, res);
                }
                return;
            }
        }
        if (split >= 0 && a.counters != nullptr) {
            // the last CTA of this tile's splits merges them (reference/attention.py:11-20)
            __shared__ int is_last;
            __threadfence();
            compute_sync();
            if (tid == 0) {
                const int chunks = (groups + 15) / 16;
                int* counter = a.counters + ((size_t)tok0 * a.nkv + kvh) * chunks + head0 / 16;
                const int ns = a.tok_nsplit[tok0];
                // more parts than the merge below has scratch for: say so rather than merge a part of them
                if (ns > MAX_MERGE_SPLITS && a.status) atomicOr(a.status, 32);
                const int prev = atomicAdd(counter, 1);
                is_last = prev == ns - 1;
                if (is_last) *counter = 0;
            }
            compute_sync();
            if (is_last) {
                // The merge is a chain of round trips to L2 on the kernel's critical path: every load
                // that does not depend on another is issued at once.
                __threadfence();
                // scratch in the ring, which nobody reads any more (12 KB + 64 bytes)
                float (*wgt_s)[MAX_MERGE_SPLITS] = (float (*)[MAX_MERGE_SPLITS])smem;
                float2 (*ml_s)[MAX_MERGE_SPLITS] = (float2 (*)[MAX_MERGE_SPLITS])(smem + 16 * MAX_MERGE_SPLITS * 4);
                float* inv_s = (float*)(smem + 16 * MAX_MERGE_SPLITS * 12);
                const int ns = min(a.tok_nsplit[tok0], MAX_MERGE_SPLITS);
                for (int idx = tid; idx < nrows * ns; idx += CWARPS * 32) {     // all (maximum, sum) pairs at once
                    const int row = idx / ns, sp = idx - row * ns;
                    const int t = tok0 + row / nheads, hq = kvh * groups + head0 + row % nheads;
                    const float* ml = a.part_ml + (((size_t)a.tok_part_row[t] + sp) * a.nq + hq) * 2;
                    ml_s[row][sp] = a.part_vec ? __ldcg((const float2*)ml) : make_float2(__ldcg(ml), __ldcg(ml + 1));
                }
                compute_sync();
                if (tid < nrows) {
                    float M = -INFINITY;
                    for (int sp = 0; sp < ns; ++sp) M = fmaxf(M, ml_s[tid][sp].x);
                    float lsum = 0.f;
                    for (int sp = 0; sp < ns; ++sp) {
                        const float ms = ml_s[tid][sp].x;
                        const float w = ms > -INFINITY ? expf(ms - M) : 0.f;
                        wgt_s[tid][sp] = w;
                        lsum += w * ml_s[tid][sp].y;
                    }
                    inv_s[tid] = lsum > 0.f ? 1.f / lsum : 0.f;
                }
                compute_sync();
                // four elements per thread and step, eight splits in flight; summed in the splits' order
                for (int idx = tid; idx < nrows * (D / 4); idx += CWARPS * 32) {
                    const int row = idx / (D / 4), e = (idx - row * (D / 4)) * 4;
                    const int t = tok0 + row / nheads, hq = kvh * groups + head0 + row % nheads;
                    const float* src = a.part_acc + ((size_t)a.tok_part_row[t] * a.nq + hq) * D + e;
                    const size_t step = (size_t)a.nq * D;
                    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
                    for (int sp = a.part_vec ? ns : 0; sp < ns; ++sp, src += step) {
                        const float w = wgt_s[row][sp];
                        acc.x += w * __ldcg(src); acc.y += w * __ldcg(src + 1); acc.z += w * __ldcg(src + 2); acc.w += w * __ldcg(src + 3);
                    }
                    for (int s0 = a.part_vec ? 0 : ns; s0 < ns; s0 += 8) {
                        float4 v[8];
#pragma unroll
                        for (int q = 0; q < 8; ++q) v[q] = __ldcg((const float4*)(src + (size_t)min(s0 + q, ns - 1) * step));
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            if (s0 + q < ns) {
                                const float w = wgt_s[row][s0 + q];
                                acc.x += w * v[q].x; acc.y += w * v[q].y; acc.z += w * v[q].z; acc.w += w * v[q].w;
                            }
                        }
                    }
                    const float inv = inv_s[row];
                    if constexpr (EXT) {
                        const float4 g = gate4_of(a, t, hq, D, e);
                        acc.x *= g.x; acc.y *= g.y; acc.z *= g.z; acc.w *= g.w;
                    }
                    store4_out(a, ((size_t)t * a.nq + hq) * D + e, make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv));
                }
            }
        }
    }
}

template <int D, bool EXT>
int configure() {
    auto kern = attention_tma_kernel<D, EXT>;
    constexpr int smem = Layout<D>::TOTAL;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return fail("attention_tma: shared memory %d: %s", smem, cudaGetErrorString(e));
        // two CTAs per SM need the large shared-memory carve-out even when one CTA would fit a small one
        cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);     // clusters of up to 16
        if (e != cudaSuccess) return fail("attention_tma: clusters of more than 8: %s", cudaGetErrorString(e));
        configured = true;
    }
    return 0;
}

template <int D, bool EXT>
int launch(const CUtensorMap& map, const AttnArgs& a, int launch_items, cudaStream_t stream) {
    auto kern = attention_tma_kernel<D, EXT>;
    constexpr int smem = Layout<D>::TOTAL;
    int rc = configure<D, EXT>();
    if (rc) return rc;
    if (a.cluster <= 1) {
        launch_kernel(kern, dim3(launch_items, a.nkv), dim3(THREADS), smem, stream, map, a);
        return check_launch("attention_tma");
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(launch_items, a.nkv);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = a.cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, map, a);
    if (e != cudaSuccess) return fail("attention_tma: launch of clusters of %d: %s", a.cluster, cudaGetErrorString(e));
    return check_launch("attention_tma");
}

// What can be read and written four elements at a time, by the addresses.
void set_widths(AttnArgs& a) {
    a.out_vec = ((uintptr_t)a.out & (a.out_f32 ? 15 : 7)) == 0;
    a.part_vec = ((uintptr_t)a.part_acc & 15) == 0 && ((uintptr_t)a.part_ml & 7) == 0;
    a.gate_vec = a.gate && !a.gate_per_head && a.gate_ld % 4 == 0 && a.gate_split_stride % 4 == 0 && ((uintptr_t)a.gate & 15) == 0;
}

// How many clusters of n CTAs of the kernel with options the device holds at once.
template <int D>
int max_clusters(int n) {
    int rc = configure<D, true>();
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n, 1);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = Layout<D>::TOTAL;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = n;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int k = 0;
    cudaError_t e = cudaOccupancyMaxActiveClusters(&k, attention_tma_kernel<D, true>, &cfg);
    if (e != cudaSuccess) return fail("attention_tma: clusters of %d: %s", n, cudaGetErrorString(e));
    return k;
}
}  // namespace

MHB_EXPORT int mhb_attention_tma_supports(int d, int P) {
    return (d == 64 || d == 128) && P >= 2 && P <= KT && KT % P == 0;
}

// Clusters of n CTAs of the kernel with options that run at once on the current device (0: none); < 0: error.
MHB_EXPORT int mhb_attention_tma_max_clusters(int d, int n) {
    if ((d != 64 && d != 128) || n < 1 || n > 16) return fail("attention_tma: head_dim %d, %d splits", d, n);
    return d == 128 ? max_clusters<128>(n) : max_clusters<64>(n);
}

// cache: one layer's pool [num_pages, 2, nkv, P, d] bfloat16; rows = 16 (items of short segments).
// fresh: the kernel launched before this one may have written the keys of the last `fresh` positions
// up to an item's first token (and later ones); older keys are loaded without waiting for it.
// 0: it may have written any key.
MHB_EXPORT int mhb_attention_tma(const void* q, const void* cache, void* out, float* part_acc, float* part_ml,
                                 const int* items, int num_items, int launch_items, int rows,
                                 const int* positions, const int* block_table, int width,
                                 const int* tok_part_row, const int* tok_nsplit, int* counters, int nq, int nkv,
                                 int d, int P, int num_pages, int window, int fresh, float scale, int* status,
                                 cudaStream_t stream) {
    if (launch_items <= 0) return 0;
    if (nkv <= 0 || nq % nkv) return fail("attention: %d query heads over %d KV heads", nq, nkv);
    if (!mhb_attention_tma_supports(d, P))
        return fail("attention_tma: head_dim %d with pages of %d keys is not built (head_dim 64 or 128, page size dividing 64)", d, P);
    const long long total_rows = (long long)num_pages * 2 * nkv * P;
    if (total_rows > 0x7fffffffLL) return fail("attention_tma: the pool has too many rows for one tensor map");
    CUtensorMap map;
    int rc = make_bf16_map(&map, cache, total_rows, d, d, P);
    if (rc) return rc;
    AttnArgs a;
    a.q = (const __nv_bfloat16*)q; a.out = (__nv_bfloat16*)out; a.part_acc = part_acc; a.part_ml = part_ml;
    a.items = items; a.positions = positions; a.block_table = block_table; a.tok_part_row = tok_part_row;
    a.tok_nsplit = tok_nsplit; a.counters = counters; a.status = status; a.num_items = num_items;
    a.width = width; a.nq = nq; a.nkv = nkv; a.P = P; a.num_pages = num_pages; a.window = window;
    a.scale = scale;
    a.fresh = fresh;
    a.gate_per_head = 0; a.shared_kv = 0; a.softcap = 0.f; a.out_f32 = 0; a.slopes = nullptr; a.cluster = 0; a.gate_vec = 0;
    a.sink = nullptr; a.gate = nullptr; a.gate_nsplit = 1; a.gate_ld = 0; a.gate_split_stride = 0;
    set_widths(a);
    if (rows == 16) return d == 128 ? launch<128, false>(map, a, launch_items, stream) : launch<64, false>(map, a, launch_items, stream);
    return fail("attention_tma: tile height %d", rows);
}

// The same with the options (see EXT at the kernel); keys and values are both d wide.  cluster > 1: the items are those of
// single tokens cut into `cluster` splits each (item = token * cluster + split, one chunk of at most 16 heads), which a
// cluster merges; partial buffers and counters are not used.
MHB_EXPORT int mhb_attention_tma_ext(const void* q, const void* cache, void* out, float* part_acc, float* part_ml,
                                     const int* items, int num_items, int launch_items, int rows,
                                     const int* positions, const int* block_table, int width,
                                     const int* tok_part_row, const int* tok_nsplit, int* counters, int nq, int nkv,
                                     int d, int P, int num_pages, int window, int fresh, float scale,
                                     const float* sink, const float* gate, int gate_nsplit,
                                     long long gate_split_stride, int gate_ld, int gate_per_head, int shared_kv,
                                     float softcap, int out_f32, const float* slopes, int cluster, int* status,
                                     cudaStream_t stream) {
    if (launch_items <= 0) return 0;
    if (nkv <= 0 || nq % nkv) return fail("attention: %d query heads over %d KV heads", nq, nkv);
    if (!mhb_attention_tma_supports(d, P))
        return fail("attention_tma: head_dim %d with pages of %d keys is not built (head_dim 64 or 128, page size dividing 64)", d, P);
    if ((sink || slopes) && !(scale > 0.f)) return fail("attention_tma: a sink and distance biases need a positive scale");
    if (slopes && softcap > 0.f) return fail("attention_tma: distance biases go with uncapped scores only");
    if (shared_kv && nkv != 1) return fail("attention_tma: rows that are key and value at once have one KV head");
    const long long total_rows = shared_kv ? (long long)num_pages * P : (long long)num_pages * 2 * nkv * P;
    if (total_rows > 0x7fffffffLL) return fail("attention_tma: the pool has too many rows for one tensor map");
    CUtensorMap map;
    int rc = make_bf16_map(&map, cache, total_rows, d, d, P);
    if (rc) return rc;
    AttnArgs a;
    a.q = (const __nv_bfloat16*)q; a.out = (__nv_bfloat16*)out; a.part_acc = part_acc; a.part_ml = part_ml;
    a.items = items; a.positions = positions; a.block_table = block_table; a.tok_part_row = tok_part_row;
    a.tok_nsplit = tok_nsplit; a.counters = counters; a.status = status; a.num_items = num_items;
    a.width = width; a.nq = nq; a.nkv = nkv; a.P = P; a.num_pages = num_pages; a.window = window;
    a.scale = scale;
    a.fresh = fresh;
    a.sink = sink; a.gate = gate; a.gate_nsplit = gate_nsplit; a.gate_ld = gate_ld;
    a.gate_split_stride = (size_t)gate_split_stride;
    a.gate_per_head = gate_per_head; a.shared_kv = shared_kv; a.softcap = softcap; a.out_f32 = out_f32;
    a.slopes = slopes;
    const int heads = nq / nkv;
    if (cluster > 1 && (cluster > 16 || heads > 16 || launch_items % cluster || launch_items != num_items ||
                        (cluster + 1) * ((heads + cluster - 1) / cluster) > Layout<128>::RECV_ROWS))
        return fail("attention_tma: clusters of %d for %d items of %d heads are not built", cluster, launch_items, heads);
    a.cluster = cluster;
    set_widths(a);
    if (rows == 16) return d == 128 ? launch<128, true>(map, a, launch_items, stream) : launch<64, true>(map, a, launch_items, stream);
    return fail("attention_tma: tile height %d", rows);
}

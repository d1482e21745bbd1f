// float32 matrix product C[M, N] = A[M, K] * W[N, K]^T for the 32-bit path: every operand enters with all of its
// 24 bits and every sum is kept in float32.  Two kernels, by the number of tokens M:
//
//  * up to 8 tokens: the weights are streamed once and multiplied on the CUDA cores (plain FFMA).  Memory sets the
//    pace, so a warp keeps NR feature rows of 16-byte loads in flight, all its lanes run along K, and the activations
//    come through L1.
//
//  * more: the tensor cores.  A float32 number is EXACTLY the sum of three bfloat16 numbers x = h + m + l: h is x rounded to 8
//    bits, m what is left rounded to 8 bits, l the rest, which has 8 bits or fewer (the splitting of a number by rounding of
//    Dekker, "A floating-point technique for extending the available precision", 1971).  |m| is at most 2^-8 and |l| at most
//    2^-17 of |h|, both of either sign.  Operands are multiplied by 2^16 first, so that the parts of the smallest float32
//    number are bfloat16 numbers too; finished sums by 2^-32.  Of the nine products of two such sums six are taken, l*h, h*l,
//    m*m, m*h, h*m, h*h; the three that are left out, m*l, l*m and l*l, come to at most 1.002 x 2^-24 of h*h, what one rounding
//    of a float32 product may cost, and have either sign.  The tensor core adds in float32 but does not round to nearest, an
//    error that would grow with the length of the sum; so an accumulator in tensor memory only ever holds ONE block of 32
//    elements of K (products of small parts first), and the warps add it to sums of their own in registers, rounded to nearest.
//    No operand is held or read in less than 32 bits outside of a CTA but as all three of its parts.
//
// Measured (us; in brackets the 64 x 64 FFMA tiles that served before), tokens x K x features: 4 x 3584 x 37888 102 [622],
// 8 x 18944 x 3584 82 [1435], 16 x 3584 x 3584 40 [210], 100 x 3584 x 37888 219 [1343], 750 x 3584 x 37888 1059 [8764] =
// 192 TFLOP/s, 750 x 18944 x 3584 564 [4936].  Errors against 64 bits there (2-norm, relative): 1.0e-7 to 2.3e-7 [1.1e-6 to
// 2.5e-6].  At K = 64, 256 and 3584 and random numbers, in units of 2^-24: 1.07, 1.34, 3.4 [2.4, 4.8, 18], of one sign 1.02, 1.13,
// 2.8 [2.0, 3.9, 15].  Parts cut from the top instead of rounded leave out up to 2^-21 of a product, always towards zero
// (1.8, 2.0, 3.7 and 1.7, 1.7, 3.1 there), and took 1168 us where 1059 stands.
//
// What bounds the second: six tensor-core products for one, i.e. 2.25 / 6 = 0.37 PFLOP/s at best, and before that shared
// memory: a 128 x 128 x 16 MMA reads 8 KB in the 64 cycles it takes, and 192 bytes a row are written per block.
//
// A result that is not finite is computed once more by one thread as a plain FFMA chain: an infinite operand is not the
// sum of its three parts (inf - inf), an operand from 2^112 or a sum from 2^96 on leaves the range when it is scaled, and the
// chain says what the result is.  The chain ends at the first NaN.
#include "common.cuh"
#include "tc_helpers.cuh"
#include "tma_helpers.cuh"

using namespace mhb;

MHB_EXPORT const char* mhb_last_error() { return error_buffer(); }

namespace {

// ---- up to 8 tokens ---------------------------------------------------------------------------------------------------
constexpr int R_WARPS = 8;

__device__ __forceinline__ float4 load4_stream(const float* p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// in program order, so that a run of them is in flight at once
__device__ __forceinline__ float4 load4_now(const float* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// KS warps of a CTA share NR features (each walks every KS-th stretch of 128 elements of K); R_WARPS / KS groups a CTA.
// GATED: W holds N / 2 gate rows and as many up rows behind them; features are pairs of one of each, and C gets
// silu(gate) * up [M, N / 2] (a launch less behind every gate/up product of a decode step: 1.5 us).
template <int MT, int NR, bool GATED>
__global__ void __launch_bounds__(R_WARPS * 32, 2)
gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                     long long lda, long long ldw, long long ldc, int KS) {
    __shared__ float part[R_WARPS][NR * MT];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int groups = R_WARPS / KS, group = warp / KS, ks = warp - group * KS;
    const int n0 = (blockIdx.x * groups + group) * NR;
    const int step = KS * 128;
    int k = ks * 128 + lane * 4;
    const float* wp[NR];
#pragma unroll
    for (int j = 0; j < NR; ++j) {
        const int n = min(n0 + j, N - 1);
        wp[j] = W + (size_t)(GATED ? (n >> 1) + (n & 1) * (N >> 1) : n) * ldw;
    }
    float4 w[NR];
    pdl_launch_dependents();
#pragma unroll
    for (int j = 0; j < NR; ++j)            // weights do not depend on the kernel before this one
        w[j] = k < K ? load4_stream(wp[j] + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    pdl_wait();
    float acc[NR][MT];
#pragma unroll
    for (int j = 0; j < NR; ++j)
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[j][m] = 0.f;
    while (k < K) {
        const int kn = k + step;
        float4 next[NR];
#pragma unroll
        for (int j = 0; j < NR; ++j) next[j] = kn < K ? load4_stream(wp[j] + kn) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 a[MT];                       // every load before the first use: one latency a step, not MT
#pragma unroll
        for (int m = 0; m < MT; ++m) a[m] = load4_now(A + (size_t)min(m, M - 1) * lda + k);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
#pragma unroll
            for (int j = 0; j < NR; ++j) {
                acc[j][m] = fmaf(a[m].x, w[j].x, acc[j][m]);
                acc[j][m] = fmaf(a[m].y, w[j].y, acc[j][m]);
                acc[j][m] = fmaf(a[m].z, w[j].z, acc[j][m]);
                acc[j][m] = fmaf(a[m].w, w[j].w, acc[j][m]);
            }
        }
#pragma unroll
        for (int j = 0; j < NR; ++j) w[j] = next[j];
        k = kn;
    }
#pragma unroll
    for (int j = 0; j < NR; ++j)
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[j][m] = warp_sum(acc[j][m]);
    if (KS == 1) {
        // lane x holds every sum: lane j * MT + m stores one of them
#pragma unroll
        for (int j = 0; j < NR; ++j)
#pragma unroll
            for (int m = 0; m < MT; ++m)
                if constexpr (GATED) {
                    if (j % 2 == 0 && lane == j * MT + m && n0 + j < N && m < M)
                        C[(size_t)m * ldc + (n0 + j) / 2] = acc[j][m] / (1.f + expf(-acc[j][m])) * acc[j + 1 < NR ? j + 1 : j][m];
                } else if (lane == j * MT + m && n0 + j < N && m < M) {
                    C[(size_t)m * ldc + n0 + j] = acc[j][m];
                }
        return;
    }
    if (lane == 0) {
#pragma unroll
        for (int j = 0; j < NR; ++j)
#pragma unroll
            for (int m = 0; m < MT; ++m) part[warp][j * MT + m] = acc[j][m];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < groups * NR * MT; i += R_WARPS * 32) {
        const int g = i / (NR * MT), jm = i - g * (NR * MT);
        const int n = (blockIdx.x * groups + g) * NR + jm / MT, m = jm % MT;
        float s = 0.f;
        for (int x = 0; x < KS; ++x) s += part[g * KS + x][jm];
        if constexpr (GATED) {
            if (n & 1) continue;
            float u = 0.f;
            for (int x = 0; x < KS; ++x) u += part[g * KS + x][jm + MT];
            if (n < N && m < M) C[(size_t)m * ldc + n / 2] = s / (1.f + expf(-s)) * u;
        } else {
            if (n < N && m < M) C[(size_t)m * ldc + n] = s;
        }
    }
}

template <int MT, int NR, bool GATED = false>
int launch_rows(const float* A, const float* W, float* C, int M, int N, int K, long long lda, long long ldw, long long ldc,
                cudaStream_t stream) {
    // Warps that share a feature's K range: enough to give every SM about two CTAs' worth of loads in flight, none with
    // fewer than two stretches of 128 elements.
    int ks = 1;
    while (ks < R_WARPS && (long long)((N + NR - 1) / NR) * ks < 148 * 2 * R_WARPS && K >= 512 * ks) ks *= 2;
    const int per_cta = R_WARPS / ks * NR;
    launch_kernel(gemm_f32_rows_kernel<MT, NR, GATED>, dim3((N + per_cta - 1) / per_cta), dim3(R_WARPS * 32), 0, stream, A, W, C,
                  M, N, K, lda, ldw, ldc, ks);
    return check_launch("gemm_f32 (rows)");
}

// ---- more tokens: three bfloat16 parts on the tensor cores ----------------------------------------------------------------
constexpr float CUT_SCALE = 65536.f, SUM_SCALE = 1.f / (65536.f * 65536.f);

__device__ __forceinline__ uint32_t round_pair(float a, float b) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
    return *(const uint32_t*)&p;
}
// 8 numbers' parts as 16 bytes each
__device__ __forceinline__ void cut(const float4& p, const float4& q, uint4& h, uint4& m, uint4& l) {
    const float x[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
    uint32_t hh[4], mm[4], ll[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float a = x[2 * i] * CUT_SCALE, b = x[2 * i + 1] * CUT_SCALE;
        hh[i] = round_pair(a, b);
        a -= __uint_as_float(hh[i] << 16);
        b -= __uint_as_float(hh[i] & 0xffff0000u);
        mm[i] = round_pair(a, b);
        ll[i] = round_pair(a - __uint_as_float(mm[i] << 16), b - __uint_as_float(mm[i] & 0xffff0000u));
    }
    h = make_uint4(hh[0], hh[1], hh[2], hh[3]);
    m = make_uint4(mm[0], mm[1], mm[2], mm[3]);
    l = make_uint4(ll[0], ll[1], ll[2], ll[3]);
}

// The tokens' parts, once per product: [3][M][K] bfloat16.  Every CTA of the product reads them, so cutting them there
// would repeat the work once per 128 features.
__global__ void __launch_bounds__(256)
cut_rows_kernel(const float* __restrict__ A, __nv_bfloat16* __restrict__ parts, int M, int K, long long lda) {
    pdl_launch_dependents();
    pdl_wait();
    const int per_row = K / 8;
    const size_t plane = (size_t)M * K;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)M * per_row; i += (size_t)gridDim.x * blockDim.x) {
        const int r = (int)(i / per_row), k = (int)(i - (size_t)r * per_row) * 8;
        const float* src = A + (size_t)r * lda + k;
        uint4 h, m, l;
        cut(vec4(src), vec4(src + 4), h, m, l);
        __nv_bfloat16* dst = parts + (size_t)r * K + k;
        *(uint4*)dst = h;
        *(uint4*)(dst + plane) = m;
        *(uint4*)(dst + 2 * plane) = l;
    }
}

// One CTA: 128 features x BN tokens.  A block is 32 elements of K; every part of it is a tile of 64-byte rows (64-byte
// swizzle).  The tokens' tiles arrive by TMA, B_STAGES blocks deep (one warp).  Eight warps load the weights as float32
// into registers, D blocks ahead, and cut them into two sets of tiles; one warp issues the MMAs.  Two accumulators: while
// one block is multiplied, the eight warps add the sums of the block before to their registers.
constexpr int T_BM = 128, T_BK = 32, T_WORKERS = 8, T_THREADS = (T_WORKERS + 2) * 32;

template <int BN, int B_STAGES>
struct SplitSmem {
    static constexpr int A_TILE = T_BM * 64, B_TILE = BN * 64;          // one part of a block
    static constexpr int A_STAGE = 3 * A_TILE, B_STAGE = 3 * B_TILE;
    static constexpr int B0 = 2 * A_STAGE;
    static constexpr int BARRIERS = B0 + B_STAGES * B_STAGE;
    static constexpr int TOTAL = BARRIERS + (5 + 2 * B_STAGES) * 8 + 16 + 1024;
};

// K-major tile of 64-byte rows with the 64-byte swizzle: groups of 8 rows 512 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_rows64(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;                 // leading offset: unused for swizzled K-major
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;                 // 64-byte swizzle
    return d;
}

template <int BN, int B_STAGES, int D, int CTAS>
__global__ void __launch_bounds__(T_THREADS, CTAS)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map, const float* __restrict__ A, const float* __restrict__ W,
                      float* __restrict__ C, int M, int N, int K, long long lda, long long ldw, long long ldc,
                      int blocks_per_split, long long split_stride, int* __restrict__ status) {
    using S = SplitSmem<BN, B_STAGES>;
    constexpr int ITEMS = T_BM * 4 / (T_WORKERS * 32);        // runs of 8 weights a thread takes from a block
    constexpr int COLS = BN / 2;                              // tokens of a warp's sums: two warps share 32 features
    constexpr uint32_t ACC = BN <= 64 ? 64 : BN <= 128 ? 128 : 256, TMEM = 2 * ACC;       // columns from accumulator to accumulator
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t base = smem_addr(smem);
    // barriers: a block's weights are cut, its MMAs are done (a set of tiles and an accumulator each); its tokens are here,
    // their stage is free again (a stage each: a wait for a phase's parity must not fall two phases behind, which a wait of
    // the loading warp on `done` could); one for leaving early
    const uint32_t full0 = base + S::BARRIERS, done0 = full0 + 16, here0 = full0 + 32, free0 = here0 + 8 * B_STAGES,
                   drain = free0 + 8 * B_STAGES;
    uint32_t* slot = (uint32_t*)(smem + S::BARRIERS + (5 + 2 * B_STAGES) * 8);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * BN, n0 = blockIdx.y * T_BM;
    const int total = (K + T_BK - 1) / T_BK;
    const int first = blockIdx.z * blocks_per_split, last = min(total, first + blocks_per_split);
    const int count = max(0, last - first);

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) { mbar_init(full0 + 8 * s, T_WORKERS); mbar_init(done0 + 8 * s, 1); }
        for (int s = 0; s < B_STAGES; ++s) { mbar_init(here0 + 8 * s, 1); mbar_init(free0 + 8 * s, 1); }
        mbar_init(drain, 1);
        mbar_fence_init();
    }
    if (warp == 0) tmem_alloc(smem_addr(slot), TMEM);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *slot;
    bool ok = true;

    if (warp == T_WORKERS) {
        if (lane == 0) {
            pdl_wait();
            int i = 0;
            for (; i < count; ++i) {
                // a stage is free when the MMAs of the block B_STAGES before have read it
                ok = i < B_STAGES || mbar_wait(free0 + 8 * (i % B_STAGES), (i / B_STAGES - 1) & 1);
                if (!ok) break;
                const uint32_t bar = here0 + 8 * (i % B_STAGES), dst = base + S::B0 + (i % B_STAGES) * S::B_STAGE;
                mbar_expect_tx(bar, S::B_STAGE);
#pragma unroll
                for (int p = 0; p < 3; ++p) tma_load_2d(dst + p * S::B_TILE, &map, (first + i) * T_BK, p * M + m0, bar);
            }
            if (!ok)                         // leaving early: no stage may still have a copy in flight
                for (int j = max(0, i - B_STAGES); j < i; ++j) mbar_wait(here0 + 8 * (j % B_STAGES), (j / B_STAGES) & 1);
        }
    } else if (warp == T_WORKERS + 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = umma_idesc(BN, false);
            for (int i = 0; i < count; ++i) {
                const int s = i & 1;
                ok = mbar_wait(here0 + 8 * (i % B_STAGES), (i / B_STAGES) & 1) && mbar_wait(full0 + 8 * s, (i >> 1) & 1);
                if (!ok) break;
                tc_fence_after();
                const uint64_t da = smem_desc_rows64(base + s * S::A_STAGE);
                const uint64_t db = smem_desc_rows64(base + S::B0 + (i % B_STAGES) * S::B_STAGE);
                // (the weights' part, the tokens' part), small products first
                constexpr int order[6][2] = {{2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}, {0, 0}};
#pragma unroll
                for (int p = 0; p < 6; ++p) {
#pragma unroll
                    for (int k = 0; k < 2; ++k)
                        umma_bf16(tmem + s * ACC, da + (order[p][0] * S::A_TILE + 32 * k) / 16,
                                  db + (order[p][1] * S::B_TILE + 32 * k) / 16, idesc, (p || k) ? 1u : 0u);
                }
                umma_commit(done0 + 8 * s);
                umma_commit(free0 + 8 * (i % B_STAGES));
            }
            if (!ok) {                       // leaving early: not before what was issued has run
                umma_commit(drain);
                mbar_wait(drain, 0);
            }
        }
    } else {
        // this thread's runs of 8 weights: four lanes a row
        const int run = lane & 3, row0 = warp * 8 + (lane >> 2);                  // run j: row0 + 64 j
        const float* wsrc = W + (size_t)(n0 + row0) * ldw + run * 8;
        const uint32_t dst0 = row0 * 64 + ((run ^ ((row0 >> 1) & 3)) << 4);
        float4 x[D][ITEMS][2];
        auto load = [&](float4 (&v)[ITEMS][2], int i) {
            const int k = (first + i) * T_BK;
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                const bool in = i < count && n0 + row0 + 64 * j < N && k + run * 8 < K;
                const float* p = wsrc + (size_t)(64 * j) * ldw + k;
                v[j][0] = in ? vec4(p) : make_float4(0.f, 0.f, 0.f, 0.f);
                v[j][1] = in ? vec4(p + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
#pragma unroll
        for (int b = 0; b < D; ++b) load(x[b], b);                                // weights are constant during the step
        pdl_wait();
        float acc[COLS];
#pragma unroll
        for (int c = 0; c < COLS; ++c) acc[c] = 0.f;
        const int quarter = warp & 3, half = warp >> 2;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        auto add_block = [&](int s) {
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < COLS; c += 32) {
                uint32_t r[2][16];
                tmem_ld16(tmem + lanes + s * ACC + half * COLS + c, r[0]);
                tmem_ld16(tmem + lanes + s * ACC + half * COLS + c + 16, r[1]);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; ++e) acc[c + e] += __uint_as_float(r[e / 16][e % 16]);
            }
            tc_fence_before();
        };
        for (int i0 = 0; i0 < count && ok; i0 += D) {
#pragma unroll
            for (int b = 0; b < D; ++b) {
                const int i = i0 + b, s = i & 1;
                if (i >= count || !ok) continue;
                if (i >= 2) {
                    ok = mbar_wait(done0 + 8 * s, ((i >> 1) - 1) & 1);
                    if (!ok) continue;
                }
#pragma unroll
                for (int j = 0; j < ITEMS; ++j) {
                    uint4 h, m, l;
                    cut(x[b][j][0], x[b][j][1], h, m, l);
                    uint8_t* at = smem + s * S::A_STAGE + dst0 + j * 64 * 64;
                    *(uint4*)at = h;
                    *(uint4*)(at + S::A_TILE) = m;
                    *(uint4*)(at + 2 * S::A_TILE) = l;
                }
                load(x[b], i + D);
                // the accumulator is free for block i once block i - 2's sums are in registers
                if (i >= 2) add_block(s);
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(full0 + 8 * s);
            }
        }
        for (int i = max(0, count - 2); i < count && ok; ++i) {
            ok = mbar_wait(done0 + 8 * (i & 1), (i >> 1) & 1);
            if (ok) add_block(i & 1);
        }
        const int n = n0 + quarter * 32 + lane;
        if (ok && n < N) {
            float* Cz = C + (size_t)blockIdx.z * split_stride + n;
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                const int m = m0 + half * COLS + c;
                if (m >= M) continue;
                float v = acc[c] * SUM_SCALE;
                if (!isfinite(v)) {              // see the top
                    const int k1 = min(K, last * T_BK);
                    v = 0.f;
                    for (int k = first * T_BK; k < k1 && v == v; ++k) v = fmaf(A[(size_t)m * lda + k], W[(size_t)n * ldw + k], v);
                }
                Cz[(size_t)m * ldc] = v;
            }
        }
    }
    if (!ok && status) atomicOr(status, 4);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, TMEM);
}

// The parts [3 M rows][K] in boxes of box_rows x 32 elements (64 bytes, 64-byte swizzle), zeros outside.
int make_parts_map(CUtensorMap* map, const void* ptr, long long rows, long long K, int box_rows) {
    EncodeTiledFn fn = tensor_map_encoder();
    if (!fn) return fail("the driver has no cuTensorMapEncodeTiled");
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    cuuint32_t box[2] = {T_BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail("cuTensorMapEncodeTiled failed with code %d (%lld rows of %lld)", (int)r, rows, K);
    return 0;
}

template <int BN, int B_STAGES, int D, int CTAS>
int launch_split(const float* A, const float* W, float* C, int M, int N, int K, long long lda, long long ldw, long long ldc,
                 int nsplit, long long split_stride, void* parts, int* status, cudaStream_t stream) {
    auto kern = gemm_f32_split_kernel<BN, B_STAGES, D, CTAS>;
    const int smem = SplitSmem<BN, B_STAGES>::TOTAL;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return fail("gemm_f32: shared memory %d: %s", smem, cudaGetErrorString(e));
    const int total = (K + T_BK - 1) / T_BK;
    dim3 grid((M + BN - 1) / BN, (N + T_BM - 1) / T_BM, nsplit);
    if (grid.y > 65535 || grid.z > 65535) return fail("gemm_f32: %d features in %d splits are too many for one launch", N, nsplit);
    CUtensorMap map;
    if (make_parts_map(&map, parts, 3LL * M, K, BN)) return -1;
    const long long runs = (long long)M * (K / 8);
    launch_kernel(cut_rows_kernel, dim3((unsigned)((runs + 255) / 256 > 1184 ? 1184 : (runs + 255) / 256)), dim3(256), 0, stream,
                  A, (__nv_bfloat16*)parts, M, K, lda);
    launch_kernel(kern, grid, dim3(T_THREADS), smem, stream, map, A, W, C, M, N, K, lda, ldw, ldc, (total + nsplit - 1) / nsplit,
                  split_stride, status);
    return check_launch("gemm_f32 (split)");
}
}  // namespace

// C[M, N] = A * W^T.  Takes K in steps of 8, 16-byte aligned operands and row strides of a multiple of 4 numbers.
// More than 8 tokens: `parts` holds 3 M K bfloat16, and with nsplit > 1 part z of K goes to C + z * split_stride.
// bn: 64, 128 or 192 tokens a CTA (0 for up to 8 tokens).
MHB_EXPORT int mhb_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, long long lda, long long ldw,
                            long long ldc, int bn, int nsplit, long long split_stride, void* parts, int* status,
                            cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 8 || lda % 4 || ldw % 4 || (((uintptr_t)A | (uintptr_t)W) & 15))
        return fail("gemm_f32: K %d in steps of 8, rows (%lld, %lld) in steps of 4, operands on 16 bytes", K, lda, ldw);
    if (nsplit < 1) nsplit = 1;
    if (bn == 0) {
        if (M > 8 || nsplit > 1) return fail("gemm_f32: %d tokens in %d splits without a tile of tokens", M, nsplit);
        // NR features a warp: four where there are features enough for every SM, one where latency counts
        const bool wide = N >= 4 * 148 * 4;
#define MHB_ROWS(MT, NR) return launch_rows<MT, NR>(A, W, C, M, N, K, lda, ldw, ldc, stream)
        if (M == 1) { if (wide) MHB_ROWS(1, 4); MHB_ROWS(1, 1); }
        if (M == 2) { if (wide) MHB_ROWS(2, 4); MHB_ROWS(2, 1); }
        if (M <= 4) { if (wide) MHB_ROWS(4, 4); MHB_ROWS(4, 1); }
        if (wide) MHB_ROWS(8, 4);
        MHB_ROWS(8, 1);
#undef MHB_ROWS
    }
    if (!parts || ((uintptr_t)parts & 15)) return fail("gemm_f32: no room for the tokens' parts, or not on 16 bytes");
    if (bn == 64) return launch_split<64, 3, 2, 2>(A, W, C, M, N, K, lda, ldw, ldc, nsplit, split_stride, parts, status, stream);
    if (bn == 128) return launch_split<128, 4, 2, 1>(A, W, C, M, N, K, lda, ldw, ldc, nsplit, split_stride, parts, status, stream);
    if (bn == 192) return launch_split<192, 4, 2, 1>(A, W, C, M, N, K, lda, ldw, ldc, nsplit, split_stride, parts, status, stream);
    return fail("gemm_f32: tiles of 64, 128 or 192 tokens, not %d", bn);
}

// C[M, I] = silu(A Wg^T) * (A Wu^T) for up to 8 tokens; W [2 I, K] holds the gate rows, then the up rows.
MHB_EXPORT int mhb_gemm_f32_glu(const float* A, const float* W, float* C, int M, int I, int K, long long lda, long long ldw,
                                long long ldc, cudaStream_t stream) {
    if (M <= 0 || I <= 0) return 0;
    if (M > 8) return fail("gemm_f32_glu: %d tokens", M);
    if (K <= 0 || K % 8 || lda % 4 || ldw % 4 || (((uintptr_t)A | (uintptr_t)W) & 15))
        return fail("gemm_f32_glu: K %d in steps of 8, rows (%lld, %lld) in steps of 4, operands on 16 bytes", K, lda, ldw);
    const int N = 2 * I;
    const bool wide = N >= 4 * 148 * 4;
#define MHB_GLU(MT) return wide ? launch_rows<MT, 4, true>(A, W, C, M, N, K, lda, ldw, ldc, stream) : launch_rows<MT, 2, true>(A, W, C, M, N, K, lda, ldw, ldc, stream)
    if (M == 1) MHB_GLU(1);
    if (M == 2) MHB_GLU(2);
    if (M <= 4) MHB_GLU(4);
    MHB_GLU(8);
#undef MHB_GLU
}

// The float32 path's product on Blackwell's 5th-generation tensor cores, with the accuracy of 32-bit arithmetic:
// C[M,N] = A[M,K] * W[N,K]^T (+ bias), all float32, for more than a few rows.
//
// A float32 value is the exact sum of three bfloat16 values (24 significant bits in pieces of 8): a = a0 + a1 + a2 with a0 the nearest bfloat16,
// a1 the rest's leading bits, a2 what is left.  Both operands are taken times 2^24, and the sums times 2^-48: so every value but 0 has its
// leading bits in a0 and all of its last ones in a2, subnormal values too (2^-149 becomes 2^-125, and bfloat16 goes down to
// 2^-133).  Of the nine products of two such sums six are taken - a0 b0, a0 b1, a1 b0, a1 b1, a0 b2, a2 b0; the other three together are below
// 2^-24 of |a b|, of either sign.  bfloat16 products are exact in the tensor core's 32-bit
// sums, whose additions are cut off, not rounded: so a sum in tensor memory spans 64 values of K only, its large products (a0 b0) come
// last, and these sums are added up in registers by ordinary rounded additions.  Error against 64 bits (2-norm over 2-norm, normal
// values; the multiply-add kernel of gemm_fp32.cu in brackets): 300 rows of K 2,048 1.0e-7 (3.3e-7), of K 8,192 1.3e-7 (4.4e-7), 33 rows of K 64
// 8.0e-8 (1.1e-7); values of one sign, K 2,048: 8.9e-8 (1.2e-7); log-normal magnitudes 5.2e-8 (1.0e-7).
//
// What bounds it: six tensor-core products for one, 1/6 of the bfloat16 rate, if everything else hides behind them.  A CTA owns 256 rows of
// W (two halves of 128, the instruction's M) times up to 160 rows of A (its N), and a range of K.  W streams once, as float32, and is
// split on the way: the halves' planes lie in tensor memory as the products' first operand, which leaves shared memory's
// bandwidth (128 bytes a clock) to the second one; the planes of A, read by every CTA, are made once by a small kernel before.
// Measured: 4,700 clocks for the 48 products of 64 values of K at 160 rows (98 a product; 80 at the tensor cores' rate; with few rows some 72,
// what reading the first operand takes), 5 us to fill the stages and 4 to 6 to store or add a tile.
// 300 rows times [2304, 2048], [2048, 2048], [16384, 2048] and [2048, 8192]: 22, 22 (as partial sums), 106 and 62 us (88, 88, 574 and 353 on
// the ordinary cores); 40 rows 13, 13, 38, 26 (36, 35, 128, 126).
//   warps 0-3, 4-7  the running sums of the first and second half, one thread per row of W and one register per row of A: they add
//                   a finished unit (one half, 64 values of K) while the tensor cores are at the other half's
//   warps 8-11      (up to 96 rows: 8-15, four for each half) split W: a thread per row reads 64 float32 from the swizzled stage and writes 3 x 32 words of tensor memory
//   then two warps  one thread each issues the TMA loads of W and of A's planes
//   and two         one thread each issues the products of a half (tcgen05.mma, kind::f16, M 128, N 16..160, K 16, first operand in tensor
//                   memory): 24 a unit.  Two threads, since one that has issued products waits for them at its next barrier
// Tensor memory: two halves' sums of 160 columns, planes of two units of 96: 512.  K ranges are CTAs of a cluster, whose
// partial tiles are added through distributed shared memory in the order of the ranges: the result does not depend on timing.
//
// What that does not hold is found and computed again by 32-bit multiply-adds: an infinity, a NaN, a value from 2^104 on or a sum from 2^80 on leaves
// a sum that is not finite.
// Every mbarrier wait is bounded by a clock deadline; one that runs out records a code and the roles leave their loops.
#include "planes.cuh"
#include "tc_ptx.cuh"
#include <atomic>
using namespace ttie;
using namespace ttie::tc;

namespace {
constexpr int HALF = 128, KB = 64, TOK_MOST = 160, MAX_RANGES = 8, MAX_PARTIAL = 16;
constexpr uint32_t W_BYTES = HALF * KB * 4, D_COL = 0, P_COL = 2 * TOK_MOST, P_COLS = 3 * KB / 2, TMEM_COLS = 512;
constexpr uint32_t SMEM_MOST = 226 * 1024;
constexpr int W_STAGES_MOST = 6;
constexpr float UP = 16777216.f, DOWN = 3.5527136788005009e-15f;          // 2^24 on the operands, 2^-48 on the sums

enum { WFULL = 0, WEMPTY = W_STAGES_MOST, XFULL = 2 * W_STAGES_MOST, XEMPTY = XFULL + 2, AFULL = XEMPTY + 2, AEMPTY = AFULL + 2, DFULL = AEMPTY + 2,
       DEMPTY = DFULL + 2, NBARS = DEMPTY + 2 };

struct F32Params {
    const float *A, *W, *bias;
    float* C;
    int M, N, K, lda, ldw, ldc;
    long long part_stride;                                       // > 0: the ranges' sums leave one by one, C + rank * part_stride (no cluster)
    int width, tok_tiles, ranges, num_kb, w_stages;
    ErrorWords err;
};

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y) : "memory");
}
// D (+)= A B: A in tensor memory (lane = row, a 32-bit column holds two consecutive values of K), B K-major in shared memory, rows of 64
// bfloat16 with 128-byte swizzle, 8-row groups 1024 bytes apart
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 db, {%2, %3};\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"((1024u >> 4) | (1u << 14) | (2u << 29)), "r"(idesc), "r"(accumulate) : "memory");
}
// Rows of A -> planes [3, M, pitch].  One block per row: memory-bound, 4 bytes read and 6 written a value (300 rows of 2,048: 2.4 us).
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ A, int lda, __nv_bfloat16* __restrict__ planes, int M, int K, int pitch) {
    TTIE_PDL_ENTRY();
    const int row = blockIdx.x;
    const float* src = A + (size_t)row * lda;
    uint32_t* dst[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) dst[i] = reinterpret_cast<uint32_t*>(planes + ((size_t)i * M + row) * pitch);
    for (int k = threadIdx.x * 4; k < K; k += 1024) {            // (K is a multiple of 4)
        const float4 v = *reinterpret_cast<const float4*>(src + k);
        float x[4] = {v.x * UP, v.y * UP, v.z * UP, v.w * UP};
        uint32_t q[3][2];
        split_values<2>(x, q[0], q[1], q[2]);
#pragma unroll
        for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(dst[i] + k / 2) = make_uint2(q[i][0], q[i][1]);
    }
}

// One output by 32-bit multiply-adds (where the planes do not hold the values)
__device__ __noinline__ float plain_dot(const float* a, const float* w, int K) {
    float4 total = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k0 = 0; k0 < K; k0 += KB) {
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k = k0; k < min(K, k0 + KB); k += 4) {
            const float4 x = *reinterpret_cast<const float4*>(a + k), y = *reinterpret_cast<const float4*>(w + k);
            s.x = fmaf(x.x, y.x, s.x); s.y = fmaf(x.y, y.y, s.y); s.z = fmaf(x.z, y.z, s.z); s.w = fmaf(x.w, y.w, s.w);
        }
        total.x += s.x; total.y += s.y; total.z += s.z; total.w += s.w;
    }
    return (total.x + total.y) + (total.z + total.w);
}

template <int TOK, int SPLIT>
__global__ void __launch_bounds__(384 + 128 * SPLIT, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const F32Params p) {
    constexpr int NTHREADS = 384 + 128 * SPLIT, ISSUE = 8 + 4 * SPLIT;                  // the first issuing warp
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) unsigned long long bars[NBARS];
    __shared__ uint32_t tmem_slot;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x % p.ranges, tile = blockIdx.x / p.ranges;               // clusters are consecutive CTAs
    const int m0 = tile % p.tok_tiles * p.width, n0 = tile / p.tok_tiles * (2 * HALF);
    const int toks = min(p.width, p.M - m0);
    const int halves = n0 + HALF < p.N ? 2 : 1;
    const int kb0 = (int)((long long)p.num_kb * rank / p.ranges), nkb = (int)((long long)p.num_kb * (rank + 1) / p.ranges) - kb0;
    const uint32_t plane = (uint32_t)p.width * 128u, x_stage = 3u * plane;             // (a multiple of 2048: 16 rows of 128 bytes)
    const uint32_t w_ring = smem_u32(smem), x_ring = w_ring + (uint32_t)p.w_stages * W_BYTES;
    const bool direct = p.ranges == 1 || p.part_stride > 0;
    float* C = p.C + (long long)rank * p.part_stride;
    const uint32_t bar0 = smem_u32(&bars[0]);
#define BAR(i) (bar0 + 8u * (uint32_t)(i))

    if (threadIdx.x == 0) {
        for (int i = 0; i < NBARS; ++i)                          // emptied by the four splitting or adding warps, else by one copy or commit
            mbar_init(BAR(i), (i >= WEMPTY && i < XFULL) || (i >= AFULL && i < AEMPTY) || i >= DEMPTY ? 4u : i >= XEMPTY && i < AFULL ? (uint32_t)halves : 1u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == ISSUE + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_slot;
    // The planes' kernel before this one has let it start early, but only after everything before the planes' kernel was done: W, and the
    // output's place, are there; only the planes have to be waited for.

    bool bad = false;                                            // a sum that is to be computed again
    if (warp < 8) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SPLIT == 1 ? 200 : 136) : "memory");
        const int h = warp >> 2, quarter = warp & 3, row = h * HALF + quarter * 32 + lane;
        const uint32_t d = tmem_base + ((uint32_t)(quarter * 32) << 16) + D_COL + (uint32_t)(h * TOK_MOST);
        float acc[TOK];
#pragma unroll
        for (int i = 0; i < TOK; ++i) acc[i] = 0.f;
        if (h < halves) {
            for (int kb = 0; kb < nkb; ++kb) {
                bool ok = mbar_wait(BAR(DFULL + h), kb & 1, 41, p.err);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int c = 0; c < TOK / 16; ++c)
                    if (c * 16 < toks) {
                        uint32_t v[16];
                        tmem_ld16(d + c * 16, v);
                        tmem_ld_wait(v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) acc[c * 16 + j] += __uint_as_float(v[j]);
                    }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(BAR(DEMPTY + h));
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(NTHREADS) : "memory");         // every product is done: the stages take the partial tile, [row of A][row of W]
        if (direct) {                                           // straight from the registers: neighbouring lanes are neighbouring columns
            const int n = n0 + row;
            if (n < p.N) {
                const float b = p.bias ? p.bias[n] : 0.f;
                float* dst = C + (size_t)m0 * p.ldc + n;
#pragma unroll
                for (int i = 0; i < TOK; ++i) {
                    if (i < toks) *dst = fmaf(acc[i], DOWN, b);
                    dst += p.ldc;
                    bad |= i < toks && !(fabsf(acc[i]) <= 3.4028234e38f);
                }
            }
        } else {
            float* part = reinterpret_cast<float*>(smem) + row;
#pragma unroll
            for (int c = 0; c < TOK / 16; ++c)
                if (c * 16 < toks) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) part[(c * 16 + j) * (2 * HALF)] = acc[c * 16 + j];
                }
        }
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(SPLIT == 1 ? 128 : 96) : "memory");
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(SPLIT == 1 ? 56 : 64) : "memory");
        if (warp < ISSUE) {
            // SPLIT 2: four warps for each half, else four for both in turn
            const int quarter = warp & 3, r = quarter * 32 + lane, own = SPLIT == 2 ? (warp - 8) >> 2 : 0;
            const uint32_t a = tmem_base + ((uint32_t)(quarter * 32) << 16) + P_COL;
            int s = 0, round = 0;
            bool ok = true;
            auto next_stage = [&]() { if (++s == p.w_stages) { s = 0; ++round; } };
            if (own == 1) next_stage();
            for (int kb = 0; kb < nkb && ok; ++kb) {
#pragma unroll
                for (int i = 0; i < 3 - SPLIT; ++i) {
                    const int h = SPLIT == 2 ? own : i;
                    if (h >= halves || !ok) break;
                    ok = mbar_wait(BAR(WFULL + s), round & 1, 42, p.err) && mbar_wait(BAR(AEMPTY + h), (kb & 1) ^ 1, 43, p.err);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t stage = w_ring + (uint32_t)s * W_BYTES + (uint32_t)r * 128;
#pragma unroll
                    for (int g = 0; g < KB / 16; ++g) {           // 16 values: four 16-byte pieces of the row's half of 32 values, swizzled
                        uint32_t q0[8], q1[8], q2[8];
                        float x[16];
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const uint32_t src = stage + (uint32_t)(g >> 1) * (HALF * 128) + (uint32_t)((((g & 1) * 4 + c) ^ (r & 7)) << 4);
                            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[4 * c]), "=f"(x[4 * c + 1]), "=f"(x[4 * c + 2]), "=f"(x[4 * c + 3]) : "r"(src));
                        }
#pragma unroll
                        for (int c = 0; c < 16; ++c) x[c] *= UP;
                        split_values<8>(x, q0, q1, q2);
                        const uint32_t dst = a + (uint32_t)h * P_COLS + (uint32_t)g * 8;
                        tmem_st8(dst, q0);
                        tmem_st8(dst + KB / 2, q1);
                        tmem_st8(dst + KB, q2);
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) { mbar_arrive(BAR(WEMPTY + s)); mbar_arrive(BAR(AFULL + h)); }
                    next_stage();
                    if (SPLIT == 2 && halves == 2) next_stage();   // (the other half's)
                }
            }
        } else if (warp == ISSUE) {
            if (lane == 0) {
                int s = 0, round = 0;
                bool ok = true;
                for (int kb = 0; kb < nkb && ok; ++kb)
                    for (int h = 0; h < halves; ++h) {
                        if (!mbar_wait(BAR(WEMPTY + s), (round & 1) ^ 1, 44, p.err)) { ok = false; break; }
                        mbar_expect_tx(BAR(WFULL + s), W_BYTES);
                        const uint32_t dst = w_ring + (uint32_t)s * W_BYTES;
                        tma_load_2d(dst, &tmW, BAR(WFULL + s), (kb0 + kb) * KB, n0 + h * HALF);
                        tma_load_2d(dst + HALF * 128, &tmW, BAR(WFULL + s), (kb0 + kb) * KB + 32, n0 + h * HALF);
                        if (++s == p.w_stages) { s = 0; ++round; }
                    }
                // nothing may land in a CTA that has left, and the other roles may have given up (each wait is bounded)
                for (int i = 0; i < p.w_stages; ++i)
                    if (round > 0 || i < s) mbar_wait(BAR(WFULL + i), (i < s ? round : round - 1) & 1, 44, p.err);
            }
        } else if (warp == ISSUE + 2) {
            if (lane == 0) {
                pdl_wait();
                pdl_launch_dependents();
                int kb = 0;
                for (; kb < nkb; ++kb) {
                    const int s = kb & 1;
                    if (!mbar_wait(BAR(XEMPTY + s), ((kb >> 1) & 1) ^ 1, 45, p.err)) break;
                    mbar_expect_tx(BAR(XFULL + s), x_stage);
                    for (int i = 0; i < 3; ++i)
                        tma_load_2d(x_ring + (uint32_t)s * x_stage + (uint32_t)i * plane, &tmX, BAR(XFULL + s), (kb0 + kb) * KB, i * p.M + m0);
                }
                for (int i = kb - 2 < 0 ? 0 : kb - 2; i < kb; ++i) mbar_wait(BAR(XFULL + (i & 1)), (i >> 1) & 1, 45, p.err);
            }
        } else if (((warp - ISSUE) >> 1) < halves) {
            if (lane == 0) {
                const int h = (warp - ISSUE) >> 1;
                // D float32, A and B bfloat16, both K-major, M 128, N the rows of A here up to a multiple of 16
                const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)((toks + 15) / 16 * 2) << 17) | ((uint32_t)(HALF >> 4) << 24);
                const uint32_t d = tmem_base + D_COL + (uint32_t)(h * TOK_MOST), a = tmem_base + P_COL + (uint32_t)h * P_COLS;
                int kb = 0;
                for (; kb < nkb; ++kb) {
                    const int s = kb & 1;
                    if (!mbar_wait(BAR(XFULL + s), (kb >> 1) & 1, 46, p.err)) break;
                    if (!mbar_wait(BAR(DEMPTY + h), (kb & 1) ^ 1, 48, p.err) || !mbar_wait(BAR(AFULL + h), kb & 1, 47, p.err)) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t b = (((x_ring + (uint32_t)s * x_stage) & 0x3FFFFu) >> 4) | (1u << 16);
#pragma unroll
                    for (int i = 0; i < 6; ++i) {                // planes of W and A: the smallest products first
                        const int wp = i == 0 ? 1 : i == 1 ? 2 : i == 3 ? 1 : 0, xp = i == 0 ? 1 : i == 2 ? 2 : i == 4 ? 1 : 0;
#pragma unroll
                        for (int k = 0; k < KB / 16; ++k)
                            umma_ts(d, a + wp * (KB / 2) + k * 8, b + ((uint32_t)xp * plane >> 4) + k * 2, idesc, (i | k) != 0);
                    }
                    umma_commit(BAR(AEMPTY + h));
                    umma_commit(BAR(XEMPTY + s));
                    umma_commit(BAR(DFULL + h));
                }
                if (kb > 0) mbar_wait(BAR(DFULL + h), (kb - 1) & 1, 48, p.err);      // (its products are done before the CTA frees their tensor memory)
            }
        }
        __syncwarp();
        asm volatile("bar.sync 1, %0;" ::"n"(NTHREADS) : "memory");
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SPLIT == 1 ? 128 : 96) : "memory");   // (what the adding warps give back)
    }
    __syncwarp();
    if (direct) {
        if (__syncthreads_or(bad))                                // (never with ordinary values)
            for (int e = threadIdx.x; e < toks * 2 * HALF; e += NTHREADS) {
                const int r = e % (2 * HALF), n = n0 + r, m = m0 + e / (2 * HALF);
                if (n >= p.N) continue;
                float* dst = C + (size_t)m * p.ldc + n;
                const int k0 = kb0 * KB;
                if (!(fabsf(*dst) <= 3.4028234e38f))
                    *dst = plain_dot(p.A + (size_t)m * p.lda + k0, p.W + (size_t)n * p.ldw + k0, min(p.K - k0, nkb * KB)) + (p.bias ? p.bias[n] : 0.f);
            }
    } else {
        // the partial tiles of the ranges, added in their order; each CTA of the cluster takes a share of the outputs
        asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
        const uint32_t mine = smem_u32(smem);
        const bool vec = p.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(p.C) & 15) == 0;
        const int share = p.ranges * NTHREADS, total = toks * (2 * HALF / 4);
        constexpr int U = SPLIT == 1 ? 2 : 1;                   // (what the registers hold)
        for (int e0 = rank * NTHREADS + threadIdx.x; e0 < total; e0 += U * share) {
            float q[U][MAX_RANGES][4];
#pragma unroll
            for (int u = 0; u < U; ++u)                          // all asked for at once: one after the other each would cost a trip to its SM
#pragma unroll
                for (int r = 0; r < MAX_RANGES; ++r)
                    if (r < p.ranges && e0 + u * share < total) {
                        uint32_t remote;
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(mine + (e0 + u * share) * 16), "r"(r));
                        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                                     : "=f"(q[u][r][0]), "=f"(q[u][r][1]), "=f"(q[u][r][2]), "=f"(q[u][r][3]) : "r"(remote));
                    }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = e0 + u * share, m = m0 + e / (2 * HALF / 4), n = n0 + e % (2 * HALF / 4) * 4;
                if (e >= total || n >= p.N) continue;
                float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int r = 0; r < MAX_RANGES; ++r)
                    if (r < p.ranges) {
#pragma unroll
                        for (int c = 0; c < 4; ++c) v[c] += q[u][r][c];
                    }
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (n + c < p.N) {
                        const float b = p.bias ? p.bias[n + c] : 0.f;
                        v[c] = fabsf(v[c]) <= 3.4028234e38f ? fmaf(v[c], DOWN, b) : plain_dot(p.A + (size_t)m * p.lda, p.W + (size_t)(n + c) * p.ldw, p.K) + b;
                    }
                float* dst = p.C + (size_t)m * p.ldc + n;
                if (vec && n + 3 < p.N) *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
                else
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (n + c < p.N) dst[c] = v[c];
            }
        }
        asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");      // no CTA leaves while its tile is read
    }
    if (warp == ISSUE + 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
}
// The most shared memory that a launch may ask for, set once per device: it is the function's, not the launch's, so setting what one launch needs would
// refuse another thread's that needs more
template <int TOK, int SPLIT>
cudaError_t allow_most() {
    static std::atomic<bool> done[64];
    int dev = 64;
    if (cudaGetDevice(&dev) == cudaSuccess && dev < 64 && done[dev].load(std::memory_order_relaxed)) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel<TOK, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MOST);
    if (e == cudaSuccess && dev < 64) done[dev].store(true, std::memory_order_relaxed);
    return e;
}
// Clusters of r CTAs, one CTA per SM, that run at the same time on this device (asked once per device and size)
int clusters_at_once(int r) {
    static std::atomic<int> known[64][MAX_RANGES + 1];
    if (r == 1) return num_sms();
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    int n = known[dev][r].load(std::memory_order_relaxed);
    if (n > 0) return n;
    const int smem = (int)SMEM_MOST;
    allow_most<160, 1>();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(r * 64); cfg.blockDim = dim3(512); cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = r; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_f32_tc_kernel<160, 1>, &cfg) != cudaSuccess || n < 1) { cudaGetLastError(); n = num_sms() / r / 2 + 1; }
    known[dev][r].store(n, std::memory_order_relaxed);
    return n;
}
}  // namespace

namespace {
struct Shape { int tok_tiles, width; long long tiles; };
Shape shape_of(int M, int N) {
    Shape s;
    s.tok_tiles = ceil_div(M, TOK_MOST);
    s.width = ceil_div(ceil_div(M, s.tok_tiles), 16) * 16;
    s.tiles = (long long)s.tok_tiles * ceil_div(N, 2 * HALF);
    return s;
}
// Ranges of K: the fewest waves times a wave's length, in blocks of 64 values, with a fixed cost per CTA (filling its stages, storing).  As
// partial sums any number of CTAs runs at once, but every range costs its reader another pass over the output.
int ranges_of(int M, int N, int K, bool partial) {
    const Shape s = shape_of(M, N);
    const int num_kb = ceil_div(K, KB), most = partial ? MAX_PARTIAL : MAX_RANGES;
    const double block_us = 0.4 + 0.0125 * s.width, pass = (double)M * N * 4 / 3e6 / block_us;
    int ranges = 1;
    double best = -1;
    for (int r = 1; r <= most && r <= num_kb; ++r) {
        if (ceil_div(num_kb, ceil_div(num_kb, r)) != r) continue;          // (no more ranges than the longest one asks for)
        const long long fit = partial ? num_sms() : clusters_at_once(r);
        const long long waves = ((partial ? s.tiles * r : s.tiles) + fit - 1) / fit;
        const double cost = (double)waves * (ceil_div(num_kb, r) + 4) + (partial ? r * pass : 0.);
        if (best < 0 || cost < best) { best = cost; ranges = r; }
    }
    return ranges;
}
}  // namespace

// C[M,N] = A[M,K] * W[N,K]^T (+ bias) with the accuracy of 32-bit multiply-adds.  K, lda and ldw multiples of 4, A and W on 16 bytes.  planes: 3 * M *
// (K up to a multiple of 8) bfloat16 of scratch, on 16 bytes.  parts > 1: C takes that many partial sums [parts, M, N] instead (ldc N, no
// bias); ttie_gemm_f32_tc_parts says how many are worth it.
extern "C" int ttie_gemm_f32_tc_parts(int M, int N, int K) { return M <= 0 || N <= 0 || K <= 0 ? 1 : ranges_of(M, N, K, true); }
extern "C" int ttie_gemm_f32_tc(const float* A, const float* W, const float* bias, float* C, void* planes, int M, int N, int K,
                                int lda, int ldw, int ldc, int parts, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 4 || lda % 4 || ldw % 4) TTIE_FAIL("gemm_f32_tc: K and the row strides must be positive multiples of 4");
    if (((uintptr_t)A | (uintptr_t)W | (uintptr_t)planes) & 15) TTIE_FAIL("gemm_f32_tc: operand pointers must be 16-byte aligned");
    const int pitch = (K + 7) / 8 * 8;
    F32Params p = {};
    p.A = A; p.W = W; p.bias = bias; p.C = C; p.M = M; p.N = N; p.K = K; p.lda = lda; p.ldw = ldw; p.ldc = ldc;
    p.num_kb = ceil_div(K, KB);
    if (parts > 1 && (bias || ldc != N || parts > p.num_kb)) TTIE_FAIL("gemm_f32_tc: %d partial sums of K %d", parts, K);
    const Shape shape = shape_of(M, N);
    p.tok_tiles = shape.tok_tiles; p.width = shape.width;
    p.ranges = parts > 1 ? parts : ranges_of(M, N, K, false);
    p.part_stride = parts > 1 ? (long long)M * N : 0;
    if (shape.tiles * p.ranges > 0x7fffffffLL || 3LL * M > 0x7fffffffLL) TTIE_FAIL("gemm_f32_tc: [%d, %d] is too large for one launch", M, N);
    // two stages of A's planes, and as many of W as fit
    const bool narrow = p.width <= 96;
    const uint32_t x_ring = 2u * 3u * (uint32_t)p.width * 128u;
    p.w_stages = (int)((SMEM_MOST - 1024 - x_ring) / W_BYTES);
    if (p.w_stages > W_STAGES_MOST) p.w_stages = W_STAGES_MOST;
    const size_t smem = (size_t)p.w_stages * W_BYTES + x_ring + 1024;
    auto kernel = narrow ? gemm_f32_tc_kernel<96, 2> : gemm_f32_tc_kernel<160, 1>;
    cudaError_t e = narrow ? allow_most<96, 2>() : allow_most<160, 1>();
    if (e != cudaSuccess) TTIE_FAIL("gemm_f32_tc: %u bytes of shared memory refused: %s", SMEM_MOST, cudaGetErrorString(e));
    CUtensorMap mw, mx;
    if (gemm_tc_make_map_of(&mw, 1, W, N, K, ldw, 32, HALF)) return -1;
    if (gemm_tc_make_map_of(&mx, 0, planes, 3LL * M, K, pitch, KB, p.width)) return -1;
    if (gemm_tc_error_words(&p.err.word, &p.err.mirror)) TTIE_FAIL("gemm_f32_tc: the error word's address is not to be had");
    cudaStream_t s = (cudaStream_t)stream;
    TTIE_LAUNCH(split_rows_kernel, M, 256, 0, s, A, lda, (__nv_bfloat16*)planes, M, K, pitch);
    TTIE_CHECK_LAUNCH("gemm_f32_tc (planes)");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(shape.tiles * p.ranges)); cfg.blockDim = dim3(narrow ? 640 : 512); cfg.dynamicSmemBytes = smem; cfg.stream = s;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (pdl_enabled()) {                                         // (with a cluster too: about 1 us here, the planes' kernel hides behind W's first blocks)
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (p.ranges > 1 && parts <= 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = p.ranges; attr[n].val.clusterDim.y = 1; attr[n++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr; cfg.numAttrs = n;
    e = cudaLaunchKernelEx(&cfg, kernel, mw, mx, p);
    if (e != cudaSuccess) TTIE_FAIL("gemm_f32_tc: launch failed: %s", cudaGetErrorString(e));
    return 0;
}

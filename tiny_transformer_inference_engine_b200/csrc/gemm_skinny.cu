// Weight-streaming matrix product for decode steps: out[M,N] = x[M,K] * W[N,K]^T with few rows
// (M <= 64), bfloat16 in, float32 accumulation.  Such a product is bound by reading W once from
// HBM; the library product launches too few CTAs for the narrow projections (N ~ 4096) to keep
// HBM busy.  Here the weight matrix takes the tensor core's M side (swap-AB): a CTA owns 16 rows
// of W, its four warps split the K range among themselves (and, optionally, CTAs split K further:
// blockIdx.y), every lane streams 16-byte pieces of its two weight rows straight from global
// memory into mma.sync A fragments, and the few activation rows ride as the B operand.
//
// Fragment trick: the sum over k does not care about order, so a lane's 16-byte load (8 consecutive
// k of one row) feeds two m16n8k16 steps; the activation fragment is cut from the same 8 k, so
// both operands agree on which k sits where and no shuffle or shared-memory staging is needed.
//
// Epilogues: (0) bfloat16 out (+bias); (1) float32 partial sums per K split, [S][M][N], for a
// consumer that adds them (add_rmsnorm, rope_store_partial) in a fixed order - so results do not
// depend on timing; (2) SwiGLU: the CTA streams gate rows n and up rows n+F together and writes
// silu(g)*u (models/mlp.py:24-32; silu in 32-bit as kernels/fused_swiglu/kernel.py:20-25);
// (3) float32 out (logits).
#include "tc_ptx.cuh"
using namespace ttie;
using namespace ttie::tc;

namespace {
struct SkinnyParams {
    const __nv_bfloat16* x; long long ldx;
    const __nv_bfloat16* w; long long ldw;
    const __nv_bfloat16* bias;
    void* out; long long ldo;
    int M, N, K;
    int kslice;            // K range of one CTA (multiple of 128)
    int up_offset;         // SwiGLU: row offset of the up projection inside w (and bias)
    // the gated unit's constants: min(g, limit) * sigmoid(alpha * min(g, limit)) * (clamp(u, -limit, limit) + shift); limit <= 0: no
    // clamps.  alpha 1, no limit, shift 0 is SwiGLU.
    float glu_alpha = 1.f, glu_limit = 0.f, glu_shift = 0.f;
    int glu_act = 0;       // 1: the gate passes the tanh form of gelu instead
};

__device__ __forceinline__ uint4 ld_stream(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// thread (lane, c) of 128 finishes accumulator element c of `lane`: the four warps' K ranges in a fixed order, then the epilogue
template <int MT, int EPI, int NSET>
__device__ __forceinline__ void finish_tile(const SkinnyParams& p, const float (&red)[4][NSET][MT][32][4], int n0, int split, int c, int lane) {
    const int r = lane >> 2, q = lane & 3;
    float up1 = 0.f;
#pragma unroll
    for (int j = 0; j < MT; ++j) {
        const int m = 8 * j + 2 * q + (c & 1);
        float v[NSET];
#pragma unroll
        for (int s = 0; s < NSET; ++s)
            v[s] = ((red[0][s][j][lane][c] + red[1][s][j][lane][c]) + red[2][s][j][lane][c]) + red[3][s][j][lane][c];
        if (m >= p.M) continue;
        if (EPI == 2) {
            // (two sets: gate rows and up rows; one: gate rows, and eight further on their up rows, which the threads of elements 0 and 1 finish)
            const int row = n0 + r + (NSET == 2 ? 8 * (c >> 1) : 0);
            if (row >= p.N || (NSET == 1 && c > 1)) continue;
            if (NSET == 1) {
                const int c2 = c + 2 < 4 ? c + 2 : c;
                up1 = ((red[0][0][j][lane][c2] + red[1][0][j][lane][c2]) + red[2][0][j][lane][c2]) + red[3][0][j][lane][c2];
            }
            float g = v[0] + (p.bias ? __bfloat162float(p.bias[row]) : 0.f);
            float u = (NSET == 1 ? up1 : v[NSET - 1]) + (p.bias ? __bfloat162float(p.bias[row + p.up_offset]) : 0.f);
            if (p.glu_limit > 0.f) { g = fminf(g, p.glu_limit); u = fminf(fmaxf(u, -p.glu_limit), p.glu_limit); }
            reinterpret_cast<__nv_bfloat16*>(p.out)[(long long)m * p.ldo + row] =
                __float2bfloat16_rn(gate_act(p.glu_act, p.glu_alpha, g) * (u + p.glu_shift));
            continue;
        }
#pragma unroll
        for (int s = 0; s < NSET; ++s) {
            const int row = n0 + 16 * s + r + 8 * (c >> 1);
            if (row >= p.N) continue;
            if (EPI == 0) {
                const float b = p.bias ? __bfloat162float(p.bias[row]) : 0.f;
                reinterpret_cast<__nv_bfloat16*>(p.out)[(long long)m * p.ldo + row] = __float2bfloat16_rn(v[s] + b);
            } else if (EPI == 4) {                                   // the square of relu, for feed-forwards of two matrices
                const float b = p.bias ? __bfloat162float(p.bias[row]) : 0.f;
                const float a = fmaxf(v[s] + b, 0.f);
                reinterpret_cast<__nv_bfloat16*>(p.out)[(long long)m * p.ldo + row] = __float2bfloat16_rn(a * a);
            } else if (EPI == 1) {
                reinterpret_cast<float*>(p.out)[((long long)split * p.M + m) * p.ldo + row] = v[s];
            } else {
                const float b = p.bias ? __bfloat162float(p.bias[row]) : 0.f;
                reinterpret_cast<float*>(p.out)[(long long)m * p.ldo + row] = v[s] + b;
            }
        }
    }
}

// SETS: sets of 16 weight rows per CTA for the plain epilogues.  Every set is multiplied with the same activation
// fragments, so the activations - which every CTA fetches for itself, through the caches - cost half as much per weight
// byte with two sets (SwiGLU has always had two: its gate rows and its up rows).
template <int MT, int EPI, int U, int SETS>
__global__ void __launch_bounds__(128)
skinny_gemm_kernel(const SkinnyParams p) {
    constexpr int NSET = EPI == 2 ? 2 : SETS;                    // SwiGLU streams two row sets: gate and up
    __shared__ float red[4][NSET][MT][32][4];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, q = lane & 3;
    const int n0 = blockIdx.x * 16 * (EPI == 2 ? 1 : SETS);
    const int set_stride = EPI == 2 ? p.up_offset : 16;           // rows from one set to the next
    const int split = blockIdx.y;
    const int kq = p.kslice / 4;
    const int k_begin = split * p.kslice + warp * kq;
    const int k_end = min(p.K, min((split + 1) * p.kslice, k_begin + kq));

    float acc[NSET][MT][4];
#pragma unroll
    for (int s = 0; s < NSET; ++s)
#pragma unroll
        for (int j = 0; j < MT; ++j) { acc[s][j][0] = acc[s][j][1] = acc[s][j][2] = acc[s][j][3] = 0.f; }

    // (SwiGLU: N counts the gate rows, and an up row exists wherever its gate row does)
    bool row_a[NSET], row_b[NSET];
    const __nv_bfloat16* wrow[NSET][2];
#pragma unroll
    for (int s = 0; s < NSET; ++s) {
        const int in_n = n0 + r + (EPI == 2 ? 0 : s * 16);
        row_a[s] = in_n < p.N; row_b[s] = in_n + 8 < p.N;
        const long long base = (long long)(n0 + r + s * set_stride);
        wrow[s][0] = p.w + (row_a[s] ? base : 0) * p.ldw;
        wrow[s][1] = p.w + (row_b[s] ? base + 8 : 0) * p.ldw;
    }
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);

    // Two register buffers: the loads of the next 32*U keys are in flight while the current ones
    // feed the tensor core, so every warp always has weight bytes on their way from HBM.  The weights
    // do not depend on the kernel before this one, so the first loads of both buffers are issued
    // before the wait for that kernel's results: the stream from HBM ramps up while it drains.
    uint4 wA[U][NSET][2], xA[U][MT], wB[U][NSET][2], xB[U][MT];
    auto load_w = [&](int k0, uint4 (&wv)[U][NSET][2]) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int kk = k0 + 32 * u + 8 * q;
            const bool ok = kk < k_end;
#pragma unroll
            for (int s = 0; s < NSET; ++s) {
                wv[u][s][0] = (ok && row_a[s]) ? ld_stream(wrow[s][0] + kk) : zero;
                wv[u][s][1] = (ok && row_b[s]) ? ld_stream(wrow[s][1] + kk) : zero;
            }
        }
    };
    auto load_x = [&](int k0, uint4 (&xv)[U][MT]) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int kk = k0 + 32 * u + 8 * q;
            const bool ok = kk < k_end;
#pragma unroll
            for (int j = 0; j < MT; ++j) {
                const int m = 8 * j + r;
                xv[u][j] = (ok && m < p.M) ? __ldg(reinterpret_cast<const uint4*>(p.x + (long long)m * p.ldx + kk)) : zero;
            }
        }
    };
    auto compute = [&](const uint4 (&wv)[U][NSET][2], const uint4 (&xv)[U][MT]) {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int s = 0; s < NSET; ++s)
#pragma unroll
                for (int j = 0; j < MT; ++j) {
                    mma_bf16(acc[s][j], wv[u][s][0].x, wv[u][s][1].x, wv[u][s][0].y, wv[u][s][1].y, xv[u][j].x, xv[u][j].y);
                    mma_bf16(acc[s][j], wv[u][s][0].z, wv[u][s][1].z, wv[u][s][0].w, wv[u][s][1].w, xv[u][j].z, xv[u][j].w);
                }
    };
    load_w(k_begin, wA);                                       // (loads past k_end give zeros)
    load_w(k_begin + 32 * U, wB);
    TTIE_PDL_ENTRY();                                          // the activations are the predecessor's output
    load_x(k_begin, xA);
    load_x(k_begin + 32 * U, xB);
    for (int k0 = k_begin; k0 < k_end; k0 += 64 * U) {
        compute(wA, xA);
        if (k0 + 64 * U < k_end) { load_w(k0 + 64 * U, wA); load_x(k0 + 64 * U, xA); }
        if (k0 + 32 * U < k_end) {
            compute(wB, xB);
            if (k0 + 96 * U < k_end) { load_w(k0 + 96 * U, wB); load_x(k0 + 96 * U, xB); }
        }
    }

    // sum the four warps' K ranges in a fixed order
#pragma unroll
    for (int s = 0; s < NSET; ++s)
#pragma unroll
        for (int j = 0; j < MT; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c) red[warp][s][j][lane][c] = acc[s][j][c];
    __syncthreads();
    finish_tile<MT, EPI, NSET>(p, red, n0, split, warp, lane);
}

// ---- up to 16 rows: the weights through shared memory, by TMA.
// What bounds such a product is HBM, and what decides how close it comes is how many bytes are on their way and that the stream does not stop
// between two tiles: copies alone, without the products, reach 6.2 TB/s with 128 KB in flight per SM and 7.0 with 192 KB, whatever the order of the
// rows (180 MB; 33 MB 5.5 and 6.1).  So a CTA stays (two per SM), walks over units (16 rows of W, or 32: two sets; a
// range of K), and one thread keeps a ring of stages filled (16 KB of W: 512 values of K of 16 rows, 256 of 32; and the activations'
// values, of which two sets need half the copies) across the units' borders; the weights of the first stages are asked for before the wait for
// the kernel before, whose results they do not depend on.  Four warps split a stage's K among themselves, take their operand fragments from
// shared memory as the other form takes them from global memory (the swizzle spreads eight rows' 16 bytes over all banks), and add up
// their ranges at the end of a unit.  Activations through the cache instead of the ring were slower (8 rows: 36 against 31 us).
constexpr int BULK_STAGES_MOST = 8;

struct BulkParams {
    SkinnyParams g;
    int tiles, units, stages, stage_bytes, dynamic;
    ErrorWords err;
    int quitter;                                             // a multiplying warp whose waits run out at once (tests of giving up), or -1
};
// Barrier of the 128 multiplying threads, each of which comes here once a unit whether its waits ran out or not: a warp that went away alone
// would leave the others waiting without a limit.  Tells all of them whether one of them gave up.
__device__ __forceinline__ bool any_of_128(bool bad) {
    uint32_t any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(any) : "r"((uint32_t)bad) : "memory");
    return any != 0;
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int row, int block) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(0), "r"(row), "r"(block) : "memory");
}

// the gated unit with SETS 1: a set's first eight rows are gate rows, the others their up rows (half as long a unit, twice the activations' copies)
__host__ __device__ constexpr int unit_columns(int epi, int sets) { return epi == 2 ? (sets == 1 ? 8 : 16) : 16 * sets; }
template <int NSET> struct BulkShape {
    static constexpr int KS = 512 / NSET, BLOCKS = KS / 64;      // K of a stage
    static constexpr uint32_t SET = BLOCKS * 16 * 128, WEIGHTS = NSET * SET;           // bytes of 16 rows, of a stage's weights (16 KB)
};

template <int MT, int EPI, int SETS>
__global__ void __launch_bounds__(160, 2) skinny_bulk_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const BulkParams bp) {
    constexpr int NSET = SETS;
    constexpr bool PAIRED = EPI == 2 && NSET == 1;
    using Sh = BulkShape<NSET>;
    constexpr int KS = Sh::KS, KW = KS / 4;                      // KW: K of a warp, in every fourth piece of 32: the same pieces with any number of sets
    const SkinnyParams& p = bp.g;
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) unsigned long long bars[2 * BULK_STAGES_MOST + 1];
    __shared__ __align__(16) uint4 next_unit;                    // the answer to the question for another unit
    __shared__ int stage_unit[BULK_STAGES_MOST], stage_k[BULK_STAGES_MOST], stage_more[BULK_STAGES_MOST];      // what a stage holds; whether a unit follows its last one
    __shared__ float red[2][4][NSET][MT][32][4];                 // (in turn: the next unit's sums need not wait for this one's to be read)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, q = lane & 3;
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * BULK_STAGES_MOST, asked = empty0 + 8 * BULK_STAGES_MOST, ring0 = smem_u32(ring);
    if (tid == 0) {
        for (int s = 0; s < bp.stages; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 4);
        }
        mbar_init(asked, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    auto range_of = [&](int unit, int& n0, int& split, int& k_begin, int& k_end) {
        split = unit / bp.tiles;
        n0 = (unit - split * bp.tiles) * unit_columns(EPI, NSET);
        k_begin = split * p.kslice;
        k_end = min(p.K, k_begin + p.kslice);
    };
    if (warp == 4) {
        if (lane != 0) return;
        const uint32_t bytes = Sh::WEIGHTS + (uint32_t)(Sh::BLOCKS * p.M * 128);
        int s = 0, round = 0, ahead = 0, turn = 0;               // ahead: stages whose activations are still to come; turn: questions answered
        bool ok = true, waited = false, open = false;               // open: a question without its answer
        auto acts = [&](int k0, int st) { tma_load_3d(ring0 + (uint32_t)st * bp.stage_bytes + Sh::WEIGHTS, &tmX, full0 + 8 * st, 0, k0 / 64); };
        auto settle = [&]() {                                    // the kernel before is done: the activations of the stages filled so far
            pdl_wait();
            pdl_launch_dependents();
            waited = true;
            for (int i = 0; i < ahead; ++i) acts(stage_k[i], i);
        };
        // a CTA that has not started yet gives its unit to one that has room for it
        auto ask = [&]() {
            open = true;
            mbar_expect_tx(asked, 16);
            asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(smem_u32(&next_unit)), "r"(asked) : "memory");
        };
        auto answer = [&]() -> int {                             // its number, or -1: all have started
            open = false;
            if (!mbar_wait(asked, turn++ & 1, 63, bp.err)) { ok = false; return -1; }
            uint32_t given, x;
            asm volatile("{\n\t.reg .b128 h;\n\t.reg .pred p;\n\tld.shared.b128 h, [%2];\n\t"
                         "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\tselp.u32 %0, 1, 0, p;\n\tmov.u32 %1, 0;\n\t"
                         "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n\t}"
                         : "=r"(given), "=r"(x) : "r"(smem_u32(&next_unit)) : "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");                  // (read before the next answer is written)
            return given ? (int)x : -1;
        };
        int unit = blockIdx.x;
        while (ok && unit >= 0) {
            if (bp.dynamic) ask();
            int n0, split, k_begin, k_end, next = -1;
            range_of(unit, n0, split, k_begin, k_end);
            for (int k0 = k_begin; k0 < k_end; k0 += KS) {
                if (!waited && ahead == bp.stages) settle();
                if (round > 0) ok = mbar_wait(empty0 + 8 * s, (round & 1) ^ 1, 61, bp.err);
                if (ok && bp.dynamic && k0 + KS >= k_end) next = answer();
                if (!ok) break;
                const uint32_t bar = full0 + 8 * s, dst = ring0 + (uint32_t)s * bp.stage_bytes;
                stage_unit[s] = unit;
                stage_k[s] = k0;
                stage_more[s] = next >= 0;
                mbar_expect_tx(bar, bytes);
#pragma unroll
                for (int i = 0; i < (PAIRED ? 2 : NSET); ++i)    // (rows and blocks past the end are zeros; blocks of the next range are not used)
                    tma_load_3d(dst + i * (PAIRED ? Sh::SET / 2 : Sh::SET), &tmW, bar, n0 + (EPI == 2 ? i * p.up_offset : i * 16), k0 / 64);
                if (waited) acts(k0, s);
                else ++ahead;
                if (++s == bp.stages) { s = 0; ++round; }
            }
            unit = next;
        }
        if (!waited) settle();
        // nothing may land in a CTA that has left, and the multiplying warps may have given up (each wait is bounded)
        for (int i = 0; i < bp.stages; ++i) if (round > 0 || i < s) mbar_wait(full0 + 8 * i, (i < s ? round : round - 1) & 1, 61, bp.err);
        if (open) mbar_wait(asked, turn & 1, 63, bp.err);
        return;
    }
    pdl_wait();                                                  // (so that a wait's limit does not count the time of the kernel before)
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    int s = 0, round = 0;
    auto arrived = [&]() { return (bool)__all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, round & 1, 62, bp.err, warp == bp.quitter)); };
    auto next_stage = [&]() { if (++s == bp.stages) { s = 0; ++round; } };
    bool more = true;
    for (int turn = 0; more; turn ^= 1) {
        bool ok = arrived();
        int n0, split, k_begin, k_end;
        range_of(ok ? stage_unit[s] : 0, n0, split, k_begin, k_end);
        float acc[NSET][MT][4];
#pragma unroll
        for (int i = 0; i < NSET; ++i)
#pragma unroll
            for (int j = 0; j < MT; ++j) { acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f; }
        for (int k0 = k_begin; k0 < k_end; k0 += KS) {
            if (k0 > k_begin) ok = arrived();
            if (!ok) break;
            const unsigned char* base = ring + (size_t)s * bp.stage_bytes;
            more = stage_more[s];
#pragma unroll
            for (int u = 0; u < KW / 32; ++u) {
                const int k = 32 * (warp + 4 * u), block = k >> 6, chunk = ((k >> 3) & 7) + q, at = (chunk ^ r) << 4;       // (row & 7 is r for all of this lane's rows)
                const bool in = k0 + k < k_end;                  // (ranges are multiples of 64)
                uint4 wv[NSET][2], xv[MT];
#pragma unroll
                for (int i = 0; i < NSET; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        wv[i][h] = in ? *reinterpret_cast<const uint4*>(base + (PAIRED ? h * (Sh::SET / 2) + (block * 8 + r) * 128 : i * Sh::SET + (block * 16 + h * 8 + r) * 128) + at) : zero;
#pragma unroll
                for (int j = 0; j < MT; ++j) {
                    const int line = block * p.M + 8 * j + r;    // (as many lines a block as there are rows)
                    xv[j] = in && 8 * j + r < p.M ? *reinterpret_cast<const uint4*>(base + Sh::WEIGHTS + line * 128 + ((chunk ^ (line & 7)) << 4)) : zero;
                }
#pragma unroll
                for (int i = 0; i < NSET; ++i)
#pragma unroll
                    for (int j = 0; j < MT; ++j) {
                        mma_bf16(acc[i][j], wv[i][0].x, wv[i][1].x, wv[i][0].y, wv[i][1].y, xv[j].x, xv[j].y);
                        mma_bf16(acc[i][j], wv[i][0].z, wv[i][1].z, wv[i][0].w, wv[i][1].w, xv[j].z, xv[j].w);
                    }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty0 + 8 * s);
            next_stage();
        }
#pragma unroll
        for (int i = 0; i < NSET; ++i)
#pragma unroll
            for (int j = 0; j < MT; ++j)
#pragma unroll
                for (int c = 0; c < 4; ++c) red[turn][warp][i][j][lane][c] = acc[i][j][c];
        if (any_of_128(!ok)) break;
        finish_tile<MT, EPI, NSET>(p, red[turn], n0, split, warp, lane);
    }
}

thread_local int g_quitter = -1;

template <int MT, int EPI, int SETS>
int launch_bulk(const SkinnyParams& p, int splits, cudaStream_t s) {
    constexpr int NSET = SETS;
    using Sh = BulkShape<NSET>;
    constexpr int ROOM = 228 * 512 - 1024 - 320 - 2 * 4 * NSET * MT * 512 - 1024;              // what two CTAs per SM leave for a ring
    BulkParams b;
    b.g = p;
    b.quitter = g_quitter;
    b.tiles = ceil_div(p.N, unit_columns(EPI, NSET));
    b.units = b.tiles * splits;
    b.stage_bytes = ((int)Sh::WEIGHTS + Sh::BLOCKS * p.M * 128 + 1023) / 1024 * 1024;
    b.stages = ROOM / b.stage_bytes < BULK_STAGES_MOST ? ROOM / b.stage_bytes : BULK_STAGES_MOST;
    CUtensorMap mw, mx;
    if (gemm_tc_make_block_map(&mw, p.w, EPI == 2 ? (long long)p.up_offset + p.N : p.N, p.K / 64, p.ldw, EPI == 2 && NSET == 1 ? 8 : 16, Sh::BLOCKS)) return -1;
    if (gemm_tc_make_block_map(&mx, p.x, p.M, p.K / 64, p.ldx, p.M, Sh::BLOCKS)) return -1;
    if (gemm_tc_error_words(&b.err.word, &b.err.mirror)) TTIE_FAIL("skinny_gemm: the error word's address is not to be had");
    auto kernel = skinny_bulk_kernel<MT, EPI, SETS>;
    static bool allowed[64] = {false};
    int dev = 64;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64 || !allowed[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ROOM + 1024);
        if (e != cudaSuccess) TTIE_FAIL("skinny_gemm: %d bytes of shared memory refused: %s", ROOM + 1024, cudaGetErrorString(e));
        if (dev < 64) allowed[dev] = true;
    }
    // A CTA per unit; where they are more than fit at once, a running one takes over the units of those that have not started.  (Equal shares
    // decided beforehand end at different times - 29 to 43 us for [32000, 4096] -, since the SMs do not get equal shares of the memory's rate.)
    b.dynamic = b.units > 2 * num_sms();
    TTIE_LAUNCH(kernel, b.units, 160, b.stages * b.stage_bytes + 1024, s, mw, mx, b);
    TTIE_CHECK_LAUNCH("skinny_gemm (bulk)");
    return 0;
}

template <int MT, int EPI, int U, int SETS>
int launch(const SkinnyParams& p, int splits, cudaStream_t s) {
    dim3 grid(ceil_div(p.N, 16 * (EPI == 2 ? 1 : SETS)), splits);
    TTIE_LAUNCH((skinny_gemm_kernel<MT, EPI, U, SETS>), grid, 128, 0, s, p);
    TTIE_CHECK_LAUNCH("skinny_gemm");
    return 0;
}

template <int EPI>
int dispatch(const SkinnyParams& p, int splits, int unroll, cudaStream_t s) {
    // unroll: low four bits 0 (chosen here), 2 or 4; + 16 asks for two row sets per CTA (plain epilogues)
    const bool two = EPI != 2 && (unroll & 16);
    unroll &= 15;
    const int mt = ceil_div(p.M, 8);
    // Through shared memory from 1 Mi weights on ([1024, 1024] in two ranges 1.9 | 2.0, [512, 2048] in four 1.9 | 2.0, whole 2.7 | 3.9).  us, this form | the other, 1 row and 8:
    // [4352, 4096] 6.7 | 7.5, 7.2 | 7.6; [4096, 4096] 6.4 | 6.7, 7.0 | 7.0; gate and up of [22016, 4096] 27.0 | 31.2, 27.5 | 31.6; [4096, 11008]
    // 13.9 | 15.5, 15.0 | 16.2; [32000, 4096] 37.8 | 44.1, 38.8 | 45.4; [256000, 2048] 146 | 145, 147 | 145 (copies alone: 5.5 us for 33 MB,
    // 25.9 for 180, 37.0 for 262).  The gated unit in sets of 8 + 8 rows where these are long enough a unit.  8 + 8 | 16 + 16 at 1 row and 8: [16384, 1024]
    // 9.4 | 8.4, 9.4 | 9.2; [16384, 2048] 12.8 | 11.7, 13.1 | 12.5; [32768, 2048] 21.0 | 21.1, 22.4 | 22.0; [13824, 2560] 12.9 | 12.8, 13.7 | 14.5;
    // [16384, 3072] 16.2 | 16.9, 17.9 | 18.2; [19456, 3584] 23.4 | 25.9, 24.6 | 26.8; [22016, 4096] 27.9 | 31.0, 28.8 | 31.9; [36352, 4544] 47.9 | 48.7,
    // 49.4 | 49.9; [57344, 8192] 131.5 | 137.0, 135.4 | 137.4.  The sums are the same to the last bit either way.
    const long long weights = (long long)p.N * (EPI == 2 ? 2 : 1) * p.K;
    // (A gated unit of fewer units than SMs stays with the other form: its caller has a product cut over K, with the activation behind it, for that.)
    if (mt <= 2 && p.K % 64 == 0 && weights >= (1LL << 20) && (EPI != 2 || p.N >= 8 * num_sms())) {
        const bool wide = EPI == 2 ? p.K < 2560 : two;
        if (mt == 1) return wide ? launch_bulk<1, EPI, 2>(p, splits, s) : launch_bulk<1, EPI, 1>(p, splits, s);
        return wide ? launch_bulk<2, EPI, 2>(p, splits, s) : launch_bulk<2, EPI, 1>(p, splits, s);
    }
    // a product that is not split over CTAs streams best with deep unrolling, a split one with more CTAs per SM
    const bool deep = EPI != 2 && (unroll ? unroll >= 4 : splits == 1);
    if (two) {
        if (mt <= 1) return deep ? launch<1, EPI, 2, 2>(p, splits, s) : launch<1, EPI, 1, 2>(p, splits, s);
        if (mt <= 2) return launch<2, EPI, 1, 2>(p, splits, s);
        if (mt <= 4) return launch<4, EPI, 1, 2>(p, splits, s);
        return launch<8, EPI, 1, 1>(p, splits, s);
    }
    if (mt <= 1) return deep ? launch<1, EPI, 4, 1>(p, splits, s) : launch<1, EPI, (EPI == 2 ? 1 : 2), 1>(p, splits, s);
    if (mt <= 2) return launch<2, EPI, (EPI == 2 ? 1 : 2), 1>(p, splits, s);
    if (mt <= 4) return launch<4, EPI, (EPI == 2 ? 1 : 2), 1>(p, splits, s);
    return launch<8, EPI, 1, 1>(p, splits, s);
}
}  // namespace

extern "C" int ttie_skinny_max_rows() { return 64; }

// epilogue: 0 bfloat16 out (4: the same after relu(.)^2), 1 float32 partial sums [splits][M][N], 2 SwiGLU (w holds gate rows then up
// rows, N = F), 3 float32 out.  kslice: K range per CTA, a multiple of 128; splits = ceil(K / kslice),
// which must be 1 unless epilogue is 1.
extern "C" int ttie_skinny_gemm_tuned(const void* x, long long ldx, const void* w, long long ldw, const void* bias, void* out,
                                      long long ldo, int M, int N, int K, int kslice, int epilogue, int up_offset, int unroll,
                                      void* stream);
extern "C" int ttie_skinny_gemm(const void* x, long long ldx, const void* w, long long ldw, const void* bias, void* out,
                                long long ldo, int M, int N, int K, int kslice, int epilogue, int up_offset, void* stream) {
    return ttie_skinny_gemm_tuned(x, ldx, w, ldw, bias, out, ldo, M, N, K, kslice, epilogue, up_offset, 0, stream);
}
// for tests: multiplying warp `warp` (0 to 3; -1: none) of this thread's launches gives up at its first wait; an error code and no hang is what follows
extern "C" void ttie_skinny_quitter(int warp) { g_quitter = warp; }
static thread_local float g_glu[3] = {1.f, 0.f, 0.f};
static thread_local int g_glu_act = 0;
// the gated-unit epilogue (2) with constants other than SwiGLU's: alpha, limit (<= 0: none), shift, act (1: gelu's tanh form on the gate);
// bias (or null): F values of the gate, then F of the up projection
extern "C" int ttie_skinny_gemm_glu(const void* x, long long ldx, const void* w, long long ldw, const void* bias, void* out, long long ldo,
                                    int M, int F, int K, float alpha, float limit, float shift, int act, void* stream) {
    if (act < 0 || act > 1) TTIE_FAIL("skinny_gemm: unknown activation %d", act);
    g_glu_act = act; g_glu[0] = alpha; g_glu[1] = limit; g_glu[2] = shift;
    const int rc = ttie_skinny_gemm_tuned(x, ldx, w, ldw, bias, out, ldo, M, F, K, (K + 127) / 128 * 128, 2, F, 0, stream);
    g_glu_act = 0; g_glu[0] = 1.f; g_glu[1] = 0.f; g_glu[2] = 0.f;
    return rc;
}
// unroll: 0 = chosen from kslice; 2 or 4 = 32-key blocks per register buffer (rows <= 8 only); + 16 = two sets of 16
// weight rows per CTA (plain epilogues; halves the 32-key blocks per buffer).
extern "C" int ttie_skinny_gemm_tuned(const void* x, long long ldx, const void* w, long long ldw, const void* bias, void* out,
                                      long long ldo, int M, int N, int K, int kslice, int epilogue, int up_offset, int unroll,
                                      void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (M > 64) TTIE_FAIL("skinny_gemm: %d rows; this kernel takes at most 64", M);
    if (K <= 0 || K % 8) TTIE_FAIL("skinny_gemm: K=%d must be a positive multiple of 8", K);
    if (ldx % 8 || ldw % 8) TTIE_FAIL("skinny_gemm: row strides must be multiples of 8 elements");
    if (((uintptr_t)x | (uintptr_t)w) & 15) TTIE_FAIL("skinny_gemm: pointers must be 16-byte aligned");
    if (kslice <= 0 || kslice % 128) TTIE_FAIL("skinny_gemm: kslice=%d must be a positive multiple of 128", kslice);
    const int splits = ceil_div(K, kslice);
    if (splits > 1 && epilogue != 1) TTIE_FAIL("skinny_gemm: K can be split over CTAs only with the partial-sum epilogue");
    if (splits > 65535) TTIE_FAIL("skinny_gemm: too many splits");
    SkinnyParams p;
    p.x = (const __nv_bfloat16*)x; p.ldx = ldx; p.w = (const __nv_bfloat16*)w; p.ldw = ldw;
    p.bias = (const __nv_bfloat16*)bias; p.out = out; p.ldo = ldo; p.M = M; p.N = N; p.K = K;
    p.kslice = kslice; p.up_offset = up_offset;
    p.glu_alpha = g_glu[0]; p.glu_limit = g_glu[1]; p.glu_shift = g_glu[2]; p.glu_act = g_glu_act;
    cudaStream_t s = (cudaStream_t)stream;
    switch (epilogue) {
        case 0: return dispatch<0>(p, splits, unroll, s);
        case 1: return dispatch<1>(p, splits, unroll, s);
        case 2: return dispatch<2>(p, splits, unroll, s);
        case 3: return dispatch<3>(p, splits, unroll, s);
        case 4: return dispatch<4>(p, splits, unroll, s);
    }
    TTIE_FAIL("skinny_gemm: unknown epilogue %d", epilogue);
}

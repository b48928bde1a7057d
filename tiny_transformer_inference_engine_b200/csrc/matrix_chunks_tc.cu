// The chunked matrix-state recurrences of matrix_chunks.cu (retention, the xLSTM matrix memory) with their products on the 5th-generation tensor
// cores, in chunks of 128 tokens: bfloat16 values of at most 128 columns and at most 128 key channels.
//
// The arithmetic is that of matrix_chunks.cu: 32-bit operands as three bfloat16, six plane products for a product of two of them.  What differs is
// where the sums lie: a CTA of 512 threads owns a (chunk, head), an instruction multiplies 128 rows by up to 128 columns from
// shared memory (the weights of the scores: from tensor memory, where the threads that computed them leave them), and its sums are in tensor
// memory, a thread per row and half of the columns.  The tensor cores cut bits off where an addition rounds: so every sum there spans 64 terms (32 in
// the chunks' own sums) with the large plane products last, and the spans are added by ordinary additions.
//
//   chunk_sum_tc   D[value column][channel] = V^T K', both operands as they lie (token by row); four spans of 32 tokens
//   chunk_out_tc   S = Q K^T, then O = Q (state)^T while the threads weigh the scores, then the weights times V; spans of 64 channels and tokens
//
// One prompt of 2,048 tokens, us of sum + carry + out: 16 heads of 128 x 128 14 + 6 + 30 (27 + 9 + 64 in chunks of 64), 16 of 64 x 128 12 + 6 + 25
// (13 + 11 + 40).  A CTA of the out kernel takes some 21,000 clocks, one after the other (one fits an SM: six planes of 32 KB): 6,000 for the rows
// of q and k, as fast as the L2 gives them to all SMs, 3,400 + 3,300 + 1,600 for the products, whose two operands come
// from shared memory at its bandwidth (73 clocks a product, 64 at the tensor cores' rate), 2,000 for splitting the state and the weights, 2,500 for the
// stores; 256 of them on 148 SMs are two rounds.  With 256 threads, a half row each, it took 31,000 (conversions and divisions wait for issue slots).
// Error against 64 bits (1,000 tokens, chunks of 64 and the walk behind it): read-out 0.97e-7 (1.0e-7, 2.4e-7), state 5.3e-8 (5.2e-8, 1.7e-7); read-out
// without CUT64 1.5e-7.
//
// Every mbarrier wait is bounded by a clock deadline; one that runs out records a code and the CTA goes on to its end.
#include "matrix_chunks.cuh"
#include "planes.cuh"
using namespace ttie;
using namespace ttie::chunks;

namespace ttie { int gemm_tc_error_words(int** word, int** mirror); }

namespace {
constexpr int CT = 128, NT = 512, DVP = 128, GROUPS = NT / 128;   // tokens of a chunk, threads, value columns (zeros behind Dv), threads of a row
constexpr int OWN = 128 / GROUPS;                                // columns of a thread
// What cutting instead of rounding leaves: a sum of 64 terms of one sign-independent size comes out 6.7e-8 of itself too small on average, one of 32
// 2.3e-8 (measured against 64 bits), the same for every sum, so it is put back.
constexpr float CUT64 = 6.7e-8f, CUT32 = 2.3e-8f;
constexpr long long WAIT_CYCLES = 2000000000LL;                 // about one second
constexpr uint32_t BLOCK = CT * 128;                             // 128 rows of 64 bfloat16, 128-byte swizzle

// a value in 64 bits as the sum of two floats (an infinity: and zero)
__device__ __forceinline__ float2 two_floats(double x) {
    const float hi = (float)x;
    return make_float2(hi, isinf(hi) ? 0.f : (float)(x - (double)hi));
}
struct ErrorWords { int* word; int* mirror; };
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool mbar_try(uint32_t bar) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar) : "memory");
    return ok != 0;
}
// each barrier here completes once
__device__ __forceinline__ void mbar_wait(uint32_t bar, int code, const ErrorWords& e) {
    if (!mbar_try(bar)) {
        const long long deadline = clock64() + WAIT_CYCLES;
        while (!mbar_try(bar)) {
            if (clock64() > deadline) {
                atomicCAS(e.word, 0, code);
                if (e.mirror) { *reinterpret_cast<volatile int*>(e.mirror) = code; __threadfence_system(); }
                break;
            }
        }
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void sync_tc() {                      // a block barrier that also orders tensor memory accesses
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Lower words of shared-memory operand descriptors.  K along the row: 64-value blocks, a step of 16 is 32 bytes.  K down the rows: a step
// of 16 is 2048 bytes, neighbouring 64-column blocks are BLOCK bytes apart.  Upper word: 8-row groups 1024 bytes apart, 128-byte swizzle.
constexpr uint32_t DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_rows(uint32_t addr, int ks) { return (((addr + (uint32_t)(ks >> 2) * BLOCK + (uint32_t)(ks & 3) * 32) & 0x3FFFFu) >> 4) | (1u << 16); }
__device__ __forceinline__ uint32_t desc_cols(uint32_t addr, int ks) { return (((addr + (uint32_t)ks * 2048) & 0x3FFFFu) >> 4) | ((BLOCK >> 4) << 16); }
__device__ __forceinline__ void umma_ss(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}"
                 ::"r"(d), "r"(a_lo), "r"(b_lo), "r"(DESC_HI), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 db, {%2, %3};\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
                 ::"r"(d), "r"(a), "r"(b_lo), "r"(DESC_HI), "r"(idesc), "r"(accumulate) : "memory");
}
// D float32, A and B bfloat16; M 128, N columns; which operands have K down the rows
__host__ __device__ constexpr uint32_t idesc_of(int n, bool a_cols, bool b_cols) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (a_cols ? 1u << 15 : 0u) | (b_cols ? 1u << 16 : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[16]) {     // (the values pass through, so that nothing that uses them moves ahead of this)
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]) :: "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
// sixteen columns of SPANS sums, `step` columns apart, added, with what their cut additions lost on average
template <int SPANS>
__device__ __forceinline__ void tmem_sum16(uint32_t taddr, int step, float (&o)[16]) {
    uint32_t v[SPANS][16];
#pragma unroll
    for (int s = 0; s < SPANS; ++s) tmem_ld16(taddr + s * step, v[s]);
#pragma unroll
    for (int s = 0; s < SPANS; ++s) tmem_ld_wait(v[s]);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        if constexpr (SPANS == 1) {
            const float t = __uint_as_float(v[0][i]);
            o[i] = fmaf(t, CUT64, t);
        } else {                                                     // (with what the last addition rounds off: the correction is about half a unit)
            float x = __uint_as_float(v[0][i]), y = __uint_as_float(v[1][i]);
            if constexpr (SPANS == 4) { x += y; y = __uint_as_float(v[2][i]) + __uint_as_float(v[3][i]); }
            const float t = x + y, u = t - x;
            o[i] = t + fmaf(t, SPANS == 4 ? CUT32 : CUT64, (x - (t - u)) + (y - u));
        }
    }
}
// byte offset of eight values (columns c .. c + 7) of row j in an operand's plane
__device__ __forceinline__ uint32_t piece_at(int j, int c) { return (uint32_t)(c >> 6) * BLOCK + (uint32_t)j * 128 + (uint32_t)((((c >> 3) & 7) ^ (j & 7)) << 4); }
// eight values into PL planes (1: they are bfloat16 already)
template <int PL>
__device__ __forceinline__ void store_piece(unsigned char* base, uint32_t plane, uint32_t at, float (&x)[8]) {
    uint32_t p0[4], p1[4], p2[4];
    split_values<4>(x, p0, p1, p2);
    *reinterpret_cast<uint4*>(base + at) = make_uint4(p0[0], p0[1], p0[2], p0[3]);
    if constexpr (PL == 3) {
        *reinterpret_cast<uint4*>(base + plane + at) = make_uint4(p1[0], p1[1], p1[2], p1[3]);
        *reinterpret_cast<uint4*>(base + 2 * plane + at) = make_uint4(p2[0], p2[1], p2[2], p2[3]);
    }
}
// 128 rows of COLS values from src + j * ld, zero where in(j, column) is false, behind scale(j, values): four pieces of a thread are on their way at a time
template <int PL, int COLS, typename E, typename In, typename Scale>
__device__ __forceinline__ void stage_rows(unsigned char* dst, const E* src, long long ld, In in, Scale scale) {
    constexpr int PIECES = COLS / 8, ITERS = CT * PIECES / NT, BATCH = ITERS < 4 ? ITERS : 4;
    static_assert(ITERS > 0 && ITERS % BATCH == 0, "128 rows of a multiple of 64 values");
#pragma unroll
    for (int i0 = 0; i0 < ITERS; i0 += BATCH) {
        float x[BATCH][8];
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
            const int e = (i0 + i) * NT + threadIdx.x, j = e / PIECES, c = (e % PIECES) * 8;
            load8(src + (size_t)j * ld + c, in(j, c), x[i]);
        }
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
            const int e = (i0 + i) * NT + threadIdx.x, j = e / PIECES, c = (e % PIECES) * 8;
            scale(j, x[i]);
            store_piece<PL>(dst, COLS / 64 * BLOCK, piece_at(j, c), x[i]);
        }
    }
}
// bfloat16 rows as they are
template <int COLS>
__device__ __forceinline__ void stage_plain(unsigned char* dst, const __nv_bfloat16* src, long long ld, int n, int cols) {
    constexpr int PIECES = COLS / 8, ITERS = CT * PIECES / NT;
    uint4 x[ITERS];
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
        const int e = i * NT + threadIdx.x, j = e / PIECES, c = (e % PIECES) * 8;
        x[i] = j < n && c < cols ? *reinterpret_cast<const uint4*>(src + (size_t)j * ld + c) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
        const int e = i * NT + threadIdx.x;
        *reinterpret_cast<uint4*>(dst + piece_at(e / PIECES, (e % PIECES) * 8)) = x[i];
    }
}
__device__ __forceinline__ unsigned char* align1024(unsigned char* p) {
    return reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~(uintptr_t)1023);
}
// rows of a tile in shared memory -> global, a warp a row (at most 128 columns, multiples of 4)
template <int LD>
__device__ __forceinline__ void copy_tile(float* dst, long long ld, const float* tile, int rows, int cols) {
    const int col = (threadIdx.x & 31) * 4;
    if (col >= cols) return;
#pragma unroll 4
    for (int r = threadIdx.x >> 5; r < rows; r += NT / 32)
        *reinterpret_cast<float4*>(dst + (size_t)r * ld + col) = *reinterpret_cast<const float4*>(tile + r * LD + col);
}
template <int NBARS>
__device__ __forceinline__ void tc_setup(unsigned long long* bars, uint32_t* slot, uint32_t cols) {      // barriers and tensor memory; ends in a block barrier
    if (threadIdx.x == 32) {
        for (int i = 0; i < NBARS; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bars + i)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // what the threads staged becomes visible to the tensor core
    sync_tc();
}
__device__ __forceinline__ void tc_free(uint32_t tmem, uint32_t cols) {
    sync_tc();
    if (threadIdx.x < 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}

// ------------------------------------------------------------------------------------------- chunk_sum
template <int KP> struct SumTc {
    static constexpr uint32_t PLANE = KP / 64 * BLOCK, COLS = 4 * KP;
    static constexpr size_t bytes = 3 * PLANE + DVP / 64 * BLOCK + 1024;
};

template <int MODE, int KP>
__global__ void __launch_bounds__(NT, KP == 64 ? 2 : 1) chunk_sum_tc_kernel(const ChunkArgs a, const ErrorWords err) {
    constexpr uint32_t PLANE = SumTc<KP>::PLANE, COLS = SumTc<KP>::COLS;
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* kd = align1024(smem_dyn);                         // [3] planes of decayed keys
    unsigned char* v_s = kd + 3 * PLANE;
    __shared__ __align__(8) unsigned long long bars[1];
    __shared__ uint32_t slot;
    __shared__ double ends[2 * CT / 32 + 2];
    __shared__ float wt[CT], norm_part[NT];
    TTIE_PDL_ENTRY();
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, quarter = (tid >> 5) & 3, group = tid >> 7;
    int s, c, t0, n;
    if (!find_chunk<CT>(a.qsl, a.num_seqs, a.slot_lo + blockIdx.x, s, c, t0, n)) return;
    const size_t unit = (size_t)blockIdx.x * a.H + h;
    stage_plain<DVP>(v_s, reinterpret_cast<const __nv_bfloat16*>(a.v) + (size_t)t0 * a.ld_v + h * a.Dv, a.ld_v, n, a.Dv);
    if constexpr (MODE == RET) {
        if (tid < CT) wt[tid] = tid < n ? (float)power((double)a.decay[h], n - 1 - tid) : 0.f;
    } else {
        double F, x, X;
        chunk_gates<CT>(a, t0, n, h, ends, F, x, X);
        if (tid < CT) wt[tid] = expf((float)(x - ends[2 * CT / 32 + 1]));
        if (tid == 0) a.span[unit] = make_double2(ends[2 * CT / 32], ends[2 * CT / 32 + 1]);
    }
    __syncthreads();
    using KT = typename std::conditional<MODE == RET, float, __nv_bfloat16>::type;
    const KT* kp = reinterpret_cast<const KT*>(a.k) + (size_t)t0 * a.ld_qk + h * a.D;
    stage_rows<3, KP>(kd, kp, a.ld_qk, [&](int j, int ch) { return j < n && ch < a.D; }, [&](int j, float (&x)[8]) {
        const float w = wt[j];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = j < n ? x[i] * w : 0.f;
    });
    tc_setup<1>(bars, &slot, COLS);
    const uint32_t tmem = slot, bar = smem_u32(bars);
    if (tid == 0) {
        constexpr uint32_t idesc = idesc_of(KP, true, true);
        const uint32_t va = smem_u32(v_s), ka = smem_u32(kd);
#pragma unroll
        for (int sp = 0; sp < 4; ++sp)
#pragma unroll
            for (int l = 2; l >= 0; --l)
#pragma unroll
                for (int ks = 0; ks < 2; ++ks)
                    umma_ss(tmem + sp * KP, desc_cols(va, sp * 2 + ks), desc_cols(ka + l * PLANE, sp * 2 + ks), idesc, l != 2 || ks != 0);
        umma_commit(bar);
    }
    __syncwarp();
    if constexpr (MODE == MLSTM) {                                   // the normaliser's sum: the same without the values
        constexpr int PARTS = NT / KP;
        const int ch = tid % KP, part = tid / KP;
        float sum = 0.f;
        for (int j = part * (CT / PARTS); j < (part + 1) * (CT / PARTS); ++j) {
            const unsigned char* at = kd + piece_at(j, ch & ~7) + (ch & 7) * 2;
            auto plane = [&](int l) { return __uint_as_float((uint32_t)*reinterpret_cast<const uint16_t*>(at + l * PLANE) << 16); };
            sum += plane(0) + (plane(1) + plane(2));
        }
        norm_part[tid] = sum;
        __syncthreads();
        if (tid < a.Dpad) {
            float t = 0.f;
#pragma unroll
            for (int i = 0; i < PARTS; ++i) t += norm_part[i * KP + tid];
            a.aux[unit * a.Dpad + tid] = t;
        }
    }
    mbar_wait(bar, 51, err);
    __syncthreads();                                                 // (the keys have been read, by the normaliser too: the sums take their place on their way out)
    constexpr int LD = KP + 4;
    float* tile = reinterpret_cast<float*>(kd);
    const int row = quarter * 32 + lane;
#pragma unroll
    for (int g = 0; g < KP / 16 / GROUPS; ++g) {
        const int col = group * (KP / GROUPS) + g * 16;
        float o[16];
        tmem_sum16<4>(tmem + ((uint32_t)(quarter * 32) << 16) + col, KP, o);
#pragma unroll
        for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(tile + row * LD + col + i) = make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]);
    }
    tc_free(tmem, COLS);
    copy_tile<LD>(a.part + unit * a.Dv * a.Dpad, a.Dpad, tile, a.Dv, a.Dpad);
}

// ------------------------------------------------------------------------------------------- chunk_out
template <int MODE, int KP> struct OutTc {
    static constexpr int QPL = MODE == MLSTM ? 1 : 3;
    static constexpr uint32_t PLANE = KP / 64 * BLOCK, COLS = 512;
    static constexpr size_t bytes = (QPL + 3) * PLANE + DVP / 64 * BLOCK + 1024;
    static_assert((QPL + 3) * PLANE + DVP / 64 * BLOCK >= CT * (DVP + 4) * 4, "the operands' place takes the output tile");
};

template <int MODE, int KP>
__global__ void __launch_bounds__(NT, 1) chunk_out_tc_kernel(const ChunkArgs a, const ErrorWords err) {
    constexpr int QPL = OutTc<MODE, KP>::QPL, SPANS = KP / 64;
    constexpr uint32_t PLANE = OutTc<MODE, KP>::PLANE, COLS = OutTc<MODE, KP>::COLS;
    constexpr uint32_t S_COL = 0, P_COL = 0, O_COL = 256;            // scores, then (over them) three planes of weights; read-outs
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* q_s = align1024(smem_dyn);                        // [QPL] planes of the queries
    unsigned char* k_s = q_s + QPL * PLANE;                          // [QPL] planes of the keys, then [3] of the state
    unsigned char* v_s = k_s + 3 * PLANE;
    __shared__ __align__(8) unsigned long long bars[3];
    __shared__ uint32_t slot;
    __shared__ double ends[2 * CT / 32 + 2], Ms[MODE == MLSTM ? CT : 1];
    __shared__ __align__(16) float2 xs[MODE == MLSTM ? CT : 1];      // mlstm: x of a token, the sum of two floats
    __shared__ float pw[MODE == RET ? CT + 1 : 1], nb[MODE == MLSTM ? KP : 1], den_s[MODE == MLSTM ? GROUPS : 1][MODE == MLSTM ? CT : 1];
    TTIE_PDL_ENTRY();
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, quarter = (tid >> 5) & 3, group = tid >> 7, row = quarter * 32 + lane;
    int s, c, t0, n;
    if (!find_chunk<CT>(a.qsl, a.num_seqs, a.slot_lo + blockIdx.x, s, c, t0, n)) return;
    const size_t unit = (size_t)blockIdx.x * a.H + h;
    using QT = typename std::conditional<MODE == RET, float, __nv_bfloat16>::type;
    const QT* qp = reinterpret_cast<const QT*>(a.q) + (size_t)t0 * a.ld_qk + h * a.D;
    const QT* kp = reinterpret_cast<const QT*>(a.k) + (size_t)t0 * a.ld_qk + h * a.D;
    float row_in = 1.f, den = 0.f, floor_ = 0.f;                     // factor of the state before the chunk; mlstm: denominator, e^-m
    if constexpr (MODE == RET) {
        auto in = [&](int j, int ch) { return j < n && ch < a.D; };
        auto as_is = [](int, float (&)[8]) {};
        stage_rows<3, KP>(q_s, qp, a.ld_qk, in, as_is);
        stage_rows<3, KP>(k_s, kp, a.ld_qk, in, as_is);
        if (tid <= CT) pw[tid] = (float)power((double)a.decay[h], tid);
    } else {
        stage_plain<KP>(q_s, qp, a.ld_qk, n, a.D);
        stage_plain<KP>(k_s, kp, a.ld_qk, n, a.D);
        double F, x, X;
        chunk_gates<CT>(a, t0, n, h, ends, F, x, X);
        const float2 mm = a.mm[unit];
        const double m = (double)mm.x;
        if (tid < CT) { xs[tid] = two_floats(x); Ms[tid] = fmax(m, X); den_s[0][tid] = expf((float)-(F + fmax(m, X))); }
        if (tid < KP) nb[tid] = tid < a.Dpad ? a.aux[unit * a.Dpad + tid] : 0.f;
        // (a chunk is the request's last of this pass if the next chunk is not there or not in the pass)
        if (tid == 0 && ((c + 1) * CT >= a.qsl[s + 1] - a.qsl[s] || (int)blockIdx.x + 1 == a.slots))
            a.mx[(size_t)state_row(a.slot_ids[s], a.state_rows) * a.H + h] = mm.y;
        __syncthreads();
        row_in = expf((float)(m - Ms[row]));
        floor_ = den_s[0][row];
    }
    stage_plain<DVP>(v_s, reinterpret_cast<const __nv_bfloat16*>(a.v) + (size_t)t0 * a.ld_v + h * a.Dv, a.ld_v, n, a.Dv);
    tc_setup<3>(bars, &slot, COLS);
    if constexpr (MODE == RET) row_in = pw[row + 1];
    const uint32_t tmem = slot, bar = smem_u32(bars), mine = tmem + ((uint32_t)(quarter * 32) << 16);
    const uint32_t qa = smem_u32(q_s), ka = smem_u32(k_s), va = smem_u32(v_s);
    // products of QPL planes of one operand and BPL of the other that matter at 32 bits, the smallest first, over a span of 64 channels
    auto products = [&](uint32_t d, uint32_t b_base, int bpl, int sp) {
        bool first = true;
        for (int sum = QPL == 3 || bpl == 3 ? 2 : 0; sum >= 0; --sum)
            for (int i = 0; i < QPL; ++i) {
                const int j = sum - i;
                if (j < 0 || j >= bpl) continue;
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    umma_ss(d, desc_rows(qa + i * PLANE, sp * 4 + ks), desc_rows(b_base + j * PLANE, sp * 4 + ks), idesc_of(128, false, false), !(first && ks == 0));
                }
                first = false;
            }
    };
    if (tid == 0) {
        for (int sp = 0; sp < SPANS; ++sp) products(tmem + S_COL + sp * 128, ka, QPL, sp);
        umma_commit(bar);
    }
    __syncwarp();
    // the state before the chunk travels meanwhile: 128 value columns of KP channels
    constexpr int PIECES = KP / 8, ITERS = DVP * PIECES / NT;
    float st[ITERS][8];
    const float* sp0 = a.part + unit * a.Dv * a.Dpad;
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
        const int e = i * NT + tid, j = e / PIECES, ch = (e % PIECES) * 8;
        load8(sp0 + (size_t)j * a.Dpad + ch, j < a.Dv && ch < a.Dpad, st[i]);
    }
    if constexpr (MODE == MLSTM) {                                   // q . n before the chunk, a quarter of the channels a thread
#pragma unroll
        for (int ch = group * (KP / GROUPS); ch < (group + 1) * (KP / GROUPS); ch += 8) {
            const uint4 q = *reinterpret_cast<const uint4*>(q_s + piece_at(row, ch));
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) { const float2 f = unpack(w[i]); den = fmaf(f.x, nb[ch + 2 * i], den); den = fmaf(f.y, nb[ch + 2 * i + 1], den); }
        }
        den *= row_in;
    }
    mbar_wait(bar, 52, err);                                         // the scores are there, the keys have been read
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
        const int e = i * NT + tid;
        store_piece<3>(k_s, PLANE, piece_at(e / PIECES, (e % PIECES) * 8), st[i]);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    sync_tc();
    if (tid == 0) {
        for (int sp = 0; sp < SPANS; ++sp) products(tmem + O_COL + sp * 128, ka, 3, sp);
        umma_commit(bar + 8);
    }
    __syncwarp();
    // the scores of this row and a quarter of the keys: weighed, masked, and back as planes
    float w[OWN];
    const float2 M = two_floats(MODE == MLSTM ? Ms[row] : 0.0);
#pragma unroll
    for (int g = 0; g < OWN / 16; ++g) {
        float o[16];
        tmem_sum16<SPANS>(mine + S_COL + group * OWN + g * 16, 128, o);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int j = group * OWN + g * 16 + i;
            float f;
            if constexpr (MODE == RET) f = pw[max(row - j, 0)];
            else f = expf((xs[j].x - M.x) + (xs[j].y - M.y));
            const float x = j <= row ? o[i] * f : 0.f;
            if constexpr (MODE == MLSTM) den += x;
            w[g * 16 + i] = x;
        }
    }
    if constexpr (MODE == MLSTM) den_s[group][row] = den;            // (its first row held e^-m, which every thread has read)
    sync_tc();                                                       // all scores have been read: the planes go over them
    if constexpr (MODE == MLSTM) den = (den_s[0][row] + den_s[1][row]) + (den_s[2][row] + den_s[3][row]);
#pragma unroll
    for (int g = 0; g < OWN / 16; ++g) {
        float x[16];
        uint32_t p0[8], p1[8], p2[8];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = w[g * 16 + i];
        split_values<8>(x, p0, p1, p2);
        const uint32_t at = mine + P_COL + group * (OWN / 2) + g * 8;
        tmem_st8(at, p0);
        tmem_st8(at + 64, p1);
        tmem_st8(at + 128, p2);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    mbar_wait(bar + 8, 53, err);                                     // what the state before the chunk gives
    float o[OWN];
#pragma unroll
    for (int g = 0; g < OWN / 16; ++g) {
        float x[16];
        tmem_sum16<SPANS>(mine + O_COL + group * OWN + g * 16, 128, x);
#pragma unroll
        for (int i = 0; i < 16; ++i) o[g * 16 + i] = x[i] * row_in;
    }
    sync_tc();
    if (tid == 0) {                                                  // weights times values, spans of 64 tokens, the small planes first
        for (int sp = 0; sp < 2; ++sp)
            for (int l = 2; l >= 0; --l)
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
                    umma_ts(tmem + O_COL + sp * 128, tmem + P_COL + l * 64 + sp * 32 + ks * 8, desc_cols(va, sp * 4 + ks), idesc_of(DVP, false, true), !(l == 2 && ks == 0));
        umma_commit(bar + 16);
    }
    __syncwarp();
    float scale = 1.f, odd = 0.f;                                    // odd: not 0 if something of this thread's is not finite
    if constexpr (MODE == MLSTM) {
        odd = den * 0.f;
        scale = a.qscale / (fmaxf(fabsf(den * a.qscale), floor_) + 1e-6f);
    }
    mbar_wait(bar + 16, 54, err);                                    // (all products are done: the output tile takes the operands' place)
    constexpr int LD = DVP + 4;
    float* tile = reinterpret_cast<float*>(q_s);
#pragma unroll
    for (int g = 0; g < OWN / 16; ++g) {
        const int col = group * OWN + g * 16;
        float x[16];
        tmem_sum16<2>(mine + O_COL + col, 128, x);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            x[i] += o[g * 16 + i];
            if constexpr (MODE == MLSTM) x[i] *= scale;
            odd = fmaf(x[i], 0.f, odd);
        }
#pragma unroll
        for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(tile + row * LD + col + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
    }
    tc_free(tmem, COLS);
    const size_t ld_o = (size_t)a.H * a.Dv;
    copy_tile<LD>(a.out + (size_t)t0 * ld_o + h * a.Dv, ld_o, tile, n, a.Dv);
    if (__syncthreads_or(row < n && !(odd == 0.f))) walk_out<MODE, CT, __nv_bfloat16>(a, unit, t0, n, h, tile);
}

template <int MODE, int KP>
int launch_tc(ChunkArgs a, int first, int slots, const ErrorWords& err, cudaStream_t st) {
    static bool allowed[64] = {false};
    int dev = 64;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64 || !allowed[dev]) {
        cudaFuncSetAttribute(chunk_sum_tc_kernel<MODE, KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SumTc<KP>::bytes);
        cudaFuncSetAttribute(chunk_out_tc_kernel<MODE, KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(OutTc<MODE, KP>::bytes));
        if (dev < 64) allowed[dev] = true;
    }
    a.slot_lo = first; a.slots = slots;
    const dim3 grid(slots, a.H);
    const dim3 carry(ceil_div(a.Dv * a.Dpad + (MODE == MLSTM ? a.Dpad : 0), 4 * CARRY), a.H, a.num_seqs);
    TTIE_LAUNCH((chunk_sum_tc_kernel<MODE, KP>), grid, NT, SumTc<KP>::bytes, st, a, err);
    TTIE_LAUNCH((chunk_carry_kernel<MODE, CT>), carry, CARRY, 0, st, a);
    TTIE_LAUNCH((chunk_out_tc_kernel<MODE, KP>), grid, NT, (OutTc<MODE, KP>::bytes), st, a, err);
    TTIE_CHECK_LAUNCH("matrix_chunks_tc");
    return 0;
}
}  // namespace

namespace ttie {
int matrix_chunks_tc(int mode, ChunkArgs a, int T, int slots, cudaStream_t st) {
    ErrorWords err;
    if (gemm_tc_error_words(&err.word, &err.mirror)) TTIE_FAIL("matrix_chunks: the error word's address is not to be had");
    const int total = T / CT + a.num_seqs;
    for (int first = 0; first < total; first += slots) {
        const int cnt = total - first < slots ? total - first : slots;
        int rc;
        if (mode == RET) rc = a.Dpad <= 64 ? launch_tc<RET, 64>(a, first, cnt, err, st) : launch_tc<RET, 128>(a, first, cnt, err, st);
        else rc = a.Dpad <= 64 ? launch_tc<MLSTM, 64>(a, first, cnt, err, st) : launch_tc<MLSTM, 128>(a, first, cnt, err, st);
        if (rc) return rc;
    }
    return 0;
}
}  // namespace ttie

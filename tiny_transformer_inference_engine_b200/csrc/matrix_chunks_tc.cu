// The chunked matrix-state recurrences of matrix_chunks.cu (retention, the xLSTM matrix memory) with their products on the 5th-generation tensor
// cores, in chunks of 128 tokens: bfloat16 values of at most 128 columns and at most 128 key channels.
//
// The arithmetic is that of matrix_chunks.cu: 32-bit operands as three bfloat16, six plane products for a product of two of them, differences of the
// gates' sums in 64 bits (as two floats).  What differs is where the sums lie: a CTA of 512 threads owns a (chunk, head), an instruction multiplies
// 128 rows by up to 128 columns from shared memory, and its sums are in tensor memory, a thread per row and quarter of the columns.  They come
// out in rounds (below): 16 terms of the leading planes at a time.
//
//   chunk_sum_tc   D[value column][channel] = V^T K', both operands as they lie (token by row); what rounding the rounds' sum leaves is kept
//   chunk_out_tc   S = Q K^T, then O = Q (state)^T while the threads weigh the scores, then the weights, in the place of queries and state, times V;
//                  with a gate the read-outs are normalised over the head and gated before they leave: the gate's rows come into the place of the
//                  state while the weights are multiplied, and leave as the results.  The whole mixer 149.4 -> 145.6 us (retention), 120.9 -> 114.9
//                  (mlstm of 64 x 128) at 2,048 tokens: the pass over the read-outs took 9 us, of which 3 to 6 more stay in this kernel.  From the
//                  sums' tile in shared memory, a warp a row, with divisions rounded to 32 bits they took 8 to 14.
//
// One prompt of 2,048 tokens, us of the scan (in chunks of 64): 16 heads of 128 x 128 retention 59 (95), mlstm 65 (100), 16 of 64 x 128 40 (54)
// and 48 (65).  One CTA of the out kernel fits an SM (six planes of 32 KB), its phases run one after the other, and 256 of them on 148 SMs are
// two turns.  With sums of 64 terms (32 in chunk_sum_tc) in one place the four took 51, 58, 34 and 43, but then the tensor cores cut off 6.7e-8 (2.3e-8)
// of each sum.  Chunk_out_tc spills 40 bytes a thread (mlstm, 128 channels) for its rows' weights and read-outs.  Tried and slower: rounds left out
// for tokens that are not there (the thread that issues the products then computes their addresses: 69 us for the 59), no sums for keys that
// no row of a warp sees (63: 300 bytes spilled).
// Error against 64 bits (mean of six inputs, 700 tokens, normal values; chunks of 64 and the walk behind it): retention of 128 x 128 read-out 8.8e-8
// (9.3e-8, 14.8e-8), state 4.0e-8 (4.4e-8, 8.7e-8); mlstm of 64 x 128 7.1e-7 (7.8e-7, 14.9e-7), 1.80e-7 (1.80e-7, 5.3e-7).  Values of one sign: 5.4e-8
// (5.0e-8, 4.1e-8), 4.2e-8 (4.1e-8, 11.8e-8).
//
// Every mbarrier wait is bounded by a clock deadline; one that runs out records a code and the CTA goes on to its end.
#include "matrix_chunks.cuh"
#include "planes.cuh"
#include "tc_ptx.cuh"
using namespace ttie;
using namespace ttie::chunks;
using namespace ttie::tc;

namespace {
constexpr int CT = 128, NT = 512, DVP = 128, GROUPS = NT / 128;   // tokens of a chunk, threads, value columns (zeros behind Dv), threads of a row
constexpr int OWN = 128 / GROUPS;                                // columns of a thread
constexpr int SLOTS = 4;                                         // sums of a round in tensor memory
constexpr uint32_t BLOCK = CT * 128;                             // 128 rows of 64 bfloat16, 128-byte swizzle

// a value in 64 bits as the sum of two floats (an infinity: and zero)
__device__ __forceinline__ float2 two_floats(double x) {
    const float hi = (float)x;
    return make_float2(hi, isinf(hi) ? 0.f : (float)(x - (double)hi));
}
// e^d for d in 64 bits: what rounding d to 32 bits leaves counts too
__device__ __forceinline__ float exp_of(double d) {
    const float2 f = two_floats(d);
    const float e = expf(f.x);
    return fmaf(e, f.y, e);
}
// each barrier here completes once; a wait that runs out leaves its code, and the thread goes on
__device__ __forceinline__ void mbar_wait(uint32_t bar, int code, const ErrorWords& e) {
    tc::mbar_wait(bar, 0, code, e);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void sync_tc() {                      // a block barrier that also orders tensor memory accesses
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
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
// D float32, A and B bfloat16; M 128, N columns; which operands have K down the rows
__host__ __device__ constexpr uint32_t idesc_of(int n, bool a_cols, bool b_cols) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (a_cols ? 1u << 15 : 0u) | (b_cols ? 1u << 16 : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
// A product of two operands of which one has, or both have, three planes, in rounds.  The tensor cores cut bits off where an addition rounds, so the
// leading planes' products - 16 bits each, 16 of them all but exact together - are summed 16 terms at a time, each 16 from zero in a
// slot of their own, and the small planes' products (at most 2^-8 of those) all in the last slot.  The slots are added in
// registers by ordinary additions.  A round is up to three 16 terms (four without small planes) and a share of the small products, which
// keep the tensor cores busy while the threads add.
template <int TERMS, bool SMALL> struct Rounds {
    static constexpr int PER = SMALL ? SLOTS - 1 : SLOTS, N = (TERMS + PER - 1) / PER, BARS = N + (SMALL ? 1 : 0);
};
// large(d, i): terms 16 i .. 16 i + 15 of the leading planes into columns d; small(d, i): the i-th of n_small small products, which adds to d unless i is 0
template <int TERMS, bool SMALL, typename Large, typename Small>
__device__ __forceinline__ void issue_round(int r, uint32_t d, int step, uint32_t bar, int n_small, Large large, Small small) {
    using R = Rounds<TERMS, SMALL>;
    for (int i = 0; i < R::PER; ++i)
        if (r * R::PER + i < TERMS) large(d + i * step, r * R::PER + i);
    umma_commit(bar + 8 * r);
    if constexpr (SMALL) {
        for (int i = n_small * r / R::N; i < n_small * (r + 1) / R::N; ++i) small(d + (SLOTS - 1) * step, i);
        if (r == R::N - 1) umma_commit(bar + 8 * R::N);
    }
}
// 16 columns of this thread's row, added
__device__ __forceinline__ void add_slot(uint32_t d, float (&acc)[16]) {
    uint32_t v[16];
    tmem_ld16(d, v);
    tmem_ld_wait(v);
#pragma unroll
    for (int c = 0; c < 16; ++c) acc[c] += __uint_as_float(v[c]);
}
// this thread's row of a round: 16 columns from `d` on of each slot, added to one another and then to acc (fewer roundings of the large sum)
template <int TERMS, bool SMALL>
__device__ __forceinline__ void add_round(int r, uint32_t d, int step, float (&acc)[16]) {
    using R = Rounds<TERMS, SMALL>;
    const int n = min(R::PER, TERMS - r * R::PER);
    uint32_t v[16];
    tmem_ld16(d, v);
    tmem_ld_wait(v);
    float t[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) t[c] = __uint_as_float(v[c]);
#pragma unroll
    for (int i = 1; i < R::PER; ++i)
        if (i < n) add_slot(d + i * step, t);
#pragma unroll
    for (int c = 0; c < 16; ++c) acc[c] += t[c];
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
        for (int i = 0; i < NBARS; ++i) mbar_init(smem_u32(bars + i), 1);
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
    static constexpr uint32_t PLANE = KP / 64 * BLOCK, COLS = SLOTS * KP;
    static constexpr size_t bytes = 3 * PLANE + DVP / 64 * BLOCK + 1024;
};

template <int MODE, int KP>
__global__ void __launch_bounds__(NT, KP == 64 ? 2 : 1) chunk_sum_tc_kernel(const ChunkArgs a, const ErrorWords err) {
    constexpr uint32_t PLANE = SumTc<KP>::PLANE, COLS = SumTc<KP>::COLS;
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* kd = align1024(smem_dyn);                         // [3] planes of decayed keys
    unsigned char* v_s = kd + 3 * PLANE;
    using R = Rounds<CT / 16, true>;
    __shared__ __align__(8) unsigned long long bars[R::BARS];
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
        if (tid < CT) wt[tid] = exp_of(x - ends[2 * CT / 32 + 1]);
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
    tc_setup<R::BARS>(bars, &slot, COLS);
    const uint32_t tmem = slot, bar = smem_u32(bars), va = smem_u32(v_s), ka = smem_u32(kd);
    auto issue = [&](int r) {
        constexpr uint32_t idesc = idesc_of(KP, true, true);
        issue_round<CT / 16, true>(r, tmem, KP, bar, 2 * (CT / 16),
            [&](uint32_t d, int i) { umma_ss(d, desc_cols(va, i), desc_cols(ka, i), idesc, 0); },
            [&](uint32_t d, int i) { umma_ss(d, desc_cols(va, i & 7), desc_cols(ka + (i < 8 ? 2 : 1) * PLANE, i & 7), idesc, i > 0); });
    };
    if (tid == 0) issue(0);
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
    constexpr int OWN_K = KP / GROUPS;                               // columns of a thread
    const int row = quarter * 32 + lane;
    const uint32_t mine = tmem + ((uint32_t)(quarter * 32) << 16) + group * OWN_K;
    float o[OWN_K / 16][16], left[OWN_K / 16][16];                   // left: what rounding the sums leaves
#pragma unroll
    for (int g = 0; g < OWN_K / 16; ++g)
#pragma unroll
        for (int i = 0; i < 16; ++i) o[g][i] = left[g][i] = 0.f;
#pragma unroll
    for (int r = 0; r < R::N; ++r) {
        mbar_wait(bar + 8 * r, 51, err);
#pragma unroll
        for (int g = 0; g < OWN_K / 16; ++g) {
            float v[16] = {};
            add_round<CT / 16, true>(r, mine + g * 16, KP, v);
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                const float t = o[g][c] + v[c], u = t - o[g][c];
                if (r > 0) left[g][c] += (o[g][c] - (t - u)) + (v[c] - u);
                o[g][c] = t;
            }
        }
        if (r + 1 < R::N) {
            sync_tc();
            if (tid == 0) issue(r + 1);
            __syncwarp();
        }
    }
    mbar_wait(bar + 8 * R::N, 51, err);
#pragma unroll
    for (int g = 0; g < OWN_K / 16; ++g) {
        add_slot(mine + (SLOTS - 1) * KP + g * 16, left[g]);
#pragma unroll
        for (int c = 0; c < 16; ++c) o[g][c] += left[g][c];
    }
    __syncthreads();                                                 // (the keys have been read, by the normaliser too: the sums take their place on their way out)
    constexpr int LD = KP + 4;
    float* tile = reinterpret_cast<float*>(kd);
#pragma unroll
    for (int g = 0; g < OWN_K / 16; ++g)
#pragma unroll
        for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(tile + row * LD + group * OWN_K + g * 16 + i) = make_float4(o[g][i], o[g][i + 1], o[g][i + 2], o[g][i + 3]);
    tc_free(tmem, COLS);
    copy_tile<LD>(a.part + unit * a.Dv * a.Dpad, a.Dpad, tile, a.Dv, a.Dpad);
}

// ------------------------------------------------------------------------------------------- chunk_out
template <int MODE, int KP> struct OutTc {
    static constexpr int QPL = MODE == MLSTM ? 1 : 3;
    static constexpr uint32_t PLANE = KP / 64 * BLOCK, COLS = 512;
    static constexpr uint32_t W_PLANE = CT / 64 * BLOCK;             // of the weights, which take the place of the queries and the state
    // behind the weights, in place of the state: the gate's rows, the rows' sums of squares and the norm's weights
    static constexpr uint32_t GATE_LD = DVP * 2 + 16, GATE = (CT * GATE_LD + (GROUPS * CT + DVP) * 4 + 1023) / 1024 * 1024;
    static constexpr uint32_t OPERANDS = (QPL + 3) * PLANE > 3 * W_PLANE + GATE ? (QPL + 3) * PLANE : 3 * W_PLANE + GATE;
    static constexpr size_t bytes = OPERANDS + DVP / 64 * BLOCK + 1024;
    static_assert(OPERANDS >= CT * (DVP + 4) * 4, "the operands' place takes the output tile");
    static_assert(OPERANDS % 1024 == 0, "the values' swizzle starts on 1024 bytes");
    // rounds of the scores, of the read-out of the state, of weights times values
    using Scores = Rounds<KP / 16, QPL == 3>;
    using State = Rounds<KP / 16, true>;
    using Values = Rounds<CT / 16, true>;
};

template <int MODE, int KP>
__global__ void __launch_bounds__(NT, 1) chunk_out_tc_kernel(const ChunkArgs a, const ErrorWords err) {
    using Tc = OutTc<MODE, KP>;
    constexpr int QPL = Tc::QPL, TERMS = KP / 16;
    constexpr uint32_t PLANE = Tc::PLANE, W_PLANE = Tc::W_PLANE, COLS = Tc::COLS, SLOT = 128;
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* q_s = align1024(smem_dyn);                        // [QPL] planes of the queries
    unsigned char* k_s = q_s + QPL * PLANE;                          // [QPL] planes of the keys, then [3] of the state
    unsigned char* v_s = q_s + Tc::OPERANDS;
    __shared__ __align__(8) unsigned long long bars[Tc::Scores::BARS + Tc::State::BARS + Tc::Values::BARS];
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
        if (tid < CT) { xs[tid] = tid < n ? two_floats(x) : make_float2(-3e38f, 0.f); Ms[tid] = fmax(m, X); den_s[0][tid] = exp_of(-(F + fmax(m, X))); }
        if (tid < KP) nb[tid] = tid < a.Dpad ? a.aux[unit * a.Dpad + tid] : 0.f;
        // (a chunk is the request's last of this pass if the next chunk is not there or not in the pass)
        if (tid == 0 && ((c + 1) * CT >= a.qsl[s + 1] - a.qsl[s] || (int)blockIdx.x + 1 == a.slots))
            a.mx[(size_t)state_row(a.slot_ids[s], a.state_rows) * a.H + h] = mm.y;
        __syncthreads();
        row_in = exp_of(m - Ms[row]);
        floor_ = den_s[0][row];
    }
    stage_plain<DVP>(v_s, reinterpret_cast<const __nv_bfloat16*>(a.v) + (size_t)t0 * a.ld_v + h * a.Dv, a.ld_v, n, a.Dv);
    tc_setup<Tc::Scores::BARS + Tc::State::BARS + Tc::Values::BARS>(bars, &slot, COLS);
    if constexpr (MODE == RET) row_in = pw[row + 1];
    const uint32_t tmem = slot, mine = tmem + ((uint32_t)(quarter * 32) << 16) + group * OWN;
    const uint32_t bar_s = smem_u32(bars), bar_o = bar_s + 8 * Tc::Scores::BARS, bar_v = bar_o + 8 * Tc::State::BARS;
    const uint32_t qa = smem_u32(q_s), ka = smem_u32(k_s), va = smem_u32(v_s);
    // queries times BPL planes of keys or state: the products of planes that matter at 32 bits, the smallest first
    auto issue_rows = [&](auto planes, int r, uint32_t bar) {
        constexpr int BPL = decltype(planes)::value;
        constexpr bool SMALL = QPL + BPL > 2;
        constexpr uint32_t idesc = idesc_of(128, false, false);
        issue_round<TERMS, SMALL>(r, tmem, SLOT, bar, (QPL == 3 && BPL == 3 ? 5 : 2) * TERMS,
            [&](uint32_t d, int i) { umma_ss(d, desc_rows(qa, i), desc_rows(ka, i), idesc, 0); },
            [&](uint32_t d, int i) {
                const int pair = i / TERMS, ks = i % TERMS;
                const int bp = QPL == 1 ? 2 - pair : pair == 0 ? 2 : pair == 1 || pair == 3 ? 1 : 0;                      // 2 1 0 1 0 of the second operand beside
                const int qp = QPL == 1 ? 0 : pair == 0 || pair == 3 ? 0 : pair == 1 || pair == 4 ? 1 : 2;                // 0 1 2 0 1 of the queries
                umma_ss(d, desc_rows(qa + qp * PLANE, ks), desc_rows(ka + bp * PLANE, ks), idesc, i > 0);
            });
    };
    using KeyPlanes = std::integral_constant<int, QPL>;
    using StatePlanes = std::integral_constant<int, 3>;
    float w[OWN / 16][16], o[OWN / 16][16];                          // scores, then weights, of this row and a quarter of the keys; read-outs of a quarter of the columns
#pragma unroll
    for (int g = 0; g < OWN / 16; ++g)
#pragma unroll
        for (int i = 0; i < 16; ++i) w[g][i] = o[g][i] = 0.f;
    if (tid == 0) issue_rows(KeyPlanes{}, 0, bar_s);
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
#pragma unroll
    for (int r = 0; r < Tc::Scores::N; ++r) {
        mbar_wait(bar_s + 8 * r, 52, err);
#pragma unroll
        for (int g = 0; g < OWN / 16; ++g) add_round<TERMS, (QPL > 1)>(r, mine + g * 16, SLOT, w[g]);
        if (r + 1 < Tc::Scores::N) {
            sync_tc();
            if (tid == 0) issue_rows(KeyPlanes{}, r + 1, bar_s);
            __syncwarp();
        }
    }
    if constexpr (QPL > 1) {
        mbar_wait(bar_s + 8 * Tc::Scores::N, 52, err);
#pragma unroll
        for (int g = 0; g < OWN / 16; ++g) add_slot(mine + (SLOTS - 1) * SLOT + g * 16, w[g]);
    }
#pragma unroll
    for (int i = 0; i < ITERS; ++i) {
        const int e = i * NT + tid;
        store_piece<3>(k_s, PLANE, piece_at(e / PIECES, (e % PIECES) * 8), st[i]);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    sync_tc();
    if (tid == 0) issue_rows(StatePlanes{}, 0, bar_o);
    __syncwarp();
    // the scores weighed and masked
    const float2 M = two_floats(MODE == MLSTM ? Ms[row] : 0.0);
#pragma unroll
    for (int g = 0; g < OWN / 16; ++g) {
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int j = group * OWN + g * 16 + i;
            float f;
            if constexpr (MODE == RET) {
                f = pw[max(row - j, 0)];
            } else {                                                 // e^(x - M): the difference, and what rounding it to 32 bits leaves
                const float2 x = xs[j];
                const float d = x.x - M.x, u = d - x.x, e = expf(d);
                f = fmaf(e, ((x.x - (d - u)) - (M.x + u)) + (x.y - M.y), e);
            }
            const float y = j <= row ? w[g][i] * f : 0.f;
            if constexpr (MODE == MLSTM) sum[i & 3] += y;
            w[g][i] = y;
        }
        if constexpr (MODE == MLSTM) den += (sum[0] + sum[1]) + (sum[2] + sum[3]);
    }
    if constexpr (MODE == MLSTM) den_s[group][row] = den;            // (its first row held e^-m, which every thread has read)
#pragma unroll
    for (int r = 0; r < Tc::State::N; ++r) {
        mbar_wait(bar_o + 8 * r, 53, err);
#pragma unroll
        for (int g = 0; g < OWN / 16; ++g) add_round<TERMS, true>(r, mine + g * 16, SLOT, o[g]);
        sync_tc();
        if (r + 1 < Tc::State::N) {
            if (tid == 0) issue_rows(StatePlanes{}, r + 1, bar_o);
            __syncwarp();
        }
    }
    if constexpr (MODE == MLSTM) den = (den_s[0][row] + den_s[1][row]) + (den_s[2][row] + den_s[3][row]);
    mbar_wait(bar_o + 8 * Tc::State::N, 53, err);                    // what the state before the chunk gives; queries and state have been read
    unsigned char* gate_s = q_s + 3 * W_PLANE;                       // [CT] rows of GATE_LD bytes
    float* squares = reinterpret_cast<float*>(gate_s + CT * Tc::GATE_LD);                            // [GROUPS][CT]
    float* norm_w = squares + GROUPS * CT;                           // [DVP]
    if (a.y) {
        const __nv_bfloat16* gp = a.gate + (size_t)t0 * a.ld_gate + h * a.Dv;
#pragma unroll
        for (int e = tid; e < CT * DVP / 8; e += NT) {
            const int r = e / (DVP / 8), col = e % (DVP / 8) * 8;
            if (r < n && col < a.Dv) copy16(gate_s + r * Tc::GATE_LD + col * 2, gp + (size_t)r * a.ld_gate + col);
        }
        if (tid < DVP) norm_w[tid] = a.norm_w && tid < a.Dv ? a.norm_w[h * a.Dv + tid] : 1.f;
    }
#pragma unroll
    for (int g = 0; g < OWN / 16; ++g) {
        add_slot(mine + (SLOTS - 1) * SLOT + g * 16, o[g]);
#pragma unroll
        for (int i = 0; i < 16; ++i) o[g][i] *= row_in;
#pragma unroll
        for (int c = 0; c < 16; c += 8) {
            float x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = w[g][c + i];
            store_piece<3>(q_s, W_PLANE, piece_at(row, group * OWN + g * 16 + c), x);
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    sync_tc();
    auto issue_values = [&](int r) {                                 // weights times values, the small planes of the weights apart
        constexpr uint32_t idesc = idesc_of(DVP, false, true);
        issue_round<CT / 16, true>(r, tmem, SLOT, bar_v, 2 * (CT / 16),
            [&](uint32_t d, int i) { umma_ss(d, desc_rows(qa, i), desc_cols(va, i), idesc, 0); },
            [&](uint32_t d, int i) { umma_ss(d, desc_rows(qa + (i < 8 ? 2 : 1) * W_PLANE, i & 7), desc_cols(va, i & 7), idesc, i > 0); });
    };
    if (tid == 0) issue_values(0);
    __syncwarp();
    float scale = 1.f, odd = 0.f;                                    // odd: not 0 if something of this thread's is not finite
    if constexpr (MODE == MLSTM) {
        odd = den * 0.f;
        scale = a.qscale / (fmaxf(fabsf(den * a.qscale), floor_) + 1e-6f);
    }
#pragma unroll
    for (int r = 0; r < Tc::Values::N; ++r) {
        mbar_wait(bar_v + 8 * r, 54, err);
#pragma unroll
        for (int g = 0; g < OWN / 16; ++g) add_round<CT / 16, true>(r, mine + g * 16, SLOT, o[g]);
        if (r + 1 < Tc::Values::N) {
            sync_tc();
            if (tid == 0) issue_values(r + 1);
            __syncwarp();
        }
    }
    mbar_wait(bar_v + 8 * Tc::Values::N, 54, err);                   // (all products are done: the output tile takes the operands' place)
    constexpr int LD = DVP + 4;
    float* tile = reinterpret_cast<float*>(q_s);
    float ss = 0.f;
#pragma unroll
    for (int g = 0; g < OWN / 16; ++g) {
        add_slot(mine + (SLOTS - 1) * SLOT + g * 16, o[g]);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if constexpr (MODE == MLSTM) o[g][i] *= scale;
            odd = fmaf(o[g][i], 0.f, odd);
            ss = fmaf(o[g][i], o[g][i], ss);
        }
        if (a.y) continue;
#pragma unroll
        for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(tile + row * LD + group * OWN + g * 16 + i) = make_float4(o[g][i], o[g][i + 1], o[g][i + 2], o[g][i + 3]);
    }
    if (a.y) {
        squares[group * CT + row] = ss;
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    tc_free(tmem, COLS);
    const size_t ld_o = (size_t)a.H * a.Dv;
    if (a.y) {                                                       // gated where the gate's row lies, then out in whole rows
        const float inv = inverse_rms(a, (squares[row] + squares[CT + row]) + (squares[2 * CT + row] + squares[3 * CT + row]));
        uint4* gr = reinterpret_cast<uint4*>(gate_s + row * Tc::GATE_LD + group * OWN * 2);
        const float2* w2 = reinterpret_cast<const float2*>(norm_w + group * OWN);
#pragma unroll
        for (int c = 0; c < OWN / 8; ++c) {
            const uint4 g4 = gr[c];
            const uint32_t g[4] = {g4.x, g4.y, g4.z, g4.w};
            uint32_t y[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) y[i] = gated_pair(a, o[c / 2][(c & 1) * 8 + 2 * i] * inv, o[c / 2][(c & 1) * 8 + 2 * i + 1] * inv, w2[c * 4 + i], g[i]);
            gr[c] = make_uint4(y[0], y[1], y[2], y[3]);
        }
        __syncthreads();
        const int col = tid % (DVP / 8) * 8;
        if (col < a.Dv)
#pragma unroll 4
            for (int r = tid / (DVP / 8); r < n; r += NT / (DVP / 8))
                *reinterpret_cast<uint4*>(a.y + (size_t)(t0 + r) * ld_o + h * a.Dv + col) = *reinterpret_cast<const uint4*>(gate_s + r * Tc::GATE_LD + col * 2);
    } else copy_tile<LD>(a.out + (size_t)t0 * ld_o + h * a.Dv, ld_o, tile, n, a.Dv);
    if (__syncthreads_or(row < n && !(odd == 0.f))) {
        walk_out<MODE, CT, __nv_bfloat16>(a, unit, t0, n, h, tile);
        if (a.y) gate_walked(a, t0, n, h);
    }
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

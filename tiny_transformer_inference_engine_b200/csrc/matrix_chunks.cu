// The matrix-state recurrences of matrix_memory.cu (retention, the xLSTM matrix memory, the RWKV-style time mix) over prompts, in
// chunks of 64 tokens instead of token by token (chunks of 128 with products on tcgen05: matrix_chunks_tc.cu; both share matrix_chunks.cuh).
//
// A token-by-token walk has no parallelism but the state's elements and waits for its own chain: one prompt of 2,048 tokens and 16
// heads of 128 x 128 took 514 us at 3 TFLOP/s.  Over a chunk the same sums are four small matrix products, and only the state
// between chunks is a chain.  Three launches:
//
//   chunk_sum     per (chunk, head): the chunk's own contribution to the state at its end, sum_j (decay from j to the end) v_j k_j^T
//   chunk_carry   per state element: walks the request's chunks; leaves the state BEFORE each chunk where the chunk's own sum lay
//                 and the request's new state in its state row
//   chunk_out     per (chunk, head): o_i = (decay to i) S q_i + sum_(j <= i) (decay from j to i) (q_i . k_j) v_j
//
// Everything stays 32-bit as in the walk.  The products run on the tensor cores as bfloat16 instructions on operands split into
// planes: a 32-bit value is the sum of three bfloat16 (8 + 8 + 8 bits; exact from 2^-110, below which the last bits fall under the smallest
// bfloat16, up to 3.39e38, above which the first plane is infinite), so a product of two of them is the six plane products
// that matter at 32 bits, in 32-bit sums; a bfloat16 operand is one plane.  Decays are never divided by: every factor is a product of
// decays over a span of tokens, or the exponential of a difference that cannot be positive, so nothing overflows however strong a
// decay is.
//
//   retention   the decay is a constant: powers from a table evaluated in 64 bits.
//   mlstm       with F_i the sum of the log forget gates up to i within the chunk, x_j = i_j - F_j and M_i = max(m before the
//               chunk, max_(j<=i) x_j), the running maximum is m_i = F_i + M_i and the weight of token j in row i is
//               exp(x_j - M_i) <= 1.  F, x and M are 64-bit: they grow with the chunk while their differences stay small.
//   wkv         the decay is per key channel, so it sits inside the product over channels.  A chunk is four blocks of 16 tokens: between
//               blocks a row is multiplied by the decays from its block's start to itself and a key by those from itself to
//               its block's end, whole blocks between them as a vector on the rows; inside a block the 136 scores are summed on the
//               ordinary cores with running products.
//
// What is not finite has no planes (an infinity leaves inf - inf in the second) and would meet rows and elements that it does not reach, as a
// zero weight times an infinity.  It always shows in the results, though: a state element of chunk_carry or a read-out of chunk_out that is not
// finite is computed again token by token, the former for its own element, the latter for its chunk and head, by the walk's operations from the
// state before the chunk.  So infinities, NaN and sums that overflow come out as the walk has them.
//
// Chunks are numbered over the whole step: request s owns the numbers from qsl[s] / 64 + s on, which leaves room for its last
// partial chunk and needs nothing of the host but the number of tokens and requests.
//
// One prompt of 2,048 tokens, us of sum + carry + out: 16 heads of 128 x 128 (retention) 30 + 12 + 69 against the walk's 514; 16 of 64 x 128
// (mlstm) 16 + 13 + 47 against 413, and 15 for its gates; 32 of 64 x 64 (wkv) 31 + 10 + 48 against 473.  What bounds the out kernels is
// latency: 12 or 16 warps per SM fit (the planes in shared memory), issue slots 30 % used, the tensor pipe 34 / 16 / 13 %.
// wkv took 41 + 12 + 85 (116 us in a row, now 89; 16 heads of 128 301, now 237): its CTAs' clocks went to products of decays in 64 bits with their conversions
// and to loads one run after the other (13,700 of 46,600), and to scores whose 16 sums at a time went through shuffles (16,600).  Now
// products are pairs of 32-bit numbers, everything a chunk needs is asked for at once by asynchronous copies, a score is a lane's own sum, and the table
// of decays is the table of the rows' products afterwards, so that four CTAs fit an SM (102 us with three).
// Error against 64 bits (2-norm; 1,000 tokens, the walk's behind it): read-out 1.0e-7 (2.3e-7), 6.4e-7 (1.1e-6), 8.4e-8 (8.6e-8); state
// 6.1e-8 (2.0e-7), 1.6e-7 (3.6e-7), 3.4e-8 (4.5e-8).
#include "matrix_chunks.cuh"
using namespace ttie;
using namespace ttie::chunks;

namespace {
constexpr int CT = 64;                       // tokens per chunk
constexpr int VT_COLS = 64, VLD = VT_COLS + 8;  // value columns per pass; row pitch of the staged values
// ---- planes
// a pair of values as three pairs of bfloat16 whose sum it is
__device__ __forceinline__ void split3(float x, float y, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    auto pack = [](float a, float b) { const __nv_bfloat162 t = __floats2bfloat162_rn(a, b); return *reinterpret_cast<const uint32_t*>(&t); };
    p0 = pack(x, y);
    const float rx = x - __uint_as_float(p0 << 16), ry = y - __uint_as_float(p0 & 0xffff0000u);
    p1 = pack(rx, ry);
    p2 = pack(rx - __uint_as_float(p1 << 16), ry - __uint_as_float(p1 & 0xffff0000u));
}
// A product of many decays as a pair of 32-bit numbers whose sum it is, some 46 bits: each multiplication keeps what it rounds (a fused
// multiply-add gives it exactly) and carries it along.  A chain of them has the latency of 32-bit multiplications; in 64 bits, with the
// conversions to and fro, the decays of a chunk took a third of a wkv read-out's time.
struct Pair {
    float hi, lo;
    __device__ __forceinline__ void operator*=(float w) {
        const float p = hi * w;
        lo = fmaf(lo, w, fmaf(hi, w, -p));
        hi = p;
    }
    __device__ __forceinline__ void operator*=(const Pair& b) {
        const float p = hi * b.hi;
        lo = fmaf(lo, b.hi, fmaf(hi, b.lo, fmaf(hi, b.hi, -p)));
        hi = p;
    }
    __device__ __forceinline__ Pair times(float power_of_two) const { return {hi * power_of_two, lo * power_of_two}; }
    __device__ __forceinline__ float value() const { return hi + lo; }
};
// planes of such a product (its third plane keeps what rounding it to 32 bits would cut)
__device__ __forceinline__ void split3(const Pair& x, uint16_t& p0, uint16_t& p1, uint16_t& p2) {
    const __nv_bfloat16 a = __float2bfloat16_rn(x.hi);
    const float r = x.hi - __bfloat162float(a);
    const __nv_bfloat16 b = __float2bfloat16_rn(r);
    p0 = __bfloat16_as_ushort(a); p1 = __bfloat16_as_ushort(b); p2 = __bfloat16_as_ushort(__float2bfloat16_rn((r - __bfloat162float(b)) + x.lo));
}

__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Two neighbouring 8-column tiles: the plane products of weight 2^-16 and up of 16 terms.  The tensor cores cut the bits below a sum's
// last instead of rounding them (accumulating everything in one place left seven times the walk's error), so the 16 products of the
// leading planes - 16 bits each, their sum all but exact - and the smaller ones are summed apart, each from zero, and
// added to the running sum by ordinary additions.
template <int NA, int NB>
__device__ __forceinline__ void mma_planes(float (&c0)[4], float (&c1)[4], const uint32_t (&a)[NA][4], const uint32_t (&b)[NB][4]) {
    float h0[4] = {0.f, 0.f, 0.f, 0.f}, h1[4] = {0.f, 0.f, 0.f, 0.f};
    mma(h0, a[0], b[0][0], b[0][1]);
    mma(h1, a[0], b[0][2], b[0][3]);
    if constexpr (NA + NB > 2) {
        float l0[4] = {0.f, 0.f, 0.f, 0.f}, l1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int sum = 2; sum >= 1; --sum)
#pragma unroll
            for (int i = 0; i < NA; ++i) {
                const int j = sum - i;
                if (j >= 0 && j < NB) {
                    mma(l0, a[i], b[j][0], b[j][1]);
                    mma(l1, a[i], b[j][2], b[j][3]);
                }
            }
#pragma unroll
        for (int i = 0; i < 4; ++i) { h0[i] += l0[i]; h1[i] += l1[i]; }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) { c0[i] += h0[i]; c1[i] += h1[i]; }
}
// The same for one plane of A and three of B, closer still: the leading products eight at a time, and what rounding the running sum
// leaves kept beside it (two-sum), with the small planes; acc + left is the result.  The wkv chunk sums take it, whose walk rounds once a
// token: the state's error against 64 bits 4.6e-8 -> 3.9e-8 (the walk's 4.5e-8) for 4 us of 30, before the last tokens were summed apart.
__device__ __forceinline__ void mma8(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(b));
}
__device__ __forceinline__ void mma_planes_kept(float (&acc)[4], float (&left)[4], const uint32_t (&a)[4], const uint32_t (&b)[3][4], int side) {
    float l[4] = {0.f, 0.f, 0.f, 0.f};
    mma(l, a, b[2][2 * side], b[2][2 * side + 1]);
    mma(l, a, b[1][2 * side], b[1][2 * side + 1]);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        float h[4] = {0.f, 0.f, 0.f, 0.f};
        mma8(h, a[2 * half], a[2 * half + 1], b[0][2 * side + half]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float t = acc[i] + h[i], u = t - acc[i];
            left[i] += (acc[i] - (t - u)) + (h[i] - u);
            acc[i] = t;
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) left[i] += l[i];
}
// A key times the decays behind it.  Below 2^-102 a pair keeps what lies above 2^-149 and no more: beside keys under 2^10 the up to 64 roundings there
// stay below 2^-133, where the planes end as well.  Larger keys beside such decays make it NaN: such states and chunks are walked.
__device__ __forceinline__ Pair decayed_key(Pair f, float k) {
    const bool lost = fabsf(k) >= 0x1p10f && fabsf(f.hi) < 0x1p-100f;
    f *= k;
    if (lost) f.hi = __int_as_float(0x7fc00000);
    return f;
}
// two 32-bit operations in one instruction
#define F32X2(name, op, ...) \
    asm(op : "=l"(reinterpret_cast<unsigned long long&>(name)) : __VA_ARGS__)
#define F32X2_IN(x) "l"(reinterpret_cast<const unsigned long long&>(x))
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { float2 d; F32X2(d, "mul.rn.f32x2 %0, %1, %2;", F32X2_IN(a), F32X2_IN(b)); return d; }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { float2 d; F32X2(d, "add.rn.f32x2 %0, %1, %2;", F32X2_IN(a), F32X2_IN(b)); return d; }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    F32X2(d, "fma.rn.f32x2 %0, %1, %2, %3;", F32X2_IN(a), F32X2_IN(b), F32X2_IN(c));
    return d;
}
#undef F32X2
#undef F32X2_IN
template <bool TRANS>
__device__ __forceinline__ void ldsm(uint32_t (&r)[4], const uint16_t* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    if (TRANS) asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
    else asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
// B operand of 16 columns (two tiles) by 16 k: stored with a row per column (k along the row) ...
__device__ __forceinline__ const uint16_t* at_cols(const uint16_t* base, int ld, int n0, int k0, int lane) {
    return base + (n0 + (lane & 7) + (lane >> 4) * 8) * ld + k0 + ((lane >> 3) & 1) * 8;
}
// ... or with a row per k (columns along the row; loaded transposed)
__device__ __forceinline__ const uint16_t* at_rows(const uint16_t* base, int ld, int n0, int k0, int lane) {
    return base + (k0 + (lane & 7) + ((lane >> 3) & 1) * 8) * ld + n0 + (lane >> 4) * 8;
}
// A operand of 16 rows by 16 k, stored with a row per k (loaded transposed)
__device__ __forceinline__ const uint16_t* at_rows_a(const uint16_t* base, int ld, int m0, int k0, int lane) {
    return base + (k0 + (lane & 7) + (lane >> 4) * 8) * ld + m0 + ((lane >> 3) & 1) * 8;
}

// eight values into PL planes at element offset `at`, planes `step` elements apart (PL 1: the values are bfloat16 already)
template <int PL>
__device__ __forceinline__ void store_planes(uint16_t* base, int step, int at, const float (&x)[8]) {
    uint32_t p[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) split3(x[2 * i], x[2 * i + 1], p[0][i], p[1][i], p[2][i]);
#pragma unroll
    for (int l = 0; l < PL; ++l) *reinterpret_cast<uint4*>(base + l * step + at) = make_uint4(p[l][0], p[l][1], p[l][2], p[l][3]);
}

// 64 rows of COLS values into PL planes: row j's columns from src + j * ld, zero where in(j, column) is false, behind scale(j, values).  The
// loads of four pieces are on their way before the first is split.
template <int PL, int COLS, int LDS, int NT = 128, typename E, typename In, typename Scale>
__device__ __forceinline__ void stage_rows(uint16_t* dst, const E* src, long long ld, In in, Scale scale) {
    constexpr int PIECES = COLS / 8, ITERS = CT * PIECES / NT, BATCH = ITERS < 4 ? ITERS : 4;
    static_assert(ITERS > 0 && ITERS % BATCH == 0, "64 rows of a multiple of 64 values");
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
            store_planes<PL>(dst, CT * LDS, j * LDS + c, x[i]);
        }
    }
}

// rows t0 .. t0 + n - 1, columns col0 .. col0 + 63 of a head's values
template <typename VT, int VPL, int NT = 128>
__device__ __forceinline__ void stage_values(uint16_t* v_s, const VT* vp, long long ld, int n, int col0, int Dv) {
    stage_rows<VPL, VT_COLS, VLD, NT>(v_s, vp + col0, ld, [&](int j, int c) { return j < n && col0 + c < Dv; }, [](int, float (&)[8]) {});
}

// ------------------------------------------------------------------------------------------- chunk_sum
// wkv: the chunk's last tokens are added in 64 bits on the ordinary cores, behind the tensor cores' sum of the others.  Under strong decays
// they are the state, and what the tensor cores cut from products of very different sizes showed there: decays of e^-1 to e^-20 a token
// 3.9e-8 without this, 2.0e-8 with it and walked; e^-0.0003 to e^-150 3.5e-8, 2.2e-8, walked 3.2e-8.  4 us of the mixer's 240 (2,048 tokens).
constexpr int TAIL = 8;
template <int MODE, int KP> struct SumSmem {
    static constexpr int LD = KP + 8;
    static constexpr int NT = MODE == WKV ? 256 : 128;               // wkv: a thread per channel and run of tokens, so more of them
    static size_t bytes(int vpl) { return (size_t)(3 * CT * LD + vpl * CT * VLD) * 2 + 64 + (MODE == WKV ? (NT + TAIL * (KP + VT_COLS)) * 8 : CT * 4); }
};

template <int MODE, int KP, typename VT>
__global__ void __launch_bounds__(SumSmem<MODE, KP>::NT, MODE == WKV && KP == 64 ? 3 : 0) chunk_sum_kernel(const ChunkArgs a) {
    constexpr int NT = SumSmem<MODE, KP>::NT, PARTS = NT / 128, LD = KP + 8, VPL = sizeof(VT) == 4 ? 3 : 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint16_t* kd = reinterpret_cast<uint16_t*>(smem_raw);                             // [3][CT][LD]: decayed keys
    uint16_t* v_s = kd + 3 * CT * LD;                                                 // [VPL][CT][VLD]
    double* half = reinterpret_cast<double*>(v_s + VPL * CT * VLD);                   // [8]
    float* wt = reinterpret_cast<float*>(half + 8);                                   // [CT]: a token's weight at the chunk's end
    double* k_tail = half + 8 + NT;                                                   // wkv: [TAIL][KP] decayed keys of the last tokens (oldest first)
    double* v_tail = k_tail + TAIL * KP;                                              // wkv: [TAIL][VT_COLS] their values
    TTIE_PDL_ENTRY();
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = (tid >> 5) & 3, part = tid >> 7;      // (part: which share of the key channels)
    int s, c, t0, n;
    if (!find_chunk<CT>(a.qsl, a.num_seqs, a.slot_lo + blockIdx.x, s, c, t0, n)) return;
    const size_t unit = (size_t)blockIdx.x * a.H + h;
    const VT* vp = reinterpret_cast<const VT*>(a.v) + (size_t)t0 * a.ld_v + h * a.Dv;
    auto stage_tail = [&]() {
        for (int e = tid; e < TAIL * VT_COLS; e += NT) {
            const int j = n - TAIL + e / VT_COLS;                                     // (the staged values; columns past the last are zeros)
            v_tail[e] = j >= 0 ? (double)__uint_as_float((uint32_t)v_s[j * VLD + e % VT_COLS] << 16) : 0.0;
        }
    };

    if constexpr (MODE == WKV) {
        // a thread per channel and run of LEN tokens: the decays of the run, its product, then keys times the decays behind them (products
        // of up to 64 decays as pairs: in 32 bits they leave more than the walk's one rounding per token)
        constexpr int LEN = CT * KP / NT, RUNS = CT / LEN;
        Pair* tot = reinterpret_cast<Pair*>(half);                                    // [RUNS][KP]: product over a run (over wt, which is not used here)
        const int ch = tid % KP, run = tid / KP;
        const bool in = ch < a.D;
        const float* wp = a.decay + (size_t)t0 * a.H * a.D + h * a.D;
        const __nv_bfloat16* kp = reinterpret_cast<const __nv_bfloat16*>(a.k) + (size_t)t0 * a.ld_qk + h * a.D;
        // decays, keys and values are all asked for at once, 16 bytes a copy; decays and keys wait where the planes will lie
        float* w_raw = reinterpret_cast<float*>(kd);
        uint16_t* k_raw = kd + 2 * CT * LD;
        const bool wide = ((uintptr_t)a.decay & 15) == 0;
        for (int e = tid; e < CT * (KP / 4); e += NT) {
            const int j = e / (KP / 4), c4 = e % (KP / 4) * 4;
            float* dst = w_raw + j * KP + c4;
            const float* src = wp + (size_t)j * a.H * a.D + c4;
            if (j >= n || c4 >= a.D) *reinterpret_cast<float4*>(dst) = make_float4(1.f, 1.f, 1.f, 1.f);
            else if (wide) copy16(dst, src);
            else *reinterpret_cast<float4*>(dst) = make_float4(src[0], src[1], src[2], src[3]);
        }
        for (int e = tid; e < CT * (KP / 8); e += NT) {
            const int j = e / (KP / 8), c8 = e % (KP / 8) * 8;
            if (j < n && c8 < a.D) copy16(k_raw + j * LD + c8, kp + (size_t)j * a.ld_qk + c8);
            else *reinterpret_cast<uint4*>(k_raw + j * LD + c8) = make_uint4(0u, 0u, 0u, 0u);
        }
        for (int e = tid; e < CT * (VT_COLS / 8); e += NT) {
            const int j = e / (VT_COLS / 8), c8 = e % (VT_COLS / 8) * 8;
            if (j < n && c8 < a.Dv) copy16(v_s + j * VLD + c8, vp + (size_t)j * a.ld_v + c8);
            else *reinterpret_cast<uint4*>(v_s + j * VLD + c8) = make_uint4(0u, 0u, 0u, 0u);
        }
        for (int e = tid; e < (TAIL - n) * KP; e += NT) k_tail[e] = 0.0;              // (fewer tokens than that)
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        float w[LEN];
        uint16_t kv[LEN];
#pragma unroll
        for (int i = 0; i < LEN; ++i) {
            w[i] = w_raw[(run * LEN + i) * KP + ch];
            kv[i] = k_raw[(run * LEN + i) * LD + ch];
        }
        stage_tail();
        // (over runs and the chunk the products are held times 2^64: the state's factor, a pair of 32-bit numbers in memory too, keeps all that these hold)
        Pair all = {0x1p64f, 0.f};
#pragma unroll
        for (int i = LEN - 1; i >= 0; --i) all *= w[i];
        tot[run * KP + ch] = all.times(0x1p-32f);
        __syncthreads();
        Pair suf = {0x1p64f, 0.f};
#pragma unroll
        for (int i = RUNS - 1; i > 0; --i)
            if (i > run) { suf = suf.times(0x1p-32f); suf *= tot[i * KP + ch]; }
        if (run == 0 && ch < a.Dpad) {
            suf = suf.times(0x1p-32f);
            all = all.times(0x1p-32f);
            all *= suf;
            const float f = all.value();
            a.aux[2 * unit * a.Dpad + ch] = in ? f * 0x1p-64f : 1.f;
            a.aux[(2 * unit + 1) * a.Dpad + ch] = in ? ((all.hi - f) + all.lo) * 0x1p-64f : 0.f;
            suf = suf.times(0x1p-32f);
        } else suf = suf.times(0x1p-64f);
#pragma unroll
        for (int i = LEN - 1; i >= 0; --i) {
            const int j = run * LEN + i;
            Pair x = decayed_key(suf, __uint_as_float((uint32_t)kv[i] << 16));
            const bool last = j >= n - TAIL && j < n;
            if (last) { k_tail[(j - (n - TAIL)) * KP + ch] = (double)x.hi + (double)x.lo; x = {0.f, 0.f}; }
            split3(x, kd[j * LD + ch], kd[CT * LD + j * LD + ch], kd[2 * CT * LD + j * LD + ch]);
            suf *= w[i];
        }
    } else {
        stage_values<VT, VPL, NT>(v_s, vp, a.ld_v, n, 0, a.Dv);
        if constexpr (MODE == RET) {
            if (tid < CT) wt[tid] = tid < n ? (float)power((double)a.decay[h], n - 1 - tid) : 0.f;
        } else {
            double F, x, X;
            chunk_gates<CT>(a, t0, n, h, half, F, x, X);
            if (tid < CT) wt[tid] = expf((float)(x - half[5]));
            if (tid == 0) a.span[unit] = make_double2(half[4], half[5]);
        }
        __syncthreads();
        using KT = typename std::conditional<MODE == RET, float, __nv_bfloat16>::type;
        const KT* kp = reinterpret_cast<const KT*>(a.k) + (size_t)t0 * a.ld_qk + h * a.D;
        stage_rows<3, KP, LD, NT>(kd, kp, a.ld_qk, [&](int j, int ch) { return j < n && ch < a.D; }, [&](int j, float (&x)[8]) {
            const float w = wt[j];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = j < n ? x[i] * w : 0.f;
        });
    }
    __syncthreads();
    if (MODE == MLSTM && tid < a.Dpad) {                                              // the normaliser's sum: the same without the values
        float sum = 0.f;
        for (int j = 0; j < CT; ++j)
            sum += __uint_as_float((uint32_t)kd[j * LD + tid] << 16) + (__uint_as_float((uint32_t)kd[CT * LD + j * LD + tid] << 16) + __uint_as_float((uint32_t)kd[2 * CT * LD + j * LD + tid] << 16));
        a.aux[unit * a.Dpad + tid] = sum;
    }
    const int g = lane >> 2, t = lane & 3;
    for (int col0 = 0; col0 < a.Dv; col0 += VT_COLS) {
        if (col0 > 0) {
            __syncthreads();
            stage_values<VT, VPL, NT>(v_s, vp, a.ld_v, n, col0, a.Dv);
            if constexpr (MODE == WKV) { __syncthreads(); stage_tail(); }
            __syncthreads();
        }
        constexpr int NP = KP / 16 / PARTS;                                           // 16-channel tiles of this warp
        float acc[2 * NP][4];
#pragma unroll
        for (int i = 0; i < 2 * NP; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
        float left[MODE == WKV ? 2 * NP : 1][4] = {};
#pragma unroll
        for (int k0 = 0; k0 < CT; k0 += 16) {
            uint32_t av[VPL][4];
#pragma unroll
            for (int l = 0; l < VPL; ++l) ldsm<true>(av[l], at_rows_a(v_s + l * CT * VLD, VLD, warp * 16, k0, lane));
#pragma unroll
            for (int np = 0; np < NP; ++np) {
                uint32_t b[3][4];
#pragma unroll
                for (int l = 0; l < 3; ++l) ldsm<true>(b[l], at_rows(kd + l * CT * LD, LD, (part * NP + np) * 16, k0, lane));
                if constexpr (MODE == WKV) {
                    mma_planes_kept(acc[2 * np], left[2 * np], av[0], b, 0);
                    mma_planes_kept(acc[2 * np + 1], left[2 * np + 1], av[0], b, 1);
                } else {
                    mma_planes<VPL, 3>(acc[2 * np], acc[2 * np + 1], av, b);
                }
            }
        }
        if constexpr (MODE == WKV) {
#pragma unroll
            for (int i = 0; i < 2 * NP; ++i) {
                double sum[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) sum[j] = (double)acc[i][j] + (double)left[i][j];
                const double* kt = k_tail + (part * NP * 2 + i) * 8 + 2 * t;
                const double* vt = v_tail + warp * 16 + g;
#pragma unroll
                for (int r = 0; r < TAIL; ++r) {
                    const double2 k = *reinterpret_cast<const double2*>(kt + r * KP);
                    const double v0 = vt[r * VT_COLS], v1 = vt[r * VT_COLS + 8];
                    sum[0] = fma(v0, k.x, sum[0]); sum[1] = fma(v0, k.y, sum[1]);
                    sum[2] = fma(v1, k.x, sum[2]); sum[3] = fma(v1, k.y, sum[3]);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = (float)sum[j];
            }
        }
        float* dst = a.part + (unit * a.Dv + col0 + warp * 16) * a.Dpad;
#pragma unroll
        for (int i = 0; i < 2 * NP; ++i) {
            const int ch = part * NP * 16 + i * 8 + 2 * t;
            if (ch < a.Dpad) {
                if (col0 + warp * 16 + g < a.Dv) *reinterpret_cast<float2*>(dst + (size_t)g * a.Dpad + ch) = make_float2(acc[i][0], acc[i][1]);
                if (col0 + warp * 16 + g + 8 < a.Dv) *reinterpret_cast<float2*>(dst + (size_t)(g + 8) * a.Dpad + ch) = make_float2(acc[i][2], acc[i][3]);
            }
        }
    }
}

// ------------------------------------------------------------------------------------------- chunk_out
template <int MODE, int KP> struct OutSmem {
    static constexpr int LD = KP + 8, FLD = KP + 4;
    static constexpr bool SHARED = MODE == WKV && KP == 64;          // wkv: one table takes first the decays, then the rows' products of them
    static constexpr int EXTRA = MODE == WKV ? ((SHARED ? 1 : 2) * CT * FLD + 4 * KP) * 4 : MODE == MLSTM ? CT * 24 + KP * 4 : (CT + 1 + 3) * 4;
    static size_t bytes(int vpl) { return (size_t)(3 * CT * LD + vpl * CT * VLD) * 2 + 64 + EXTRA; }
};

template <int MODE, int KP, typename VT, int CTAS = MODE == WKV && KP == 128 ? 1 : sizeof(VT) == 4 ? 2 : 3>
__global__ void __launch_bounds__(128, CTAS) chunk_out_kernel(const ChunkArgs a) {
    constexpr int LD = KP + 8, FLD = KP + 4, VPL = sizeof(VT) == 4 ? 3 : 1;
    constexpr int QPL = MODE == MLSTM ? 1 : 3, KPL = MODE == MLSTM ? 1 : 3, KS = KP / 16;
    constexpr bool GATES = OutSmem<MODE, KP>::SHARED;                // (the gate's rows take the place of the table, one tile of columns)
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint16_t* pl = reinterpret_cast<uint16_t*>(smem_raw);                             // [3][CT][LD]: keys, then 64 columns of the state
    uint16_t* v_s = pl + 3 * CT * LD;                                                 // [VPL][CT][VLD]
    double* half = reinterpret_cast<double*>(v_s + VPL * CT * VLD);                   // [8]
    unsigned char* extra = reinterpret_cast<unsigned char*>(half + 8);
    TTIE_PDL_ENTRY();
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    int s, c, t0, n;
    if (!find_chunk<CT>(a.qsl, a.num_seqs, a.slot_lo + blockIdx.x, s, c, t0, n)) return;
    const size_t unit = (size_t)blockIdx.x * a.H + h;
    using QT = typename std::conditional<MODE == RET, float, __nv_bfloat16>::type;
    const QT* qp = reinterpret_cast<const QT*>(a.q) + (size_t)t0 * a.ld_qk + h * a.D;
    const QT* kp = reinterpret_cast<const QT*>(a.k) + (size_t)t0 * a.ld_qk + h * a.D;
    const VT* vp = reinterpret_cast<const VT*>(a.v) + (size_t)t0 * a.ld_v + h * a.Dv;
    const int r0 = warp * 16 + g, r1 = r0 + 8;                                        // this lane's rows (tokens of the chunk)
    bool odd = false;                                                                 // something of this lane's is not finite
    if (MODE != WKV) stage_values<VT, VPL>(v_s, vp, a.ld_v, n, 0, a.Dv);

    // a lane's part of a 16 x 16 piece of the query rows: rows r0 / r1, channels c0 + 2t, + 1 and those + 8
    auto load_q = [&](int c0, float (&f)[8]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = i & 1 ? r1 : r0, ch = c0 + 2 * t + (i & 2 ? 8 : 0);
            const bool in = r < n && ch < a.D;
            if constexpr (MODE == RET) {
                const float2 x = in ? *reinterpret_cast<const float2*>(qp + (size_t)r * a.ld_qk + ch) : make_float2(0.f, 0.f);
                f[2 * i] = x.x; f[2 * i + 1] = x.y;
            } else {
                const float2 x = unpack(in ? *reinterpret_cast<const uint32_t*>(qp + (size_t)r * a.ld_qk + ch) : 0u);
                f[2 * i] = x.x; f[2 * i + 1] = x.y;
            }
        }
    };
    auto planes_of = [&](const float (&f)[8], uint32_t (&q)[QPL][4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t p0, p1, p2;
            split3(f[2 * i], f[2 * i + 1], p0, p1, p2);
            q[0][i] = p0;
            if constexpr (QPL == 3) { q[1][i] = p1; q[2][i] = p2; }
        }
    };

    float P[8][4];                                                                    // scores, then weights: rows r0, r0, r1, r1; columns 8 i + 2t, + 1
#pragma unroll
    for (int i = 0; i < 8; ++i) P[i][0] = P[i][1] = P[i][2] = P[i][3] = 0.f;
    float rq[MODE == WKV ? KS : 1][8];                                                // wkv: the rows with their decays from the chunk's start
    float row_in[2], den[2] = {0.f, 0.f}, floor_[2] = {0.f, 0.f};                     // factor of the state before the chunk; mlstm: denominator, e^-m

    if constexpr (MODE == WKV) {
        float* ws = reinterpret_cast<float*>(extra);                                  // [CT][FLD] decays
        constexpr bool SHARED = OutSmem<MODE, KP>::SHARED;
        float* pre = SHARED ? ws : ws + CT * FLD;                                     // [CT][FLD] product of the block's decays before the token
        float* blk = pre + CT * FLD;                                                  // [4][KP] product over a block
        // decays, keys and query rows are all asked for at once, 16 bytes a copy; the keys wait where their last plane will lie, the query rows (64
        // channels of them) where the values will
        uint16_t* k_raw = pl + 2 * CT * LD;
        const float* wp = a.decay + (size_t)t0 * a.H * a.D + h * a.D;
        const bool wide = ((uintptr_t)a.decay & 15) == 0;
        for (int e = tid; e < CT * (KP / 4); e += 128) {
            const int j = e / (KP / 4), ch = e % (KP / 4) * 4;
            float* dst = ws + j * FLD + ch;
            const float* src = wp + (size_t)j * a.H * a.D + ch;
            if (j >= n || ch >= a.D) *reinterpret_cast<float4*>(dst) = make_float4(1.f, 1.f, 1.f, 1.f);
            else if (wide) copy16(dst, src);
            else *reinterpret_cast<float4*>(dst) = make_float4(src[0], src[1], src[2], src[3]);
        }
        for (int e = tid; e < CT * (KP / 8); e += 128) {
            const int j = e / (KP / 8), ch = e % (KP / 8) * 8;
            const bool in = j < n && ch < a.D;
            uint16_t* dst = k_raw + j * LD + ch;
            if (in) copy16(dst, kp + (size_t)j * a.ld_qk + ch);
            else *reinterpret_cast<uint4*>(dst) = make_uint4(0u, 0u, 0u, 0u);
            if (ch >= 64) continue;
            if (in) copy16(v_s + j * VLD + ch, qp + (size_t)j * a.ld_qk + ch);
            else *reinterpret_cast<uint4*>(v_s + j * VLD + ch) = make_uint4(0u, 0u, 0u, 0u);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        constexpr int ITEMS = 4 * KP / 128;                                           // (block, channel) pairs of a thread
        uint16_t k[ITEMS][16];
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
            const int e = it * 128 + tid, J = e / KP, ch = e % KP;
#pragma unroll
            for (int i = 0; i < 16; ++i) k[it][i] = k_raw[(J * 16 + i) * LD + ch];
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
            const int e = it * 128 + tid, J = e / KP, ch = e % KP;
            const float* w = ws + J * 16 * FLD + ch;
            Pair f = {1.f, 0.f};                                                      // (as in chunk_sum)
            if (!SHARED) {
#pragma unroll
                for (int i = 0; i < 16; ++i) { pre[(J * 16 + i) * FLD + ch] = f.value(); f *= w[i * FLD]; }
                blk[J * KP + ch] = f.value();
                f = {1.f, 0.f};
            }
#pragma unroll
            for (int i = 15; i >= 0; --i) {
                const int at = (J * 16 + i) * LD + ch;
                split3(decayed_key(f, __uint_as_float((uint32_t)k[it][i] << 16)), pl[at], pl[CT * LD + at], pl[2 * CT * LD + at]);
                f *= w[i * FLD];
            }
        }
        auto row_products = [&]() {                                                   // of decays before a token within its block, and over whole blocks
#pragma unroll
            for (int it = 0; it < ITEMS; ++it) {
                const int e = it * 128 + tid, J = e / KP, ch = e % KP;
                Pair f = {1.f, 0.f};
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int at = (J * 16 + i) * FLD + ch;
                    const float w = ws[at];
                    pre[at] = f.value();
                    f *= w;
                }
                blk[J * KP + ch] = f.value();
            }
        };
        __syncthreads();
        // inside the block: a lane owns a key j and 32 channels, the rows come one after the other; the key's running product moves on with each
        // row behind it.  The 32 terms of a score are added as pairs, then in a tree (as when lanes owned channels and 16 sums at a time
        // went through shuffles; those were two thirds of the scores' instructions, 16,600 clocks of a CTA's 46,600).  The scores of key j take
        // the place of query row j, which nothing reads from row j + 1 on (more than 64 channels: of the row of decays).
        const float* dw = ws + warp * 16 * FLD;
        uint16_t* rows = v_s + warp * 16 * VLD;
        constexpr int GLD = SHARED ? VLD / 2 : FLD;
        float* dg = SHARED ? reinterpret_cast<float*>(rows) : ws + warp * 16 * FLD;
        const int jl = lane & 15, side = (lane >> 4) * 32;
        for (int ch0 = 0; ch0 < KP; ch0 += 64) {
            if (ch0 > 0) {
                __syncwarp();                                                         // (the last channels' rows have been read)
#pragma unroll
                for (int e = lane; e < 16 * 8; e += 32) {
                    const int i = e >> 3, c = (e & 7) * 8;
                    const bool in = warp * 16 + i < n && ch0 + c < a.D;
                    *reinterpret_cast<uint4*>(rows + i * VLD + c) =
                        in ? *reinterpret_cast<const uint4*>(qp + (size_t)(warp * 16 + i) * a.ld_qk + ch0 + c) : make_uint4(0u, 0u, 0u, 0u);
                }
            }
            float2 p[16];                                                             // the key's channels side + 2 m, + 1, times the decays up to the row
#pragma unroll
            for (int m = 0; m < 16; m += 4) {
                const int c = ch0 + side + 2 * m;
                const bool in = warp * 16 + jl < n && c < a.D;
                const uint4 x = in ? *reinterpret_cast<const uint4*>(kp + (size_t)(warp * 16 + jl) * a.ld_qk + c) : make_uint4(0u, 0u, 0u, 0u);
                p[m] = unpack(x.x); p[m + 1] = unpack(x.y); p[m + 2] = unpack(x.z); p[m + 3] = unpack(x.w);
            }
            __syncwarp();
            // sum over this lane's channels of row i (its pieces at `row`) times `x`, as a tree
            auto dot = [&](const uint16_t* row, auto x) {
                float2 t[8];
#pragma unroll
                for (int m = 0; m < 8; ++m) {
                    const uint2 r = *reinterpret_cast<const uint2*>(row + side + 4 * m);
                    t[m] = fma2(unpack(r.y), x(2 * m + 1), mul2(unpack(r.x), x(2 * m)));
                }
#pragma unroll
                for (int d = 1; d < 8; d *= 2)
#pragma unroll
                    for (int m = 0; m < 8; m += 2 * d) t[m] = add2(t[m], t[m + d]);
                const float sum = t[0].x + t[0].y;
                return sum + __shfl_xor_sync(0xffffffffu, sum, 16);
            };
            const float* up = a.u + h * a.D + ch0 + side;
            const float own = dot(rows + jl * VLD, [&](int m) {
                const bool in = ch0 + side + 2 * m < a.D;                             // (a multiple of 8)
                return mul2(p[m], in ? make_float2(up[2 * m], up[2 * m + 1]) : make_float2(0.f, 0.f));
            });
#pragma unroll 1
            for (int i = 1; i < 16; ++i) {
                const float sum = dot(rows + i * VLD, [&](int m) { return p[m]; });
                if (i > jl) {
                    const float4* w = reinterpret_cast<const float4*>(dw + i * FLD + ch0 + side);
#pragma unroll
                    for (int m = 0; m < 8; ++m) {
                        const float4 x = w[m];
                        p[2 * m] = mul2(p[2 * m], make_float2(x.x, x.y));
                        p[2 * m + 1] = mul2(p[2 * m + 1], make_float2(x.z, x.w));
                    }
                }
                __syncwarp();
                if (i > jl && lane < 16) { float* o = dg + jl * GLD + i; *o = ch0 == 0 ? sum : *o + sum; }
            }
            __syncwarp();
            if (lane < 16) { float* o = dg + jl * GLD + jl; *o = ch0 == 0 ? own : *o + own; }
        }
        if (SHARED) {
            __syncthreads();                                                          // (every warp's decays have been read)
            row_products();
            __syncthreads();
        } else __syncwarp();
        // between blocks: rows times the decays from their block's start, then times whole blocks going back
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            load_q(ks * 16, rq[ks]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = (i >> 1) & 1 ? r1 : r0, ch = ks * 16 + 2 * t + (i & 4 ? 8 : 0) + (i & 1);
                rq[ks][i] *= pre[r * FLD + ch];
            }
        }
#pragma unroll
        for (int J = 2; J >= 0; --J) {
            if (J >= warp) continue;
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) {
                uint32_t q[QPL][4], b[3][4];
                planes_of(rq[ks], q);
#pragma unroll
                for (int l = 0; l < 3; ++l) ldsm<false>(b[l], at_cols(pl + l * CT * LD, LD, J * 16, ks * 16, lane));
                mma_planes<3, 3>(P[2 * J], P[2 * J + 1], q, b);
#pragma unroll
                for (int i = 0; i < 8; ++i) rq[ks][i] *= blk[J * KP + ks * 16 + 2 * t + (i & 4 ? 8 : 0) + (i & 1)];
            }
        }
#pragma unroll
        for (int J = 0; J < 4; ++J)
            if (J == warp)
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        const int r = g + (b & 2 ? 8 : 0), col = i * 8 + 2 * t + (b & 1);
                        P[2 * J + i][b] = col <= r ? dg[col * GLD + r] : 0.f;
                    }
        if (SHARED) {                                                                 // the rows wait in their own places of the table
            __syncwarp();
#pragma unroll
            for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    const int r = (i >> 1) & 1 ? r1 : r0, ch = ks * 16 + 2 * t + (i & 4 ? 8 : 0);
                    *reinterpret_cast<float2*>(pre + r * FLD + ch) = make_float2(rq[ks][i], rq[ks][i + 1]);
                }
        }
        row_in[0] = row_in[1] = 1.f;
    } else {
        stage_rows<KPL, KP, LD>(pl, kp, a.ld_qk, [&](int j, int ch) { return j < n && ch < a.D; }, [](int, float (&)[8]) {});
        float* pw = reinterpret_cast<float*>(extra);                                  // retention: powers 0 .. CT of the decay
        double* xs = reinterpret_cast<double*>(extra);                                // mlstm: x, M and F of every token; the normaliser before the chunk
        double* Ms = xs + CT;
        double* Fs = Ms + CT;
        float* nb = reinterpret_cast<float*>(Fs + CT);
        if constexpr (MODE == RET) {
            if (tid <= CT) pw[tid] = (float)power((double)a.decay[h], tid);
            __syncthreads();
        } else {
            double F, x, X;
            chunk_gates<CT>(a, t0, n, h, half, F, x, X);
            const float2 mm = a.mm[unit];
            const double m = (double)mm.x;
            if (tid < CT) { xs[tid] = x; Ms[tid] = fmax(m, X); Fs[tid] = F; }
            if (tid < KP) nb[tid] = tid < a.Dpad ? a.aux[unit * a.Dpad + tid] : 0.f;
            // (a chunk is the request's last of this pass if the next chunk is not there or not in the pass)
            if (tid == 0 && ((c + 1) * CT >= a.qsl[s + 1] - a.qsl[s] || (int)blockIdx.x + 1 == a.slots))
                a.mx[(size_t)state_row(a.slot_ids[s], a.state_rows) * a.H + h] = mm.y;
            __syncthreads();
            row_in[0] = expf((float)(m - Ms[r0])); row_in[1] = expf((float)(m - Ms[r1]));
            floor_[0] = expf((float)-(Fs[r0] + Ms[r0])); floor_[1] = expf((float)-(Fs[r1] + Ms[r1]));
        }
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            float f[8];
            uint32_t q[QPL][4];
            load_q(ks * 16, f);
            planes_of(f, q);
            if constexpr (MODE == MLSTM) {                                            // q . n before the chunk
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float x = f[i] * nb[ks * 16 + 2 * t + (i & 4 ? 8 : 0) + (i & 1)];
                    if ((i >> 1) & 1) den[1] += x; else den[0] += x;
                }
            }
#pragma unroll
            for (int J = 0; J < 4; ++J) {
                if (J > warp) continue;                                               // keys behind all of the warp's rows
                uint32_t b[KPL][4];
#pragma unroll
                for (int l = 0; l < KPL; ++l) ldsm<false>(b[l], at_cols(pl + l * CT * LD, LD, J * 16, ks * 16, lane));
                mma_planes<QPL, KPL>(P[2 * J], P[2 * J + 1], q, b);
            }
        }
        if constexpr (MODE == RET) {
            row_in[0] = pw[r0 + 1]; row_in[1] = pw[r1 + 1];
        } else {
            den[0] *= row_in[0]; den[1] *= row_in[1];
        }
        const double M0 = MODE == MLSTM ? Ms[r0] : 0.0, M1 = MODE == MLSTM ? Ms[r1] : 0.0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int r = b & 2 ? r1 : r0, j = i * 8 + 2 * t + (b & 1);
                float w = 0.f;
                if (j <= r) {
                    if constexpr (MODE == RET) w = P[i][b] * pw[r - j];
                    else { w = P[i][b] * expf((float)(xs[j] - (b & 2 ? M1 : M0))); den[b >> 1] += w; }
                }
                P[i][b] = w;
            }
        if constexpr (MODE == MLSTM) {
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                den[b] += __shfl_xor_sync(0xffffffffu, den[b], 1);
                den[b] += __shfl_xor_sync(0xffffffffu, den[b], 2);
                odd = odd || ((b ? r1 : r0) < n && !isfinite(den[b]));
                den[b] = fmaxf(fabsf(den[b] * a.qscale), floor_[b]) + 1e-6f;
            }
        }
    }

    for (int col0 = 0; col0 < a.Dv; col0 += VT_COLS) {
        __syncthreads();                                                              // the keys (or the last columns) have been read by everyone
        if (col0 > 0 || MODE == WKV) stage_values<VT, VPL>(v_s, vp, a.ld_v, n, col0, a.Dv);
        const float* sp = a.part + (unit * a.Dv + col0) * a.Dpad;
        stage_rows<3, KP, LD>(pl, sp, a.Dpad, [&](int j, int ch) { return col0 + j < a.Dv && ch < a.Dpad; }, [](int, float (&)[8]) {});
        __syncthreads();
        float acc[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            uint32_t q[QPL][4];
            if constexpr (MODE == WKV && OutSmem<MODE, KP>::SHARED) {
                const float* pre = reinterpret_cast<const float*>(extra);
                float f[8];
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    const int r = (i >> 1) & 1 ? r1 : r0, ch = ks * 16 + 2 * t + (i & 4 ? 8 : 0);
                    const float2 x = *reinterpret_cast<const float2*>(pre + r * FLD + ch);
                    f[i] = x.x; f[i + 1] = x.y;
                }
                planes_of(f, q);
            } else if constexpr (MODE == WKV) planes_of(rq[ks], q);
            else { float f[8]; load_q(ks * 16, f); planes_of(f, q); }
#pragma unroll
            for (int np = 0; np < 4; ++np) {
                uint32_t b[3][4];
#pragma unroll
                for (int l = 0; l < 3; ++l) ldsm<false>(b[l], at_cols(pl + l * CT * LD, LD, np * 16, ks * 16, lane));
                mma_planes<QPL, 3>(acc[2 * np], acc[2 * np + 1], q, b);
            }
        }
        if (GATES && a.y) {                                                           // the warp's rows of the table have been read: the gate's, while the values are multiplied
            __syncwarp();
            const __nv_bfloat16* gp = a.gate + (size_t)t0 * a.ld_gate + h * a.Dv;
#pragma unroll
            for (int e = lane; e < 16 * VT_COLS / 8; e += 32) {
                const int r = warp * 16 + e / 8, piece = e % 8;
                if (r < n && piece * 8 < a.Dv) copy16(reinterpret_cast<float*>(extra) + r * FLD + piece * 4, gp + (size_t)r * a.ld_gate + piece * 8);
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            acc[i][0] *= row_in[0]; acc[i][1] *= row_in[0]; acc[i][2] *= row_in[1]; acc[i][3] *= row_in[1];
        }
#pragma unroll
        for (int J = 0; J < 4; ++J) {
            if (J > warp) continue;
            uint32_t p[3][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) split3(P[2 * J + (i >> 1)][(i & 1) * 2], P[2 * J + (i >> 1)][(i & 1) * 2 + 1], p[0][i], p[1][i], p[2][i]);
#pragma unroll
            for (int np = 0; np < 4; ++np) {
                uint32_t b[VPL][4];
#pragma unroll
                for (int l = 0; l < VPL; ++l) ldsm<true>(b[l], at_rows(v_s + l * CT * VLD, VLD, np * 16, J * 16, lane));
                mma_planes<3, VPL>(acc[2 * np], acc[2 * np + 1], p, b);
            }
        }
        const size_t ld_o = (size_t)a.H * a.Dv;
        float* op = a.out + (size_t)t0 * ld_o + h * a.Dv + col0;
        // Gated where the gate's row lies, then out in whole rows.  With the products over, a row's 64 values are in four lanes: no tile is needed.
        // 101 -> 97 us of a scan of 2,048 tokens and 32 heads (the pass apart: 8).
        if (GATES && a.y) {
            float s0 = 0.f, s1 = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                s0 = fmaf(acc[i][0], acc[i][0], fmaf(acc[i][1], acc[i][1], s0));
                s1 = fmaf(acc[i][2], acc[i][2], fmaf(acc[i][3], acc[i][3], s1));
                odd = odd || (r0 < n && !finite4(acc[i][0], acc[i][1], 0.f, 0.f)) || (r1 < n && !finite4(acc[i][2], acc[i][3], 0.f, 0.f));
            }
#pragma unroll
            for (int k = 1; k < 4; k <<= 1) { s0 += __shfl_xor_sync(0xffffffffu, s0, k); s1 += __shfl_xor_sync(0xffffffffu, s1, k); }
            s0 = inverse_rms(a, s0); s1 = inverse_rms(a, s1);
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();
            uint32_t* gate = reinterpret_cast<uint32_t*>(extra);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int col = i * 8 + 2 * t;
                if (col >= a.Dv) continue;
                const float2 w = a.norm_w ? *reinterpret_cast<const float2*>(a.norm_w + h * a.Dv + col) : make_float2(1.f, 1.f);
                uint32_t* g0 = gate + r0 * FLD + i * 4 + t;
                uint32_t* g1 = gate + r1 * FLD + i * 4 + t;
                *g0 = gated_pair(a, acc[i][0] * s0, acc[i][1] * s0, w, *g0);
                *g1 = gated_pair(a, acc[i][2] * s1, acc[i][3] * s1, w, *g1);
            }
            __syncwarp();
#pragma unroll
            for (int e = lane; e < 16 * VT_COLS / 8; e += 32) {
                const int r = warp * 16 + e / 8, piece = e % 8;
                if (r < n && piece * 8 < a.Dv)
                    *reinterpret_cast<uint4*>(a.y + (size_t)(t0 + r) * ld_o + h * a.Dv + piece * 8) = *reinterpret_cast<const uint4*>(gate + r * FLD + piece * 4);
            }
            continue;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int col = i * 8 + 2 * t;
            if (col0 + col >= a.Dv) continue;
            float y[4] = {acc[i][0], acc[i][1], acc[i][2], acc[i][3]};
            if constexpr (MODE == MLSTM) {
                y[0] = y[0] * a.qscale / den[0]; y[1] = y[1] * a.qscale / den[0]; y[2] = y[2] * a.qscale / den[1]; y[3] = y[3] * a.qscale / den[1];
            }
            if (r0 < n) *reinterpret_cast<float2*>(op + (size_t)r0 * ld_o + col) = make_float2(y[0], y[1]);
            if (r1 < n) *reinterpret_cast<float2*>(op + (size_t)r1 * ld_o + col) = make_float2(y[2], y[3]);
            odd = odd || (r0 < n && !finite4(y[0], y[1], 0.f, 0.f)) || (r1 < n && !finite4(y[2], y[3], 0.f, 0.f));
        }
    }
    if (__syncthreads_or(odd)) {
        walk_out<MODE, CT, VT>(a, unit, t0, n, h, reinterpret_cast<float*>(pl));
        if (GATES && a.y) gate_walked(a, t0, n, h);
    }
}

template <int MODE, int KP, typename VT>
int launch_chunks(ChunkArgs a, int first, int slots, cudaStream_t st) {
    constexpr int VPL = sizeof(VT) == 4 ? 3 : 1;
    constexpr bool MANY = OutSmem<MODE, KP>::SHARED;
    const size_t sum_smem = SumSmem<MODE, KP>::bytes(VPL), out_smem = OutSmem<MODE, KP>::bytes(VPL);
    static bool allowed[64] = {false};
    int dev = 64;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64 || !allowed[dev]) {
        cudaFuncSetAttribute(chunk_sum_kernel<MODE, KP, VT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sum_smem);
        cudaFuncSetAttribute(chunk_out_kernel<MODE, KP, VT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)out_smem);
        if constexpr (MANY) cudaFuncSetAttribute(chunk_out_kernel<MODE, KP, VT, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)out_smem);
        if (dev < 64) allowed[dev] = true;
    }
    a.slot_lo = first; a.slots = slots;
    const dim3 grid(slots, a.H);
    const dim3 carry(ceil_div(a.Dv * a.Dpad + (MODE == MLSTM ? a.Dpad : 0), 4 * CARRY), a.H, a.num_seqs);
    TTIE_LAUNCH((chunk_sum_kernel<MODE, KP, VT>), grid, (SumSmem<MODE, KP>::NT), sum_smem, st, a);
    TTIE_LAUNCH((chunk_carry_kernel<MODE, CT>), carry, CARRY, 0, st, a);
    // wkv, heads of up to 64: four CTAs an SM with 128 registers where three with 168 do not hold the grid at once
    if constexpr (MANY) {
        if ((long long)slots * a.H > 3LL * num_sms()) {
            TTIE_LAUNCH((chunk_out_kernel<MODE, KP, VT, 4>), grid, 128, out_smem, st, a);
            TTIE_CHECK_LAUNCH("matrix_chunks");
            return 0;
        }
    }
    TTIE_LAUNCH((chunk_out_kernel<MODE, KP, VT>), grid, 128, out_smem, st, a);
    TTIE_CHECK_LAUNCH("matrix_chunks");
    return 0;
}
}  // namespace

// mode: 0 retention (q, k float32; v either type), 1 mlstm, 2 wkv (q, k, v bfloat16).  T: rows of the step.  D and Dv multiples of
// 8, D at most 128, rows that start on 16 bytes.  part / aux / span / mm hold `slots` chunk numbers' worth; a step of more chunk
// numbers (T / chunk + requests) is done in passes.  chunk: tokens of one, 64 or (modes 0 and 1, bfloat16 values of at most 128 columns) 128.
// pre_bias (chunks of 128): bfloat16 [2H] on mlstm's gate pre-activations.  y (or null; chunks of 128, or mode 2 with at most 64 channels):
// bfloat16 [T, H*Dv], the read-outs normalised over a head, times norm_w [H*Dv] (or null) and act(gate) (0 silu, 1 sigmoid); `out` is scratch then.
extern "C" int ttie_matrix_chunks(int mode, const void* q, const void* k, long long ld_qk, const void* v, long long ld_v, int v_dtype,
                                  const float* pre, long long ld_pre, float cap, const float* decay, const float* u, float* S, float* nrm,
                                  float* mx, int state_rows, const void* x, long long ld_x, int d, float* prev, int prev_rows, const int* qsl,
                                  const int* slot_ids, int num_seqs, int T, float* out, int H, int D, int Dv, int Dpad, float qscale,
                                  float* part, float* aux, void* span, void* mm, int slots, int chunk, const void* pre_bias, void* y,
                                  const void* gate, long long ld_gate, const float* norm_w, float eps, int act, void* stream) {
    if (num_seqs <= 0 || T <= 0) return 0;
    if (chunk != CT && (chunk != 128 || mode == WKV || v_dtype != kBF16 || Dv > 128)) TTIE_FAIL("matrix_chunks: chunks of %d tokens, mode %d, %d value channels", chunk, mode, Dv);
    if (pre_bias && (chunk != 128 || mode != MLSTM)) TTIE_FAIL("matrix_chunks: a gate bias goes with mlstm in chunks of 128 tokens");
    if (mode < 0 || mode > 2 || (v_dtype != kBF16 && !(v_dtype == kF32 && mode == RET))) TTIE_FAIL("matrix_chunks: mode %d with values of type %d", mode, v_dtype);
    const int ce = mode == RET ? 4 : 8, ve = v_dtype == kF32 ? 4 : 8;                 // values per 16 bytes
    if (D < 8 || D > 128 || D % 8 || Dv < 8 || Dv % 8 || Dpad < D || Dpad > 128 || Dpad % 8 || ld_qk % ce || ld_v % ve || (mode == WKV && D != Dv)
        || (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)S | (uintptr_t)nrm | (uintptr_t)part | (uintptr_t)aux) & 15))
        TTIE_FAIL("matrix_chunks: heads of %d key channels (padded %d) and %d value channels, strides %lld and %lld: multiples of 8, at most 128 key channels, rows on 16 bytes", D, Dpad, Dv, ld_qk, ld_v);
    if (slots < 1 || H > 65535 || num_seqs > 65535) TTIE_FAIL("matrix_chunks: %d chunks a pass, %d heads, %d requests", slots, H, num_seqs);
    if (y && (!(chunk == 128 || (mode == WKV && Dpad <= 64)) || !gate || ld_gate % 8 || (((uintptr_t)gate | (uintptr_t)y) & 15) || ((uintptr_t)norm_w & 7)))
        TTIE_FAIL("matrix_chunks: a gate with mode %d in chunks of %d, its rows %lld apart", mode, chunk, ld_gate);
    ChunkArgs a = {};
    a.y = (__nv_bfloat16*)y; a.gate = (const __nv_bfloat16*)gate; a.ld_gate = ld_gate; a.norm_w = norm_w; a.eps = eps; a.act = act;
    a.q = q; a.k = k; a.ld_qk = ld_qk; a.v = v; a.ld_v = ld_v; a.pre = pre; a.ld_pre = ld_pre; a.cap = cap; a.decay = decay; a.u = u;
    a.v_f32 = v_dtype == kF32;
    a.S = S; a.nrm = nrm; a.mx = mx; a.state_rows = state_rows; a.x = x; a.ld_x = ld_x; a.d = d; a.prev = prev; a.prev_rows = prev_rows;
    a.qsl = qsl; a.slot_ids = slot_ids; a.num_seqs = num_seqs; a.out = out; a.H = H; a.D = D; a.Dv = Dv; a.Dpad = Dpad; a.qscale = qscale;
    a.part = part; a.aux = aux; a.span = (double2*)span; a.mm = (float2*)mm;
    a.pre_bias = (const __nv_bfloat16*)pre_bias;
    cudaStream_t st = (cudaStream_t)stream;
    if (chunk == 128) return matrix_chunks_tc(mode, a, T, slots, st);
    const int total = T / CT + num_seqs;
    for (int first = 0; first < total; first += slots) {
        const int cnt = total - first < slots ? total - first : slots;
        int rc;
        if (mode == RET && v_dtype == kF32) rc = Dpad <= 64 ? launch_chunks<RET, 64, float>(a, first, cnt, st) : launch_chunks<RET, 128, float>(a, first, cnt, st);
        else if (mode == RET) rc = Dpad <= 64 ? launch_chunks<RET, 64, __nv_bfloat16>(a, first, cnt, st) : launch_chunks<RET, 128, __nv_bfloat16>(a, first, cnt, st);
        else if (mode == MLSTM) rc = Dpad <= 64 ? launch_chunks<MLSTM, 64, __nv_bfloat16>(a, first, cnt, st) : launch_chunks<MLSTM, 128, __nv_bfloat16>(a, first, cnt, st);
        else rc = Dpad <= 64 ? launch_chunks<WKV, 64, __nv_bfloat16>(a, first, cnt, st) : launch_chunks<WKV, 128, __nv_bfloat16>(a, first, cnt, st);
        if (rc) return rc;
    }
    return 0;
}

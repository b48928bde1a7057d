// The selective scan (a diagonal state-space recurrence whose step size and in/out projections depend on the token), for any
// split of a sequence into steps.  Per channel c and state n, with dt = softplus(low-rank product + bias) per token and channel,
//     S[c, n] <- exp(dt_c A[c, n]) S[c, n] + dt_c u_c B_n          y_c = sum_n S[c, n] C_n + D_c u_c          out = y * silu(z)
// A is negative, [channels, states]; B and C are one row of states per token that all channels share; u is the output of a short
// convolution and z a gate branch.  Step sizes, decays, state and read-out are 32-bit in every run.
//
// A thread owns four consecutive states of one channel, the slices of a channel are adjacent lanes, and a CTA of 128 threads takes
// 128 / slices channels of one request.  The kernel is bound by the exponentials (one per state and token; the unit does 16 a
// clock and SM) as long as nothing else shows, so a run of TB tokens is taken in phases: all its decays and inputs first (independent
// of each other), then the chain of the state (two multiply-adds a token), then the read-outs of the whole run reduced over the
// slices at once.  The lanes of a channel share what belongs to a token and channel alone: each loads the step sizes, inputs
// and gates of its share of the run's tokens, evaluates them, and finishes those tokens' outputs.  B and C, which all channels
// share, go through two buffers of shared memory (one barrier per run); all of the next run's values travel into registers
// while this one is computed.  A state row is [channels][padded states].
//
// Long prompts in parts.  The decay over a part is exp(A * sum of dt), so what a part adds to the state needs no other part:
// with ``parts`` > 1 the kernel runs twice over requests x parts.  Mode 1 walks every part but a request's last from a zero
// state without reading out and leaves that sum and the part's summed step sizes in scratch (the unit of the last part copies
// the request's state row there meanwhile, so that the second launch reads nothing that it also writes).  Mode 0 builds each
// part's first state from those, walks the part with read-out, and the request's last part writes the state row.
// The last unit of a request also moves the short convolution's last inputs into their state row (that kernel ran before).
#include "common.cuh"
#include <math.h>
using namespace ttie;

namespace {

constexpr int NT = 128, TB = 8, KPT = 4;    // threads of a CTA; tokens of a run; states of a thread
constexpr int DIRECT_TOKENS = 2;            // a request that brings this few tokens (decoded ones) is walked straight from global memory
constexpr int PART_MIN_TOKENS = 64;

__device__ __forceinline__ int slot_row_(int slot, int num_rows) { return slot < 0 ? num_rows - 1 : slot; }
// The step of a state, S <- exp(dt A) S + du B.
// A slow state (dt * A near 0) lives for thousands of tokens, and the rounding of a factor just below 1 repeats itself with every
// token: a 32-bit run adds expm1(dt * A) S + du B to S instead, which leaves only the sum's own rounding.  A bfloat16 run uses the
// hardware's 2^x on A * log2(e), which the thread then holds for A (relative error about 2^-22, far below the rounding of the
// bfloat16 operands around it).
__device__ __forceinline__ float ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
// softplus and silu: the library's accurate functions in a 32-bit run; else the hardware's exponential, logarithm and reciprocal
// (relative error about 1e-6 as well: log(1 + e) of a small e, where 1 + e has lost its digits, by the series e - e^2/2 + e^3/3; a step size below
// 2^-126 counts as none: with such ones kept the scan takes 1 % longer).
template <typename T> struct Act {
    static __device__ __forceinline__ float softplus(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }
    static __device__ __forceinline__ float silu(float x) { return x / (1.0f + expf(-x)); }
};
__device__ __forceinline__ float lg2(float x) { float y; asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float rcp(float x) { float y; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
template <> struct Act<__nv_bfloat16> {
    static __device__ __forceinline__ float softplus(float x) {
        const float e = ex2(-1.4426950408889634f * fabsf(x));
        const float small = e * fmaf(e, fmaf(e, 0.33333334f, -0.5f), 1.0f);
        return fmaxf(x, 0.f) + (e < 0.01f ? small : 0.6931471805599453f * lg2(1.0f + e));
    }
    static __device__ __forceinline__ float silu(float x) { return x * rcp(1.0f + ex2(-1.4426950408889634f * x)); }
};
template <typename T> struct Decay {
    static __device__ __forceinline__ float hold(float a) { return a; }
    static __device__ __forceinline__ float of(float dt, float a) { return expm1f(dt * a); }
    static __device__ __forceinline__ float step(float e, float S, float x) { return S + fmaf(e, S, x); }
};
template <> struct Decay<__nv_bfloat16> {
    static __device__ __forceinline__ float hold(float a) { return a * 1.4426950408889634f; }
    static __device__ __forceinline__ float of(float dt, float a) { return ex2(dt * a); }
    static __device__ __forceinline__ float step(float e, float S, float x) { return fmaf(e, S, x); }
};

struct SelArgs {
    const void* u; long long ld_u;                                    // [T, I] compute dtype
    const float* dt; long long ld_dt; const float* dt_bias;           // [T, I] before bias and softplus, [I]
    const float* A; const float* D;                                   // [I, Np], [I]
    const void* bc; long long ld_bc; int col_b, col_c;                // rows that hold B and C at these columns, compute dtype
    const void* z; long long ld_z;                                    // [T, I] compute dtype
    float* state; int state_rows;                                     // [rows, I, Np]
    const void* xin; long long ld_x; float* tail; int tail_rows, taps; // the convolution's inputs [T, I] and its state rows [rows, taps - 1, I]
    const int* qsl; const int* slot_ids;
    void* out;                                                        // [T, I] compute dtype
    int I, N, Np;
    float* scratch; float* scratch_dt; int parts, mode;               // [requests * parts, I, Np], [requests * parts, I]
    int copies16, pairs;                                              // u, dt and z rows lie on 16 bytes (channels a multiple of 8); pairs of u and z on 4 (an even number)
};

template <int SL> __device__ __forceinline__ float slices_sum(float v) {
#pragma unroll
    for (int o = 1; o < SL; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// Sums over the SL adjacent lanes of a channel of CNT values per lane at once (the read-outs of a run of tokens): at every step
// a lane hands half of its values to the partner and adds the partner's other half to the half it keeps; once a lane is down to
// one value the remaining steps are butterfly additions.  Afterwards v[0 ..] holds the totals of tokens slice * CNT / SL ..
template <int O, int CNT>
__device__ __forceinline__ void run_reduce(float* v, int slice) {
    if constexpr (O >= 1) {
        if constexpr (CNT > 1) {
            constexpr int HALF = CNT / 2;
            const bool upper = (slice & O) != 0;
#pragma unroll
            for (int i = 0; i < HALF; ++i) {
                const float send = upper ? v[i] : v[i + HALF];
                const float keep = upper ? v[i + HALF] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, O);
            }
            run_reduce<O / 2, HALF>(v, slice);
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
            run_reduce<O / 2, 1>(v, slice);
        }
    }
}
__device__ __forceinline__ void ld4(const float* p, float* o) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    o[0] = x.x; o[1] = x.y; o[2] = x.z; o[3] = x.w;
}

// Walks n tokens.  READ: with read-out (writes out); without, only the state moves.  Returns the sum of the step sizes.
template <typename T, int SL, bool READ>
__device__ __forceinline__ float walk(const SelArgs& a, int t0, int n, int c, bool cv, int slice, const float (&A)[KPT], float (&S)[KPT], float* smem) {
    constexpr int NP = SL * KPT, PC = TB / SL > 0 ? TB / SL : 1, SAME = SL / TB > 0 ? SL / TB : 1, PB = (TB * NP + NT - 1) / NT;
    const int cc = cv ? c : 0, n0 = slice * KPT;
    const T* up = reinterpret_cast<const T*>(a.u) + (size_t)t0 * a.ld_u + cc;
    const T* zp = reinterpret_cast<const T*>(a.z) + (size_t)t0 * a.ld_z + cc;
    const T* bp = reinterpret_cast<const T*>(a.bc) + (size_t)t0 * a.ld_bc + a.col_b;
    const T* cp = reinterpret_cast<const T*>(a.bc) + (size_t)t0 * a.ld_bc + a.col_c;
    const float* dp = a.dt + (size_t)t0 * a.ld_dt + cc;
    T* op = reinterpret_cast<T*>(a.out) + (size_t)t0 * a.I + cc;
    const float bias = a.dt_bias[cc], Dc = a.D[cc];
    float sum_dt = 0.f;
    if (n <= DIRECT_TOKENS) {
        for (int tt = 0; tt < n; ++tt) {
            const float dt = Act<T>::softplus(dp[(size_t)tt * a.ld_dt] + bias), u = to_f32(up[(size_t)tt * a.ld_u]), du = dt * u;
            float acc = 0.f;
#pragma unroll
            for (int i = 0; i < KPT; ++i) {
                const bool in = n0 + i < a.N;
                S[i] = Decay<T>::step(Decay<T>::of(dt, A[i]), S[i], du * (in ? to_f32(bp[(size_t)tt * a.ld_bc + n0 + i]) : 0.f));
                acc = fmaf(S[i], READ && in ? to_f32(cp[(size_t)tt * a.ld_bc + n0 + i]) : 0.f, acc);
            }
            sum_dt += dt;
            if (!READ) continue;
            acc = slices_sum<SL>(acc);
            if (slice == 0 && cv) op[(size_t)tt * a.I] = from_f32<T>(fmaf(Dc, u, acc) * Act<T>::silu(to_f32(zp[(size_t)tt * a.ld_z])));
        }
        return sum_dt;
    }
    // the lanes of a channel share the tokens of a run: lane `slice` holds step size, input and gate of tokens own .. own + PC - 1
    // (with more slices than tokens, SAME lanes hold the same one)
    const int own = slice / SAME * PC;
    float d_next[PC], d[PC], u[PC], b_next[PB], c_next[PB];
    T u_next[PC], z_next[PC], z[PC];
    auto fetch = [&](int r0, int nb) {
#pragma unroll
        for (int j = 0; j < PC; ++j) {
            const int tt = own + j;
            const bool ok = tt < nb;
            d_next[j] = ok ? dp[(size_t)(r0 + tt) * a.ld_dt] : 0.f;
            u_next[j] = ok ? up[(size_t)(r0 + tt) * a.ld_u] : from_f32<T>(0.f);
            if (READ) z_next[j] = ok ? zp[(size_t)(r0 + tt) * a.ld_z] : from_f32<T>(0.f);
        }
#pragma unroll
        for (int i = 0; i < PB; ++i) {
            const int e = i * NT + threadIdx.x, tt = e / NP, k = e - tt * NP;
            const bool ok = tt < nb && k < a.N;
            b_next[i] = ok ? to_f32(bp[(size_t)(r0 + tt) * a.ld_bc + k]) : 0.f;
            if (READ) c_next[i] = ok ? to_f32(cp[(size_t)(r0 + tt) * a.ld_bc + k]) : 0.f;
        }
    };
    auto settle = [&](int buf, int nb) {                             // what has arrived becomes the current run
        float* bs = smem + buf * 2 * TB * NP;
#pragma unroll
        for (int i = 0; i < PB; ++i) {
            const int e = i * NT + threadIdx.x;
            if (e < TB * NP) { bs[e] = b_next[i]; if (READ) bs[TB * NP + e] = c_next[i]; }
        }
#pragma unroll
        for (int j = 0; j < PC; ++j) {                               // (a token behind the last one: step size 0, which moves nothing)
            d[j] = own + j < nb ? Act<T>::softplus(d_next[j] + bias) : 0.f;
            u[j] = to_f32(u_next[j]);
            if (READ) z[j] = z_next[j];
        }
        __syncthreads();
    };
    fetch(0, min(TB, n));
    settle(0, min(TB, n));
    for (int r0 = 0, it = 0; r0 < n; r0 += TB, ++it) {
        const int nb = min(TB, n - r0);
        const bool more = r0 + TB < n;
        if (more) fetch(r0 + TB, min(TB, n - r0 - TB));
        const float* bs = smem + (it & 1) * 2 * TB * NP + n0;
        float e[TB][KPT], x[TB][KPT], y[TB];
#pragma unroll
        for (int tt = 0; tt < TB; ++tt) {
            float dt = d[tt % PC], du = d[tt % PC] * u[tt % PC], b[KPT];
            if (SL > 1) {
                dt = __shfl_sync(0xffffffffu, dt, tt / PC * SAME, SL);
                du = __shfl_sync(0xffffffffu, du, tt / PC * SAME, SL);
            }
            ld4(bs + tt * NP, b);
#pragma unroll
            for (int i = 0; i < KPT; ++i) { e[tt][i] = Decay<T>::of(dt, A[i]); x[tt][i] = du * b[i]; }
            if (!READ) sum_dt += dt;
        }
#pragma unroll
        for (int tt = 0; tt < TB; ++tt) {
#pragma unroll
            for (int i = 0; i < KPT; ++i) S[i] = Decay<T>::step(e[tt][i], S[i], x[tt][i]);
            if (READ) {
                float q[KPT];
                ld4(bs + TB * NP + tt * NP, q);
                y[tt] = fmaf(S[0], q[0], S[1] * q[1]) + fmaf(S[2], q[2], S[3] * q[3]);
            }
        }
        if (READ) {
            run_reduce<SL / 2, TB>(y, slice);
            if (cv && slice % SAME == 0) {
#pragma unroll
                for (int j = 0; j < PC; ++j)
                    if (own + j < nb) op[(size_t)(r0 + own + j) * a.I] = from_f32<T>(fmaf(Dc, u[j], y[j]) * Act<T>::silu(to_f32(z[j])));
            }
        }
        if (more) settle((it & 1) ^ 1, min(TB, n - r0 - TB));
    }
    return sum_dt;
}

// the convolution's last taps - 1 inputs of a channel, oldest first: those of this step, and before them what the row held
template <typename T>
__device__ __forceinline__ void move_tail(const SelArgs& a, int s, int q0, int n, int ch) {
    const T* x = reinterpret_cast<const T*>(a.xin) + ch;
    float* mine = a.tail + (size_t)slot_row_(a.slot_ids[s], a.tail_rows) * (a.taps - 1) * a.I + ch;
    for (int i = 0; i < a.taps - 1; ++i) {                           // ascending: row i takes from an old row behind it, or from the step
        const int idx = n - (a.taps - 1) + i;
        mine[(size_t)i * a.I] = idx >= 0 ? to_f32(x[(size_t)(q0 + idx) * a.ld_x]) : mine[(size_t)(a.taps - 1 + idx) * a.I];
    }
}

template <typename T, int SL>
__global__ void __launch_bounds__(NT) selective_scan_kernel(const SelArgs a) {
    pdl_wait();                                                      // (the successor is let in at the end: its waiting CTAs would sit on the SMs of a long, latency-bound walk)
    constexpr int CH = NT / SL, NP = SL * KPT;                       // channels per CTA, padded states
    __shared__ __align__(16) float smem[4 * TB * NP];                // two buffers of B and C
    const int s = blockIdx.y / a.parts, p = blockIdx.y - s * a.parts;
    const int q0 = a.qsl[s], n = a.qsl[s + 1] - q0;
    int L = n, p_last = 0;                                           // tokens of a part, the part of the request's last token
    if (a.parts > 1 && n > 0) {
        L = max(PART_MIN_TOKENS, ((n + a.parts - 1) / a.parts + TB - 1) / TB * TB);
        p_last = (n - 1) / L;                                        // (< parts)
    }
    const bool local = a.mode == 1;
    const bool copies = local && p_last > 0 && p == a.parts - 1;     // (never a part that mode 1 walks: those lie before p_last)
    if (n <= 0 || (local ? (p >= p_last && !copies) : p > p_last)) return;
    const int slice = threadIdx.x % SL, c0 = blockIdx.x * CH, c = c0 + threadIdx.x / SL;
    const bool cv = c < a.I;
    const int cc = cv ? c : 0, n0 = slice * KPT;
    float* sp = a.state + ((size_t)slot_row_(a.slot_ids[s], a.state_rows) * a.I + cc) * NP + n0;
    auto scratch_at = [&](int part) { return a.scratch + (((size_t)s * a.parts + part) * a.I + cc) * NP + n0; };
    if (copies) {
        if (cv) *reinterpret_cast<float4*>(scratch_at(p)) = *reinterpret_cast<const float4*>(sp);
        return;
    }
    float A[KPT], S[KPT] = {0.f, 0.f, 0.f, 0.f}, sum_dt;
    ld4(a.A + (size_t)cc * NP + n0, A);
#pragma unroll
    for (int i = 0; i < KPT; ++i) A[i] = Decay<T>::hold(A[i]);
    if (local) {
        sum_dt = walk<T, SL, false>(a, q0 + p * L, min(L, n - p * L), c, cv, slice, A, S, smem);
    } else {
        ld4(p_last == 0 ? sp : scratch_at(a.parts - 1), S);          // the state row as it was before the step
        for (int j = 0; j < p; ++j) {                                // then the parts before this one: S <- exp(A * sum of dt) S + what the part adds
            float add[KPT];
            ld4(scratch_at(j), add);
            const float sdt = a.scratch_dt[((size_t)s * a.parts + j) * a.I + cc];
#pragma unroll
            for (int i = 0; i < KPT; ++i) S[i] = Decay<T>::step(Decay<T>::of(sdt, A[i]), S[i], add[i]);
        }
        walk<T, SL, true>(a, q0 + p * L, min(L, n - p * L), c, cv, slice, A, S, smem);
    }
    pdl_launch_dependents();
    if (cv && (local || p == p_last)) {
        *reinterpret_cast<float4*>(local ? scratch_at(p) : sp) = make_float4(S[0], S[1], S[2], S[3]);
        if (local && slice == 0) a.scratch_dt[((size_t)s * a.parts + p) * a.I + c] = sum_dt;
    }
    if (!local && p == p_last && threadIdx.x < CH && c0 + (int)threadIdx.x < a.I) move_tail<T>(a, s, q0, n, c0 + threadIdx.x);
}

// ---- bfloat16 prompt portions of up to 16 states: a thread owns a channel with all its states (NS of them, padded to 4, 8 or 16).
// What a token costs besides its states - loads, softplus, silu, the store - is then paid once per channel instead of being
// dealt out to the lanes of a channel with shuffles and predicates (that was seven of twelve instructions per state), rows
// of a warp's 32 channels are 64 and 128 contiguous bytes, and the states' multiplications go in pairs (one instruction for two;
// the exponentials have no such form).  Step sizes, inputs and gates travel into shared memory by asynchronous copies three runs ahead, B
// and C of a run lie there widened, read by every thread at the same address; so a thread's registers are its states and the
// values of several tokens at once: a whole run is straight-line code in which the next tokens' exponentials go ahead of this one's sums (with a branch per
// token and the next run in registers 117 us, so 101 in as many parts, with the parts of _even_parts 99; two walks of 2,048 tokens of 4,096 channels).
// What bounds it: without the states' exponentials 72 us, with nothing but loads, sums and loop 65; the exponential unit alone needs 69 (16 a token for the
// states, four for softplus and silu).  Two channels a thread 139, a quarter of the exponentials as polynomials on the multiply-add pipe 114, more CTAs an SM with fewer
// registers 105 to 121.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<unsigned long long&>(d)) : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
    return d;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)), "l"(reinterpret_cast<const unsigned long long&>(c)));
    return d;
}

// What a CTA's walk keeps in shared memory: STAGES runs of its 128 channels' step sizes (before bias and softplus), inputs and gates, which
// come from memory three runs ahead, and two runs of B and C, which all CTAs share.
constexpr int STAGES = 4, WIDE_CTAS = 4;      // runs in shared memory; CTAs of an SM (of 128 registers a thread)
template <int NS>
struct __align__(16) WideRuns {
    float d[STAGES][TB][NT];
    unsigned short u[STAGES][TB][NT], z[STAGES][TB][NT];
    float b[2][TB][NS], c[2][TB][NS];
};
__device__ __forceinline__ void copy16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void copy4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <int NS, bool READ>
__device__ __forceinline__ float wide_walk(const SelArgs& a, int t0, int n, int c, bool cv, const float2 (&A)[NS / 2], float2 (&S)[NS / 2], WideRuns<NS>& w) {
    using T = __nv_bfloat16;
    using Raw = unsigned short;
    const int tid = threadIdx.x, c0 = c - tid, cc = cv ? c : 0;
    const float bias = a.dt_bias[cc], Dc = READ ? a.D[cc] : 0.f;
    T* o = reinterpret_cast<T*>(a.out) + (size_t)t0 * a.I + cc;
    auto wide = [](Raw r) { return __uint_as_float((unsigned)r << 16); };
    // asks for step sizes, inputs and gates of run r (an empty group of copies past the last run)
    auto fetch = [&](int r) {
        const int r0 = r * TB, nb = min(TB, n - r0), st = r % STAGES;
        if (nb > 0) {
            const float* d = a.dt + (size_t)(t0 + r0) * a.ld_dt + c0;
            const Raw* u = reinterpret_cast<const Raw*>(a.u) + (size_t)(t0 + r0) * a.ld_u + c0;
            const Raw* z = reinterpret_cast<const Raw*>(a.z) + (size_t)(t0 + r0) * a.ld_z + c0;
            if (a.copies16) {
                const int dk = tid % 32 * 4, uk = tid % 16 * 8;
                static_assert(NT / 16 == TB, "16 threads a row of inputs");
                if (c0 + dk < a.I)
#pragma unroll
                    for (int tt = tid / 32; tt < TB; tt += NT / 32)
                        if (tt < nb) copy16(&w.d[st][tt][dk], d + (size_t)tt * a.ld_dt + dk);
                if (c0 + uk < a.I && tid / 16 < nb) {
                    copy16(&w.u[st][tid / 16][uk], u + (size_t)(tid / 16) * a.ld_u + uk);
                    if (READ) copy16(&w.z[st][tid / 16][uk], z + (size_t)(tid / 16) * a.ld_z + uk);
                }
            } else {                                                  // rows that do not lie on 16 bytes: two channels a copy, or one
#pragma unroll
                for (int tt = 0; tt < TB; ++tt)
                    if (tt < nb && cv) copy4(&w.d[st][tt][tid], d + (size_t)tt * a.ld_dt + tid);
                if (a.pairs) {
                    const int uk = tid % 64 * 2;
                    if (c0 + uk < a.I)
#pragma unroll
                        for (int tt = tid / 64; tt < TB; tt += NT / 64)
                            if (tt < nb) {
                                copy4(&w.u[st][tt][uk], u + (size_t)tt * a.ld_u + uk);
                                if (READ) copy4(&w.z[st][tt][uk], z + (size_t)tt * a.ld_z + uk);
                            }
                } else if (cv) {
                    Raw ur[TB], zr[TB];
#pragma unroll
                    for (int tt = 0; tt < TB; ++tt) {
                        ur[tt] = tt < nb ? u[(size_t)tt * a.ld_u + tid] : (Raw)0;
                        if (READ) zr[tt] = tt < nb ? z[(size_t)tt * a.ld_z + tid] : (Raw)0;
                    }
#pragma unroll
                    for (int tt = 0; tt < TB; ++tt) { w.u[st][tt][tid] = ur[tt]; if (READ) w.z[st][tt][tid] = zr[tt]; }
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // B and C of a run, through a register each (they are widened)
    constexpr int PB = (TB * NS + NT - 1) / NT;
    Raw b_next[PB], c_next[PB];
    auto fetch_bc = [&](int r) {
        const int r0 = r * TB, nb = min(TB, n - r0);
        const Raw* bc = reinterpret_cast<const Raw*>(a.bc) + (size_t)(t0 + r0) * a.ld_bc;
#pragma unroll
        for (int i = 0; i < PB; ++i) {
            const int e = i * NT + tid, tt = e / NS, k = e % NS;
            const bool ok = tt < nb && k < a.N;
            b_next[i] = ok ? bc[(size_t)tt * a.ld_bc + a.col_b + k] : (Raw)0;
            if (READ) c_next[i] = ok ? bc[(size_t)tt * a.ld_bc + a.col_c + k] : (Raw)0;
        }
    };
    // makes run r readable for all threads; what was read before may be overwritten behind it
    auto settle = [&](int r) {
#pragma unroll
        for (int i = 0; i < PB; ++i) {
            const int e = i * NT + tid;
            if (e < TB * NS) { (&w.b[r & 1][0][0])[e] = wide(b_next[i]); if (READ) (&w.c[r & 1][0][0])[e] = wide(c_next[i]); }
        }
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();
    };
    float sum_dt = 0.f;
    const int nruns = (n + TB - 1) / TB;
#pragma unroll
    for (int r = 0; r < STAGES - 1; ++r) fetch(r);
    fetch_bc(0);
    for (int r = 0; r < nruns; ++r) {
        settle(r);
        fetch(r + STAGES - 1);                                        // (into the run before r, which every thread has read)
        if (r + 1 < nruns) fetch_bc(r + 1);
        const int nb = min(TB, n - r * TB), st = r % STAGES, bb = r & 1;
        auto token = [&](int tt) {
            const float dt = Act<T>::softplus(w.d[st][tt][tid] + bias), uv = wide(w.u[st][tt][tid]);
            const float2 dt2 = make_float2(dt, dt), du2 = make_float2(dt * uv, dt * uv);
            float2 y2 = make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < NS / 2; i += 2) {
                const float4 b = *reinterpret_cast<const float4*>(&w.b[bb][tt][2 * i]);
                const float2 e0 = mul2(dt2, A[i]), e1 = mul2(dt2, A[i + 1]);
                S[i] = fma2(make_float2(ex2(e0.x), ex2(e0.y)), S[i], mul2(du2, make_float2(b.x, b.y)));
                S[i + 1] = fma2(make_float2(ex2(e1.x), ex2(e1.y)), S[i + 1], mul2(du2, make_float2(b.z, b.w)));
                if (READ) {
                    const float4 q = *reinterpret_cast<const float4*>(&w.c[bb][tt][2 * i]);
                    y2 = fma2(S[i], make_float2(q.x, q.y), y2);
                    y2 = fma2(S[i + 1], make_float2(q.z, q.w), y2);
                }
            }
            if (READ) {
                if (cv) *o = from_f32<T>(fmaf(Dc, uv, y2.x + y2.y) * Act<T>::silu(wide(w.z[st][tt][tid])));
                o += a.I;
            } else sum_dt += dt;
        };
        if (nb == TB) {                                               // (without a branch per token: the next token's loads and exponentials go ahead of this one's sums)
#pragma unroll
            for (int tt = 0; tt < TB; ++tt) token(tt);
        } else {
#pragma unroll 1
            for (int tt = 0; tt < nb; ++tt) token(tt);
        }
    }
    return sum_dt;
}

template <int NS>
__global__ void __launch_bounds__(NT, WIDE_CTAS) selective_wide_kernel(const SelArgs a) {
    pdl_wait();                                                      // (the successor is let in at the end, as in the other form)
    __shared__ WideRuns<NS> smem;
    // the last request first: a prompt portion stands behind the decoded tokens of a step, and its CTAs spread over idle SMs only if they are
    // the first to be placed (8,192 channels, 23 requests of one token and one of 2,000: 405 us in four parts, now 265)
    const int y = blockIdx.y / a.parts, s = gridDim.y / a.parts - 1 - y, p = blockIdx.y - y * a.parts;
    const int q0 = a.qsl[s], n = a.qsl[s + 1] - q0;
    int L = n, p_last = 0;                                           // tokens of a part, the part of the request's last token
    if (a.parts > 1 && n > 0) {
        L = max(PART_MIN_TOKENS, ((n + a.parts - 1) / a.parts + TB - 1) / TB * TB);
        p_last = (n - 1) / L;
    }
    const bool local = a.mode == 1;
    const bool copies = local && p_last > 0 && p == a.parts - 1;     // (never a part that mode 1 walks: those lie before p_last)
    if (n <= 0 || (local ? (p >= p_last && !copies) : p > p_last)) return;
    const int c = blockIdx.x * NT + threadIdx.x;
    const bool cv = c < a.I;
    const int cc = cv ? c : 0;
    float* sp = a.state + ((size_t)slot_row_(a.slot_ids[s], a.state_rows) * a.I + cc) * NS;
    auto scratch_at = [&](int part) { return a.scratch + (((size_t)s * a.parts + part) * a.I + cc) * NS; };
    float2 A[NS / 2], S[NS / 2];
    auto load = [&](const float* src, float2 (&v)[NS / 2]) {
#pragma unroll
        for (int i = 0; i < NS / 2; i += 2) {
            const float4 x = *reinterpret_cast<const float4*>(src + 2 * i);
            v[i] = make_float2(x.x, x.y); v[i + 1] = make_float2(x.z, x.w);
        }
    };
    auto store = [&](float* dst) {
#pragma unroll
        for (int i = 0; i < NS / 2; i += 2) *reinterpret_cast<float4*>(dst + 2 * i) = make_float4(S[i].x, S[i].y, S[i + 1].x, S[i + 1].y);
    };
    if (copies) {
        load(sp, S);
        if (cv) store(scratch_at(p));
        return;
    }
    load(a.A + (size_t)cc * NS, A);
#pragma unroll
    for (int i = 0; i < NS / 2; ++i) {
        A[i] = make_float2(Decay<__nv_bfloat16>::hold(A[i].x), Decay<__nv_bfloat16>::hold(A[i].y));
        S[i] = make_float2(0.f, 0.f);
    }
    float sum_dt = 0.f;
    if (local) {
        sum_dt = wide_walk<NS, false>(a, q0 + p * L, min(L, n - p * L), c, cv, A, S, smem);
    } else {
        load(p_last == 0 ? sp : scratch_at(a.parts - 1), S);         // the state row as it was before the step
        constexpr int AHEAD = 4;                                     // then the parts before this one, the loads of AHEAD of them at once
        for (int j0 = 0; j0 < p; j0 += AHEAD) {
            float2 add[AHEAD][NS / 2];
            float sdt[AHEAD];
#pragma unroll
            for (int k = 0; k < AHEAD; ++k) {
                const int j = min(j0 + k, p - 1);
                load(scratch_at(j), add[k]);
                sdt[k] = a.scratch_dt[((size_t)s * a.parts + j) * a.I + cc];
            }
#pragma unroll
            for (int k = 0; k < AHEAD; ++k) {
                if (j0 + k >= p) break;
#pragma unroll
                for (int i = 0; i < NS / 2; ++i) S[i] = fma2(make_float2(ex2(sdt[k] * A[i].x), ex2(sdt[k] * A[i].y)), S[i], add[k][i]);
            }
        }
        wide_walk<NS, true>(a, q0 + p * L, min(L, n - p * L), c, cv, A, S, smem);
    }
    pdl_launch_dependents();
    if (cv && (local || p == p_last)) {
        store(local ? scratch_at(p) : sp);
        if (local) a.scratch_dt[((size_t)s * a.parts + p) * a.I + c] = sum_dt;
    }
    if (!local && p == p_last && cv) move_tail<__nv_bfloat16>(a, s, q0, n, c);
}

int state_slices(int N) {
    int sl = 1;
    while (sl * KPT < N) sl <<= 1;
    return sl;
}
}  // namespace

// padded states of a state row (0: more states than the kernel takes)
extern "C" int ttie_selective_state_pad(int N) { return N < 1 || N > 128 ? 0 : state_slices(N) * KPT; }

// wide: a thread per channel (16-bit operands, up to 16 states), else a thread per four states.
// parts > 1: scratch holds requests * parts * channels * (padded states + 1) floats
extern "C" int ttie_selective_scan(const void* u, long long ld_u, const float* dt, long long ld_dt, const float* dt_bias, const float* A,
                                   const float* D, const void* bc, long long ld_bc, int col_b, int col_c, const void* z, long long ld_z,
                                   float* state, int state_rows, const void* xin, long long ld_x, float* tail, int tail_rows, int taps,
                                   const int* qsl, const int* slot_ids, int num_seqs, void* out, int I, int N, int parts, float* scratch,
                                   int wide, int dtype, void* stream) {
    if (num_seqs <= 0) return 0;
    if (wide && (dtype != kBF16 || N > 16)) TTIE_FAIL("selective_scan: a thread per channel takes 16-bit operands and up to 16 states (%d)", N);
    if (N < 1 || N > 128) TTIE_FAIL("selective_scan: %d states per channel (1 to 128)", N);
    if (parts < 1 || (parts > 1 && !scratch) || (long long)num_seqs * parts > 65535)
        TTIE_FAIL("selective_scan: %d parts for %d requests", parts, num_seqs);
    if (taps > 1 && (!tail || !xin)) TTIE_FAIL("selective_scan: %d taps need state rows and inputs", taps);
    if (dtype != kF32 && dtype != kBF16) TTIE_FAIL("selective_scan: unknown dtype %d", dtype);
    SelArgs a;
    a.u = u; a.ld_u = ld_u; a.dt = dt; a.ld_dt = ld_dt; a.dt_bias = dt_bias; a.A = A; a.D = D; a.bc = bc; a.ld_bc = ld_bc; a.col_b = col_b;
    a.col_c = col_c; a.z = z; a.ld_z = ld_z; a.state = state; a.state_rows = state_rows; a.xin = xin; a.ld_x = ld_x; a.tail = tail;
    a.tail_rows = tail_rows; a.taps = taps; a.qsl = qsl; a.slot_ids = slot_ids; a.out = out; a.I = I; a.N = N;
    a.copies16 = I % 8 == 0 && ld_u % 8 == 0 && ld_z % 8 == 0 && ld_dt % 4 == 0 && (((uintptr_t)u | (uintptr_t)z | (uintptr_t)dt) & 15) == 0;
    a.pairs = I % 2 == 0 && ld_u % 2 == 0 && ld_z % 2 == 0 && (((uintptr_t)u | (uintptr_t)z) & 3) == 0;
    const int sl = state_slices(N);
    a.Np = KPT * sl; a.parts = parts; a.scratch = scratch;
    a.scratch_dt = scratch ? scratch + (size_t)num_seqs * parts * I * a.Np : nullptr;
    const dim3 grid(wide ? ceil_div(I, NT) : ceil_div(I, NT / sl), num_seqs * parts);
    cudaStream_t s = (cudaStream_t)stream;
    for (int mode = parts > 1 ? 1 : 0; mode >= 0; --mode) {          // (mode 1: every part's own sum, from a zero state)
        a.mode = mode;
        if (wide) {
            if (sl == 1) TTIE_LAUNCH(selective_wide_kernel<4>, grid, NT, 0, s, a);
            else if (sl == 2) TTIE_LAUNCH(selective_wide_kernel<8>, grid, NT, 0, s, a);
            else TTIE_LAUNCH(selective_wide_kernel<16>, grid, NT, 0, s, a);
            TTIE_CHECK_LAUNCH("selective_scan");
            continue;
        }
#define SEL_CASE(L_)                                                                                                      \
        if (sl == L_) {                                                                                                   \
            if (dtype == kF32) TTIE_LAUNCH((selective_scan_kernel<float, L_>), grid, NT, 0, s, a);                        \
            else TTIE_LAUNCH((selective_scan_kernel<__nv_bfloat16, L_>), grid, NT, 0, s, a);                              \
        }
        SEL_CASE(1) SEL_CASE(2) SEL_CASE(4) SEL_CASE(8) SEL_CASE(16) SEL_CASE(32)
#undef SEL_CASE
        TTIE_CHECK_LAUNCH("selective_scan");
    }
    return 0;
}

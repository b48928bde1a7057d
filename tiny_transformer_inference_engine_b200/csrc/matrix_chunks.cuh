// What the two forms of the chunked matrix-state recurrences share (matrix_chunks.cu: 64 tokens a chunk, mma.sync; matrix_chunks_tc.cu: 128 tokens,
// tcgen05): arguments, chunk numbering, gates, the carry between chunks, and the walk's operations for what is not finite.
#pragma once
#include "common.cuh"
#include <math.h>
#include <type_traits>

namespace ttie {
namespace chunks {
constexpr int CARRY = 128;                   // threads of a carry block
enum Mode { RET = 0, MLSTM = 1, WKV = 2 };

struct ChunkArgs {
    const void* q; const void* k; long long ld_qk;                    // [T, H*D]; float32 (retention) or bfloat16
    const void* v; long long ld_v;                                    // [T, H*Dv], bfloat16 or (retention) float32
    const float* pre; long long ld_pre; float cap;                    // mlstm: gate pre-activations [T, 2H]
    const float* decay;                                               // retention [H]; wkv [T, H*D]
    const float* u;                                                   // wkv [H*D]
    bool v_f32;                                                       // v is float32
    float* S; float* nrm; float* mx; int state_rows;                  // state rows (mlstm: normaliser and running maximum too)
    const void* x; long long ld_x; int d; float* prev; int prev_rows; // wkv: the mixer's input and the rows that keep its last token
    const int* qsl; const int* slot_ids; int num_seqs;
    float* out;                                                       // [T, H*Dv]
    int H, D, Dv, Dpad; float qscale;
    int slot_lo, slots;                                               // the chunk numbers of this pass
    float* part;                                                      // [slots, H, Dv, Dpad]
    float* aux;                                                       // mlstm: [slots, H, Dpad] normaliser sums; wkv: [slots, H, 2, Dpad] chunk decays and what rounding them left
    double2* span;                                                    // mlstm: [slots, H] (F at the end, max of x)
    float2* mm;                                                       // mlstm: [slots, H] the running maximum before and behind the chunk
    const __nv_bfloat16* pre_bias;                                    // mlstm in chunks of 128 tokens: [2H] on the gates' pre-activations, or null
    // the read-outs normalised over a head and gated (head_norm_gate of matrix_memory.cu), where y is not null: `out` then only holds what is walked
    __nv_bfloat16* y; const __nv_bfloat16* gate; long long ld_gate; const float* norm_w; float eps; int act;
};

__device__ __forceinline__ int state_row(int slot, int num_rows) { return slot < 0 ? num_rows - 1 : slot; }

// chunk number -> request, chunk of the request, first token (of the step's rows) and number of tokens; false: the number is not in use
template <int CT>
__device__ __forceinline__ bool find_chunk(const int* qsl, int num_seqs, int number, int& s, int& c, int& t0, int& n) {
    int lo = 0, hi = num_seqs - 1;
    while (lo < hi) {                                                 // the last request whose first number is <= number
        const int mid = (lo + hi + 1) >> 1;
        if (qsl[mid] / CT + mid <= number) lo = mid; else hi = mid - 1;
    }
    s = lo;
    c = number - qsl[s] / CT - s;
    const int len = qsl[s + 1] - qsl[s];
    t0 = qsl[s] + c * CT;
    n = min(CT, len - c * CT);
    return c >= 0 && n > 0;
}

// x^n for 0 <= n <= 128 in 64 bits by squaring (0^0 = 1: a head that keeps nothing still sees the token itself): eight roundings at most, a
// tenth of the time of the general function
__device__ __forceinline__ double power(double x, int n) {
    double r = 1.0;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        if (n >> b & 1) r *= x;
        x *= x;
    }
    return r;
}

__device__ __forceinline__ float2 unpack(uint32_t p) { return make_float2(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u)); }

__device__ __forceinline__ void copy16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
// eight consecutive values of a row as floats (zeros where `in` is false)
__device__ __forceinline__ void load8(const float* p, bool in, float (&o)[8]) {
    const float4 a = in ? *reinterpret_cast<const float4*>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 b = in ? *reinterpret_cast<const float4*>(p + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, bool in, float (&o)[8]) {
    const uint4 a = in ? *reinterpret_cast<const uint4*>(p) : make_uint4(0u, 0u, 0u, 0u);
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 f = unpack(w[i]); o[2 * i] = f.x; o[2 * i + 1] = f.y; }
}
// log input gate and log forget gate of a token
template <int CT>
__device__ __forceinline__ float2 log_gates(const ChunkArgs& a, int token, int h) {
    const float* g = a.pre + (size_t)token * a.ld_pre;
    float i = g[h], f = g[a.H + h];
    if (CT == 128 && a.pre_bias) { i += __bfloat162float(a.pre_bias[h]); f += __bfloat162float(a.pre_bias[a.H + h]); }
    const float z = a.cap * tanhf(f / a.cap);
    return make_float2(a.cap * tanhf(i / a.cap), fminf(z, 0.f) - log1pf(expf(-fabsf(z))));
}

// ---- the walk's operations, for what is not finite
__device__ __forceinline__ bool finite4(float x, float y, float z, float w) { return (x - x) + (y - y) + ((z - z) + (w - w)) == 0.f; }

// four state elements (dv, ch .. ch + 3) of a head over the chunk's tokens; normaliser: its elements ch .. ch + 3.  mlstm: m is the running maximum
// before the chunk, m_end the one that the result is scaled to
template <int MODE, int CT>
__device__ __forceinline__ float4 walk_state(const ChunkArgs& a, int t0, int n, int h, int dv, int ch, bool normaliser, float4 S4, float m, float m_end) {
    float S[4] = {S4.x, S4.y, S4.z, S4.w};
    const float decay = MODE == RET ? a.decay[h] : 0.f;
#pragma unroll 1
    for (int t = t0; t < t0 + n; ++t) {
        const size_t at = (size_t)t * a.ld_v + h * a.Dv + dv;
        float v = 1.f, fa = decay, ib = 1.f;
        if (!normaliser) v = a.v_f32 ? reinterpret_cast<const float*>(a.v)[at] : to_f32(reinterpret_cast<const __nv_bfloat16*>(a.v)[at]);
        if constexpr (MODE == MLSTM) {
            const float2 g = log_gates<CT>(a, t, h);
            const float next = fmaxf(g.y + m, g.x);
            fa = expf(g.y + m - next); ib = expf(g.x - next);
            m = next;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const bool in = ch + i < a.D;                                             // (padded channels have keys and decays of zero)
            const size_t kat = (size_t)t * a.ld_qk + h * a.D + ch + i;
            const float k = !in ? 0.f : MODE == RET ? reinterpret_cast<const float*>(a.k)[kat] : to_f32(reinterpret_cast<const __nv_bfloat16*>(a.k)[kat]);
            if constexpr (MODE == WKV) fa = in ? a.decay[(size_t)t * a.H * a.D + h * a.D + ch + i] : 0.f;
            const float bk = ib * k;
            S[i] = fmaf(fa, S[i], normaliser ? bk : bk * v);
        }
    }
    if constexpr (MODE == MLSTM) {
        const float f = expf(m - m_end);
#pragma unroll
        for (int i = 0; i < 4; ++i) S[i] *= f;
    }
    return make_float4(S[0], S[1], S[2], S[3]);
}

// the read-outs of a chunk and head, the block's first 128 threads (all of them call): a thread per value column, eight key channels of its state at a time over all tokens.  `sm`: 7 * CT
// floats of shared memory that nothing else uses any more
template <int MODE, int CT, typename VT>
__device__ __forceinline__ void walk_out(const ChunkArgs& a, size_t unit, int t0, int n, int h, float* sm) {
    using QT = typename std::conditional<MODE == RET, float, __nv_bfloat16>::type;
    const QT* qp = reinterpret_cast<const QT*>(a.q) + (size_t)t0 * a.ld_qk + h * a.D;
    const QT* kp = reinterpret_cast<const QT*>(a.k) + (size_t)t0 * a.ld_qk + h * a.D;
    const VT* vp = reinterpret_cast<const VT*>(a.v) + (size_t)t0 * a.ld_v + h * a.Dv;
    const size_t ld_o = (size_t)a.H * a.Dv;
    float* op = a.out + (size_t)t0 * ld_o + h * a.Dv;
    const int tid = threadIdx.x;
    float* gate = sm;                                                                 // mlstm: [CT][3] state decay, input weight, e^-m
    float* den = sm + 3 * CT;                                                         // mlstm: [4][CT] the warps' shares of n . q
    if constexpr (MODE == MLSTM) {
        if (tid == 0) {
            double m = (double)a.mm[unit].x;                                           // (in 64 bits, as the chunks have it: over 128 tokens it drifts otherwise)
#pragma unroll 1
            for (int t = 0; t < n; ++t) {
                const float2 g = log_gates<CT>(a, t0 + t, h);
                const double next = fmax((double)g.y + m, (double)g.x);
                gate[3 * t] = expf((float)((double)g.y + m - next)); gate[3 * t + 1] = expf((float)((double)g.x - next)); gate[3 * t + 2] = expf((float)-next);
                m = next;
            }
        }
        __syncthreads();
        float nv = tid < a.Dpad ? a.aux[unit * a.Dpad + tid] : 0.f;
#pragma unroll 1
        for (int t = 0; t < n; ++t) {
            const float k = tid < a.D ? to_f32(kp[(size_t)t * a.ld_qk + tid]) : 0.f, q = tid < a.D ? to_f32(qp[(size_t)t * a.ld_qk + tid]) * a.qscale : 0.f;
            nv = fmaf(gate[3 * t], nv, gate[3 * t + 1] * k);
            const float p = warp_sum(tid < a.Dpad ? nv * q : 0.f);
            if ((tid & 31) == 0 && tid < 128) den[(tid >> 5) * CT + t] = p;
        }
        __syncthreads();
    }
    for (int dv = tid < 128 ? tid : a.Dv; dv < a.Dv; dv += 128) {
#pragma unroll 1
        for (int c0 = 0; c0 < a.Dpad; c0 += 8) {
            const bool in = c0 < a.D;                                                 // (both are multiples of 8)
            float S[8];
            load8(a.part + (unit * a.Dv + dv) * a.Dpad + c0, true, S);
#pragma unroll 1
            for (int t = 0; t < n; ++t) {
                float k[8], q[8], acc = 0.f;
                load8(kp + (size_t)t * a.ld_qk + c0, in, k);
                load8(qp + (size_t)t * a.ld_qk + c0, in, q);
                const float v = to_f32(vp[(size_t)t * a.ld_v + dv]);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if constexpr (MODE == WKV) {
                        const float kv = k[i] * v;
                        acc = fmaf(q[i], fmaf(in ? a.u[h * a.D + c0 + i] : 0.f, kv, S[i]), acc);
                        S[i] = fmaf(in ? a.decay[(size_t)(t0 + t) * a.H * a.D + h * a.D + c0 + i] : 0.f, S[i], kv);
                    } else {
                        S[i] = MODE == RET ? fmaf(a.decay[h], S[i], k[i] * v) : fmaf(gate[3 * t], S[i], gate[3 * t + 1] * k[i] * v);
                        acc = fmaf(S[i], MODE == MLSTM ? q[i] * a.qscale : q[i], acc);
                    }
                }
                float* o = op + (size_t)t * ld_o + dv;
                if (c0 > 0) acc += *o;
                if (MODE == MLSTM && c0 + 8 >= a.Dpad)
                    acc /= fmaxf(fabsf((den[t] + den[CT + t]) + (den[2 * CT + t] + den[3 * CT + t])), gate[3 * t + 2]) + 1e-6f;
                *o = acc;
            }
        }
    }
}

// ---- normalised and gated read-outs: o * weight / rms(o over the head) * act(gate), 32-bit until the result is rounded to bfloat16 (2^-9; gates are
// good to 2^-21 down to -87 and end there, 1 / rms to two units in the last place)
__device__ __forceinline__ float inverse_rms(const ChunkArgs& a, float squares) { return rsqrtf(squares / (float)a.Dv + a.eps); }
__device__ __forceinline__ float gate_of(const ChunkArgs& a, float g) {
    const float s = sigmoid_close(g);
    return a.act == 0 ? g * s : s;
}
__device__ __forceinline__ uint32_t gated_pair(const ChunkArgs& a, float x, float y, float2 w, uint32_t gate) {
    const float2 g = unpack(gate);
    const __nv_bfloat162 p = __floats2bfloat162_rn(x * w.x * gate_of(a, g.x), y * w.y * gate_of(a, g.y));
    return *reinterpret_cast<const uint32_t*>(&p);
}
// the chunk's rows behind the walk, which leaves its read-outs in `out`; the whole block calls
__device__ __forceinline__ void gate_walked(const ChunkArgs& a, int t0, int n, int h) {
    __syncthreads();
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int r = threadIdx.x >> 5; r < n; r += blockDim.x >> 5) {
        const size_t at = ((size_t)(t0 + r) * a.H + h) * a.Dv;
        const __nv_bfloat16* gate = a.gate + (size_t)(t0 + r) * a.ld_gate + h * a.Dv;
        float ss = 0.f;
        for (int c = lane; c < a.Dv; c += 32) ss = fmaf(a.out[at + c], a.out[at + c], ss);
        const float inv = inverse_rms(a, warp_sum(ss));
        for (int c = lane; c < a.Dv; c += 32)
            a.y[at + c] = __float2bfloat16(a.out[at + c] * inv * (a.norm_w ? a.norm_w[h * a.Dv + c] : 1.f) * gate_of(a, __bfloat162float(gate[c])));
    }
}

// ---- the matrix memory's gates over a chunk: threads 0 .. CT - 1 (whole warps), thread = token.  F: inclusive sum of the log forget gates,
// x = i - F, X: inclusive maximum of x.  Tokens behind the chunk's n-th: F stays, x = -inf.  `ends` holds 2 * CT / 32 + 2 doubles in shared memory;
// the last two are F and X at the chunk's end.
template <int CT>
__device__ __forceinline__ void chunk_gates(const ChunkArgs& a, int t0, int n, int h, double* ends, double& F, double& x, double& X) {
    constexpr int W = CT / 32;
    const int j = threadIdx.x, lane = j & 31, warp = j >> 5;
    double f = 0.0, ig = -INFINITY;
    x = X = 0.0;
    if (j < n) {
        const float2 g = log_gates<CT>(a, t0 + j, h);
        ig = (double)g.x;
        f = (double)g.y;
    }
    F = f;
    if (j < CT) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const double y = __shfl_up_sync(0xffffffffu, F, o); if (lane >= o) F += y; }
        if (lane == 31) ends[warp] = F;
    }
    __syncthreads();
    if (j < CT) {
        for (int w = 0; w < W - 1; ++w) if (w < warp) F += ends[w];
        x = ig - F;
        X = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const double y = __shfl_up_sync(0xffffffffu, X, o); if (lane >= o) X = fmax(X, y); }
        if (lane == 31) ends[W + warp] = X;
    }
    __syncthreads();
    if (j < CT) for (int w = 0; w < W - 1; ++w) if (w < warp) X = fmax(X, ends[W + w]);
    if (j == CT - 1) { ends[2 * W] = F; ends[2 * W + 1] = X; }
    __syncthreads();
}

// ---- the chain between chunks
// A thread per four elements of a (request, head)'s state; the request's chunks of this pass one after the other, the next chunks'
// sums on their way meanwhile.  mlstm: the elements behind the state are the normaliser's.
template <int MODE, int CT>
__global__ void __launch_bounds__(CARRY) chunk_carry_kernel(const ChunkArgs a) {
    __shared__ float powers[2];
    TTIE_PDL_ENTRY();
    const int h = blockIdx.y, s = blockIdx.z;
    const int q0 = a.qsl[s], len = a.qsl[s + 1] - q0;
    const int base = q0 / CT + s;
    const int c_lo = max(0, a.slot_lo - base), c_hi = min((len + CT - 1) / CT, a.slot_lo + a.slots - base);
    if (c_lo >= c_hi) return;
    if (MODE == RET) {
        const int last = len - (c_hi - 1) * CT;
        if (threadIdx.x < 2) powers[threadIdx.x] = (float)power((double)a.decay[h], threadIdx.x == 0 ? CT : min(CT, last));
        __syncthreads();
    }
    const size_t row = state_row(a.slot_ids[s], a.state_rows);
    if (MODE == WKV && h == 0 && blockIdx.x == 0 && c_hi == (len + CT - 1) / CT) {     // the request's last input is the next step's previous token
        const __nv_bfloat16* x = reinterpret_cast<const __nv_bfloat16*>(a.x) + (size_t)(q0 + len - 1) * a.ld_x;
        float* p = a.prev + (size_t)state_row(a.slot_ids[s], a.prev_rows) * a.d;
        for (int i = threadIdx.x; i < a.d; i += blockDim.x) p[i] = to_f32(x[i]);
    }
    const int state = a.Dv * a.Dpad;
    const int e = (blockIdx.x * CARRY + threadIdx.x) * 4;
    if (e >= state + (MODE == MLSTM ? a.Dpad : 0)) return;
    const bool in_state = e < state;                                                  // (only mlstm has elements behind it)
    float* sp = in_state ? a.S + (row * a.H + h) * state + e : a.nrm + (row * a.H + h) * a.Dpad + (e - state);
    float* pp = in_state ? a.part + e : a.aux + (e - state);
    const size_t step = (size_t)a.H * (in_state ? state : a.Dpad);
    const size_t unit = (size_t)(base + c_lo - a.slot_lo) * a.H + h;                  // of chunk c_lo
    pp += (in_state ? state : a.Dpad) * unit;
    float4 S = *reinterpret_cast<const float4*>(sp);
    // the running maximum as the request's state row has it; every CTA reads the row here, so the new one is written by chunk_out
    double m = MODE == MLSTM ? (double)a.mx[row * a.H + h] : 0.0;
    // two batches of chunks in registers: the next one's sums are on their way while this one is worked off
    constexpr int AHEAD = MODE == RET ? 8 : 4;
    float4 p[2][AHEAD], w[2][MODE == WKV ? AHEAD : 1], wl[2][MODE == WKV ? AHEAD : 1];
    double2 sc[2][MODE == MLSTM ? AHEAD : 1];
    auto fetch = [&](int b, int c0) {
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            if (c0 + i >= c_hi) continue;
            const size_t off = (size_t)(c0 + i - c_lo);
            p[b][i] = *reinterpret_cast<const float4*>(pp + off * step);
            if constexpr (MODE == WKV) {
                const float* f = a.aux + 2 * (unit + off * a.H) * a.Dpad + e % a.Dpad;
                w[b][i] = *reinterpret_cast<const float4*>(f);
                wl[b][i] = *reinterpret_cast<const float4*>(f + a.Dpad);
            }
            if constexpr (MODE == MLSTM) sc[b][i] = a.span[unit + off * a.H];
        }
    };
    auto work = [&](int b, int c0) {
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            if (c0 + i >= c_hi) continue;
            const size_t off = (size_t)(c0 + i - c_lo);
            *reinterpret_cast<float4*>(pp + off * step) = S;
            const float4 before = S;
            const double m_before = m;
            float4 f, x = p[b][i];
            if constexpr (MODE == RET) {
                const float d = powers[c0 + i == c_hi - 1 ? 1 : 0];
                f = make_float4(d, d, d, d);
            } else if constexpr (MODE == WKV) {
                f = w[b][i];
                const float4 l = wl[b][i];
                x = make_float4(fmaf(l.x, S.x, x.x), fmaf(l.y, S.y, x.y), fmaf(l.z, S.z, x.z), fmaf(l.w, S.w, x.w));
            } else {
                const double next = (double)(float)(sc[b][i].x + fmax(m, sc[b][i].y));      // as the state row will hold it
                const float d = expf((float)(sc[b][i].x + m - next)), own = expf((float)(sc[b][i].x + sc[b][i].y - next));
                f = make_float4(d, d, d, d);
                x = make_float4(x.x * own, x.y * own, x.z * own, x.w * own);
                if (e == 0) a.mm[unit + off * a.H] = make_float2((float)m, (float)next);
                m = next;
            }
            S.x = fmaf(f.x, S.x, x.x); S.y = fmaf(f.y, S.y, x.y); S.z = fmaf(f.z, S.z, x.z); S.w = fmaf(f.w, S.w, x.w);
            if (!finite4(S.x, S.y, S.z, S.w)) {
                const int el = in_state ? e : e - state;
                S = walk_state<MODE, CT>(a, q0 + (c0 + i) * CT, min(CT, len - (c0 + i) * CT), h, in_state ? el / a.Dpad : 0, el % a.Dpad, !in_state, before, (float)m_before, (float)m);
            }
        }
    };
    fetch(0, c_lo);
    for (int c0 = c_lo; c0 < c_hi; c0 += 2 * AHEAD) {
        fetch(1, c0 + AHEAD);
        work(0, c0);
        fetch(0, c0 + 2 * AHEAD);
        work(1, c0 + AHEAD);
    }
    *reinterpret_cast<float4*>(sp) = S;
}

}  // namespace chunks

// matrix_chunks_tc.cu: retention (mode 0) and the matrix memory (1), bfloat16 values of at most 128 columns
int matrix_chunks_tc(int mode, chunks::ChunkArgs a, int T, int slots, cudaStream_t st);
}  // namespace ttie

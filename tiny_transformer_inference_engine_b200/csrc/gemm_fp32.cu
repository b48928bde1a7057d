// True 32-bit matrix product for the float32 path: C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]).
// Plain FFMA with float32 accumulation.  Any M, N, K; larger products of aligned operands run on the tensor cores with three
// bfloat16 a value and a smaller error (gemm_fp32_tc.cu; the rule is the caller's, ops/__init__.py).
// Two kernels: tiles of 64 x 128 or 64 x 64 for prompt portions, and for up to 16 rows (decode steps) a form that streams the weight
// matrix once: a warp owns four weight rows at a time, its lanes walk K in 16-byte steps, and the activations - a few
// rows that every warp reads - come through the cache.
#include "common.cuh"
using namespace ttie;

namespace {
// ---- the tile form.  What bounds it is the FMA pipe (74 TFLOP/s nominal), so everything else has to hide behind it: a thread
// owns 8 x 8 outputs (one shared-memory load of 16 bytes feeds 16 multiply-adds), both operands lie in shared memory as they
// do in memory, K along the row, so that they travel as asynchronous 16-byte copies through three stages without a register or
// a transposition in between, and a load's four values along K are two pairs for the packed multiply-add.  Accumulators are
// pairs too (even and odd K), added at the end.  Rows are 20 floats apart: the eight rows that a warp reads at once fall into
// different banks.  Too few tiles for the GPU: a cluster of CTAs shares a tile, each walks a range of K, and the partial tiles
// are added through distributed shared memory in the order of the ranges.  Two widths: 64 columns (8 x 4 outputs) where a 128-wide tile would be
// half empty or, with few tiles and a K too short to cut, the whole time is one tile's: us, 64 columns | 128, 300 rows of K 64 to N 2,048 7.0 | 7.6,
// of K 128 to N 128 8.0 | 12.1, of K 2,048 to N 64 15.3 | 22.5, 32 products of [2,048, 128] with [64, 128] 33 | 59.
// 300 rows times [2304, 2048], [2048, 2048], [16384, 2048] and [2048, 8192] (36 GFLOP): 1,121 us, 32 TFLOP/s; 2,393 us as a 64 x 64
// tile of 4 x 4 outputs staged through registers.
constexpr int BM = 64, BK = 16, PITCH = BK + 4, STAGES = 3, MAX_RANGES = 8;

__device__ __forceinline__ void fma_pair(float2& d, float2 a, float2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
}

// VEC: rows start on 16 bytes and K is a multiple of 4, so a row travels in 16-byte copies; else value by value.
template <bool VEC>
__device__ __forceinline__ void stage_operand(float* dst, const float* src, int ld, int rows, int row0, int row_end, int k0, int k_end) {
    constexpr int W = VEC ? 4 : 1, PER_ROW = BK / W;
    for (int e = threadIdx.x; e < rows * PER_ROW; e += 128) {
        const int r = e / PER_ROW, k = (e % PER_ROW) * W;
        const bool in = row0 + r < row_end && k0 + k < k_end;
        const float* p = in ? src + (size_t)(row0 + r) * ld + k0 + k : src;        // (nothing is read where the size is 0)
        const unsigned d = (unsigned)__cvta_generic_to_shared(dst + r * PITCH + k);
        if (VEC) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(d), "l"(p), "r"(in ? 16 : 0) : "memory");
        else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" :: "r"(d), "l"(p), "r"(in ? 4 : 0) : "memory");
    }
}

// TN: columns per thread (8 rows); a tile has 16 TN columns
template <bool VEC, int TN>
__global__ void __launch_bounds__(128, TN == 8 ? 2 : 3)
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                float* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc,
                long long batch_a, long long batch_w, long long batch_c, int ranges, int range_len) {
    constexpr int BN = 16 * TN, STAGE_FLOATS = (BM + BN) * PITCH;
    static_assert(STAGES * STAGE_FLOATS >= BM * BN, "the stages hold a partial tile at the end");
    __shared__ __align__(16) float smem[STAGES * STAGE_FLOATS];           // 46,080 bytes (TN 8), 30,720
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = blockIdx.x % ranges;                                                 // clusters are consecutive CTAs along x
    A += blockIdx.z * batch_a; W += blockIdx.z * batch_w; C += blockIdx.z * batch_c;      // (a batch of products: grid z)
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x / ranges * BN;
    const int k_lo = rank * range_len, k_hi = min(K, k_lo + range_len);
    const int tm = (warp >> 1) * 32 + (lane >> 3), tn = (warp & 1) * 8 * TN + (lane & 7);     // the thread's rows tm + 4 i, columns tn + 8 j
    float2 acc[8][TN];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
    const int steps = (k_hi - k_lo + BK - 1) / BK;
    auto stage = [&](int it) {
        if (it < steps) {
            float* s = smem + it % STAGES * STAGE_FLOATS;
            stage_operand<VEC>(s, A, lda, BM, m0, M, k_lo + it * BK, k_hi);
            stage_operand<VEC>(s + BM * PITCH, W, ldw, BN, n0, N, k_lo + it * BK, k_hi);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int it = 0; it < STAGES - 1; ++it) stage(it);
    for (int it = 0; it < steps; ++it) {
        asm volatile("cp.async.wait_group %0;" :: "n"(STAGES - 2) : "memory");
        __syncthreads();                                              // this step's rows are there, and everyone is done with the stage refilled next
        stage(it + STAGES - 1);
        const float* as = smem + it % STAGES * STAGE_FLOATS + tm * PITCH;
        const float* ws = smem + it % STAGES * STAGE_FLOATS + (BM + tn) * PITCH;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 a[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float4*>(as + 4 * i * PITCH + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const float4 w = *reinterpret_cast<const float4*>(ws + 8 * j * PITCH + k);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    fma_pair(acc[i][j], make_float2(a[i].x, a[i].y), make_float2(w.x, w.y));
                    fma_pair(acc[i][j], make_float2(a[i].z, a[i].w), make_float2(w.z, w.w));
                }
            }
        }
    }
    if (ranges == 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int gm = m0 + tm + 4 * i;
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int gn = n0 + tn + 8 * j;
                if (gm < M && gn < N) C[(size_t)gm * ldc + gn] = acc[i][j].x + acc[i][j].y + (bias ? bias[gn] : 0.f);
            }
        }
        return;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                                  // the stages are free: they take the partial tile
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) smem[(tm + 4 * i) * BN + tn + 8 * j] = acc[i][j].x + acc[i][j].y;
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(smem);
    for (int e = rank * 128 + tid; e < BM * BN / 4; e += ranges * 128) {
        const int gm = m0 + e / (BN / 4), gn = n0 + e % (BN / 4) * 4;
        if (gm >= M || gn >= N) continue;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        for (int r = 0; r < ranges; ++r) {
            uint32_t remote;
            float p[4];
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(mine + e * 16), "r"(r));
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(p[0]), "=f"(p[1]), "=f"(p[2]), "=f"(p[3]) : "r"(remote) : "memory");
#pragma unroll
            for (int c = 0; c < 4; ++c) v[c] += p[c];
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (gn + c < N) C[(size_t)gm * ldc + gn + c] = v[c] + (bias ? bias[gn + c] : 0.f);
    }
    // no CTA leaves while its tile is read.  (Not the .aligned form, which every lane of a warp has to reach together: at the tiles' edges lanes
    // come out of the loop at different times)
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}

int launch_tiles(const float* A, const float* W, const float* bias, float* C, int B, int M, int N, int K, int lda, int ldw, int ldc,
                 long long batch_a, long long batch_w, long long batch_c, cudaStream_t s) {
    const long long wide_tiles = (long long)B * ceil_div(M, BM) * ceil_div(N, 128), slots = 2LL * num_sms();
    const bool narrow = N <= 64 || (K <= 240 && wide_tiles <= num_sms());
    const int BN = narrow ? 64 : 128;
    const long long tiles = (long long)B * ceil_div(M, BM) * ceil_div(N, BN);
    // K ranges per tile: the fewest waves of two CTAs per SM times a wave's length, a range's fixed cost taken as 64 values of K
    // (filling the stages) and 48 more for adding the partial tiles.  [300, 2048] x [2304, 2048]: 90 tiles alone leave half
    // of the SMs' places empty.
    int ranges = 1;
    long long best = -1;
    for (int r = 1; r <= MAX_RANGES; ++r) {
        const int len = ceil_div(ceil_div(K, r), BK) * BK;
        if (r > 1 && (len < 128 || ceil_div(K, len) != r)) continue;
        const long long cost = (tiles * r + slots - 1) / slots * (len + 64 + (r > 1 ? 48 : 0));
        if (best < 0 || cost < best) { best = cost; ranges = r; }
    }
    const int range_len = ceil_div(ceil_div(K, ranges), BK) * BK;
    const dim3 grid(ceil_div(N, BN) * ranges, ceil_div(M, BM), B);
    const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && batch_a % 4 == 0 && batch_w % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    // (an ordinary launch, as the tile kernel always was: it reads its operands from the first instruction on)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = dim3(128); cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ranges; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = ranges > 1 ? 1 : 0;
    auto launch = [&](auto kernel) { return cudaLaunchKernelEx(&cfg, kernel, A, W, bias, C, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c, ranges, range_len); };
    const cudaError_t e = narrow ? (vec ? launch(gemm_f32_kernel<true, 4>) : launch(gemm_f32_kernel<false, 4>))
                                 : (vec ? launch(gemm_f32_kernel<true, 8>) : launch(gemm_f32_kernel<false, 8>));
    if (e != cudaSuccess) TTIE_FAIL("gemm_f32: launch failed: %s", cudaGetErrorString(e));
    return 0;
}

// ---- up to 16 activation rows.  acc[m][r]: lane-partial dot product of activation row m with weight row r of the warp's
// four; the lanes' partial sums are added by shuffles in a fixed order.  Rows of 4-element-aligned length and stride only.
constexpr int GV_WARPS = 8, GV_ROWS = 4;
template <int MT>
__global__ void __launch_bounds__(GV_WARPS * 32, MT <= 8 ? 3 : 1)     // (a long matrix streams best with many warps per SM)
gemv_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                float* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = (blockIdx.x * GV_WARPS + warp) * GV_ROWS;
    if (n0 >= N) return;
    const float* wrow[GV_ROWS];
#pragma unroll
    for (int r = 0; r < GV_ROWS; ++r) wrow[r] = W + (size_t)min(n0 + r, N - 1) * ldw;       // (a row past the end repeats the last one; it is not stored)
    float acc[MT][GV_ROWS];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int r = 0; r < GV_ROWS; ++r) acc[m][r] = 0.f;
    TTIE_PDL_ENTRY();
#pragma unroll(MT <= 4 ? 2 : 1)
    for (int k = lane * 4; k < K; k += 128) {
        float4 w[GV_ROWS];
#pragma unroll
        for (int r = 0; r < GV_ROWS; ++r) w[r] = __ldcs(reinterpret_cast<const float4*>(wrow[r] + k));   // streamed once
        // all activation loads of the step are asked for at once (a row past the last repeats it and is not stored): every
        // one of them is new to this SM's cache, and one after the other they would cost a trip to L2 each
        float4 x[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) x[m] = __ldg(reinterpret_cast<const float4*>(A + (size_t)min(m, M - 1) * lda + k));
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int r = 0; r < GV_ROWS; ++r)
                acc[m][r] = fmaf(x[m].w, w[r].w, fmaf(x[m].z, w[r].z, fmaf(x[m].y, w[r].y, fmaf(x[m].x, w[r].x, acc[m][r]))));
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int r = 0; r < GV_ROWS; ++r) {
            float v = acc[m][r];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            acc[m][r] = v;
        }
    if (lane == 0) {
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int r = 0; r < GV_ROWS; ++r)
                if (m < M && n0 + r < N) C[(size_t)m * ldc + n0 + r] = acc[m][r] + (bias ? bias[n0 + r] : 0.f);
    }
}

template <int MT>
int launch_gemv(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t s) {
    TTIE_LAUNCH(gemv_f32_kernel<MT>, ceil_div(N, GV_WARPS * GV_ROWS), GV_WARPS * 32, 0, s, A, W, bias, C, M, N, K, lda, ldw, ldc);
    TTIE_CHECK_LAUNCH("gemm_f32 (few rows)");
    return 0;
}
}  // namespace

extern "C" int ttie_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K,
                             int lda, int ldw, int ldc, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) TTIE_FAIL("gemm_f32: K must be positive, got %d", K);
    if (M <= 32 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0) {
        cudaStream_t s = (cudaStream_t)stream;
        if (M <= 2) return launch_gemv<2>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
        if (M <= 4) return launch_gemv<4>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
        if (M <= 8) return launch_gemv<8>(A, W, bias, C, M, N, K, lda, ldw, ldc, s);
        // 17 to 32 rows: twice 16 (measured against the tile kernel at 32 rows: 13 against 38 us on a [512, 512] matrix,
        // 137 against 170 on [50257, 512])
        for (int m0 = 0; m0 < M; m0 += 16) {
            const int rc = launch_gemv<16>(A + (size_t)m0 * lda, W, bias, C + (size_t)m0 * ldc, M - m0 < 16 ? M - m0 : 16, N, K, lda, ldw, ldc, s);
            if (rc) return rc;
        }
        return 0;
    }
    if (ceil_div(M, BM) > 65535) TTIE_FAIL("gemm_f32: M=%d too large for one launch", M);
    return launch_tiles(A, W, bias, C, 1, M, N, K, lda, ldw, ldc, 0, 0, 0, (cudaStream_t)stream);
}

// A batch of products of one shape: C[b] = A[b] * W[b]^T, the operands of batch b at b * batch_a / batch_w / batch_c elements
// (per-head and per-block weights: strided views of one activation matrix on the A side).
extern "C" int ttie_gemm_f32_batched(const float* A, const float* W, float* C, int B, int M, int N, int K, long long lda,
                                     long long ldw, long long ldc, long long batch_a, long long batch_w, long long batch_c,
                                     void* stream) {
    if (B <= 0 || M <= 0 || N <= 0) return 0;
    if (K <= 0) TTIE_FAIL("gemm_f32_batched: K must be positive, got %d", K);
    if (ceil_div(M, BM) > 65535 || B > 65535) TTIE_FAIL("gemm_f32_batched: M=%d, B=%d too large for one launch", M, B);
    return launch_tiles(A, W, nullptr, C, B, M, N, K, (int)lda, (int)ldw, (int)ldc, batch_a, batch_w, batch_c, (cudaStream_t)stream);
}

// Instructions of the 5th-generation tensor cores and of barriers in shared memory, and the error word, for the kernels that are written with
// them directly (gemm_fp32_tc.cu, gemm_skinny.cu, matrix_chunks_tc.cu).
#pragma once
#include <cuda.h>
#include "common.cuh"

namespace ttie {
// gemm_tcgen05.cu: the product kernels' error word and its mirror; tensor maps of rows and of blocks of 64 columns
int gemm_tc_error_words(int** word, int** mirror);
int gemm_tc_make_map_of(CUtensorMap* map, int f32, const void* base, long long rows, long long cols, long long ld, int box_cols, int box_rows);
int gemm_tc_make_block_map(CUtensorMap* map, const void* base, long long rows, long long blocks, long long ld, int box_rows, int box_blocks);

namespace tc {
constexpr long long WAIT_CYCLES = 2000000000LL;                  // about one second
struct ErrorWords { int *word, *mirror; };

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// false: the phase did not come within the limit; the code is recorded.  quits: the limit is over at once (tests of giving up)
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int code, const ErrorWords& e, bool quits = false) {
    if (!quits && mbar_try(bar, parity)) return true;
    const long long deadline = clock64() + WAIT_CYCLES;
    while (quits || !mbar_try(bar, parity)) {
        if (quits || clock64() > deadline) {
            atomicCAS(e.word, 0, code);
            if (e.mirror) { *reinterpret_cast<volatile int*>(e.mirror) = code; __threadfence_system(); }
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
// the loads before have arrived (the values pass through, so that nothing that uses them moves ahead of this)
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]) :: "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
}  // namespace tc
}  // namespace ttie

// Device and host helpers shared by the tcgen05 kernels: mbarriers, TMA loads, tensor-memory access,
// UMMA issue and descriptors, int8 -> bf16 dequantisation, tensor maps.
#pragma once

#include "q3t_common.cuh"

#include <cuda.h>

namespace q3t {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// 1 if that phase is complete; does not wait
__device__ __forceinline__ uint32_t mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok;
}

// One lane of a converged warp.  Unlike a test of the lane index, this tells the compiler that
// the code below runs in exactly one thread, which the instructions that take their operands
// from uniform registers (TMA copies, MMA issue) need in order to be emitted without a loop
// over the active lanes.
__device__ __forceinline__ bool elect_one() {
    uint32_t chosen;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(chosen));
    return chosen != 0;
}

// Shared by all roles of a CTA: deadline and an abort flag that turns every later wait into a no-op.
struct Guard {
    unsigned long long deadline;
    volatile int* abort_flag;
    __device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity) const {
        // the clock is read once per 1024 polls: a read of the global timer costs about as much
        // as a whole pipeline stage
        uint32_t polls = 0;
        while (!mbar_try_wait(bar, parity)) {
            if ((++polls & 63u) != 0) continue;
            if (*abort_flag) return false;
            if ((polls & 1023u) == 0 && now_ns() > deadline) {
                *abort_flag = 1;
                return false;
            }
        }
        return true;
    }
};

// How many steps have all of their operands, for the thread that issues the products.  A look at a barrier costs 110 cycles even
// when it is complete (200 and more at cluster scope), twice a step, and the tensor cores' queue holds only a few products;
// a thread of its own looks at the barriers, and the issuing one at a word.
__device__ __forceinline__ void publish_steps(uint32_t* word, uint32_t steps) {
    asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_u32(word)), "r"(steps) : "memory");
}
__device__ __forceinline__ uint32_t published_steps(const uint32_t* word) {
    uint32_t steps;
    asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(steps) : "r"(smem_u32(word)) : "memory");
    return steps;
}
// until `word` has passed `step`; `seen` is what it was at the last look
__device__ __forceinline__ bool await_step(const Guard& g, const uint32_t* word, uint32_t step, uint32_t& seen) {
    uint32_t polls = 0;
    while (seen <= step) {
        seen = published_steps(word);
        if (seen > step) break;
        if ((++polls & 255u) != 0) continue;
        if (*g.abort_flag) return false;
        if ((polls & 16383u) == 0 && now_ns() > g.deadline) {
            *g.abort_flag = 1;
            return false;
        }
    }
    return true;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// a tensor map is 128 bytes of kernel parameters that the first copy would otherwise wait for
__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// Hardware barrier over every thread of the cluster (one CTA per K-slice of a channel tile).
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// address of the same shared-memory location in the CTA of another rank of the cluster
__device__ __forceinline__ uint32_t peer_smem(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
// the two halves of cluster_sync(); a thread that has exited counts as arrived
// (relaxed: what it announces, barriers set up, has its own fence, and a release would wait for loads in flight)
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// sixteen bytes to another CTA's shared memory, counted on an mbarrier of that CTA
__device__ __forceinline__ void st_async_v4(uint32_t addr, float a, float b, float c, float d, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar) : "memory");
}

// K-major, 128-byte-swizzled operand tile: rows at a 128-byte pitch, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

// A (128 x 16 bf16) from TMEM columns, B from shared memory
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}

// 32 consecutive columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_store_32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr),
          "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
          "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
          "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(smem_u32(bar)) : "memory");
}


// Four int8 (one word) -> four bf16 (two words), exact.  Behind the byte 0x43 the low seven bits of a weight read as
// 128 + those bits, and its sign bit alone as 128 or, set, 256: their difference is the weight.  Six integer instructions
// and two subtractions; by way of fp32 (2^23 + byte, minus the bias, high halves) it was seven and two, and the integer
// pipe bounds a step of the skinny GEMM (16 projections of 48 rows 123.9 against 119.9 us).
__device__ __forceinline__ void dequant4(uint32_t word, uint32_t& lo, uint32_t& hi) {
    const uint32_t p = __byte_perm(word, 0x43434343u, 0x4140), q = __byte_perm(word, 0x43434343u, 0x4342);
    asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(lo) : "r"(p & 0xff7fff7fu), "r"(p & 0xff80ff80u));
    asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(hi) : "r"(q & 0xff7fff7fu), "r"(q & 0xff80ff80u));
}

// Keeps the computation of these values ahead of what follows (the compiler would move it behind a wait, next to the store).
__device__ __forceinline__ void compute_now(uint32_t (&r)[32]) {
#pragma unroll
    for (int i = 0; i < 32; ++i) asm volatile("" : "+r"(r[i]));
}

// NCOL consecutive fp32 accumulator columns of this thread's TMEM lane
template <int NCOL>
__device__ __forceinline__ void tmem_load_row(uint32_t taddr, float (&v)[NCOL]) {
#pragma unroll
    for (int c = 0; c < NCOL; c += 8) {
        uint32_t r[8];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
            : "r"(taddr + c));
#pragma unroll
        for (int i = 0; i < 8; ++i) v[c + i] = __uint_as_float(r[i]);
    }
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---- host side ---------------------------------------------------------------------------------

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                 CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                 CUtensorMapFloatOOBfill);

inline EncodeTiled encode_tiled() {
    static EncodeTiled fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &result) != cudaSuccess
            || result != cudaDriverEntryPointSuccess) {
            p = nullptr;
        }
        return reinterpret_cast<EncodeTiled>(p);
    }();
    return fn;
}

inline bool make_map(CUtensorMap* map, CUtensorMapDataType type, const void* base, uint64_t inner, uint64_t outer,
              uint64_t row_bytes, uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle swizzle) {
    EncodeTiled fn = encode_tiled();
    if (fn == nullptr) return false;
    const cuuint64_t dims[2] = {inner, outer};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {box_inner, box_outer};
    const cuuint32_t elem[2] = {1, 1};
    return fn(map, type, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace tc
}  // namespace q3t

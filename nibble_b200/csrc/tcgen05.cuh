// Shared pieces of the kernels on the 5th-generation tensor cores: mbarriers with bounded waits, operand descriptors, the
// MMA and its commits, tensor maps.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace w4a16 {

// Status word of the tensor-core kernels: set when a bounded wait gives up (which barrier: low byte).  One per library,
// defined in linear_gemm.cu; kernels of other files get its address as a parameter.
unsigned* tcgen05_status_address();

namespace {

constexpr unsigned kSpinLimit = 1u << 20;

__device__ __forceinline__ unsigned smem_u32(const void* p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Bounded wait for the phase with the given parity to complete.  False (and a status code) on give-up.  `kCluster`: of a barrier at
// which threads or copies of the cluster's other CTAs arrive.
template <bool kCluster = false>
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, unsigned code, unsigned* status) {
    for (unsigned spin = 0; spin < kSpinLimit; ++spin) {
        unsigned done;
        if constexpr (kCluster) {
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(bar), "r"(parity)
                : "memory");
        } else {
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(bar), "r"(parity)
                : "memory");
        }
        if (done) return true;
    }
    atomicMax(status, code);
    return false;
}
// Whether that phase has completed, without waiting.
template <bool kCluster = false>
__device__ __forceinline__ bool mbar_test(unsigned bar, unsigned parity) {
    unsigned done;
    if constexpr (kCluster) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
    }
    return done != 0;
}

// Shared-memory operand descriptor: K-major tile, 128-byte swizzle, rows 128 bytes apart, 8-row
// groups 1024 bytes apart, descriptor version 1 (sm_100).
__device__ __forceinline__ uint64_t operand_desc(unsigned smem_address) {
    uint64_t desc = (smem_address & 0x3FFFFu) >> 4;   // start address, 16-byte units
    desc |= static_cast<uint64_t>(1) << 16;           // leading byte offset (unused with swizzle): 1
    desc |= static_cast<uint64_t>(1024 >> 4) << 32;   // stride byte offset between 8-row groups
    desc |= static_cast<uint64_t>(1) << 46;           // version
    desc |= static_cast<uint64_t>(2) << 61;           // SWIZZLE_128B
    return desc;
}

// D (TMEM) += A (TMEM) x B (shared memory).
__device__ __forceinline__ void umma_f16_tmem_a(unsigned tmem_d, unsigned tmem_a, uint64_t b_desc, uint32_t instr_desc,
                                                uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(instr_desc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// A 2-d tile copy into shared memory that counts its bytes on an mbarrier.
__device__ __forceinline__ void tma_load_2d(unsigned dst, const CUtensorMap* map, int x, int y, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// 16 columns of this thread's TMEM lane.  Load and wait are one statement: between two, the compiler could move (or spill)
// registers that have not arrived yet.
__device__ __forceinline__ void tmem_load16(unsigned address, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(address)
        : "memory");
}

// True in one lane of a converged warp, always the same one.
__device__ __forceinline__ bool elect_one() {
    uint32_t chosen;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(chosen));
    return chosen != 0;
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's tensor-map encoder, looked up through the runtime so that libcuda is not a link dependency.
inline EncodeTiledFn tensor_map_encoder() {
    static EncodeTiledFn fn = [] {
        void* entry = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &entry, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess) {
            entry = nullptr;
        }
        return reinterpret_cast<EncodeTiledFn>(entry);
    }();
    return fn;
}

// A row-major matrix [rows, row_bytes] seen as boxes of box_rows x box_bytes; rows past the end read as zero.
inline bool encode_rows(CUtensorMap* map, CUtensorMapDataType type, int element_bytes, const void* base, int64_t rows,
                        int64_t row_bytes, int box_bytes, int box_rows, CUtensorMapSwizzle swizzle,
                        CUtensorMapL2promotion promotion) {
    const EncodeTiledFn encode = tensor_map_encoder();
    if (encode == nullptr) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(row_bytes / element_bytes), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(row_bytes)};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_bytes / element_bytes), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t element_strides[2] = {1, 1};
    return encode(map, type, 2, const_cast<void*>(base), dims, strides, box, element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  swizzle, promotion, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace
}  // namespace w4a16

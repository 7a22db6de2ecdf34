// What the two GEMMs with weights in tensor memory share: codes to FP16 weights in memory order, and their way into TMEM.
#pragma once

#include <stdint.h>

#include "tcgen05.cuh"
#include "unpack.cuh"

namespace w4a16 {
namespace {

// One word of eight codes as four FP16 pairs in memory order, exact.  The byte that holds a pair is put into both halves
// under the exponent of 1024: its low nibble stays in the low half, its high nibble, 16 times as large, in the high one.
__device__ __forceinline__ void unpack8_ordered(uint32_t word, uint32_t* out) {
    constexpr uint32_t kSelect[4] = {0x4040u, 0x4141u, 0x4242u, 0x4343u};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t both = prmt(word, 0x64u, kSelect[i]);
        out[i] = hfma2_u32(and_xor(both, 0xFFF0FF0Fu, 0x00800008u), 0x2C003C00u, 0xD480E408u);   // x (1, 1/16) - (1032, 72)
    }
}

// The same times the scale, rounded once as half(code * scale) is, three instructions of sixteen fewer: the nibbles (code + 8) lie
// in bits 4..7 of halves whose other bits are zero, FP16 values of (code + 8) * 2^-20, and one FMA with scale * 2^20 and
// -8 * scale, both exact, gives the product.  For scales whose 2^20-fold FP16 can hold (weights of a group below 0.43).  8192 ->
// 28672, 64 rows: 45.9 -> 44.5 us; 8192 x 8192, 48 rows: 19.2 -> 18.6, 1024 rows: 116 -> 112.
__device__ __forceinline__ void unpack8_scaled(uint32_t word, uint32_t scale_2_20, uint32_t minus_8_scale, uint32_t* out) {
    constexpr uint32_t kSelect[4] = {0x4400u, 0x5511u, 0x6622u, 0x7733u};
    const uint32_t low = word << 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        out[i] = hfma2_u32(and_xor(prmt(low, word, kSelect[i]), 0x00F000F0u, 0x00800080u), scale_2_20, minus_8_scale);
    }
}
constexpr uint32_t kLargestScaled = 0x2BFFu;   // FP16 bits of the largest scale for it: 65504 / 2^20

// 16 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_store16(unsigned address, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(address), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
          "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Its two halves, by each thread for itself.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
}  // namespace
}  // namespace w4a16

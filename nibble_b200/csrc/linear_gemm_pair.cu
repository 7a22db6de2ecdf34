// W4A16 linear for prompts on pairs of SMs: the weights are dequantised into tensor memory (TMEM), as in linear_gemm.cu, and one
// MMA of the pair (cta_group::2) multiplies them by up to 256 batch rows, half of which each of the two SMs holds.
//
//   D[128 x BN] (TMEM of each SM, FP32)  +=  A[128 x 128] (its TMEM: FP16 weights)  x  B[BN x 128] (BN / 2 rows in each shared memory)
//
// Weights are half(code * scale), accumulated in FP32 over K: the arithmetic of dequantise-then-matmul.
//
// What bounds it.  At 256 batch rows the MMAs: 1021 of 1024 clocks a K block measured over a tile, and with that the power limit
// (8192 -> 28672, 2048 rows in long runs: 730 to 740 us; dequantise and cuBLAS 930 to 990, linear_gemm.cu 910 to 1060).  Against
// linear_gemm.cu a weight is dequantised half as often and a row of x is brought to half as many SMs, for the same MMAs; with a
// row of x in every SM, 256 batch rows would take 64 bytes a clock out of L2, more than it gives.  At small batches the chain of
// waits, unpacking and stores of the four dequantiser groups: 0.4 us a block.
//
// Roles of a CTA's 28 warps, one CTA per SM, two to a cluster:
//   warp 0        loads its half of x (TMA), one K block per ring slot, counted on the first CTA's barrier
//   warp 1        loads the packed codes of its 128 rows (TMA)
//   warp 2        of the first CTA: issues the pair's MMAs, whose commits reach both CTAs
//   warps 4-11    drain: two per quarter of the TMEM lanes
//   warps 12-27   dequantisers: four groups of four warps taking the K blocks in turn, a thread per weight row
// The second CTA's dequantisers arrive at the first one's barrier themselves: a warp that waited there and passed the word on, with
// the fence at cluster scope that a single arrival for all of them needs, took 0.7 us a block.
//
// A pair takes every 74th tile, whole.  So at any time the pairs work on neighbours: 9 batch tiles (kBand) by about 8 of N, whose x
// and weights come out of HBM once and are shared in L2.  When a pair took neighbouring tiles itself, the 74 read 74 different tiles
// of weights at a time, each again for every batch tile: 1.23 GB out of HBM at 2048 rows of 8192 -> 28672 instead of 0.17, which the
// power limit turned into time (in runs of 0.15 s 794 -> 737 us; 4096 rows 1618 -> 1463; 8192 rows of 8192 x 8192 927 -> 849;
// without bands the last two 1517 and 928; bands of 5 as these; 600 and 1024 rows unchanged).
//
// Tiles cut between pairs through a workspace, as linear_gemm.cu cuts them, were built as well: 0.07 % faster over 442 shapes, each
// by the better of the two.  There is room for one accumulator beside the weights, so the MMAs wait for a tile's drain, 3300 clocks
// of 69000 at K = 8192; with the dequantisers' help 2600, which no call showed.
//
// Every wait is bounded; one that gives up sets the status word and the CTA still runs to its end.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "gemm_weights.cuh"
#include "kernels.h"
#include "per_device.h"
#include "tcgen05.cuh"
#include "unpack.cuh"

namespace w4a16 {
namespace {

constexpr int kRows = 128;               // output channels of a CTA (TMEM lanes)
constexpr int kTileRows = 2 * kRows;     // ... and of a tile
constexpr int kBlockK = 128;             // K per pipeline block
constexpr int kRing = 8;                 // blocks the barriers tell apart
constexpr int kMaxCodeSlots = 8;
constexpr int kCodeBytes = kRows * kBlockK / 2;
constexpr int kMaxBatch = 256;           // batch rows per tile (MMA N)
constexpr int kSlotColumns = kBlockK / 2;             // TMEM columns of a block's weights
constexpr int kWeightColumn = kMaxBatch;
constexpr int kSlots = (512 - kWeightColumn) / kSlotColumns;
constexpr int kFirstDrainWarp = 4, kDrainWarps = 8;
constexpr int kFirstDequantWarp = kFirstDrainWarp + kDrainWarps;
constexpr int kDequantGroups = 4, kGroupWarps = 4;
constexpr int kShares = kDrainWarps / 4;                // warps that drain a quarter of the lanes
constexpr int kThreads = (kFirstDequantWarp + kDequantGroups * kGroupWarps) * 32;
constexpr int kBarrierBytes = 512;
constexpr int kPairs = 74;               // of a B200
constexpr int kBand = 9;                 // batch tiles side by side: 74 pairs then work on about as many tiles of N
constexpr int kSmem = 194 * 1024;        // as in linear_gemm.cu: leaves the L1 that keeps a tile's scales

struct PairParams {
    const __half* scales;
    __half* y;
    const __half* bias;
    unsigned* status;
    int M, N;
    int k_blocks;            // of one tile
    int bn, m_tiles;
    int x_slots, code_slots;
    int tiles;
    int band, band_tiles;    // batch tiles side by side, and tiles of that many batch tiles and all of N
};

// Where a tile is.  Pair i takes tiles i, i + pairs, ...: at any time the pairs work on neighbours.
struct Place {
    int n0, m0;
};
__device__ __forceinline__ Place place_of(const PairParams& p, int tile) {
    const int band = tile / p.band_tiles, in_band = tile - band * p.band_tiles;
    const int width = max(1, min(p.band, p.m_tiles - band * p.band)), n = in_band / width;       // (1 for a tile past the end)
    return {n * kTileRows, (band * p.band + in_band - n * width) * p.bn};
}

__device__ __forceinline__ unsigned first_cta_address(unsigned local) {
    unsigned remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote) : "r"(local));
    return remote;
}
// At a barrier of the first CTA, by threads of both.  What such an arrival hands over is tensor memory, never ordinary memory, and that is
// ordered by the tcgen05 fences either side of it and the arrival being seen; for threads of two CTAs that takes the scope of the
// cluster (the default is the CTA).  A release would wait for the scales that are on their way as well (2048 -> 12000, 96 rows: 10.7 ->
// 12.6 us; 1024 -> 8192, 1024 rows: 19.6 -> 21.4).
__device__ __forceinline__ void mbar_arrive_remote(unsigned bar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// A tile copy into this CTA's shared memory that counts its bytes on a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_pair(unsigned dst, const CUtensorMap* map, int x, int y, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t instr_desc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a), "l"(b_desc), "r"(instr_desc), "r"(accumulate)
        : "memory");
}
// Arrives at the barrier of both CTAs once all MMAs issued so far have finished.
__device__ __forceinline__ void commit_pair(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"(static_cast<uint16_t>(3))
                 : "memory");
}
template <int GROUP>
__global__ void __launch_bounds__(kThreads, 1)
linear_gemm_pair_kernel(const PairParams p, const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map) {
    constexpr int kScales = kBlockK / GROUP;                               // per row and K block
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const unsigned base = (smem_u32(smem_raw) + 1023u) & ~1023u;           // the same in both CTAs
    const unsigned x_half_bytes = static_cast<unsigned>(p.bn) * 64;        // 64 K of this CTA's batch rows, 128-byte swizzled
    auto x_slot = [&](int s) { return base + s * 2 * x_half_bytes; };
    const unsigned codes_ring = base + p.x_slots * 2 * x_half_bytes;
    auto code_slot = [&](int c) { return codes_ring + c * kCodeBytes; };
    const unsigned bars = codes_ring + p.code_slots * kCodeBytes;
    // The first CTA's counts for the pair: both halves of x have landed, and both CTAs' weights are in TMEM.
    auto full_bar = [&](int r) { return bars + r * 8; };
    auto done_bar = [&](int r) { return bars + (kRing + r) * 8; };         // the block's MMAs have finished
    auto codes_bar = [&](int c) { return bars + (2 * kRing + c) * 8; };
    auto codes_free_bar = [&](int c) { return bars + (2 * kRing + kMaxCodeSlots + c) * 8; };
    constexpr int kRingBars = 2 * kRing + 2 * kMaxCodeSlots;
    const unsigned acc_full_bar = bars + kRingBars * 8, acc_free_bar = bars + (kRingBars + 1) * 8;
    const unsigned tmem_word = bars + (kRingBars + 2) * 8;
    static_assert((kRingBars + 2) * 8 + 4 <= kBarrierBytes);

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int pair = static_cast<int>(blockIdx.x) >> 1, rank = static_cast<int>(blockIdx.x) & 1;
    const int pairs = static_cast<int>(gridDim.x) >> 1;
    const int blocks = (p.tiles - pair + pairs - 1) / pairs * p.k_blocks;

    if (tid == 0) {
        for (int r = 0; r < kRing; ++r) {
            mbar_init(full_bar(r), 2 * kGroupWarps + 1);       // the warps of one dequantiser group of each CTA, and x
            mbar_init(done_bar(r), 1);
        }
        for (int c = 0; c < p.code_slots; ++c) {
            mbar_init(codes_bar(c), 1);
            mbar_init(codes_free_bar(c), kGroupWarps);
        }
        mbar_init(acc_full_bar, 1);
        mbar_init(acc_free_bar, 2 * kDrainWarps);      // of both CTAs
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&x_map)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&w_map)) : "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tmem_word) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    if (warp == 1 && lane < p.code_slots && lane < blocks) {
        // the first codes travel to L2 while the kernel in front finishes (a prefetch cannot go stale there)
        const int ahead = lane / p.k_blocks;
        asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];"
                     ::"l"(reinterpret_cast<uint64_t>(&w_map)), "r"((lane - ahead * p.k_blocks) * (kBlockK / 2)),
                       "r"(place_of(p, pair + ahead * pairs).n0 + rank * kRows)
                     : "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_barrier();                                 // the other CTA's barriers are in place too
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    unsigned tmem;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_word));
    pdl_release_downstream();
    pdl_wait_for_upstream();

    const bool issuer = elect_one();
    const unsigned first_full = first_cta_address(full_bar(0));
    if (warp == 0) {                                   // ---- this CTA's half of x
        bool healthy = true;
        int xs = 0, tile = pair, kb = 0;
        int m0 = place_of(p, tile).m0 + rank * (p.bn / 2);
        for (unsigned it = 0; it < static_cast<unsigned>(blocks); ++it) {
            const unsigned r = it % kRing;
            if (it >= static_cast<unsigned>(p.x_slots)) {
                const unsigned old = it - p.x_slots;
                healthy = mbar_wait(done_bar(old % kRing), (old / kRing) & 1, 0x10u + r, p.status);
                healthy = __all_sync(0xffffffffu, healthy);
            }
            if (!healthy) break;
            if (issuer) {
                const int k = kb * kBlockK;
                if (rank == 0) mbar_arrive_expect_tx(full_bar(r), 4 * x_half_bytes);
                tma_load_pair(x_slot(xs), &x_map, k, m0, first_full + r * 8);
                tma_load_pair(x_slot(xs) + x_half_bytes, &x_map, k + 64, m0, first_full + r * 8);
            }
            __syncwarp();
            if (++xs == p.x_slots) xs = 0;
            if (++kb == p.k_blocks) {
                kb = 0;
                tile += pairs;
                m0 = place_of(p, tile).m0 + rank * (p.bn / 2);
            }
        }
    } else if (warp == 1) {                            // ---- packed codes
        bool healthy = true;
        int c = 0, tile = pair, kb = 0;
        int n0 = place_of(p, tile).n0 + rank * kRows;
        unsigned round = 0;
        for (int it = 0; it < blocks; ++it) {
            if (round > 0) {
                healthy = mbar_wait(codes_free_bar(c), (round - 1) & 1, 0x60u + c, p.status);
                healthy = __all_sync(0xffffffffu, healthy);
            }
            if (!healthy) break;
            if (issuer) {
                mbar_arrive_expect_tx(codes_bar(c), kCodeBytes);
                tma_load_2d(code_slot(c), &w_map, kb * (kBlockK / 2), n0, codes_bar(c));
            }
            __syncwarp();
            if (++c == p.code_slots) {
                c = 0;
                ++round;
            }
            if (++kb == p.k_blocks) {
                kb = 0;
                tile += pairs;
                n0 = place_of(p, tile).n0 + rank * kRows;
            }
        }
    } else if (warp == 2 && rank == 0) {               // ---- the pair's MMAs
        const uint32_t instr_desc = (1u << 4)                                            // FP32 accumulate
                                    | (static_cast<uint32_t>(p.bn >> 3) << 17)           // N
                                    | (static_cast<uint32_t>(kTileRows >> 4) << 24);     // M, of both; FP16, K-major B
        bool healthy = true, peeked = false;
        int xs = 0, s = 0, kb = 0;
        unsigned tiles = 0;
        for (unsigned it = 0; it < static_cast<unsigned>(blocks); ++it) {
            const unsigned r = it % kRing, next = it + 1;
            if (kb == 0 && tiles > 0) healthy = mbar_wait<true>(acc_free_bar, (tiles - 1) & 1, 0x40u, p.status);
            if (!peeked && healthy) healthy = mbar_wait<true>(full_bar(r), (it / kRing) & 1, 0x20u + r, p.status);
            healthy = __all_sync(0xffffffffu, healthy);
            if (!healthy) break;
            peeked = mbar_test<true>(full_bar(next % kRing), (next / kRing) & 1);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned a = tmem + kWeightColumn + s * kSlotColumns;
            const uint64_t b0 = operand_desc(x_slot(xs)), b1 = operand_desc(x_slot(xs) + x_half_bytes);
            if (++xs == p.x_slots) xs = 0;
            if (++s == kSlots) s = 0;
            if (issuer) {
#pragma unroll
                for (int j = 0; j < kBlockK / 16; ++j) {
                    // 16 k = 8 columns of weights, and 32 bytes further along the swizzled row of x
                    umma_pair(tmem, a + 8 * j, (j < 4 ? b0 : b1) + 2 * (j & 3), instr_desc, kb > 0 || j > 0 ? 1u : 0u);
                }
                commit_pair(done_bar(r));
                if (kb + 1 == p.k_blocks) commit_pair(acc_full_bar);
            }
            __syncwarp();
            peeked = __all_sync(0xffffffffu, peeked);
            if (kb == 0) ++tiles;
            if (++kb == p.k_blocks) kb = 0;
        }
    } else if (warp >= kFirstDequantWarp) {            // ---- dequantisers
        const int group = (warp - kFirstDequantWarp) / kGroupWarps;
        const int r = (warp & 3) * 32 + lane;          // weight row of this CTA's half
        const unsigned row_offset = r * 64;
        const unsigned swizzle = (r >> 1) & 3;         // 64-byte swizzle of the code tile
        const int groups_per_row = p.k_blocks * kScales;
        const unsigned lane_base = tmem + (static_cast<unsigned>((warp & 3) * 32) << 16) + kWeightColumn;
        uint32_t next_scale[kScales] = {};             // (a register each: packed in pairs they would be waited for at once)
        // Where the scales of the group's next block are: walked along, a division per block showed.
        int next_tile = pair + group / p.k_blocks * pairs, next_kb = group % p.k_blocks;
        int left = blocks - group;                     // blocks of the run from that one on
        const __half* scale_row = nullptr;
        auto point_at_row = [&]() {                    // rows past N hold zero codes
            scale_row = p.scales + static_cast<size_t>(min(place_of(p, next_tile).n0 + rank * kRows + r, p.N - 1)) * groups_per_row;
        };
        auto fetch_scales = [&]() {
            if (left > 0) {
                const __half* src = scale_row + next_kb * kScales;
#pragma unroll
                for (int i = 0; i < kScales; ++i) asm volatile("ld.global.nc.u16 %0, [%1];" : "=r"(next_scale[i]) : "l"(src + i));
            }
            left -= kDequantGroups;
            next_kb += kDequantGroups;
            if (next_kb >= p.k_blocks) {
                do {
                    next_kb -= p.k_blocks;
                    next_tile += pairs;
                } while (next_kb >= p.k_blocks);
                if (left > 0) point_at_row();
            }
        };
        // A wait that gives up is recorded and not repeated; the loop goes on with whatever is there, so the warps stay together.
        bool healthy = true;
        unsigned c = group % p.code_slots, code_round = group / p.code_slots;
        if (left > 0) point_at_row();
        fetch_scales();
        for (unsigned it = group; it < static_cast<unsigned>(blocks); it += kDequantGroups) {
            uint32_t scale2[kScales], scale_2_20[kScales], minus_8_scale[kScales];
            bool scaled = true;                        // all scales of the warp's rows are such that unpack8_scaled may be used
#pragma unroll
            for (int i = 0; i < kScales; ++i) {
                scale2[i] = next_scale[i] * 0x10001u;
                scaled = scaled && (next_scale[i] & 0x7FFFu) <= kLargestScaled;
                scale_2_20[i] = hmul2_u32(hmul2_u32(scale2[i], 0x64006400u), 0x64006400u);
                minus_8_scale[i] = hmul2_u32(scale2[i], 0xC800C800u);
            }
            scaled = __all_sync(0xffffffffu, scaled);
            if (healthy) healthy = mbar_wait(codes_bar(c), code_round & 1, 0x50u + c, p.status);
            __syncwarp();
            uint4 words[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                             : "=r"(words[q].x), "=r"(words[q].y), "=r"(words[q].z), "=r"(words[q].w)
                             : "r"(code_slot(c) + row_offset + ((q ^ swizzle) << 4))
                             : "memory");
            }
            fetch_scales();
            auto weights_of = [&](auto is_scaled, int q, uint32_t (&v)[16]) {
                const uint32_t word[4] = {words[q].x, words[q].y, words[q].z, words[q].w};
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    if constexpr (decltype(is_scaled)::value) {
                        unpack8_scaled(word[w], scale_2_20[q * 32 / GROUP], minus_8_scale[q * 32 / GROUP], v + 4 * w);
                    } else {
                        unpack8_ordered(word[w], v + 4 * w);
#pragma unroll
                        for (int j = 0; j < 4; ++j) v[4 * w + j] = hmul2_u32(v[4 * w + j], scale2[q * 32 / GROUP]);
                    }
                }
            };
            uint32_t v[16];
            if (scaled) {
                weights_of(std::true_type{}, 0, v);
            } else {
                weights_of(std::false_type{}, 0, v);
            }
            // The slot is next written by a TMA copy, through another proxy: the arrival alone does not order this lane's reads
            // before it.
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();                                                  // every lane has its codes
            if (lane == 0) mbar_arrive(codes_free_bar(c));
            if ((c += kDequantGroups) >= static_cast<unsigned>(p.code_slots)) {
                c -= p.code_slots;
                ++code_round;
            }
            // the weights of this slot's last block are no longer needed once its MMAs are done
            if (it >= kSlots) {
                const unsigned old = it - kSlots;
                if (healthy) healthy = mbar_wait(done_bar(old % kRing), (old / kRing) & 1, 0x70u, p.status);
            }
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned to = lane_base + it % kSlots * kSlotColumns;
            tmem_store16(to, v);
            auto store_rest = [&](auto is_scaled) {
#pragma unroll
                for (int q = 1; q < 4; ++q) {
                    weights_of(is_scaled, q, v);
                    tmem_store16(to + q * 16, v);
                }
            };
            if (scaled) {
                store_rest(std::true_type{});
            } else {
                store_rest(std::false_type{});
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(first_full + it % kRing * 8);
        }
    } else if (warp >= kFirstDrainWarp) {              // ---- drain
        const int row = (warp & 3) * 32 + lane;
        const int share = warp / 4 - kFirstDrainWarp / 4;                  // of a quarter of the rows: every other 16 columns
        auto emit = [&](const Place& at, int col, const uint32_t (&sum)[16]) {
            const int n = at.n0 + rank * kRows + row, m = at.m0 + col;
            if (n >= p.N) return;
            char* out = reinterpret_cast<char*>(p.y + static_cast<size_t>(m) * p.N + n);
            const unsigned stride = static_cast<unsigned>(p.N) * 2u;
            __half2 two[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) two[j] = __floats2half2_rn(__uint_as_float(sum[2 * j]), __uint_as_float(sum[2 * j + 1]));
            if (p.bias != nullptr) {
                const __half2 bias = __half2half2(p.bias[n]);
#pragma unroll
                for (int j = 0; j < 8; ++j) two[j] = __hadd2(two[j], bias);
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (m + j < p.M) *reinterpret_cast<__half*>(out) = j % 2 == 0 ? __low2half(two[j / 2]) : __high2half(two[j / 2]);
                out += stride;
            }
        };
        bool healthy = true;
        unsigned done = 0;
        for (int tile = pair; tile < p.tiles; tile += pairs, ++done) {
            const Place at = place_of(p, tile);
            if (healthy) healthy = mbar_wait(acc_full_bar, done & 1, 0x30u, p.status);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int col = share * 16; col < p.bn; col += kShares * 16) {
                uint32_t v[16];
                tmem_load16(tmem + (static_cast<unsigned>((warp & 3) * 32) << 16) + col, v);
                emit(at, col, v);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0 && tile + pairs < p.tiles) mbar_arrive_remote(first_cta_address(acc_free_bar));
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_barrier();                                 // the pair's MMAs read both CTAs' memory
    if (warp == 2) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

const void* pair_kernel(int64_t group) {
    static const void* const kernels[3] = {reinterpret_cast<const void*>(linear_gemm_pair_kernel<128>),
                                           reinterpret_cast<const void*>(linear_gemm_pair_kernel<64>),
                                           reinterpret_cast<const void*>(linear_gemm_pair_kernel<32>)};
    return kernels[group == 128 ? 0 : group == 64 ? 1 : 2];
}

int learn_device(int& pairs) {
    for (const int group : {128, 64, 32}) {
        if (cudaFuncSetAttribute(pair_kernel(group), cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) return W4A16_ERR_LAUNCH;
    }
    cudaLaunchConfig_t shape = {};
    shape.gridDim = dim3(2);
    shape.blockDim = dim3(kThreads);
    shape.dynamicSmemBytes = kSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    shape.attrs = attr;
    shape.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&pairs, pair_kernel(128), &shape) != cudaSuccess || pairs <= 0) return W4A16_ERR_LAUNCH;
    return W4A16_OK;
}

int current_pairs(int* pairs) {
    static PerDevice<int> devices;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices) return W4A16_ERR_LAUNCH;
    const int* known = nullptr;
    const int status = devices.get(device, [](int& n) { return learn_device(n); }, &known);
    if (status == W4A16_OK) *pairs = std::min(*known, kPairs);
    return status;
}

// Batch tile and rounds of pairs of a call.
struct PairPlan {
    int bn, m_tiles, k_blocks;
    long long tiles;
};
PairPlan plan_pair(int64_t M, int64_t N, int64_t K) {
    PairPlan g;
    g.m_tiles = static_cast<int>((M + kMaxBatch - 1) / kMaxBatch);
    g.bn = static_cast<int>(((M + g.m_tiles - 1) / g.m_tiles + 31) / 32 * 32);
    g.k_blocks = static_cast<int>(K / kBlockK);
    g.tiles = (N + kTileRows - 1) / kTileRows * g.m_tiles;
    return g;
}

}  // namespace

// Fitted, with the time that linear_gemm.cu plans by, to 617 calls on 72 layers of 512 to 28672 -> 1024 to 28672 at 65 to 8192 rows, in
// runs of 12 ms and more: choosing by the two is 0.5 % slower than the better kernel on average.
double gemm_pair_time(int64_t M, int64_t N, int64_t K) {
    const PairPlan g = plan_pair(M, N, K);
    const double rounds = static_cast<double>((g.tiles + kPairs - 1) / kPairs);
    return 5.0 + rounds * g.k_blocks * std::max(0.4, 0.0032 * g.bn) + 2.0 * (rounds - 1.0);
}
int gemm_pair_rounds(int64_t M, int64_t N) { return static_cast<int>(std::min<long long>(INT32_MAX, (plan_pair(M, N, kBlockK).tiles + kPairs - 1) / kPairs)); }

int launch_linear_gemm_pair(const LinearProblem& prob, cudaStream_t stream) {
    if (prob.K % kBlockK != 0 || prob.K <= 0 || !is_stream_group(prob.group)) return W4A16_ERR_BAD_CONFIG;
    if (prob.M > INT32_MAX || prob.N > INT32_MAX || prob.K > INT32_MAX) return W4A16_ERR_TOO_LARGE;
    if (reinterpret_cast<uintptr_t>(prob.x) % 16 != 0 || reinterpret_cast<uintptr_t>(prob.packed) % 16 != 0) {
        return W4A16_ERR_MISALIGNED;
    }
    int pairs = 0;
    const int known = current_pairs(&pairs);
    if (known != W4A16_OK) return known;
    const PairPlan g = plan_pair(prob.M, prob.N, prob.K);
    if (g.tiles * g.k_blocks > INT32_MAX) return W4A16_ERR_TOO_LARGE;
    const long long grid = std::min<long long>(pairs, g.tiles);
    PairParams params;
    params.m_tiles = g.m_tiles;
    params.bn = g.bn;
    params.k_blocks = g.k_blocks;
    CUtensorMap x_map, w_map;
    if (!encode_rows(&x_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, prob.x, prob.M, prob.K * 2, 128, params.bn / 2, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B) ||
        !encode_rows(&w_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, prob.packed, prob.N, prob.K / 2, kBlockK / 2, kRows,
                     CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B)) {
        return W4A16_ERR_LAUNCH;
    }
    params.scales = prob.scales;
    params.y = static_cast<__half*>(prob.y);
    params.bias = prob.bias;
    params.status = tcgen05_status_address();
    if (params.status == nullptr) return W4A16_ERR_LAUNCH;
    params.M = static_cast<int>(prob.M);
    params.N = static_cast<int>(prob.N);
    params.tiles = static_cast<int>(g.tiles);
    const int bands = (g.m_tiles + kBand - 1) / kBand;
    params.band = (g.m_tiles + bands - 1) / bands;
    params.band_tiles = static_cast<int>(g.tiles / g.m_tiles) * params.band;
    // 256 batch rows: 4 blocks of x and 8 of codes.
    const int x_bytes = params.bn * 128;
    const int room = kSmem - kBarrierBytes - 1024;
    params.x_slots = std::min(6, (room - 6 * kCodeBytes) / x_bytes);
    params.code_slots = std::min(kMaxCodeSlots, (room - params.x_slots * x_bytes) / kCodeBytes);

    cudaLaunchConfig_t launch = {};
    launch.gridDim = dim3(static_cast<unsigned>(2 * grid));
    launch.blockDim = dim3(kThreads);
    launch.dynamicSmemBytes = static_cast<size_t>(params.x_slots) * x_bytes + params.code_slots * kCodeBytes + kBarrierBytes + 1024;
    launch.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    launch.attrs = attr;
    launch.numAttrs = 2;
    void* args[] = {&params, &x_map, &w_map};
    if (cudaLaunchKernelExC(&launch, pair_kernel(prob.group), args) != cudaSuccess) return W4A16_ERR_LAUNCH;
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    return W4A16_OK;
}

}  // namespace w4a16

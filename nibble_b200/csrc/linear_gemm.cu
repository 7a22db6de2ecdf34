// W4A16 linear for prompts and medium batches on the 5th-generation tensor cores: the weights are dequantised straight into
// tensor memory (TMEM) and enter the MMA from there, and the K blocks of output tiles are shared between SMs where that pays.
//
//   D[2 x 128 x BN] (TMEM, FP32)  +=  A[2 x 128 x 128] (TMEM: FP16 weights)  x  B[BN x 128] (shared memory: rows of x)
//
// Weights are half(code * scale), accumulated in FP32 over K: the arithmetic of dequantise-then-matmul.
//
// What bounds it.  A K block of 256 weight rows is 32768 weights: 500 issue slots of each SM quarter to unpack (thirteen
// instructions per word of eight codes), 8 clocks of MMA per batch row, 16 MMAs to issue at about 40 clocks each, and 16 KB
// of codes plus 256 bytes per batch row out of L2, which gives an SM some 50 bytes per clock.  Hence 256 rows: with 128, the x
// tile of a 128-row batch alone took the whole of that.  Measured from the time against K (one tile a CTA, 37888 channels, K from 2048 to
// 16384, calls back to back): a block at 64 batch rows 0.56 us while the weights stay in L2, 0.71 to 0.97 out of HBM (the chain of waits,
// unpacking and stores of the three dequantiser groups; two groups took a quarter more), at 128 rows 0.69, and 0.89 to 1.17, of which
// the MMAs are 0.55; and 5 to 11 us of start and end beside them: tensor pipe active 48 % of the time (128 rows, 8192 -> 28672).
//
// (A GEMM with the FP16 tile in shared memory, since given up, was 1.2 to 1.9 times slower by the store, a proxy
// fence and the space that takes.)
//
// Roles of a CTA's 32 warps, one CTA per SM:
//   warp 0        loads x (TMA), one K block per ring slot
//   warp 1        loads the packed codes (TMA), as far ahead as shared memory allows
//   warp 2        allocates TMEM and issues the MMAs: one commit per K block frees its slots
//   warps 4-7     drain: one per quarter of the TMEM lanes, for all tiles of a run but the last
//   warps 8-31    dequantisers: three groups of eight warps taking the K blocks in turn, a thread per weight row
//   all           the last tile of a run
// A barrier's phase cannot complete twice before each of its waiters has seen it once, because every waiter is needed
// for the phase after: so parity waits are exact whichever group takes which block.
//
// Work split.  Layers of few tiles: the CTAs of a cluster (2 to 8) share the K blocks of a tile, leave their sums in their own
// shared memory and each adds up its share of the columns over distributed shared memory.  Layers of many tiles: the
// (tile, K block) pairs of all tiles in a row are cut into equal runs, one per CTA.  A run that holds part of a tile leaves
// FP32 sums in the caller's workspace; the CTA that arrives last at a tile adds the parts in order (no one waits).  It is
// nearly always the one that reaches the tile at the end of its run, finds the others' parts in place and adds them to its
// own accumulator.  Without a workspace, runs are whole tiles.  plan_gemm() weighs the three.
//
// Every wait is bounded; one that gives up sets the status word and the CTA still runs to its TMEM deallocation.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "gemm_weights.cuh"
#include "kernels.h"
#include "per_device.h"
#include "tcgen05.cuh"
#include "unpack.cuh"

namespace w4a16 {
namespace {

// Set when a bounded wait inside a tensor-core kernel gives up (which barrier: low byte).
__device__ unsigned g_tcgen05_status = 0;

constexpr int kHalfRows = 128;           // output channels of one MMA (TMEM lanes)
constexpr int kRows = 2 * kHalfRows;     // ... and of a tile
constexpr int kBlockK = 128;             // K per pipeline block
constexpr int kRing = 8;                 // blocks the barriers tell apart; also the most blocks of x in flight
constexpr int kMaxCodeSlots = 8;         // blocks of packed codes in flight at most
constexpr int kCodeBytes = kRows * kBlockK / 2;
constexpr int kMaxBatch = 128;           // batch rows per tile (MMA N)
constexpr int kHalfColumns = kBlockK / 2;             // TMEM columns of one half's weights
constexpr int kSlotColumns = 2 * kHalfColumns;
constexpr int kDrainWarps = 4;
constexpr int kFirstDrainWarp = 4;
constexpr int kDequantGroups = 3;
constexpr int kGroupWarps = kRows / 32;
constexpr int kFirstDequantWarp = kFirstDrainWarp + kDrainWarps;
constexpr int kGemmThreads = (kFirstDequantWarp + kDequantGroups * kGroupWarps) * 32;   // 1024
constexpr int kMaxCluster = 8;
constexpr int kBarrierBytes = 512;

struct GemmParams {
    const __half* scales;
    __half* y;
    const __half* bias;
    float* partial;          // two parts of 256 x bn sums per CTA, or null: runs are whole tiles
    unsigned* counters;      // arrivals per tile, zero between calls
    unsigned* status;
    int M, N;
    int k_blocks;            // of one tile
    int bn, m_tiles;
    int x_slots, code_slots; // blocks of x and of codes in flight
    int slots;               // blocks of weights in TMEM
    int cluster;             // CTAs that share a tile (1: runs)
    int run, longer;         // units (tile, K block) of a CTA's run, or its tiles where runs are whole tiles; the first `longer` CTAs
                             // take one more
};

// CTA c takes units first_unit(c) .. first_unit(c + 1) - 1.  The host has divided: a 64-bit division here took each CTA a
// microsecond at its start, and the search for a unit's owner several while a tile's parts waited (8192 -> 28672, 128 rows: 64.0
// -> 60.4 us; 8192 x 8192, 512 rows: 61.7 -> 57.8).
__device__ __forceinline__ int first_unit(const GemmParams& p, int c) {
    if (p.cluster > 1) return c / p.cluster * p.k_blocks + p.k_blocks * (c % p.cluster) / p.cluster;
    const int first = c * p.run + min(c, p.longer);
    return p.partial != nullptr ? first : first * p.k_blocks;
}
// The CTA whose run holds unit u, where runs may cut tiles (they are never empty).
__device__ __forceinline__ int owner_of(const GemmParams& p, int u) {
    const unsigned unit = u, in_longer = static_cast<unsigned>(p.longer) * (p.run + 1);
    return unit < in_longer ? unit / (p.run + 1) : p.longer + (unit - in_longer) / p.run;
}

// Which CTAs hold parts of a tile, and where the first of them keeps it (the others: part 0, they start inside the tile).
struct TileParts {
    int first, last, first_which;
};
__device__ __forceinline__ TileParts parts_of(const GemmParams& p, int tile) {
    const int begin = tile * p.k_blocks;
    TileParts t;
    t.first = owner_of(p, begin);
    t.last = owner_of(p, begin + p.k_blocks - 1);
    t.first_which = first_unit(p, t.first) == begin ? 0 : 1;   // a run's last segment is its second part
    return t;
}
// Parts keep four columns of a row together and rows side by side: 16-byte accesses, 512 bytes a warp.
__device__ __forceinline__ float4* part_of(const GemmParams& p, int cta, int which) {
    return reinterpret_cast<float4*>(p.partial + (static_cast<size_t>(cta) * 2 + which) * (static_cast<size_t>(kRows) * p.bn));
}
__device__ __forceinline__ void add_to(float4& sum, const float4& q) {
    sum.x += q.x;
    sum.y += q.y;
    sum.z += q.z;
    sum.w += q.w;
}

// A contiguous run of K blocks of one tile.
struct Segment {
    int tile, k_begin, k_count;
};

__device__ __forceinline__ void drain_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kDrainWarps * 32) : "memory"); }

// Sixteen bytes at the same place in the shared memory of the cluster's CTA `rank`.
__device__ __forceinline__ float4 load_cluster(unsigned local, int rank) {
    unsigned remote;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
    return v;
}

template <int GROUP>
__global__ void __launch_bounds__(kGemmThreads, 1)
linear_gemm_kernel(const GemmParams p, const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map) {
    constexpr int kScales = kBlockK / GROUP;                               // per row and K block
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // Whether all parts of a tile are in place: for the drain warps, and for all warps at the end (both may be at it at once).
    __shared__ int drain_verdict, verdict;
    __shared__ TileParts drain_parts, shared_parts;
    const unsigned base = (smem_u32(smem_raw) + 1023u) & ~1023u;           // swizzle patterns are a function of the address
    const unsigned x_half_bytes = static_cast<unsigned>(p.bn) * 128;       // 64 K of every batch row, 128-byte swizzled
    auto x_slot = [&](int s) { return base + s * 2 * x_half_bytes; };
    const unsigned codes_ring = base + p.x_slots * 2 * x_half_bytes;
    auto code_slot = [&](int c) { return codes_ring + c * kCodeBytes; };
    const unsigned bars = codes_ring + p.code_slots * kCodeBytes;
    auto full_bar = [&](int r) { return bars + r * 8; };                   // x has landed and the weights are in TMEM
    auto done_bar = [&](int r) { return bars + (kRing + r) * 8; };         // the block's MMAs have finished
    auto codes_bar = [&](int c) { return bars + (2 * kRing + c) * 8; };    // the codes have landed
    auto codes_free_bar = [&](int c) { return bars + (2 * kRing + kMaxCodeSlots + c) * 8; };
    constexpr int kRingBars = 2 * kRing + 2 * kMaxCodeSlots;
    const unsigned acc_full_bar = bars + kRingBars * 8, acc_free_bar = bars + (kRingBars + 1) * 8;
    const unsigned finished_bar = bars + (kRingBars + 2) * 8;              // the run's last tile has been accumulated
    const unsigned tmem_word = bars + (kRingBars + 3) * 8;
    static_assert((kRingBars + 3) * 8 + 4 <= kBarrierBytes);
    const int acc_columns = p.bn <= 64 ? 64 : kMaxBatch;                   // TMEM: two accumulators, then the weight slots
    const int weight_column = 2 * acc_columns;

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // the same in all lanes, and known to be: addresses stay uniform
    const int run_begin = first_unit(p, blockIdx.x), run_end = first_unit(p, blockIdx.x + 1);
    auto segment_at = [&](int u) {
        Segment s;
        s.tile = u / p.k_blocks;
        s.k_begin = u - s.tile * p.k_blocks;
        s.k_count = min(p.k_blocks - s.k_begin, run_end - u);
        return s;
    };

    if (tid == 32 * 3) {                               // (a warp without other work here)
        for (int r = 0; r < kRing; ++r) {
            mbar_init(full_bar(r), kGroupWarps + 1);   // the warps of one dequantiser group, and x
            mbar_init(done_bar(r), 1);
        }
        for (int c = 0; c < p.code_slots; ++c) {
            mbar_init(codes_bar(c), 1);
            mbar_init(codes_free_bar(c), kGroupWarps);
        }
        mbar_init(acc_full_bar, 1);
        mbar_init(acc_free_bar, kDrainWarps);
        mbar_init(finished_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tmem_word) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (warp == 0 && lane == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&x_map)) : "memory");
    if (p.cluster > 1 && p.m_tiles == 1 && warp >= kFirstDequantWarp && warp < kFirstDequantWarp + kGroupWarps) {
        // and so do the first scales of short calls (8192 x 8192, 48 rows: 18.2 -> 17.7 us; of long ones they were 2 % in the way)
        const Segment at = segment_at(run_begin);
        const int n = min(at.tile / p.m_tiles * kRows + (warp - kFirstDequantWarp) * 32 + lane, p.N - 1);
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p.scales + static_cast<size_t>(n) * (p.k_blocks * kScales) + at.k_begin * kScales));
    }
    if (warp == 1 && lane < p.code_slots && run_begin + lane < run_end) {
        // the first codes travel to L2 while the kernel in front finishes (a prefetch cannot go stale there)
        const Segment at = segment_at(run_begin + lane);
        asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];"
                     ::"l"(reinterpret_cast<uint64_t>(&w_map)), "r"(at.k_begin * (kBlockK / 2)), "r"(at.tile / p.m_tiles * kRows)
                     : "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    unsigned tmem;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_word));
    pdl_release_downstream();
    pdl_wait_for_upstream();

    // Sums of a finished tile are handled 16 columns of a row at a time: thread and warp give the row (a quarter of the TMEM
    // lanes is all that a warp may read), `i` counts the columns of both halves.
    struct Chunk {
        int row, col;
        unsigned tmem;
    };
    auto chunk_at = [&](int i) {
        const int half = i >= p.bn ? 1 : 0;
        Chunk c;
        c.col = i - half * p.bn;
        c.row = half * kHalfRows + (warp & 3) * 32 + lane;
        c.tmem = tmem + (static_cast<unsigned>((warp & 3) * 32) << 16) + half * acc_columns + c.col;
        return c;
    };
    auto load_sums = [&](const Chunk& at, float (&sum)[16]) {
        uint32_t v[16];
        tmem_load16(at.tmem, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) sum[j] = __uint_as_float(v[j]);
    };
    // Rounded, to the output.  Few instructions per element: the drain warps share their schedulers with 24 dequantisers.
    auto emit = [&](int tile, const float (&sum)[16], const Chunk& at) {
        const int n = tile / p.m_tiles * kRows + at.row, m = tile % p.m_tiles * p.bn + at.col;
        if (n >= p.N) return;
        char* out = reinterpret_cast<char*>(p.y + static_cast<size_t>(m) * p.N + n);
        const unsigned stride = static_cast<unsigned>(p.N) * 2u;
        __half2 pair[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) pair[j] = __floats2half2_rn(sum[2 * j], sum[2 * j + 1]);
        if (p.bias != nullptr) {
            const __half2 bias = __half2half2(p.bias[n]);
#pragma unroll
            for (int j = 0; j < 8; ++j) pair[j] = __hadd2(pair[j], bias);
        }
        if (m + 16 <= p.M) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                *reinterpret_cast<__half*>(out) = j % 2 == 0 ? __low2half(pair[j / 2]) : __high2half(pair[j / 2]);
                out += stride;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (m + j < p.M) *reinterpret_cast<__half*>(out) = j % 2 == 0 ? __low2half(pair[j / 2]) : __high2half(pair[j / 2]);
                out += stride;
            }
        }
    };
    auto store_part = [&](int which, const float (&sum)[16], const Chunk& at) {
        float4* part = part_of(p, blockIdx.x, which) + at.col / 4 * kRows + at.row;
#pragma unroll
        for (int j = 0; j < 4; ++j) part[j * kRows] = make_float4(sum[4 * j], sum[4 * j + 1], sum[4 * j + 2], sum[4 * j + 3]);
    };
    // The parts of a tile in the order of their CTAs; this CTA's own comes from TMEM or, with the others, from memory.
    auto add_parts = [&](const TileParts& parts, bool own_in_tmem, const Chunk& at, float (&sum)[16]) {
        for (int cta = parts.first; cta <= parts.last; ++cta) {
            float q[16];
            if (own_in_tmem && cta == static_cast<int>(blockIdx.x)) {
                load_sums(at, q);
            } else {
                const float4* src = part_of(p, cta, cta == parts.first ? parts.first_which : 0) + at.col / 4 * kRows + at.row;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 four = __ldcg(src + j * kRows);
                    q[4 * j] = four.x;
                    q[4 * j + 1] = four.y;
                    q[4 * j + 2] = four.z;
                    q[4 * j + 3] = four.w;
                }
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) sum[j] = cta == parts.first ? q[j] : sum[j] + q[j];
        }
    };

    // The producers and the MMA issuer walk their loops with all lanes and elect one to issue: addresses and descriptors then
    // live in uniform registers.  (With the loops inside `if (lane == 0)` a 128-row block took 1300 clocks instead of 900.)
    const bool issuer = elect_one();
    if (warp == 0) {                                   // ---- x, one K block after the other
        bool healthy = true;
        unsigned it = 0;
        int xs = 0;
        for (int u = run_begin; u < run_end && healthy;) {
            const Segment seg = segment_at(u);
            u += seg.k_count;
            const int m0 = seg.tile % p.m_tiles * p.bn;
            for (int kb = 0; kb < seg.k_count; ++kb, ++it) {
                const unsigned r = it % kRing;
                if (it >= static_cast<unsigned>(p.x_slots)) {      // the block that had this slot
                    const unsigned old = it - p.x_slots;
                    healthy = mbar_wait(done_bar(old % kRing), (old / kRing) & 1, 0x10u + r, p.status);
                    healthy = __all_sync(0xffffffffu, healthy);
                }
                if (!healthy) break;
                if (issuer) {
                    const int k = (seg.k_begin + kb) * kBlockK;
                    mbar_arrive_expect_tx(full_bar(r), 2 * x_half_bytes);
                    tma_load_2d(x_slot(xs), &x_map, k, m0, full_bar(r));
                    tma_load_2d(x_slot(xs) + x_half_bytes, &x_map, k + 64, m0, full_bar(r));
                }
                __syncwarp();
                if (++xs == p.x_slots) xs = 0;
            }
        }
    } else if (warp == 1) {                            // ---- packed codes
        bool healthy = true;
        int c = 0;
        unsigned round = 0;
        for (int u = run_begin; u < run_end && healthy;) {
            const Segment seg = segment_at(u);
            u += seg.k_count;
            const int n0 = seg.tile / p.m_tiles * kRows;
            for (int kb = 0; kb < seg.k_count; ++kb) {
                if (round > 0) {
                    healthy = mbar_wait(codes_free_bar(c), (round - 1) & 1, 0x60u + c, p.status);
                    healthy = __all_sync(0xffffffffu, healthy);
                }
                if (!healthy) break;
                if (issuer) {
                    mbar_arrive_expect_tx(codes_bar(c), kCodeBytes);
                    tma_load_2d(code_slot(c), &w_map, (seg.k_begin + kb) * (kBlockK / 2), n0, codes_bar(c));
                }
                __syncwarp();
                if (++c == p.code_slots) {
                    c = 0;
                    ++round;
                }
            }
        }
    } else if (warp == 2) {                            // ---- MMAs
        const uint32_t instr_desc = (1u << 4)                                            // FP32 accumulate
                                    | (static_cast<uint32_t>(p.bn >> 3) << 17)           // N
                                    | (static_cast<uint32_t>(kHalfRows >> 4) << 24);     // M; FP16, K-major B
        bool healthy = true, peeked = false;
        unsigned it = 0, tiles_done = 0;
        int xs = 0, s = 0;
        for (int u = run_begin; u < run_end && healthy; ++tiles_done) {
            const Segment seg = segment_at(u);
            u += seg.k_count;
            if (tiles_done > 0) healthy = mbar_wait(acc_free_bar, (tiles_done - 1) & 1, 0x40u, p.status);
            for (int kb = 0; kb < seg.k_count && healthy; ++kb, ++it) {
                const unsigned r = it % kRing, next = it + 1;
                if (!peeked) healthy = mbar_wait(full_bar(r), (it / kRing) & 1, 0x20u + r, p.status);
                healthy = __all_sync(0xffffffffu, healthy);
                if (!healthy) break;
                // whether the next block is ready too: asked now, so that the answer's latency hides under these MMAs
                peeked = mbar_test(full_bar(next % kRing), (next / kRing) & 1);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned a = tmem + weight_column + s * kSlotColumns;
                const uint64_t b0 = operand_desc(x_slot(xs)), b1 = operand_desc(x_slot(xs) + x_half_bytes);
                if (++xs == p.x_slots) xs = 0;
                if (++s == p.slots) s = 0;
                if (issuer) {
#pragma unroll
                    for (int j = 0; j < kBlockK / 16; ++j) {
                        // 16 k = 8 columns of weights, and 32 bytes further along the swizzled row of x
                        const uint64_t b = (j < 4 ? b0 : b1) + 2 * (j & 3);
                        const uint32_t accumulate = kb > 0 || j > 0 ? 1u : 0u;
                        umma_f16_tmem_a(tmem, a + 8 * j, b, instr_desc, accumulate);
                        umma_f16_tmem_a(tmem + acc_columns, a + kHalfColumns + 8 * j, b, instr_desc, accumulate);
                    }
                    umma_commit(done_bar(r));
                    if (kb == seg.k_count - 1) umma_commit(u < run_end ? acc_full_bar : finished_bar);
                }
                __syncwarp();
                peeked = __all_sync(0xffffffffu, peeked);
            }
        }
    } else if (warp >= kFirstDequantWarp) {            // ---- dequantisers
        const int group = (warp - kFirstDequantWarp) / kGroupWarps;
        const int half = ((warp - kFirstDequantWarp) >> 2) & 1;
        const int r = half * kHalfRows + (warp & 3) * 32 + lane;           // weight row of the tile
        const unsigned row_offset = r * 64;
        const unsigned swizzle = (r >> 1) & 3;         // 64-byte swizzle of the code tile
        const int groups_per_row = p.k_blocks * kScales;
        const unsigned lane_base = tmem + (static_cast<unsigned>((warp & 3) * 32) << 16) + weight_column + half * kHalfColumns;
        uint32_t next_scale[kScales] = {};             // (a register each: packed in pairs they would be waited for at once)
        // Where the scales of the group's next block are: walked along, a division per block showed.
        int next_tile = (run_begin + group) / p.k_blocks, next_kb = run_begin + group - next_tile * p.k_blocks;
        int left = run_end - run_begin - group;        // blocks of the run from that one on
        const __half* scale_row = nullptr;
        auto point_at_row = [&]() {                    // rows past N hold zero codes
            scale_row = p.scales + static_cast<size_t>(min(next_tile / p.m_tiles * kRows + r, p.N - 1)) * groups_per_row;
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
                    ++next_tile;
                } while (next_kb >= p.k_blocks);
                point_at_row();
            }
        };
        // A wait that gives up is recorded and not repeated; the loop goes on with whatever is there, so the warps stay together.
        bool healthy = true;
        unsigned it = group, c = group, code_round = 0;
        int s = group % p.slots;
        point_at_row();
        fetch_scales();
        for (int blocks = run_end - run_begin; static_cast<int>(it) < blocks; it += kDequantGroups) {
            uint32_t scale2[kScales];
#pragma unroll
            for (int i = 0; i < kScales; ++i) scale2[i] = next_scale[i] * 0x10001u;
            bool scaled = true;                        // all scales of the warp's rows are such that unpack8_scaled may be used
            uint32_t scale_2_20[kScales], minus_8_scale[kScales];
#pragma unroll
            for (int i = 0; i < kScales; ++i) {
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
            // 32 K of the row as FP16 pairs; which way, the warp decides twice a block.
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
            // before it.  (Without the fence a few rows of a call in some ten were read after the refill; it costs 0 to 0.6 %.)
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();                                                  // every lane has its codes
            if (lane == 0) mbar_arrive(codes_free_bar(c));
            if ((c += kDequantGroups) >= static_cast<unsigned>(p.code_slots)) {
                c -= p.code_slots;
                ++code_round;
            }
            // the weights of this slot's last block are no longer needed once its MMAs are done
            if (it >= static_cast<unsigned>(p.slots)) {
                const unsigned old = it - p.slots;
                if (healthy) healthy = mbar_wait(done_bar(old % kRing), (old / kRing) & 1, 0x70u + s, p.status);
            }
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned to = lane_base + s * kSlotColumns;
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
            if (lane == 0) mbar_arrive(full_bar(it % kRing));
            s += kDequantGroups;
            while (s >= p.slots) s -= p.slots;
        }
    } else if (warp >= kFirstDrainWarp) {              // ---- drain: every tile of the run but the last
        bool healthy = true;
        unsigned tiles_done = 0;
        for (int u = run_begin; u + segment_at(u).k_count < run_end; ++tiles_done) {
            const Segment seg = segment_at(u);
            const bool starts_run = u == run_begin, whole = seg.k_count == p.k_blocks;
            u += seg.k_count;
            if (healthy) healthy = mbar_wait(acc_full_bar, tiles_done & 1, 0x30u, p.status);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int i = 0; i < 2 * p.bn; i += 16) {
                const Chunk at = chunk_at(i);
                float sum[16];
                load_sums(at, sum);
                if (whole) {
                    emit(seg.tile, sum, at);
                } else {
                    store_part(starts_run ? 0 : 1, sum, at);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_free_bar);
            if (!whole) {
                __threadfence();
                drain_barrier();
                if (tid == kFirstDrainWarp * 32) {
                    drain_parts = parts_of(p, seg.tile);
                    drain_verdict = atomicAdd(p.counters + seg.tile, 1u) == static_cast<unsigned>(drain_parts.last - drain_parts.first);
                    if (drain_verdict) p.counters[seg.tile] = 0u;                // ready for the next call
                }
                drain_barrier();
                if (drain_verdict != 0) {
                    __threadfence();
                    for (int i = 0; i < 2 * p.bn; i += 16) {
                        float sum[16];
                        add_parts(drain_parts, false, chunk_at(i), sum);
                        emit(seg.tile, sum, chunk_at(i));
                    }
                }
                drain_barrier();                       // the verdict may be rewritten by the next segment
            }
        }
    }

    // ---- the run's last tile: all warps take part, eight to a quarter of the TMEM lanes
    __syncwarp();
    mbar_wait(finished_bar, 0, 0x38u, p.status);
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int last_tile = (run_end - 1) / p.k_blocks;
    const int first_chunk = warp / 4 * 16, chunk_step = kGemmThreads / 128 * 16;
    if (p.cluster > 1) {                               // every CTA adds up and writes its share of the columns
        for (int i = first_chunk; i < 2 * p.bn; i += chunk_step) {
            const Chunk at = chunk_at(i);
            float sum[16];
            load_sums(at, sum);
#pragma unroll
            for (int j = 0; j < 4; ++j) {              // to shared memory, whose rings have served
                asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};"
                             ::"r"(base + ((at.col / 4 + j) * kRows + at.row) * 16), "f"(sum[4 * j]), "f"(sum[4 * j + 1]), "f"(sum[4 * j + 2]),
                               "f"(sum[4 * j + 3])
                             : "memory");
            }
        }
        __syncwarp();
        cluster_barrier();
        const int rank = static_cast<int>(blockIdx.x) % p.cluster;
        const int first_quad = p.bn / 4 * rank / p.cluster, last_quad = p.bn / 4 * (rank + 1) / p.cluster;
        const int n0 = last_tile / p.m_tiles * kRows, m0 = last_tile % p.m_tiles * p.bn;
        bool reading = first_quad * kRows + tid < last_quad * kRows;
        if (!reading) cluster_arrive();
        for (int i = first_quad * kRows + tid; reading; i += kGemmThreads) {
            // every CTA starts with its own sums and goes round, so that no one's memory is read by all at once; the order
            // in which an element's parts are added is fixed all the same
            float4 q[kMaxCluster];
#pragma unroll
            for (int c = 0; c < kMaxCluster; ++c) {
                if (c < p.cluster) q[c] = load_cluster(base + i * 16, rank + c < p.cluster ? rank + c : rank + c - p.cluster);
            }
#pragma unroll
            for (int c = 1; c < kMaxCluster; ++c) {
                if (c < p.cluster) add_to(q[0], q[c]);
            }
            reading = i + kGemmThreads < last_quad * kRows;
            if (!reading) cluster_arrive();            // as far as this thread goes, the others may leave
            const int n = n0 + i % kRows, m = m0 + i / kRows * 4;
            if (n < p.N) {
                const float value[4] = {q[0].x, q[0].y, q[0].z, q[0].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    __half out = __float2half_rn(value[j]);
                    if (p.bias != nullptr) out = __hadd(out, p.bias[n]);
                    if (m + j < p.M) p.y[static_cast<size_t>(m + j) * p.N + n] = out;
                }
            }
        }
        cluster_wait();                                // no CTA leaves while another may still read its memory
        __syncwarp();
    } else if (run_begin <= last_tile * p.k_blocks && run_end == (last_tile + 1) * p.k_blocks) {
        for (int i = first_chunk; i < 2 * p.bn; i += chunk_step) {
            float sum[16];
            load_sums(chunk_at(i), sum);
            emit(last_tile, sum, chunk_at(i));
        }
    } else {
        if (tid == 0) {
            shared_parts = parts_of(p, last_tile);
            unsigned arrived;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(arrived) : "l"(p.counters + last_tile) : "memory");
            verdict = arrived == static_cast<unsigned>(shared_parts.last - shared_parts.first);
            if (verdict) p.counters[last_tile] = 0u;
        }
        __syncthreads();
        bool complete = verdict != 0;
        const bool own_in_tmem = complete;
        if (!complete) {                               // other parts are still to come: leave this one, and look again
            for (int i = first_chunk; i < 2 * p.bn; i += chunk_step) {
                float sum[16];
                load_sums(chunk_at(i), sum);
                store_part(run_begin >= last_tile * p.k_blocks ? 0 : 1, sum, chunk_at(i));
            }
            __threadfence();
            __syncthreads();
            if (tid == 0) {
                verdict = atomicAdd(p.counters + last_tile, 1u) == static_cast<unsigned>(shared_parts.last - shared_parts.first);
                if (verdict) p.counters[last_tile] = 0u;
            }
            __syncthreads();
            complete = verdict != 0;
        }
        if (complete) {
            __threadfence();
            for (int i = first_chunk; i < 2 * p.bn; i += chunk_step) {
                float sum[16];
                add_parts(shared_parts, own_in_tmem, chunk_at(i), sum);
                emit(last_tile, sum, chunk_at(i));
            }
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 2) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

// What a call does: batch tile, grid, and how tiles are shared.
struct GemmPlan {
    int bn, m_tiles, k_blocks;
    long long tiles;
    int cluster;             // > 1: CTAs per tile
    int grid;                // of the runs (cluster == 1)
    bool cut;                // runs may hold parts of tiles
    double time;             // us, by the model that chose them
    double whole_time;       // ... of runs of whole tiles
};

// `clusters[s]`: clusters of s CTAs that run at once (0 where unknown or none).
GemmPlan plan_gemm(int64_t M, int64_t N, int64_t K, int sms, const int* clusters) {
    GemmPlan g;
    g.m_tiles = static_cast<int>((M + kMaxBatch - 1) / kMaxBatch);
    g.bn = static_cast<int>(((M + g.m_tiles - 1) / g.m_tiles + 15) / 16 * 16);
    g.k_blocks = static_cast<int>(K / kBlockK);
    g.tiles = (N + kRows - 1) / kRows * g.m_tiles;
    // Times in us, fitted to 65..512 rows on sixteen layers from 1024 x 1024 to 8192 -> 28672 (mostly within 15 %): a K block, a
    // CTA's start and end, going on to another tile, the exchange inside a cluster (13 bytes a clock), the exchange through
    // the workspace (parts of 256 x bn sums written and read back).
    const double block = 0.62 + 0.0045 * std::max(0, g.bn - 64), ends = 4.5, next_tile = 1.0 + 0.012 * g.bn;
    auto by_cluster = [&](int s) { return 1.2 + 0.043 * g.bn * (s - 1) / s; };
    const double by_workspace = 1.5 + 0.025 * g.bn;
    const long long units = g.tiles * g.k_blocks;
    g.cluster = 1;
    g.cut = false;
    g.grid = static_cast<int>(std::min<long long>(sms, g.tiles));
    const double rounds = static_cast<double>((g.tiles + sms - 1) / sms);
    double best = rounds * g.k_blocks * block + ends + (rounds - 1.0) * next_tile;
    g.whole_time = best;
    for (int s = 2; s <= kMaxCluster && s <= g.k_blocks; ++s) {
        if (clusters == nullptr || clusters[s] <= 0 || g.tiles * s > INT32_MAX) continue;
        const long long waves = (g.tiles + clusters[s] - 1) / clusters[s];
        const double time = waves * ((g.k_blocks + s - 1) / s * block + ends + by_cluster(s));
        if (time < best) {
            best = time;
            g.cluster = s;
        }
    }
    if (K >= 2048 && g.tiles <= 65536) {
        // runs of at least four K blocks, on all SMs where there is that much work
        const long long grid = std::min<long long>(sms, std::max<long long>(g.tiles, units / 4));
        const double time = static_cast<double>((units + grid - 1) / grid) * block + ends + static_cast<double>(g.tiles) / sms * next_tile +
                            by_workspace * ((g.k_blocks * grid + units - 1) / units);
        if (time < best && grid != g.tiles) {
            best = time;
            g.cluster = 1;
            g.cut = true;
            g.grid = static_cast<int>(grid);
        }
    }
    g.time = best;
    return g;
}

// At most 38 MB: two parts of 256 x 128 sums for each SM.
size_t gemm_partial_bytes(const GemmPlan& g) { return g.cut ? static_cast<size_t>(g.grid) * 2 * kRows * g.bn * sizeof(float) : 0; }

// Shared memory of a CTA, with the 1 KB that the system adds: one carve-out (196 KB) below the largest, which leaves 60 KB of L1.
// The scales of a tile lie in 256 lines, of which the 28 KB beside 228 KB hold too few from one block to the next (8192 -> 28672,
// 64 rows: 45.7 -> 44.5 us, 128 rows: 61.0 -> 59.4; 162 KB: 45.4, 59.7).
constexpr int kSmem = 194 * 1024;

const void* gemm_kernel(int64_t group) {
    static const void* const kernels[3] = {reinterpret_cast<const void*>(linear_gemm_kernel<128>),
                                           reinterpret_cast<const void*>(linear_gemm_kernel<64>),
                                           reinterpret_cast<const void*>(linear_gemm_kernel<32>)};
    return kernels[group == 128 ? 0 : group == 64 ? 1 : 2];
}

// SM count and resident clusters of each size.  As initialised: a B200.
struct GemmDevice {
    int sms = 148;
    int clusters[kMaxCluster + 1] = {0, 0, 74, 45, 33, 26, 22, 15, 15};
};

int learn_device(int device, GemmDevice& d) {
    for (const int group : {128, 64, 32}) {
        if (cudaFuncSetAttribute(gemm_kernel(group), cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) {
            return W4A16_ERR_LAUNCH;
        }
    }
    if (cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || d.sms <= 0) return W4A16_ERR_LAUNCH;
    for (int s = 2; s <= kMaxCluster; ++s) {
        cudaLaunchConfig_t shape = {};
        shape.gridDim = dim3(static_cast<unsigned>(s));
        shape.blockDim = dim3(kGemmThreads);
        shape.dynamicSmemBytes = kSmem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = static_cast<unsigned>(s);
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        shape.attrs = attr;
        shape.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&d.clusters[s], gemm_kernel(128), &shape) != cudaSuccess) {
            d.clusters[s] = 0;
            (void)cudaGetLastError();
        }
    }
    return W4A16_OK;
}

int current_device(const GemmDevice** dev) {
    static PerDevice<GemmDevice> devices;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices) return W4A16_ERR_LAUNCH;
    return devices.get(device, [device](GemmDevice& d) { return learn_device(device, d); }, dev);
}

// What a call with this much workspace does: runs that may not cut tiles are whole ones.
GemmPlan plan_on(const GemmDevice& dev, int64_t M, int64_t N, int64_t K, size_t workspace_bytes) {
    const int sms = std::min(dev.sms, 148);
    GemmPlan g = plan_gemm(M, N, K, sms, dev.clusters);
    if (g.cut && workspace_bytes < linear_counter_bytes(M, N) + gemm_partial_bytes(g)) {
        g.cut = false;
        g.grid = static_cast<int>(std::min<long long>(sms, g.tiles));
        g.time = g.whole_time;
    }
    return g;
}

}  // namespace

// The status word's device address, looked up once per device.
unsigned* tcgen05_status_address() {
    static std::atomic<unsigned*> cached[kMaxDevices] = {};
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices) return nullptr;
    unsigned* address = cached[device].load(std::memory_order_relaxed);
    if (address == nullptr) {
        void* found = nullptr;
        if (cudaGetSymbolAddress(&found, g_tcgen05_status) != cudaSuccess) return nullptr;
        address = static_cast<unsigned*>(found);
        cached[device].store(address, std::memory_order_relaxed);
    }
    return address;
}

// Reads (and clears) the status word of the tensor-core kernels.  Synchronises the device.
int read_tcgen05_status(unsigned* value) {
    unsigned zero = 0;
    if (cudaMemcpyFromSymbol(value, g_tcgen05_status, sizeof(unsigned)) != cudaSuccess) return W4A16_ERR_LAUNCH;
    if (cudaMemcpyToSymbol(g_tcgen05_status, &zero, sizeof(unsigned)) != cudaSuccess) return W4A16_ERR_LAUNCH;
    return W4A16_OK;
}

// The plan for the current device, or where there is none, for a B200.
static GemmPlan plan_here(int64_t M, int64_t N, int64_t K, size_t workspace_bytes) {
    static const GemmDevice b200;
    const GemmDevice* dev = nullptr;
    if (current_device(&dev) != W4A16_OK) {
        (void)cudaGetLastError();
        dev = &b200;
    }
    return plan_on(*dev, M, N, K, workspace_bytes);
}

size_t gemm_scratch_bytes(int64_t M, int64_t N, int64_t K) {
    if (M > INT32_MAX || N > INT32_MAX || K > INT32_MAX) return 0;
    const GemmPlan g = plan_here(M, N, K, SIZE_MAX);
    return g.cut ? linear_counter_bytes(M, N) + gemm_partial_bytes(g) : 0;
}

double gemm_time(int64_t M, int64_t N, int64_t K, size_t workspace_bytes) { return plan_here(M, N, K, workspace_bytes).time; }

int launch_linear_gemm(const LinearProblem& prob, cudaStream_t stream) {
    if (prob.K % kBlockK != 0 || prob.K <= 0 || !is_stream_group(prob.group)) return W4A16_ERR_BAD_CONFIG;
    if (prob.M > INT32_MAX || prob.N > INT32_MAX || prob.K > INT32_MAX) return W4A16_ERR_TOO_LARGE;
    if (reinterpret_cast<uintptr_t>(prob.x) % 16 != 0 || reinterpret_cast<uintptr_t>(prob.packed) % 16 != 0) {
        return W4A16_ERR_MISALIGNED;
    }
    const GemmDevice* dev = nullptr;
    const int known = current_device(&dev);
    if (known != W4A16_OK) return known;
    const GemmPlan g = plan_on(*dev, prob.M, prob.N, prob.K, usable_workspace(prob));
    if (g.tiles * g.k_blocks > INT32_MAX) return W4A16_ERR_TOO_LARGE;
    const size_t counters = linear_counter_bytes(prob.M, prob.N);
    CUtensorMap x_map, w_map;
    if (!encode_rows(&x_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, prob.x, prob.M, prob.K * 2, 128, g.bn, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B) ||
        !encode_rows(&w_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, prob.packed, prob.N, prob.K / 2, kBlockK / 2, kRows,
                     CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B)) {
        return W4A16_ERR_LAUNCH;
    }
    GemmParams params;
    params.scales = prob.scales;
    params.y = static_cast<__half*>(prob.y);
    params.bias = prob.bias;
    params.partial = g.cut ? reinterpret_cast<float*>(static_cast<char*>(prob.workspace) + counters) : nullptr;
    params.counters = static_cast<unsigned*>(prob.workspace);
    params.status = tcgen05_status_address();
    if (params.status == nullptr) return W4A16_ERR_LAUNCH;
    params.M = static_cast<int>(prob.M);
    params.N = static_cast<int>(prob.N);
    params.k_blocks = g.k_blocks;
    params.bn = g.bn;
    // Codes come from HBM and want the most blocks in flight; x comes out of L2.  128 batch rows: 3 blocks of x, 6 of codes;
    // 64 rows: 4 and 8.
    const int x_bytes = 2 * g.bn * 128;
    const int room = kSmem - kBarrierBytes - 1024;
    params.code_slots = std::min(kMaxCodeSlots, (room - 3 * x_bytes) / kCodeBytes);
    params.x_slots = std::min(kRing, (room - params.code_slots * kCodeBytes) / x_bytes);
    params.slots = g.bn <= 64 ? 3 : 2;
    params.cluster = g.cluster;
    params.m_tiles = g.m_tiles;
    const long long pieces = params.partial != nullptr ? g.tiles * g.k_blocks : g.tiles;
    params.run = static_cast<int>(pieces / g.grid);
    params.longer = static_cast<int>(pieces % g.grid);

    const void* kernel = gemm_kernel(prob.group);
    cudaLaunchConfig_t launch = {};
    launch.gridDim = dim3(static_cast<unsigned>(g.cluster > 1 ? g.tiles * g.cluster : g.grid));
    launch.blockDim = dim3(kGemmThreads);
    // (a cluster keeps its sums where the rings were: 1 KB per batch row, less than x and codes take)
    launch.dynamicSmemBytes = static_cast<size_t>(params.x_slots) * x_bytes + params.code_slots * kCodeBytes + kBarrierBytes + 1024;
    launch.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = static_cast<unsigned>(g.cluster);
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    launch.attrs = attr;
    launch.numAttrs = g.cluster > 1 ? 2 : 1;
    void* args[] = {&params, &x_map, &w_map};
    if (cudaLaunchKernelExC(&launch, kernel, args) != cudaSuccess) return W4A16_ERR_LAUNCH;
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    return W4A16_OK;
}

}  // namespace w4a16

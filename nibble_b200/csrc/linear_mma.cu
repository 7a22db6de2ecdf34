// Fused W4A16 linear for sm_100a: packed INT4 weights are streamed from HBM, unpacked to exact FP16
// integers with two-instruction-per-pair bit tricks, and fed to the tensor cores as the 16-row
// operand of m16n8k16 MMAs whose 8-wide axis carries the batch.  The group scale multiplies the
// FP32 accumulator once per 128 k, never the individual weights.
//
// Replaces the reference's M=1 decode kernel (csrc/int4_linear_kernel.cu:325-404), its M=2..8
// small-batch kernel (:542-617) and, for larger M, its dequantise-then-cuBLAS route
// (w4a16/linear.py:132-152); one design covers all of them because the work per weight byte is
// independent of M as long as the batch fits the MMA's n axis.
//
// Shape of a launch
//   CTA        : 8 warps = RW row groups x KW warps; the KW warps of a group split the K range of
//                one row tile between them (contiguous sub-ranges), the RW groups own different
//                row tiles.  CTAs are persistent: the grid is what is resident at once and every
//                group strides over the row tiles.
//   row tile   : 16*TILES consecutive output rows.  Row-major [N, K/2] makes a row's K range one
//                contiguous byte run; lane (g, t) owns 16 bytes of rows g and g+8 per 128-wide K
//                chunk, so a quad covers the 64 bytes of one scale group.
//   weights    : each thread keeps a ring of STAGES slots in shared memory, filled with 16-byte
//                cp.async copies of exactly the bytes its own MMAs will consume (plus one 4-byte
//                scale pair per row).  The thread's own cp.async.wait_group is the only
//                synchronisation of the stream, and the bytes in flight per SM are set by the ring
//                depth, not by registers.  Slot addresses are compile-time offsets: the step loop
//                is unrolled over the ring.
//   x          : copied once per CTA into shared memory, already permuted to the (k, k+4) pairing
//                the unpack produces; a warp's B-fragment read is one conflict-free 512-byte row.
//   reduction  : warps of a group combine through shared memory (one named barrier per group and
//                tile); optional K-split CTAs (grid.y) combine through an FP32 workspace, the
//                group that arrives last summing the partials in split order.
//
// The instruction budget is what bounds this kernel on B200: at 6.5 TB/s an SM has about 43 clocks
// per KB of packed weights, lop3/shf/prmt and fma.f16x2 each issue at 2 warp-instructions per clock
// per SM, and the unpack alone needs 40 + 32 of them per KB.  Hence no per-step address arithmetic,
// no register clearing and no register-to-register copies in the step loop.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <tuple>
#include <utility>

#include "kernels.h"
#include "linear_mma_body.cuh"
#include "linear_mma_variants.cuh"
#include "unpack.cuh"

namespace w4a16 {
namespace {

// What a kernel needs to be the reader of a sharded layer's publication.
struct ReaderParams {
    const unsigned* epoch;
    unsigned* const* consumed;
    unsigned* staged_counter;
    unsigned* status;
    long long stride;
    long long max_polls;
    long long col0, cols_per_rank;
    int rank, world;
};

// Block-wide: the last block of the grid to get here gives the buffers back to the senders.
__device__ __forceinline__ void reader_release(const ReaderParams& r, unsigned epoch) {
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned blocks = gridDim.x * gridDim.y * gridDim.z;
        if (atomicAdd(r.staged_counter, 1u) == blocks - 1) {
            *r.staged_counter = 0u;
            release_buffers(r.consumed, r.rank, r.world, epoch);
        }
    }
}

// A reader as a kernel of its own: copies `units` groups of eight FP16 values of the publication out of the
// result buffer (tagged elements -> plain FP16), re-reading what has not arrived yet, then releases the buffer.
// `ld` is the row length of the gathered result in elements (names the sender of a missing element).
__global__ void wait_peers_kernel(const ReaderParams r, const uint4* buffer0, uint4* out, long long units, long long ld) {
    pdl_release_downstream();
    pdl_wait_for_upstream();
    const unsigned epoch = __ldcg(r.epoch);
    const unsigned tag = tag_of(epoch);
    const unsigned tag2 = tag | (tag << 16);
    const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(buffer0) + (epoch & 1u) * r.stride);
    for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < units;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        Tagged8 t = load_tagged8(src + 2 * i);
        if (!wait_tagged8(src + 2 * i, tag2, r.max_polls, r.status, t)) {
            const long long column = r.col0 + (ld > 0 ? (i * 8) % ld : 0);
            atomicMax(r.status, sender_of(column, r.cols_per_rank, r.world) + 1u);
        }
        out[i] = values_of(t);
    }
    reader_release(r, epoch);
}

// y = half(sum over ranks of partials[rank]), summed in rank order so every rank gets identical bits.
// With a reader description the partials are tagged 64-bit elements of a publication: each is re-read
// (bounded) until it has arrived, and the buffer is released afterwards.
__global__ void sum_partials_kernel(const void* __restrict__ partials, __half* __restrict__ y, long long count,
                                    int world, const ReaderParams r) {
    pdl_release_downstream();
    pdl_wait_for_upstream();
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r.epoch == nullptr) {
        if (i < count) {
            float sum = 0.f;
            for (int k = 0; k < world; ++k) sum += __ldcg(static_cast<const float*>(partials) + static_cast<long long>(k) * count + i);
            y[i] = __float2half_rn(sum);
        }
        return;
    }
    const unsigned epoch = __ldcg(r.epoch);
    const unsigned long long tag = tag_of(epoch);
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(
        static_cast<const char*>(partials) + (epoch & 1u) * r.stride);
    if (i < count) {
        float sum = 0.f;
        for (int k0 = 0; k0 < world; k0 += 8) {
            unsigned long long v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (k0 + j < world) {
                    asm volatile("ld.volatile.global.u64 %0, [%1];" : "=l"(v[j]) : "l"(src + static_cast<long long>(k0 + j) * count + i));
                }
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (k0 + j < world) {
                    const unsigned long long* at = src + static_cast<long long>(k0 + j) * count + i;
                    long long poll = 0;
                    while ((v[j] >> 32) != tag && poll++ < r.max_polls) {
                        if ((poll & 255) == 255 && already_failed(r.status)) break;
                        __nanosleep(20);
                        asm volatile("ld.volatile.global.u64 %0, [%1];" : "=l"(v[j]) : "l"(at));
                    }
                    if ((v[j] >> 32) != tag) atomicMax(r.status, static_cast<unsigned>(k0 + j) + 1u);
                    sum += __uint_as_float(static_cast<unsigned>(v[j]));
                }
            }
        }
        y[i] = __float2half_rn(sum);
    }
    reader_release(r, epoch);
}

// ------------------------------------------------------------------------------------------------
template <int NT, int XB, int TILES, int KW>
bool pick_pipeline(int unroll, int stages, Variant* v) {
    if (unroll == 1) {   // odd K/128: the slow-scale path, one tile per warp and one ring depth only
        if constexpr (TILES == 1) {
            if (stages != 3) return false;
            *v = variant_of<NT, XB, 1, KW, 1, 3, kGroup>();
            return true;
        } else {
            return false;
        }
    }
    if (unroll != 2) return false;
    if (stages == 3) { *v = variant_of<NT, XB, TILES, KW, 2, 3, kGroup>(); return true; }
    if (stages == 4) { *v = variant_of<NT, XB, TILES, KW, 2, 4, kGroup>(); return true; }
    return false;
}

template <int NT, int XB, int TILES>
bool pick_kw(int kw, int unroll, int stages, Variant* v) {
    switch (kw) {
        case 1: return pick_pipeline<NT, XB, TILES, 1>(unroll, stages, v);
        case 2: return pick_pipeline<NT, XB, TILES, 2>(unroll, stages, v);
        case 4: return pick_pipeline<NT, XB, TILES, 4>(unroll, stages, v);
        case 8: return pick_pipeline<NT, XB, TILES, 8>(unroll, stages, v);
        default: return false;
    }
}

template <int NT, int XB>
bool pick_tiles(const w4a16_linear_config& c, Variant* v) {
    switch (c.row_tiles) {
        case 1: return pick_kw<NT, XB, 1>(c.k_warps, c.unroll, c.stages, v);
        case 2:
            if constexpr (NT <= 2) {
                return pick_kw<NT, XB, 2>(c.k_warps, c.unroll, c.stages, v);
            } else {
                return false;
            }
        default: return false;
    }
}

bool pick_variant(int64_t group, int nt, bool single_row, const w4a16_linear_config& c, Variant* v) {
    if (group != kGroup) return pick_group_variant(static_cast<int>(group), nt, single_row, c, v);
    switch (nt) {
        case 1: return single_row ? pick_tiles<1, 1>(c, v) : pick_tiles<1, 8>(c, v);
        case 2: return pick_tiles<2, 16>(c, v);
        case 4: return pick_tiles<4, 32>(c, v);
        default: return false;
    }
}

int batch_tiles_for(int64_t M) { return M <= 8 ? 1 : (M <= 16 ? 2 : 4); }
int x_rows_for(int64_t M) { return M == 1 ? 1 : 8 * batch_tiles_for(M); }

constexpr int kMaxDevices = 64;

// SM count of `device`, looked up once per device.
int sm_count(int device) {
    static std::atomic<int> cached[kMaxDevices] = {};
    if (device < 0 || device >= kMaxDevices) return 148;
    int count = cached[device].load(std::memory_order_relaxed);
    if (count == 0) {
        if (cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || count <= 0) return 148;
        cached[device].store(count, std::memory_order_relaxed);
    }
    return count;
}

// Bytes of x a CTA holds for `rows` stored batch rows of a K slice of `chunks` chunks.
size_t x_slice_bytes(int rows, int chunks) { return static_cast<size_t>(rows) * chunks * kGroup * sizeof(__half); }

}  // namespace

// The arrival counters occupy a prefix of the workspace whose size does not depend on the problem (as long as
// the problem has at most kCounterSlots row-tile x batch-block pairs): one workspace may then serve calls of
// different shapes one after the other, because the FP32 partial sums of one call can never land where another
// call keeps its counters (they used to, when the prefix was sized per problem: leftover partials of an N = 2048
// call sat in the counter slots of tiles 128.. of a following N = 2560 call, whose last arriver was then never
// recognised and whose outputs were never written).
constexpr int64_t kCounterSlots = 65536;

size_t linear_counter_bytes(int64_t M, int64_t N) {
    const int64_t row_blocks = (N + 15) / 16;
    const int64_t batch_blocks = (M + 7) / 8;
    const int64_t slots = std::max<int64_t>(row_blocks * batch_blocks, kCounterSlots);
    const size_t bytes = static_cast<size_t>(slots) * sizeof(unsigned);
    return (bytes + 255) & ~static_cast<size_t>(255);
}

size_t linear_workspace_bytes_for(int64_t M, int64_t N, int splits) {
    if (M <= 0 || N <= 0 || splits <= 1) return 0;
    return linear_counter_bytes(M, N) + static_cast<size_t>(splits) * M * N * sizeof(float);
}

namespace {

// Launch shape of a single row.
//   - Up to about three row tiles per resident CTA: all eight warps on each tile.  In a chain of dependent layers the whole share
//     of a CTA is then prefetched before its activations arrive, and at most three short steps per warp remain after
//     the wait (2 us per launch on a fused gate/up layer inside a decode step).
//   - More tiles: as many warps per tile as leave each of them four steps (3072 -> 16000: two warps 8.5 us, eight 10.2;
//     8192 -> 28672: eight 25.6, one 29.3).
//   - An activation slice above 32 KB would crowd the copy ring out of shared memory at two CTAs per SM: K is split four ways, and
//     the fewest warps that still give 12 streaming ones per SM share a tile (28672 -> 8192: 28.2 us, 30.5 split two ways).
//   - Fewer tiles than a quarter of the SMs and K to spare: K is split until two CTAs per SM have work (16384 -> 512: 5.0 us, 6.6
//     unsplit).  With 64 tiles unsplit is already faster (8192 -> 1024: 4.6 against 5.2 us).
w4a16_linear_config choose_single_row(int64_t tiles, int chunks, int sms, int max_splits) {
    w4a16_linear_config c{};
    int kw = 1, splits = 1;
    if (x_slice_bytes(1, chunks) > 32u * 1024 && max_splits > 1) {
        splits = std::min(4, max_splits);
        while (kw < 8 && tiles * kw * splits < static_cast<int64_t>(sms) * 12) kw *= 2;
    } else if (tiles <= 6 * sms) {
        while (kw < 8 && chunks >= kw * 4) kw *= 2;
        while (4 * tiles <= sms && splits * 2 <= max_splits && tiles * splits * 2 <= 2 * sms && chunks >= splits * 32) splits *= 2;
    } else {
        while (kw < 8 && chunks >= kw * 16 + (kw == 1 ? 8 : 0)) kw *= 2;
    }
    c.k_warps = kw;
    c.k_splits = splits;
    return c;
}

// Launch shape of a batch: the cheapest by a model fitted to measurements (25 layers from 1024 x 1024 to 28672 -> 8192, batches of 2
// to 64 rows, every k_warps x k_splits; the pick is on average within 2 % of the fastest).  What the model knows: a CTA's
// start; the batch rows it stages; its steps, each as long as the step's own chain or the SM's issue slots allow,
// whichever is longer; the end of a tile; the hand-over of a tile between CTAs that split its K.
// (28672 -> 8192 at 13 rows: 95 -> 62 us against the rule it replaces; 11008 -> 4096 at 2 rows: 18.8 -> 10.7.)
w4a16_linear_config choose_batch(int64_t M, int64_t tiles, int chunks, int unroll, int sms, int max_splits, bool small_group) {
    struct Costs {   // us; steps of 256 K
        double start, stage_per_kb, stage_per_8_rows, step_issue, step_chain, tile_end, split, split_per_row, split_per_cta;
    };
    static const Costs costs[3] = {{1.13, 0.0133, 2.19, 0.382, 0.672, 0.132, 5.34, 0.0021, 0.083},
                                   {1.74, 0.0010, 2.09, 0.414, 0.488, 0.216, 2.52, 0.0006, 0.0},
                                   {0.07, 0.0006, 1.67, 0.841, 0.306, 1.195, 1.10, 0.0031, 0.0}};
    const int nt = batch_tiles_for(M), x_rows = x_rows_for(M);
    const Costs& cost = costs[nt == 1 ? 0 : nt == 2 ? 1 : 2];
    const int64_t batch_blocks = (M + 8 * nt - 1) / (8 * nt);
    const int rows = static_cast<int>(std::min<int64_t>(M, 8 * nt));
    const size_t slot = unroll == 1 ? 8192 : small_group ? 18432 : 16896;
    const size_t reduction = static_cast<size_t>(nt) * 8192;
    w4a16_linear_config best{};
    double best_time = 1e30;
    int fitting = 0;                // the fewest splits whose slice of x fits
    // Up to eight rows on large layers (two row tiles per SM and more), where the model is least sure of splits.  Slower than the
    // fastest of sixteen shapes, on average over 2 to 8 rows: K that fits unsplit (140 shapes), never split 0.5 %, by the model 1.2
    // (5632 -> 16384, 8 rows: 15.9 / 18.8 us); K that only fits four ways (19), always four 0 %, by the model 4.3 (28672 -> 8192, 8
    // rows: 40.1 / 42.8); K that fits two ways (306 shapes of 10752 to 20480 -> 4864 to 20480), by the model with four ways a fifth
    // dearer 1.4 %, as it is 3.3, always two 6.5 (20480 -> 10240, 4 rows: 39.3 / 39.3 / 45.2).
    const bool large = nt == 1 && tiles >= 2 * static_cast<int64_t>(sms);
    best.k_warps = 8;
    best.k_splits = 1;
    for (int splits = 1; splits <= std::min(max_splits, kMaxKSplits) && splits <= chunks; splits *= 2) {
        const int per_split = ((chunks + splits - 1) / splits + unroll - 1) / unroll * unroll;
        if ((splits - 1) * per_split >= chunks) break;                    // an empty split
        const size_t slice = x_slice_bytes(x_rows, per_split);
        // (smaller scale groups are built for two and eight warps)
        for (int kw = small_group ? 2 : 1; kw <= 8; kw *= small_group ? 4 : 2) {
            const size_t smem = kFlagBytes + (kw > 1 ? reduction : 0) + slice + 3 * slot;
            if (smem > static_cast<size_t>(kSmemBudget)) continue;
            const int per_sm = nt <= 2 && smem <= static_cast<size_t>(kSmemPerSm / 2 - 1024) ? 2 : 1;
            const int64_t tile_ctas = (tiles * kw + 7) / 8;
            const int64_t resident = std::max<int64_t>(1, static_cast<int64_t>(sms) * per_sm / (splits * batch_blocks));
            const int64_t grid_x = std::min(tile_ctas, resident);
            const int64_t ctas = grid_x * splits * batch_blocks;
            const double rounds = static_cast<double>((tile_ctas + grid_x - 1) / grid_x);
            const double active = static_cast<double>(std::min<int64_t>(per_sm, (ctas + sms - 1) / sms));
            const double waves = static_cast<double>((ctas + static_cast<int64_t>(sms) * per_sm - 1) / (static_cast<int64_t>(sms) * per_sm));
            const double steps = 0.5 * (((per_split + kw - 1) / kw + unroll - 1) / unroll * unroll);
            double tile = steps * std::max(cost.step_chain, cost.step_issue * active) + cost.tile_end;
            if (splits > 1) tile += cost.split + cost.split_per_row * rows * splits + cost.split_per_cta * splits;
            double time = waves * (cost.start + cost.stage_per_8_rows * rows / 8.0 +
                                   cost.stage_per_kb * rows * per_split * 0.25 * active + rounds * tile);
            if (large && fitting == 2 && splits == 4) time *= 1.2;
            if (time < best_time) {
                best_time = time;
                best.k_warps = kw;
                best.k_splits = splits;
            }
        }
        if (fitting == 0 && best_time < 1e30) fitting = splits;
        if (large && fitting != 0 && fitting != 2) break;
    }
    // Nothing fits shared memory: the most splits, for the launch to refuse (and its caller to take another kernel).
    if (best_time == 1e30) {
        while (best.k_splits * 2 <= std::min(max_splits, kMaxKSplits) && chunks >= best.k_splits * 2) best.k_splits *= 2;
    }
    return best;
}

}  // namespace

w4a16_linear_config choose_linear_config(int64_t M, int64_t N, int64_t K, int max_splits, bool small_group) {
    // A model calls with a few dozen shapes over and over: each thread keeps its recent answers.
    struct Answer {
        int64_t M = -1, N = 0, K = 0;
        int max_splits = 0;
        bool small_group = false;
        w4a16_linear_config config{};
    };
    static thread_local Answer answers[64];
    const uint64_t mixed = (static_cast<uint64_t>(M) * 31 + static_cast<uint64_t>(N)) * 0x9E3779B97F4A7C15ull ^
                           (static_cast<uint64_t>(K) * 0xC2B2AE3D27D4EB4Full + static_cast<uint64_t>(max_splits * 2 + small_group));
    Answer& answer = answers[mixed >> 58];
    if (answer.M == M && answer.N == N && answer.K == K && answer.max_splits == max_splits &&
        answer.small_group == small_group) {
        return answer.config;
    }

    const int sms = 148;
    const int chunks = static_cast<int>(K / kGroup);
    const int64_t tiles = (N + 15) / 16;
    const int unroll = chunks % 2 == 0 ? 2 : 1;
    w4a16_linear_config c = M == 1 ? choose_single_row(tiles, chunks, sms, max_splits)
                                   : choose_batch(M, tiles, chunks, unroll, sms, max_splits, small_group);
    c.row_tiles = 1;     // (two 16-row tiles per warp were never the fastest)
    c.unroll = unroll;
    c.stages = 0;        // chosen at launch from the shared memory left over
    answer = {M, N, K, max_splits, small_group, c};
    return c;
}

namespace {

int reader_params(const w4a16_peer_source* source, ReaderParams* r) {
    *r = ReaderParams{};
    if (source == nullptr) return W4A16_OK;
    if (source->epoch == nullptr || source->consumed == nullptr || source->staged_counter == nullptr ||
        source->status == nullptr) {
        return W4A16_ERR_NULL_POINTER;
    }
    if (source->world < 1 || source->world > 32 || source->rank < 0 || source->rank >= source->world ||
        source->max_polls <= 0 || source->buffer_stride < 0 || source->first_column < 0 || source->columns_per_rank < 0) {
        return W4A16_ERR_BAD_SHAPE;
    }
    *r = ReaderParams{source->epoch, source->consumed, source->staged_counter, source->status, source->buffer_stride,
                      source->max_polls, source->first_column, source->columns_per_rank, source->rank, source->world};
    return W4A16_OK;
}

template <typename Kernel, typename... Args>
int launch_small(Kernel kernel, unsigned blocks, unsigned threads, bool programmatic, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t launch = {};
    launch.gridDim = dim3(blocks, 1, 1);
    launch.blockDim = dim3(threads, 1, 1);
    launch.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    launch.attrs = attr;
    launch.numAttrs = programmatic ? 1 : 0;
    if (cudaLaunchKernelEx(&launch, kernel, args...) != cudaSuccess) return W4A16_ERR_LAUNCH;
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    return W4A16_OK;
}

}  // namespace

int launch_wait_peers(const w4a16_peer_source* source, const void* buffer0, void* out, int64_t count, int64_t ld,
                      bool programmatic, cudaStream_t stream) {
    if (source == nullptr) return W4A16_ERR_NULL_POINTER;
    ReaderParams r;
    const int status = reader_params(source, &r);
    if (status != W4A16_OK) return status;
    if (count < 0 || count % 8 != 0) return W4A16_ERR_BAD_SHAPE;
    if (count > 0) {
        if (buffer0 == nullptr || out == nullptr) return W4A16_ERR_NULL_POINTER;
        if (reinterpret_cast<uintptr_t>(buffer0) % 32 != 0 || reinterpret_cast<uintptr_t>(out) % 16 != 0 ||
            source->buffer_stride % 32 != 0) {
            return W4A16_ERR_MISALIGNED;
        }
    }
    const long long units = count / 8;
    const unsigned blocks = static_cast<unsigned>(std::min<long long>(64, std::max<long long>(1, (units + 255) / 256)));
    return launch_small(wait_peers_kernel, blocks, 256, programmatic, stream, r, static_cast<const uint4*>(buffer0),
                        static_cast<uint4*>(out), units, static_cast<long long>(ld));
}

int launch_sum_partials(const void* partials, __half* y, int64_t count, int world, const w4a16_peer_source* source,
                        bool programmatic, cudaStream_t stream) {
    if (count <= 0) return W4A16_OK;
    ReaderParams r;
    const int status = reader_params(source, &r);
    if (status != W4A16_OK) return status;
    if (source != nullptr && (reinterpret_cast<uintptr_t>(partials) % 8 != 0 || source->buffer_stride % 8 != 0)) {
        return W4A16_ERR_MISALIGNED;
    }
    const int threads = 256;
    const int64_t blocks = (count + threads - 1) / threads;
    if (blocks > INT32_MAX) return W4A16_ERR_TOO_LARGE;
    return launch_small(sum_partials_kernel, static_cast<unsigned>(blocks), threads, programmatic, stream, partials, y,
                        static_cast<long long>(count), world, r);
}

// Reads and clears the bounds-check word of the streaming kernel (builds with -DW4A16_BOUNDS_CHECK only).
int read_bounds_check(unsigned* site, unsigned* count) {
#ifdef W4A16_BOUNDS_CHECK
    unsigned word[2] = {0u, 0u};
    const unsigned zero[2] = {0u, 0u};
    if (cudaMemcpyFromSymbol(word, g_bounds_word, sizeof(word)) != cudaSuccess ||
        cudaMemcpyToSymbol(g_bounds_word, zero, sizeof(zero)) != cudaSuccess) {
        return W4A16_ERR_LAUNCH;
    }
    *site = word[0];
    *count = word[1];
    return W4A16_OK;
#else
    *site = 0u;
    *count = 0u;
    return W4A16_ERR_BAD_CONFIG;
#endif
}

int launch_linear_mma(const LinearProblem& prob, const w4a16_linear_config& cfg_in, bool early_weights,
                      bool out_f32, cudaStream_t stream) {
    if (!is_stream_group(prob.group) || prob.K % kGroup != 0) return W4A16_ERR_BAD_CONFIG;
    if (prob.M > INT32_MAX || prob.N > INT32_MAX || prob.K > INT32_MAX) return W4A16_ERR_TOO_LARGE;
    w4a16_linear_config cfg = cfg_in;
    const int nt = batch_tiles_for(prob.M);
    const int x_rows = x_rows_for(prob.M);
    const int chunks = static_cast<int>(prob.K / kGroup);
    const int splits = cfg.k_splits;
    if (splits < 1 || splits > kMaxKSplits || splits > chunks) return W4A16_ERR_BAD_CONFIG;
    // With unroll 2 the two scales of a step travel as one 4-byte copy: that needs K/128 even and
    // the scale matrix 4-byte aligned.
    if (cfg.unroll == 2 && (chunks % 2 != 0 || reinterpret_cast<uintptr_t>(prob.scales) % 4 != 0)) {
        return W4A16_ERR_BAD_CONFIG;
    }
    if (cfg.unroll != 1 && cfg.unroll != 2) return W4A16_ERR_BAD_CONFIG;
    if (prob.group != kGroup) {
        // several scales of a row travel together: 16-byte copies at most
        if (reinterpret_cast<uintptr_t>(prob.scales) % 16 != 0) return W4A16_ERR_BAD_CONFIG;
        cfg.row_tiles = 1;
        cfg.k_warps = cfg.k_warps <= 2 ? 2 : 8;
    }
    if (cfg.stages != 0 && cfg.stages != 3 && cfg.stages != 4) return W4A16_ERR_BAD_CONFIG;

    const int per_split = (chunks + splits - 1) / splits;
    const int chunks_per_split = (per_split + cfg.unroll - 1) / cfg.unroll * cfg.unroll;
    if ((splits - 1) * chunks_per_split >= chunks) return W4A16_ERR_BAD_CONFIG;   // an empty split

    // Ring depth: four slots when two CTAs still fit on an SM with them; else three if that is what lets two CTAs fit;
    // and when the activation slice is so large that only one CTA fits either way, four again (as many bytes in flight
    // as the budget allows, and the step loop is unrolled over 4 positions instead of 6: with eight warps per SM the
    // longer loop showed up as instruction-fetch stalls, `no_instruction` 1.26 per issue at M = 8 on 8192-wide layers).
    Variant variant;
    if (cfg.stages == 0) {
        cfg.stages = cfg.unroll == 1 ? 3 : 4;
        if (cfg.unroll == 2) {
            if (!pick_variant(prob.group, nt, prob.M == 1, cfg, &variant)) return W4A16_ERR_BAD_CONFIG;
            const size_t fixed = kFlagBytes + variant.red_bytes + x_slice_bytes(x_rows, chunks_per_split);
            const size_t half_sm = static_cast<size_t>(kSmemPerSm / 2 - 1024);
            const bool two_with_four = fixed + 4u * variant.stage_bytes <= half_sm;
            const bool two_with_three = fixed + 3u * variant.stage_bytes <= half_sm;
            const bool four_fit = fixed + 4u * variant.stage_bytes <= static_cast<size_t>(kSmemBudget);
            if (!two_with_four && (two_with_three || !four_fit)) cfg.stages = 3;
        }
    }
    if (!pick_variant(prob.group, nt, prob.M == 1, cfg, &variant)) return W4A16_ERR_BAD_CONFIG;

    MmaParams params;
    params.x = prob.x;
    params.packed = prob.packed;
    params.scales = prob.scales;
    params.y = prob.y;
    params.partial = nullptr;
    params.counters = nullptr;
    params.M = static_cast<int>(prob.M);
    params.N = static_cast<int>(prob.N);
    params.K = static_cast<int>(prob.K);
    params.chunks = chunks;
    params.chunks_per_split = chunks_per_split;
    params.k_splits = splits;
    params.row_tiles_total = static_cast<int>((prob.N + 16 * cfg.row_tiles - 1) / (16 * cfg.row_tiles));
    params.out_f32 = out_f32 ? 1 : 0;
    params.peer_out = nullptr;
    params.done_counter = nullptr;
    params.send_epoch = nullptr;
    params.peer_status = nullptr;
    params.wait_polls = 0;
    params.ld_out = 0;
    params.col_out = 0;
    params.rank = 0;
    params.world = 1;
    params.x_mode = W4A16_INPUT_PLAIN;
    params.x_ld = prob.K;
    params.x_row_index = nullptr;
    params.x_second = nullptr;
    params.norm_weight = nullptr;
    params.stream_out = nullptr;
    params.eps = 0.0f;
    params.early_weights = early_weights ? 1 : 0;
    params.bias = prob.bias;
    if (prob.input != nullptr && prob.input->kind != W4A16_INPUT_PLAIN) {
        const w4a16_input_transform& in = *prob.input;
        auto aligned = [](const void* q) { return reinterpret_cast<uintptr_t>(q) % 16 == 0; };
        if (in.kind == W4A16_INPUT_SILU_MUL) {
            params.x_ld = 2 * prob.K;
        } else if (in.kind == W4A16_INPUT_ADD_RMSNORM) {
            if (prob.M != 1) return W4A16_ERR_BAD_SHAPE;
            if (in.norm_weight == nullptr) return W4A16_ERR_NULL_POINTER;
            if (!aligned(in.second) || !aligned(in.norm_weight) || !aligned(in.stream_out)) return W4A16_ERR_MISALIGNED;
            if (in.stream_out != nullptr && (in.stream_out == prob.x || in.stream_out == in.second)) return W4A16_ERR_BAD_CONFIG;
            params.x_second = static_cast<const __half*>(in.second);
            params.norm_weight = static_cast<const __half*>(in.norm_weight);
            params.stream_out = static_cast<__half*>(in.stream_out);
            params.eps = in.eps;
        } else {
            return W4A16_ERR_BAD_CONFIG;
        }
        params.x_mode = in.kind;
    }
    params.consumed = nullptr;
    params.out_stride = 0;
    params.src_epoch = nullptr;
    params.src_consumed = nullptr;
    params.src_col0 = 0;
    params.src_cols_per_rank = 0;
    params.staged_counter = nullptr;
    params.src_stride = 0;
    if (prob.x_ld != 0) {
        if (prob.x_ld < prob.K || prob.x_ld % 8 != 0 || params.x_mode != W4A16_INPUT_PLAIN) return W4A16_ERR_BAD_SHAPE;
        params.x_ld = prob.x_ld;
    }
    if (prob.peers != nullptr) {
        const w4a16_peer_target& t = *prob.peers;
        if (t.outputs == nullptr || t.consumed == nullptr || t.done_counter == nullptr ||
            t.send_epoch == nullptr || t.status == nullptr) {
            return W4A16_ERR_NULL_POINTER;
        }
        if (t.world < 1 || t.world > 32 || t.rank < 0 || t.rank >= t.world || t.ld < prob.N || t.column_offset < 0 ||
            t.max_polls <= 0 || t.buffer_stride < 0) {
            return W4A16_ERR_BAD_SHAPE;
        }
        params.peer_out = t.outputs;
        params.consumed = t.consumed;
        params.done_counter = t.done_counter;
        params.send_epoch = t.send_epoch;
        params.peer_status = t.status;
        params.out_stride = t.buffer_stride;
        params.wait_polls = t.max_polls;
        params.ld_out = t.ld;
        params.col_out = t.column_offset;
        params.rank = t.rank;
        params.world = t.world;
    }
    if (prob.source != nullptr) {
        ReaderParams r;
        const int status = reader_params(prob.source, &r);
        if (status != W4A16_OK) return status;
        // tagged elements are 4 bytes each and are read 32 bytes at a time
        if (params.x_mode != W4A16_INPUT_PLAIN || r.stride % 32 != 0 || reinterpret_cast<uintptr_t>(prob.x) % 32 != 0) {
            return W4A16_ERR_BAD_CONFIG;
        }
        if (prob.peers != nullptr && (prob.peers->world != r.world || prob.peers->rank != r.rank)) return W4A16_ERR_BAD_SHAPE;
        params.src_epoch = r.epoch;
        params.src_col0 = r.col0;
        params.src_cols_per_rank = r.cols_per_rank;
        params.src_consumed = r.consumed;
        params.staged_counter = r.staged_counter;
        params.src_stride = r.stride;
        params.rank = r.rank;
        params.world = r.world;
        if (params.peer_status == nullptr) params.peer_status = r.status;
        if (params.wait_polls == 0) params.wait_polls = r.max_polls;
    }
    if (splits > 1) {
        const size_t need = linear_workspace_bytes_for(prob.M, prob.N, splits);
        if (prob.workspace == nullptr || prob.workspace_bytes < need) return W4A16_ERR_WORKSPACE;
        if (reinterpret_cast<uintptr_t>(prob.workspace) % 16 != 0) return W4A16_ERR_MISALIGNED;
        params.counters = static_cast<unsigned*>(prob.workspace);
        params.partial = reinterpret_cast<float*>(static_cast<char*>(prob.workspace) +
                                                  linear_counter_bytes(prob.M, prob.N));
    }

    const size_t smem = kFlagBytes + static_cast<size_t>(variant.red_bytes) + x_slice_bytes(x_rows, chunks_per_split) +
                        static_cast<size_t>(variant.stages) * variant.stage_bytes;
    if (smem > static_cast<size_t>(kSmemBudget)) return W4A16_ERR_WORKSPACE;   // x slice too large: more K splits

    // Opt in to large dynamic shared memory once per device and kernel variant (the attribute belongs to
    // the function as loaded on one device), and learn its occupancy there (cached per device, variant
    // and shared-memory size).
    const void* kernel = variant.fn;
    if (prob.peers != nullptr || prob.source != nullptr) {
        if (variant.fn_exchange == nullptr) return W4A16_ERR_BAD_CONFIG;
        kernel = variant.fn_exchange;
    } else if (early_weights && prob.bias == nullptr && !prob.among_transforms && variant.fn_early != nullptr) {
        kernel = variant.fn_early;
    }
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return W4A16_ERR_LAUNCH;
    static std::mutex mutex;
    static std::map<std::tuple<int, const void*, size_t>, int> occupancy;
    int blocks_per_sm = 0;
    {
        std::lock_guard<std::mutex> lock(mutex);
        const auto key = std::make_tuple(device, kernel, smem);
        const auto found = occupancy.find(key);
        if (found != occupancy.end()) {
            blocks_per_sm = found->second;
        } else {
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget) !=
                cudaSuccess) {
                return W4A16_ERR_LAUNCH;
            }
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm, kernel, kThreads, smem) !=
                    cudaSuccess || blocks_per_sm < 1) {
                return W4A16_ERR_LAUNCH;
            }
            occupancy.emplace(key, blocks_per_sm);
        }
    }

    const int rw = kWarpsPerCta / cfg.k_warps;
    const int64_t batch_blocks = (prob.M + 8 * nt - 1) / (8 * nt);
    if (batch_blocks > 65535) return W4A16_ERR_TOO_LARGE;
    const int64_t tile_ctas = (params.row_tiles_total + rw - 1) / rw;
    int64_t resident = static_cast<int64_t>(sm_count(device)) * blocks_per_sm / (splits * batch_blocks);
    if (resident < 1) resident = 1;
    const int64_t grid_x = tile_ctas < resident ? tile_ctas : resident;
    const dim3 grid(static_cast<unsigned>(grid_x), static_cast<unsigned>(splits), static_cast<unsigned>(batch_blocks));

    cudaLaunchConfig_t launch = {};
    launch.gridDim = grid;
    launch.blockDim = dim3(kThreads, 1, 1);
    launch.dynamicSmemBytes = smem;
    launch.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    launch.attrs = attr;
    // Always programmatic: with the weights waited for (early_weights false) the kernel still starts, and its first weights
    // travel to L2, while the one before it drains; a kernel of another kind in front completes before this one starts.
    // Not so the tensor-parallel launches, whose CTAs would hold SMs while they wait for other GPUs.
    launch.numAttrs = early_weights || kernel == variant.fn ? 1 : 0;
    void* args[] = {const_cast<MmaParams*>(&params)};
    if (cudaLaunchKernelExC(&launch, kernel, args) != cudaSuccess) return W4A16_ERR_LAUNCH;
    g_launch_count.fetch_add(1, std::memory_order_relaxed);
    return W4A16_OK;
}

}  // namespace w4a16

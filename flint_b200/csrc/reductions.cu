// Deterministic reductions over rows: flint_bias_gradient, flint_layernorm_backward,
// flint_embedding_backward and their workspace queries.
//
// Column sums (a bias gradient, LayerNorm's dgamma/dbeta, the position table's
// gradient) share one two-pass scheme whose addition order depends only on the
// matrix shape, never on the GPU: rows are cut into chunks of 256; inside a
// chunk, lane-row y (0..7) adds rows y, y+8, ... with a compensated FP32 sum,
// the eight lane-rows are merged in order of y, and the chunk's (sum, error)
// pair per column goes to the workspace as two FP32 rows; a second pass merges
// the chunks (lane l takes chunks l, l+32, ..., then a butterfly) and writes
// sum + error. There are no floating-point atomics anywhere.
// Reference for the order and the workspace layout:
// src/kernels/bias_gradient.cu:82-178, src/kernels/layernorm_backward.cu:119-233,
// src/kernels/embedding_backward.cu:131-345 and embedding_backward.cuh:31-79.
//
// Argument checks follow src/api/bias_gradient.cpp:11-67,
// src/api/layernorm.cpp:55-119 and src/api/embedding.cpp:55-134.
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <type_traits>

#include <cuda.h>
#include <cuda_fp16.h>

#include "common.h"
#include "device_utils.cuh"
#include "flint/flint_b200.h"

namespace {

using fb::Comp;

constexpr size_t kChunkRows = 256;
constexpr int kLaneRows = 8;    // interleaved row streams per chunk
constexpr size_t kMaxCols = size_t{65535} * 256;            // 16,776,960
constexpr size_t kMaxBiasRows = size_t{0x7fffffff} * 256;   // 549,755,813,632
constexpr size_t kMaxRows8 = size_t{0x7fffffff} * 8;

constexpr size_t column_sum_workspace(size_t rows, size_t cols) {
    return (rows + kChunkRows - 1) / kChunkRows * cols * 8;
}

enum class Source { kHalf, kHalfTimesXhat, kFloat };

// First pass. CTA (chunk, tile of 64 kPairs columns): warp ly adds row stream ly, a lane the
// column pairs 64 i + 2 lane of the tile, and a ninth warp fetches.
//
// A chunk's adding is a chain of 32 rows per stream, seven (with a product eleven) dependent
// FP32 operations each. A small matrix needs many CTAs with that chain alone, 64 columns each
// (in the place of 256: 300 x 768 with a product 8.8 -> 5.7 us, 8,192 x 768 FP16 9.0 -> 6.4 us). Once
// there are more than three CTAs per SM the chains of two column pairs a lane hide each other
// better than more CTAs do, and the CTAs pass in fewer rounds: see wide_tiles().
//
// The chunk's rows reach the CTA through shared memory, 32 to a stage: one TMA tensor load
// per operand, or (where the row count does not fit a tensor map) a bulk copy per row segment
// by the fetching warp's lanes. The next stages load while this one is added, so the memory
// has many bytes in flight although every stream takes its rows strictly in order. (A thread
// that loaded its own rows would add each one as it arrived, paying one memory latency per
// row.) The additions run on packed FP32 pairs, a lane's two neighbouring columns.
constexpr int kPairPieces = 8;                         // pieces that a warp's column pairs cover
constexpr int kAddThreads = 32 * kLaneRows;            // a warp per stream; and a fetching warp
constexpr unsigned kTilesY = 32768;                    // tiles per grid layer

template <Source kSource, int kPairs>
struct Staging {
    static constexpr int kTilePieces = kPairPieces * kPairs;
    static constexpr int kTileColumns = kTilePieces * 8;
    static constexpr int kMainBytes = kSource == Source::kFloat ? 32 : 16;  // per piece and row
    static constexpr int kXBytes = kSource == Source::kHalfTimesXhat ? 32 : 0;
    static constexpr int kRows = 32;                                        // rows per stage
    static constexpr int kMainStage = kRows * kTilePieces * kMainBytes;
    static constexpr int kStage = kMainStage + kRows * kTilePieces * kXBytes;
    // All of a chunk's 256 rows at once (FP16, 64 columns), or half of them.
    static constexpr int kStages = kSource == Source::kHalf && kPairs == 1 ? 8 : 4;
    static constexpr int kBytes = kStages * kStage + 128;
};
__device__ int g_reduction_error = 0;

__device__ __forceinline__ uint32_t shared_address(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool staged_try(uint32_t bar, uint32_t parity) {
    uint32_t done = 0;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

// Bounded mbarrier wait: false (and the flag set) after about a second of SM clocks.
__device__ __forceinline__ bool staged_wait(uint32_t bar, uint32_t parity, volatile int* abort) {
    const long long start = clock64();
    for (uint32_t spin = 0;; ++spin) {
        if (staged_try(bar, parity)) {
            return true;
        }
        if ((spin & 63u) == 63u && (*abort != 0 || clock64() - start > 2000000000LL)) {
            *abort = 1;
            return false;
        }
    }
}

// The same for a whole warp, with one outcome for all its lanes (a lane that left alone would
// leave the others waiting for it in the next __syncwarp).
__device__ __forceinline__ bool staged_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort) {
    const long long start = clock64();
    bool done = false;
    for (uint32_t spin = 0;; ++spin) {
        done = done || staged_try(bar, parity);
        if (__all_sync(fb::kFullMask, done)) {
            return true;
        }
        if ((spin & 63u) == 63u &&
            __any_sync(fb::kFullMask, *abort != 0 || clock64() - start > 2000000000LL)) {
            *abort = 1;
            return false;
        }
    }
}

// Tensor maps of the source (and of x for the dgamma sums): one TMA tensor load
// then brings a whole 32-row stage. `use` is 0 for matrices whose row count does
// not fit a tensor map; those stages are fetched row by row.
struct ColumnMaps {
    CUtensorMap main;
    CUtensorMap x;
    int use;
};

// The barriers and statistics of a CTA that adds a tile of a chunk.
template <Source kSource, int kPairs>
struct PartialsShared {
    float mean[kSource == Source::kHalfTimesXhat ? kChunkRows : 1];
    float rstd[kSource == Source::kHalfTimesXhat ? kChunkRows : 1];
    alignas(8) unsigned long long barriers[2 * Staging<kSource, kPairs>::kStages];
    int abort_flag;

    // By one thread, before the CTA waits for earlier kernels.
    __device__ void init() {
        using S = Staging<kSource, kPairs>;
        const uint32_t bar0 = shared_address(barriers);
        abort_flag = 0;
        for (int i = 0; i < S::kStages; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8u * i) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar0 + 8u * (S::kStages + i)),
                         "r"(kLaneRows)
                         : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
};

// Where a CTA's tile lies: worked out before it waits for earlier kernels (behind the wait: 0.03 to 0.1 us of the 2.5 to
// 7 us that sums over a few rows take).
template <Source kSource, int kPairs>
struct PartialsPlace {
    size_t chunk, first;      // chunk of rows, its first row
    int first_piece, width;   // 8-column pieces
    int chunk_rows, stages_total;
    uint32_t staging;

    __device__ PartialsPlace(size_t chunk_, unsigned tile, size_t rows, int pieces, const unsigned char* staging_raw) {
        using S = Staging<kSource, kPairs>;
        chunk = chunk_;
        first_piece = static_cast<int>(tile) * S::kTilePieces;
        width = min(S::kTilePieces, pieces - first_piece);
        first = chunk * kChunkRows;
        chunk_rows = static_cast<int>(rows - first < kChunkRows ? rows - first : kChunkRows);
        stages_total = (chunk_rows + S::kRows - 1) / S::kRows;
        staging = (shared_address(staging_raw) + 127u) & ~127u;
    }
};

// One tile of a chunk, by kAddThreads + 32 threads. (The pointers are after_wait() ones.)
// kPlain: a stream adds its rows with ordinary FP32 adds (one instruction per pair
// instead of seven); the eight streams, the chunks and the lanes are still merged with
// compensated adds in the same fixed order. This is not the reference's pinned
// arithmetic (the public entry points never use it); the model built on the fused
// attention kernels does, where it makes these kernels bandwidth-bound.
// The FP16-times-xhat kernel (LayerNorm's dgamma) also sums the FP16 values themselves
// (dbeta) from the same staged rows, with the operations the FP16 kernel would use, and
// writes those partial sums to `second` (unless kAlso is false).
template <Source kSource, bool kPlain, bool kAlso, int kPairs>
__device__ __forceinline__ void add_tile(const ColumnMaps& maps, float* partial, float* second, const void* src,
                                         const float4* x, const float* mean, const float* rstd, int pieces,
                                         const PartialsPlace<kSource, kPairs>& place,
                                         PartialsShared<kSource, kPairs>& shared, unsigned char* staging_raw) {
    using S = Staging<kSource, kPairs>;
    constexpr int kTilePieces = S::kTilePieces;
    constexpr int kTileColumns = S::kTileColumns;
    // After the last stage the ring's memory holds the eight streams' sums for the merge.
    static_assert(S::kStages * S::kStage >= 2 * kLaneRows * kTileColumns * 4 &&
                      kTileColumns <= kAddThreads,
                  "the merge buffers must fit in the ring, and a thread merge a column");
    const int lane = threadIdx.x % 32;
    const int ly = threadIdx.x / 32;     // 0-7: the row stream; 8: fetching
    const int first_piece = place.first_piece, width = place.width;
    const size_t chunk = place.chunk, first = place.first;
    const int chunk_rows = place.chunk_rows, stages_total = place.stages_total;
    const uint32_t staging = place.staging;
    const uint32_t bar0 = shared_address(shared.barriers);
    auto full_bar = [&](int slot) { return bar0 + 8u * slot; };
    auto empty_bar = [&](int slot) { return bar0 + 8u * (S::kStages + slot); };
    if constexpr (kSource == Source::kHalfTimesXhat) {
        for (int t = threadIdx.x; t < chunk_rows; t += kAddThreads + 32) {
            shared.mean[t] = mean[first + t];
            shared.rstd[t] = rstd[first + t];
        }
    }
    __syncthreads();
    volatile int* abort = &shared.abort_flag;
    bool ok = true;
    int issued = 0;  // fetching warp: stages whose copies have been started
    fb::Comp2 sums[kPairs];
    // LayerNorm's two parameter gradients come from one reading of dy.
    constexpr bool kAlsoSums = kAlso && kSource == Source::kHalfTimesXhat;
    fb::Comp2 also_sums[kPairs];

    if (ly == kLaneRows) {
        // ---- fetching warp: lane l copies row l of each stage (and its x segment) ----
        const uint32_t main_bytes = static_cast<uint32_t>(width) * S::kMainBytes;
        const uint32_t x_bytes = static_cast<uint32_t>(width) * S::kXBytes;
        for (int k = 0; k < stages_total; ++k) {
            const int slot = k % S::kStages;
            if (k >= S::kStages &&
                !staged_wait_warp(empty_bar(slot), static_cast<uint32_t>(k / S::kStages - 1) & 1u,
                             abort)) {
                ok = false;
                break;
            }
            issued = k + 1;
            const int here = min(S::kRows, chunk_rows - k * S::kRows);
            if (maps.use != 0) {
                // One tensor load per operand: the box is always delivered whole (zeros
                // past the matrix's edges, which the adding warps never read).
                if (lane == 0) {
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                                     full_bar(slot)),
                                 "r"(static_cast<uint32_t>(S::kStage))
                                 : "memory");
                    const int column = first_piece * 8;
                    const int row = static_cast<int>(first) + k * S::kRows;
                    const uint32_t dst = staging + slot * S::kStage;
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
                        " [%0], [%1, {%3, %4}], [%2];"
                        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(&maps.main)),
                          "r"(full_bar(slot)), "r"(column), "r"(row)
                        : "memory");
                    if constexpr (S::kXBytes != 0) {
                        asm volatile(
                            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
                            " [%0], [%1, {%3, %4}], [%2];"
                            ::"r"(dst + S::kMainStage), "l"(reinterpret_cast<uint64_t>(&maps.x)),
                              "r"(full_bar(slot)), "r"(column), "r"(row)
                            : "memory");
                    }
                }
                continue;
            }
            if (lane == 0) {
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                                 full_bar(slot)),
                             "r"(static_cast<uint32_t>(here) * (main_bytes + x_bytes))
                             : "memory");
            }
            if (lane < here) {
                const size_t at =
                    (first + static_cast<size_t>(k) * S::kRows + lane) * pieces + first_piece;
                const uint32_t dst =
                    staging + slot * S::kStage + lane * (kTilePieces * S::kMainBytes);
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                    ::"r"(dst), "l"(static_cast<const unsigned char*>(src) + at * S::kMainBytes),
                      "r"(main_bytes), "r"(full_bar(slot))
                    : "memory");
                if constexpr (S::kXBytes != 0) {
                    const uint32_t xdst = staging + slot * S::kStage + S::kMainStage +
                                          lane * (kTilePieces * S::kXBytes);
                    asm volatile(
                        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                        ::"r"(xdst),
                          "l"(reinterpret_cast<const unsigned char*>(x) + at * S::kXBytes),
                          "r"(x_bytes), "r"(full_bar(slot))
                        : "memory");
                }
            }
        }
    } else {
        // ---- adding warps ----
        const int at_main = lane * (S::kMainBytes / 4);   // two columns' bytes
        const int at_x = S::kMainStage + lane * (S::kXBytes / 4);
        for (int k = 0; k < stages_total; ++k) {
            const int slot = k % S::kStages;
            // (A lane that gives up goes on with the others, who would wait for it in __syncwarp;
            // what it adds is thrown away.)
            ok = staged_wait(full_bar(slot), static_cast<uint32_t>(k / S::kStages) & 1u, abort) && ok;
            const int here = min(S::kRows, chunk_rows - k * S::kRows);
            const uint32_t stage = staging + slot * S::kStage;
            // The first `pairs` of this lane's column pairs, whose rows are added in step.
            auto add_rows = [&](auto pairs) {
#pragma unroll
                for (int j = 0; j < S::kRows / kLaneRows; ++j) {
                    const int row = ly + kLaneRows * j;  // row inside the stage
                    if (row >= here) {
                        break;
                    }
#pragma unroll
                    for (int i = 0; i < pairs.value; ++i) {
                        fb::Comp2& acc = sums[i];
                        [[maybe_unused]] fb::Comp2& also = also_sums[i];
                        fb::F2 v;
                        const uint32_t at = stage + row * (kTilePieces * S::kMainBytes) + at_main +
                                            i * (kPairPieces * S::kMainBytes);
                        if constexpr (kSource == Source::kFloat) {
                            asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(at));
                        } else {
                            unsigned bits;
                            asm volatile("ld.shared.b32 %0, [%1];" : "=r"(bits) : "r"(at));
                            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&bits));
                            v = fb::f2_pack(f.x, f.y);
                        }
                        if constexpr (kSource == Source::kHalfTimesXhat) {
                            fb::F2 xs;
                            asm volatile("ld.shared.b64 %0, [%1];"
                                         : "=l"(xs)
                                         : "r"(stage + row * (kTilePieces * S::kXBytes) + at_x +
                                               i * (kPairPieces * S::kXBytes)));
                            const float m = shared.mean[k * S::kRows + row];
                            const float rs = shared.rstd[k * S::kRows + row];
                            const fb::F2 xhat =
                                fb::f2_mul(fb::f2_sub(xs, fb::f2_pack(m, m)), fb::f2_pack(rs, rs));
                            if constexpr (kPlain) {
                                acc.s = fb::f2_fma(v, xhat, acc.s);
                            } else {
                                fb::comp_add_product2(acc, v, xhat);
                            }
                            if constexpr (kAlsoSums && kPlain) {
                                also.s = fb::f2_add(also.s, v);
                            } else if constexpr (kAlsoSums) {
                                fb::comp_add2(also, v);
                            }
                        } else if constexpr (kPlain) {
                            acc.s = fb::f2_add(acc.s, v);
                        } else {
                            fb::comp_add2(acc, v);
                        }
                    }
                }
            };
            if (lane + 32 * (kPairs - 1) < 4 * width) {
                add_rows(std::integral_constant<int, kPairs>{});
            } else if (kPairs == 2 && lane < 4 * width) {
                add_rows(std::integral_constant<int, 1>{});
            }
            // This stream is done with the slot; the fetching warp refills it once all eight are.
            __syncwarp();
            if (lane == 0) {
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty_bar(slot))
                             : "memory");
            }
        }
    }
    if (!__all_sync(fb::kFullMask, ok) && lane == 0) {
        atomicExch(&g_reduction_error, 1);
    }
    __syncthreads();
    if (shared.abort_flag != 0) {
        // A wait gave up (the flag was written before the barrier above, so every thread
        // sees the same value). The error word is set; this CTA writes no sums. Before it
        // leaves, the fetching warp waits, again with a limit, for the copies it started
        // into the ring: shared memory must not be handed to another CTA with a copy
        // still on its way.
        if (ly == kLaneRows && lane == 0) {
            for (int k = max(0, issued - S::kStages); k < issued; ++k) {
                int unused = 0;
                staged_wait(full_bar(k % S::kStages), static_cast<uint32_t>(k / S::kStages) & 1u,
                            &unused);
            }
        }
        return;
    }
    // Every stage has been consumed: the ring's memory now carries the eight streams'
    // (sum, error) pairs to a thread per column, which merges them in stream order.
    float* sh_s = reinterpret_cast<float*>(staging_raw + (staging - shared_address(staging_raw)));
    float* sh_e = sh_s + kLaneRows * kTileColumns;
#pragma unroll
    for (int set = 0; set < (kAlsoSums ? 2 : 1); ++set) {
        if (set == 1) {
            __syncthreads();  // the first set has been read
        }
        if (ly < kLaneRows) {
#pragma unroll
            for (int i = 0; i < kPairs; ++i) {
                const int at = ly * kTileColumns + 64 * i + 2 * lane;
                const fb::Comp2& from = set == 0 ? sums[i] : also_sums[i];
                fb::f2_unpack(from.s, sh_s[at], sh_s[at + 1]);
                fb::f2_unpack(from.e, sh_e[at], sh_e[at + 1]);
            }
        }
        __syncthreads();
        const int column = threadIdx.x;
        if (column >= width * 8) {
            continue;
        }
        Comp total;
        total.s = sh_s[column];
        total.e = sh_e[column];
#pragma unroll
        for (int other = 1; other < kLaneRows; ++other) {
            fb::comp_merge(total, sh_s[other * kTileColumns + column],
                           sh_e[other * kTileColumns + column]);
        }
        // Chunk c occupies rows 2c (sums) and 2c+1 (errors) of a [2*chunks, cols] FP32 matrix.
        float* out = (set == 0 ? partial : second) + chunk * pieces * 16 + first_piece * 8 + column;
        out[0] = total.s;
        out[size_t(pieces) * 8] = total.e;
    }
}

template <Source kSource, bool kPlain, bool kAlso, int kPairs>
__global__ void __launch_bounds__(kAddThreads + 32)
    fb_column_partials(const __grid_constant__ ColumnMaps maps, float* __restrict__ partial,
                       float* __restrict__ second, const void* __restrict__ src, const float4* __restrict__ x,
                       const float* __restrict__ mean, const float* __restrict__ rstd, size_t rows,
                       int pieces) {
    extern __shared__ unsigned char staging_raw[];
    __shared__ PartialsShared<kSource, kPairs> shared;
    const unsigned tile = blockIdx.z * kTilesY + blockIdx.y;
    if (tile * static_cast<unsigned>(Staging<kSource, kPairs>::kTilePieces) >= static_cast<unsigned>(pieces)) {
        return;
    }
    const PartialsPlace<kSource, kPairs> place(blockIdx.x, tile, rows, pieces, staging_raw);
    if (threadIdx.x == 0) {
        shared.init();
    }
    fb::dependency_wait();
    if (threadIdx.x == 0) {
        fb::dependency_release();
    }
    src = fb::after_wait(src);
    x = fb::after_wait(x);
    mean = fb::after_wait(mean);
    rstd = fb::after_wait(rstd);
    add_tile<kSource, kPlain, kAlso, kPairs>(maps, partial, second, src, x, mean, rstd, pieces, place, shared,
                                             staging_raw);
}

// Second pass: a warp per 4 columns.
constexpr int kFinishWarps = 8;

// The sums of columns [4 quad, 4 quad + 4) over all chunks, by one warp.
__device__ __forceinline__ void finish_quad(float4* __restrict__ out,
                                            const float4* __restrict__ partial, size_t chunks,
                                            int quads, int quad, bool accumulate) {
    const int lane = threadIdx.x % 32;
    Comp total[4];
    for (size_t chunk = lane; chunk < chunks; chunk += 32) {
        const float4* row = partial + chunk * quads * 2;
        const float4 s = row[quad];
        const float4 e = row[quads + quad];
        fb::comp_merge(total[0], s.x, e.x);
        fb::comp_merge(total[1], s.y, e.y);
        fb::comp_merge(total[2], s.z, e.z);
        fb::comp_merge(total[3], s.w, e.w);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        float os[4];
        float oe[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            os[j] = __shfl_xor_sync(fb::kFullMask, total[j].s, off);
            oe[j] = __shfl_xor_sync(fb::kFullMask, total[j].e, off);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            fb::comp_merge(total[j], os[j], oe[j]);
        }
    }
    if (lane != 0) {
        return;
    }
    float4 result = make_float4(fb::comp_value(total[0]), fb::comp_value(total[1]),
                                fb::comp_value(total[2]), fb::comp_value(total[3]));
    if (accumulate) {
        const float4 old = out[quad];
        result = make_float4(__fadd_rn(old.x, result.x), __fadd_rn(old.y, result.y),
                             __fadd_rn(old.z, result.z), __fadd_rn(old.w, result.w));
    }
    out[quad] = result;
}

__global__ void __launch_bounds__(32 * kFinishWarps)
    fb_column_finish(float4* __restrict__ out, const float4* __restrict__ partial, size_t chunks,
                     int quads, bool accumulate) {
    fb::dependency_wait();
    fb::dependency_release();
    partial = fb::after_wait(partial);
    const int quad = blockIdx.x * kFinishWarps + threadIdx.x / 32;
    if (quad < quads) {
        finish_quad(out, partial, chunks, quads, quad, accumulate);
    }
}

// Several second passes in one launch: job j owns blocks [first_block[j], first_block[j + 1]).
struct FinishJobs {
    float4* out[fb::ColumnFinishList::kMost];
    const float4* partial[fb::ColumnFinishList::kMost];
    int quads[fb::ColumnFinishList::kMost];
    int first_block[fb::ColumnFinishList::kMost + 1];
    unsigned accumulate;  // bit j
    int count;
};

__global__ void __launch_bounds__(32 * kFinishWarps)
    fb_column_finish_many(const __grid_constant__ FinishJobs jobs, size_t chunks) {
    fb::dependency_wait();
    fb::dependency_release();
    int j = 0;
    while (j + 1 < jobs.count && static_cast<int>(blockIdx.x) >= jobs.first_block[j + 1]) {
        ++j;
    }
    const int quad =
        (static_cast<int>(blockIdx.x) - jobs.first_block[j]) * kFinishWarps + threadIdx.x / 32;
    if (quad < jobs.quads[j]) {
        finish_quad(jobs.out[j], fb::after_wait(jobs.partial[j]), chunks, jobs.quads[j], quad,
                    ((jobs.accumulate >> j) & 1u) != 0);
    }
}

template <Source kSource, bool kPlain, bool kAlso, int kPairs>
cudaError_t launch_partials_of(void* workspace, const void* src, const void* x, const void* mean,
                               const void* rstd, size_t rows, size_t cols, cudaStream_t stream,
                               void* second) {
    constexpr int kTilePieces = Staging<kSource, kPairs>::kTilePieces;
    const unsigned chunks = static_cast<unsigned>((rows + kChunkRows - 1) / kChunkRows);
    const int pieces = static_cast<int>(cols / 8);
    const unsigned tiles = static_cast<unsigned>((pieces + kTilePieces - 1) / kTilePieces);
    constexpr int kDynamic = Staging<kSource, kPairs>::kBytes;
    static std::atomic<bool> configured[64] = {};  // per instantiation and device
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) {
        return e;
    }
    if (device >= 64 || !configured[device].load(std::memory_order_relaxed)) {
        e = cudaFuncSetAttribute(fb_column_partials<kSource, kPlain, kAlso, kPairs>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, kDynamic);
        if (e != cudaSuccess) {
            return e;
        }
        if (device < 64) {
            configured[device].store(true, std::memory_order_relaxed);
        }
    }
    ColumnMaps maps;
    maps.use = rows < (size_t{1} << 31) ? 1 : 0;
    if (maps.use != 0) {
        using S = Staging<kSource, kPairs>;
        e = fb::encode_rows_map(&maps.main, src, rows, cols, S::kMainBytes / 8, kTilePieces * 8,
                                S::kRows);
        if (e == cudaSuccess && S::kXBytes != 0) {
            e = fb::encode_rows_map(&maps.x, x, rows, cols, 4, kTilePieces * 8, S::kRows);
        }
        if (e != cudaSuccess) {
            return e;
        }
    }
    return fb::launch_dependent(fb_column_partials<kSource, kPlain, kAlso, kPairs>,
                                dim3(chunks, std::min(tiles, kTilesY), (tiles + kTilesY - 1) / kTilesY),
                                dim3(kAddThreads + 32), kDynamic, stream, maps,
                                static_cast<float*>(workspace), static_cast<float*>(second), src,
                                static_cast<const float4*>(x),
                                static_cast<const float*>(mean), static_cast<const float*>(rstd),
                                rows, pieces);
}

// Whether FP16 sums take 128 columns per CTA: where 64 would make more than three CTAs per SM.
// Bias gradient, 64 -> 128 columns: 8,192 x 2,304 (1,152 CTAs) 14.0 -> 12.4 us, x 1,600 (800)
// 11.4 -> 10.3, x 3,072 17.7 -> 16.1, 4,096 x 2,304 (576) 8.9 -> 8.1, 2,048 x 4,096 (512)
// 8.8 -> 8.0; but 4,096 x 1,600 (400) 7.5 -> 8.0, 8,192 x 768 (384) 7.6 -> 8.1, 1,024 x 768 (48)
// 5.8 -> 6.8. 256 columns lie between or behind (8,192 x 2,304 12.1 us, x 3,072 16.5). LayerNorm's
// sums, 12 bytes per element to stage, are slower in wide tiles (8,192 x 768 backward 25 -> 31 us).
cudaError_t wide_tiles(size_t rows, size_t cols, bool* wide) {
    int sms = 0;
    const cudaError_t e = fb::sm_count(&sms);
    *wide = (rows + kChunkRows - 1) / kChunkRows * ((cols + 63) / 64) > 3 * static_cast<size_t>(sms);
    return e;
}

template <Source kSource, bool kPlain = false, bool kAlso = true>
cudaError_t launch_partials(void* workspace, const void* src, const void* x, const void* mean,
                            const void* rstd, size_t rows, size_t cols, cudaStream_t stream,
                            void* second = nullptr) {
    if constexpr (kSource == Source::kHalf) {
        bool wide = false;
        const cudaError_t e = wide_tiles(rows, cols, &wide);
        if (e != cudaSuccess) {
            return e;
        }
        if (wide) {
            return launch_partials_of<kSource, kPlain, kAlso, 2>(workspace, src, x, mean, rstd, rows, cols,
                                                                 stream, second);
        }
    }
    return launch_partials_of<kSource, kPlain, kAlso, 1>(workspace, src, x, mean, rstd, rows, cols, stream,
                                                         second);
}

cudaError_t launch_finish(void* out, const void* workspace, size_t rows, size_t cols,
                          bool accumulate, cudaStream_t stream) {
    const size_t chunks = (rows + kChunkRows - 1) / kChunkRows;
    const int quads = static_cast<int>(cols / 4);
    const unsigned blocks = static_cast<unsigned>((quads + kFinishWarps - 1) / kFinishWarps);
    return fb::launch_dependent(fb_column_finish, dim3(blocks), dim3(32 * kFinishWarps), 0, stream,
                                static_cast<float4*>(out), static_cast<const float4*>(workspace),
                                chunks, quads, accumulate);
}

// ---- LayerNorm backward: dx -----------------------------------------------------

constexpr int kWarpsPerBlock = 8;

// A warp per row, lane l owning the 8-column pieces l, l+32, ... kPieces > 0:
// the lane keeps its pieces of dy and x in registers (rows up to 256*kPieces
// wide) and the row is read once; kPieces == 0 re-reads the row for the
// second pass. (The pointers are after_wait() ones.)
template <int kPieces>
__device__ __forceinline__ void layernorm_dx_row(float4* dx, const uint4* dy, const float4* x, const float* mean,
                                                 const float* rstd, const float4* gamma, size_t row, int pieces,
                                                 bool accumulate, uint4* dx_half) {
    const int lane = threadIdx.x % 32;
    const uint4* dyr = dy + row * pieces;
    const float4* xr = x + row * pieces * 2;
    float4* dxr = dx + row * pieces * 2;
    const float m = mean[row];
    const float rs = rstd[row];
    const float n = static_cast<float>(pieces * 8);

    float g_sum = 0.0f;
    float gx_sum = 0.0f;
    if constexpr (kPieces > 0) {
        float g[kPieces][8];
        float xh[kPieces][8];
#pragma unroll
        for (int k = 0; k < kPieces; ++k) {
            const int i = lane + 32 * k;
            if (i < pieces) {
                float d[8];
                float xs[8];
                float gs[8];
                fb::unpack8(d, dyr[i]);
                fb::load8(xs, xr + 2 * i);
                fb::load8(gs, gamma + 2 * i);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    g[k][j] = __fmul_rn(d[j], gs[j]);
                    xh[k][j] = __fmul_rn(__fsub_rn(xs[j], m), rs);
                    g_sum = __fadd_rn(g_sum, g[k][j]);
                    gx_sum = __fadd_rn(gx_sum, __fmul_rn(g[k][j], xh[k][j]));
                }
            }
        }
        const float g_mean = __fdiv_rn(fb::warp_sum_rn(g_sum), n);
        const float gx_mean = __fdiv_rn(fb::warp_sum_rn(gx_sum), n);
#pragma unroll
        for (int k = 0; k < kPieces; ++k) {
            const int i = lane + 32 * k;
            if (i < pieces) {
                float o[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    o[j] = __fmul_rn(rs, __fsub_rn(__fsub_rn(g[k][j], g_mean),
                                                   __fmul_rn(xh[k][j], gx_mean)));
                }
                if (accumulate) {
                    float old[8];
                    fb::load8(old, dxr + 2 * i);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        o[j] = __fadd_rn(old[j], o[j]);
                    }
                }
                fb::store8(dxr + 2 * i, o);
                if (dx_half != nullptr) {
                    dx_half[row * pieces + i] = fb::pack8(o);  // the same values, rounded once
                }
            }
        }
    } else {
        for (int i = lane; i < pieces; i += 32) {
            float d[8];
            float xs[8];
            float gs[8];
            fb::unpack8(d, fb::load_input(dyr + i));
            fb::load8_input(xs, xr + 2 * i);
            fb::load8_input(gs, gamma + 2 * i);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float g = __fmul_rn(d[j], gs[j]);
                g_sum = __fadd_rn(g_sum, g);
                gx_sum = __fadd_rn(gx_sum, __fmul_rn(g, __fmul_rn(__fsub_rn(xs[j], m), rs)));
            }
        }
        const float g_mean = __fdiv_rn(fb::warp_sum_rn(g_sum), n);
        const float gx_mean = __fdiv_rn(fb::warp_sum_rn(gx_sum), n);
        for (int i = lane; i < pieces; i += 32) {
            float d[8];
            float xs[8];
            float gs[8];
            fb::unpack8(d, fb::load_input(dyr + i));
            fb::load8_input(xs, xr + 2 * i);
            fb::load8_input(gs, gamma + 2 * i);
            float o[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float g = __fmul_rn(d[j], gs[j]);
                const float xhat = __fmul_rn(__fsub_rn(xs[j], m), rs);
                o[j] = __fmul_rn(rs, __fsub_rn(__fsub_rn(g, g_mean), __fmul_rn(xhat, gx_mean)));
            }
            if (accumulate) {
                float old[8];
                fb::load8(old, dxr + 2 * i);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    o[j] = __fadd_rn(old[j], o[j]);
                }
            }
            fb::store8(dxr + 2 * i, o);
            if (dx_half != nullptr) {
                dx_half[row * pieces + i] = fb::pack8(o);
            }
        }
    }
}

template <int kPieces>
__global__ void __launch_bounds__(32 * kWarpsPerBlock)
    fb_layernorm_backward_dx(float4* __restrict__ dx, const uint4* __restrict__ dy,
                             const float4* __restrict__ x, const float* __restrict__ mean,
                             const float* __restrict__ rstd, const float4* __restrict__ gamma,
                             size_t first, size_t rows, int pieces, bool accumulate,
                             uint4* __restrict__ dx_half) {
    fb::dependency_wait();
    fb::dependency_release();
    dy = fb::after_wait(dy);
    x = fb::after_wait(x);
    mean = fb::after_wait(mean);
    rstd = fb::after_wait(rstd);
    gamma = fb::after_wait(gamma);
    const size_t row = first + size_t{blockIdx.x} * kWarpsPerBlock + threadIdx.x / 32;
    if (row < rows) {
        layernorm_dx_row<kPieces>(dx, dy, x, mean, rstd, gamma, row, pieces, accumulate, dx_half);
    }
}

// The parameter gradients' partial sums and dx side by side: the former are chains of additions
// on 64-column tiles, the latter moves bytes, and both read dy and x, which then come from
// memory once. CTA 2 i (i < sums) adds tile i / chunks of chunk i % chunks, the others take eight
// rows of dx each, up to `dx_rows`.
// Two launches -> one (all of the backward): 8,192 x 768 26.2 -> 24.0 us, 16,384 x 768 46.7 -> 41.7,
// 1,000 x 768 13.3 -> 10.2, 8,192 x 256 16.6 -> 12.5; in the training step (plain sums) 25 -> 22.9.
template <bool kPlain, int kPieces>
__global__ void __launch_bounds__(kAddThreads + 32)
    fb_layernorm_backward_both(const __grid_constant__ ColumnMaps maps, float* __restrict__ partial,
                               float* __restrict__ second, float4* __restrict__ dx,
                               const uint4* __restrict__ dy, const float4* __restrict__ x,
                               const float* __restrict__ mean, const float* __restrict__ rstd,
                               const float4* __restrict__ gamma, size_t rows, int pieces, unsigned chunks,
                               unsigned sums, size_t dx_rows, bool accumulate, uint4* __restrict__ dx_half) {
    extern __shared__ unsigned char staging_raw[];
    __shared__ PartialsShared<Source::kHalfTimesXhat, 1> shared;
    const unsigned block = blockIdx.x;
    const bool adds = block / 2 < sums && block % 2 == 0;
    if (adds && threadIdx.x == 0) {
        shared.init();
    }
    fb::dependency_wait();
    if (threadIdx.x == 0) {
        fb::dependency_release();
    }
    dy = fb::after_wait(dy);
    x = fb::after_wait(x);
    mean = fb::after_wait(mean);
    rstd = fb::after_wait(rstd);
    gamma = fb::after_wait(gamma);
    if (adds) {
        const PartialsPlace<Source::kHalfTimesXhat, 1> place(block / 2 % chunks, block / 2 / chunks, rows, pieces,
                                                             staging_raw);
        add_tile<Source::kHalfTimesXhat, kPlain, true, 1>(maps, partial, second, dy, x, mean, rstd, pieces, place,
                                                          shared, staging_raw);
        return;
    }
    const size_t index = block / 2 < sums ? block / 2 : block - sums;
    const size_t row = index * kWarpsPerBlock + threadIdx.x / 32;
    if (threadIdx.x < 32 * kWarpsPerBlock && row < dx_rows) {
        layernorm_dx_row<kPieces>(dx, dy, x, mean, rstd, gamma, row, pieces, accumulate, dx_half);
    }
}

template <bool kPlain, int kPieces>
cudaError_t launch_both(void* dx, const void* dy, const void* x, const void* mean, const void* rstd,
                        const void* gamma, size_t rows, size_t cols, bool accumulate, void* partial,
                        void* second, size_t dx_rows, void* dx_half, cudaStream_t stream) {
    using S = Staging<Source::kHalfTimesXhat, 1>;
    const unsigned chunks = static_cast<unsigned>((rows + kChunkRows - 1) / kChunkRows);
    const int pieces = static_cast<int>(cols / 8);
    const unsigned sums = chunks * static_cast<unsigned>((pieces + S::kTilePieces - 1) / S::kTilePieces);
    const unsigned row_blocks = static_cast<unsigned>((dx_rows + kWarpsPerBlock - 1) / kWarpsPerBlock);
    ColumnMaps maps;
    maps.use = 1;
    cudaError_t e = fb::encode_rows_map(&maps.main, dy, rows, cols, S::kMainBytes / 8, S::kTilePieces * 8, S::kRows);
    if (e == cudaSuccess) {
        e = fb::encode_rows_map(&maps.x, x, rows, cols, 4, S::kTilePieces * 8, S::kRows);
    }
    static std::atomic<bool> configured[64] = {};
    const auto kernel = fb_layernorm_backward_both<kPlain, kPieces>;
    if (e == cudaSuccess) {
        e = fb::allow_shared_memory(kernel, S::kBytes, configured);
    }
    if (e != cudaSuccess) {
        return e;
    }
    // (Whichever kind there are more of, the last of them follow one another.)
    const unsigned blocks = std::max(2 * sums, sums + row_blocks);
    return fb::launch_dependent(kernel, dim3(blocks), dim3(kAddThreads + 32), S::kBytes, stream, maps,
                                static_cast<float*>(partial), static_cast<float*>(second),
                                static_cast<float4*>(dx), static_cast<const uint4*>(dy),
                                static_cast<const float4*>(x), static_cast<const float*>(mean),
                                static_cast<const float*>(rstd), static_cast<const float4*>(gamma), rows, pieces,
                                chunks, sums, dx_rows, accumulate, static_cast<uint4*>(dx_half));
}

template <bool kPlain>
cudaError_t launch_both(void* dx, const void* dy, const void* x, const void* mean, const void* rstd,
                        const void* gamma, size_t rows, size_t cols, bool accumulate, void* partial,
                        void* second, size_t dx_rows, void* dx_half, cudaStream_t stream) {
    const auto launch = cols <= 256 ? launch_both<kPlain, 1> : launch_both<kPlain, 3>;
    return launch(dx, dy, x, mean, rstd, gamma, rows, cols, accumulate, partial, second, dx_rows, dx_half, stream);
}

cudaError_t launch_dx(void* dx, const void* dy, const void* x, const void* mean, const void* rstd,
                      const void* gamma, size_t first, size_t rows, size_t cols, bool accumulate, void* dx_half,
                      cudaStream_t stream) {
    const auto kernel = cols <= 256    ? fb_layernorm_backward_dx<1>
                        : cols <= 768  ? fb_layernorm_backward_dx<3>
                        : cols <= 1536 ? fb_layernorm_backward_dx<6>
                                       : fb_layernorm_backward_dx<0>;
    const unsigned blocks = static_cast<unsigned>((rows - first + kWarpsPerBlock - 1) / kWarpsPerBlock);
    return fb::launch_dependent(kernel, dim3(blocks), dim3(32 * kWarpsPerBlock), 0, stream,
                                static_cast<float4*>(dx), static_cast<const uint4*>(dy),
                                static_cast<const float4*>(x), static_cast<const float*>(mean),
                                static_cast<const float*>(rstd), static_cast<const float4*>(gamma), first, rows,
                                static_cast<int>(cols / 8), accumulate, static_cast<uint4*>(dx_half));
}

// ---- embedding backward: bucket the rows by token -----------------------------------
//
// A stable least-significant-digit radix sort of (token, row) pairs by the
// 16-bit token, in two passes of 8 bits. Rows start in ascending order and both
// passes are stable, so a token's rows end up ascending, which fixes the order
// of its sum. Per pass: count digits per tile of 2,048 rows, one exclusive scan
// over (digit, tile), then a ranked scatter. Integer counting only.

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr size_t kSortTileRows = 2048;
constexpr int kRowsPerWarp = static_cast<int>(kSortTileRows) / kSortWarps;
constexpr int kDigits = 256;
constexpr unsigned kNoDigit = 0xffffffffu;

struct EmbeddingLayout {
    size_t sorted_tokens, sorted_rows, offsets, pass_tokens, pass_rows, counts, bytes;
};

constexpr size_t align16(size_t v) { return (v + 15) / 16 * 16; }

// Byte offsets of the workspace's parts: position partials first, then the
// sorted tokens (u16) and rows (u32), offsets[vocab + 1] (u32), the first
// pass's tokens and rows, and 256 u32 counters per tile.
EmbeddingLayout embedding_layout(size_t sequences, size_t length, size_t vocab, size_t width) {
    const size_t rows = sequences * length;
    const size_t tiles = (rows + kSortTileRows - 1) / kSortTileRows;
    EmbeddingLayout l{};
    size_t at = align16(column_sum_workspace(sequences, length * width));
    l.sorted_tokens = at;
    at += align16(rows * 2);
    l.sorted_rows = at;
    at += align16(rows * 4);
    l.offsets = at;
    at += align16((vocab + 1) * 4);
    l.pass_tokens = at;
    at += align16(rows * 2);
    l.pass_rows = at;
    at += align16(rows * 4);
    l.counts = at;
    at += align16(tiles * kDigits * 4);
    l.bytes = at;
    return l;
}

// The lowest lane of a group of lanes that share a digit.
__device__ __forceinline__ bool rank_leader(unsigned peers, int lane) {
    return lane == __ffs(peers) - 1;
}

__device__ __forceinline__ unsigned digit_at(const uint16_t* tokens, size_t i, size_t rows,
                                             int shift) {
    return i < rows ? (static_cast<unsigned>(tokens[i]) >> shift) & (kDigits - 1) : kNoDigit;
}

// counts[digit * tiles + tile] = rows of this tile with that digit.
__global__ void __launch_bounds__(kSortThreads)
    fb_sort_count(unsigned* __restrict__ counts, const uint16_t* __restrict__ tokens, size_t rows,
                  int shift) {
    __shared__ unsigned histogram[kDigits];
    histogram[threadIdx.x] = 0;
    __syncthreads();
    const size_t base = size_t{blockIdx.x} * kSortTileRows;
    for (int i = threadIdx.x; i < static_cast<int>(kSortTileRows); i += kSortThreads) {
        const unsigned digit = digit_at(tokens, base + i, rows, shift);
        if (digit != kNoDigit) {
            atomicAdd(&histogram[digit], 1u);  // integer: the total is order-independent
        }
    }
    __syncthreads();
    counts[size_t{threadIdx.x} * gridDim.x + blockIdx.x] = histogram[threadIdx.x];
}

// In-place exclusive prefix sum of `entries` counters by one CTA of 1,024 threads.
__global__ void __launch_bounds__(1024) fb_sort_scan(unsigned* __restrict__ counts, size_t entries) {
    __shared__ unsigned warp_totals[32];
    __shared__ unsigned carry_shared;
    const int lane = threadIdx.x % 32;
    const int warp = threadIdx.x / 32;
    if (threadIdx.x == 0) {
        carry_shared = 0;
    }
    __syncthreads();
    for (size_t base = 0; base < entries; base += 1024) {
        const size_t i = base + threadIdx.x;
        const unsigned v = i < entries ? counts[i] : 0;
        unsigned inc = v;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const unsigned o = __shfl_up_sync(fb::kFullMask, inc, off);
            if (lane >= off) {
                inc += o;
            }
        }
        if (lane == 31) {
            warp_totals[warp] = inc;
        }
        __syncthreads();
        if (warp == 0) {
            unsigned w = warp_totals[lane];
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const unsigned o = __shfl_up_sync(fb::kFullMask, w, off);
                if (lane >= off) {
                    w += o;
                }
            }
            warp_totals[lane] = w;  // inclusive over warps
        }
        __syncthreads();
        const unsigned carry = carry_shared;
        const unsigned before = warp == 0 ? 0 : warp_totals[warp - 1];
        if (i < entries) {
            counts[i] = carry + before + inc - v;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            carry_shared = carry + warp_totals[31];
        }
        __syncthreads();
    }
}

// Moves a tile's (token, row) pairs to their positions for this digit. Warp w
// handles rows [256 w, 256 w + 256) of the tile, 32 at a time in order, so
// equal digits keep their input order.
__global__ void __launch_bounds__(kSortThreads)
    fb_sort_scatter(uint16_t* __restrict__ out_tokens, unsigned* __restrict__ out_rows,
                    const uint16_t* __restrict__ in_tokens, const unsigned* __restrict__ in_rows,
                    const unsigned* __restrict__ starts, size_t rows, int shift) {
    __shared__ unsigned next[kSortWarps][kDigits];
    const int lane = threadIdx.x % 32;
    const int warp = threadIdx.x / 32;
    for (int w = 0; w < kSortWarps; ++w) {
        next[w][threadIdx.x] = 0;
    }
    __syncthreads();
    const size_t first = size_t{blockIdx.x} * kSortTileRows + size_t(warp) * kRowsPerWarp;
    // Each warp's digit counts.
    for (int step = 0; step < kRowsPerWarp / 32; ++step) {
        const unsigned digit = digit_at(in_tokens, first + step * 32 + lane, rows, shift);
        if (digit != kNoDigit) {
            atomicAdd(&next[warp][digit], 1u);
        }
    }
    __syncthreads();
    // Thread d turns digit d's per-warp counts into per-warp start positions.
    unsigned position = starts[size_t{threadIdx.x} * gridDim.x + blockIdx.x];
    for (int w = 0; w < kSortWarps; ++w) {
        const unsigned c = next[w][threadIdx.x];
        next[w][threadIdx.x] = position;
        position += c;
    }
    __syncthreads();
    for (int step = 0; step < kRowsPerWarp / 32; ++step) {
        const size_t i = first + step * 32 + lane;
        const unsigned digit = digit_at(in_tokens, i, rows, shift);
        const unsigned peers = __match_any_sync(fb::kFullMask, digit);
        if (digit != kNoDigit) {
            const unsigned rank = __popc(peers & ((1u << lane) - 1u));
            const unsigned at = next[warp][digit] + rank;
            out_tokens[at] = in_tokens[i];
            out_rows[at] = in_rows == nullptr ? static_cast<unsigned>(i) : in_rows[i];
        }
        __syncwarp();
        if (digit != kNoDigit && rank_leader(peers, lane)) {
            next[warp][digit] += __popc(peers);
        }
        __syncwarp();
    }
}

// ---- embedding backward: two launches --------------------------------------------------
//
// The bytes are dwte's 4 * vocab * width written and dx read twice; what the path spent its
// time on was a chain of nine small launches and, on tokens distributed like text, one CTA
// that walked the most frequent word's rows one memory latency at a time. So the first
// launch does everything that does not need the sorted order, with the sort itself on one
// CTA beside it: that CTA sorts and lists the words in use while the others write dwte's
// zeros (most of the bytes; the rows in use are written again later) and the position
// table. The second launch adds up the listed words.
// 8 x 1,024 tokens x 768, words as frequent as in text: 678 us -> 53 us (prepare 32.6: 188 MB,
// 5.8 TB/s; words 18.9); uniform tokens 175 us before.

constexpr int kPrepareThreads = 512;
constexpr int kPrepareWarps = kPrepareThreads / 32;
// Keys per lane of the one-CTA sort: 32 registers hold 16,384 keys. More rows (or row
// numbers that do not fit 16 bits) take the multi-launch sort, which costs about 25 us more (text-like
// tokens x 768: 12 x 1,024 67 us, 16 x 1,024 85, 17 x 1,024 115, 20 x 1,024 127, 32 x 1,024 173).
constexpr int kSortSteps = 32;
constexpr size_t kOneCtaRows = size_t{kPrepareThreads} * kSortSteps;
constexpr size_t kZeroQuads = size_t{kPrepareThreads} * 8;  // float4s a zeroing CTA writes

// Runs of one token's rows by length: a warp adds a short run whole, a warp per 128 columns
// a middling one, a CTA per 128 columns a long one.
constexpr unsigned kMiddleRun = 9;
constexpr unsigned kLongRun = 96;

// The sorted positions at which runs begin. Short runs from the front of heads[rows], long
// ones from its back; middling ones (at most rows / 9) in middle[rows / 2].
struct RunLists {
    unsigned* heads;
    unsigned* middle;
    unsigned* counts;   // short, middling, long
};

struct PrepareParams {
    float4* dwte;
    float4* dwpe;
    float4* partial;          // position partial sums: cols sums, then cols errors
    const float4* dx;
    const uint16_t* tokens;
    uint16_t* sorted_tokens;
    unsigned* sorted_rows;
    RunLists lists;
    unsigned rows, sequences;
    unsigned sort_blocks, position_blocks;  // 0 or 1; 0 when launch_partials does the table
    size_t word_quads, position_quads;
    bool accumulate_wpe;
};

// Lists sorted position i if a run begins there. The order in a list is whatever the atomics
// make it; every run is added up on its own, so no result depends on it.
template <typename Token>
__device__ __forceinline__ void list_head(const RunLists& lists, unsigned* counts, size_t i,
                                          size_t rows, Token token_at) {
    const unsigned token = token_at(i);
    if (i > 0 && token_at(i - 1) == token) {
        return;
    }
    auto reaches = [&](unsigned n) { return i + n <= rows && token_at(i + n - 1) == token; };
    const unsigned value = static_cast<unsigned>(i);
    if (!reaches(kMiddleRun)) {
        lists.heads[atomicAdd(&counts[0], 1u)] = value;
    } else if (!reaches(kLongRun)) {
        lists.middle[atomicAdd(&counts[1], 1u)] = value;
    } else {
        lists.heads[rows - 1 - atomicAdd(&counts[2], 1u)] = value;
    }
}

__global__ void __launch_bounds__(256)
    fb_list_heads(const RunLists lists, const uint16_t* __restrict__ sorted_tokens, size_t rows) {
    const size_t i = size_t{blockIdx.x} * 256 + threadIdx.x;
    if (i < rows) {
        list_head(lists, lists.counts, i, rows,
                  [&](size_t k) -> unsigned { return sorted_tokens[k]; });
    }
}

// Stable sort of rows <= kOneCtaRows (token, row) pairs packed as token << 16 | row. Warp w
// owns keys [w * share, (w + 1) * share), 32 at a time in order: the order within a digit is
// (warp, step, lane), i.e. the input's.
__device__ void sort_tokens(const PrepareParams& p, unsigned* keys, unsigned (*next)[kDigits],
                            unsigned* warp_totals) {
    const int lane = threadIdx.x % 32;
    const int warp = threadIdx.x / 32;
    const int steps = static_cast<int>((p.rows + kPrepareThreads - 1) / kPrepareThreads);
    const unsigned first = static_cast<unsigned>(warp * steps * 32 + lane);
    unsigned held[kSortSteps];
#pragma unroll
    for (int step = 0; step < kSortSteps; ++step) {
        const unsigned i = first + step * 32;
        held[step] = 0;
        if (step < steps && i < p.rows) {
            held[step] = (static_cast<unsigned>(p.tokens[i]) << 16) | i;
        }
    }
    for (int pass = 0; pass < 2; ++pass) {
        const int shift = 16 + 8 * pass;
        for (int i = threadIdx.x; i < kPrepareWarps * kDigits; i += kPrepareThreads) {
            (&next[0][0])[i] = 0;
        }
        __syncthreads();
        if (pass == 1) {
#pragma unroll
            for (int step = 0; step < kSortSteps; ++step) {
                const unsigned i = first + step * 32;
                if (step < steps && i < p.rows) {
                    held[step] = keys[i];
                }
            }
        }
#pragma unroll
        for (int step = 0; step < kSortSteps; ++step) {
            if (step < steps && first + step * 32 < p.rows) {
                atomicAdd(&next[warp][(held[step] >> shift) & (kDigits - 1)], 1u);
            }
        }
        __syncthreads();
        // Thread d: digit d's total, its exclusive prefix over the digits, then each warp's start.
        unsigned total = 0;
        unsigned inclusive = 0;
        if (threadIdx.x < kDigits) {
            for (int w = 0; w < kPrepareWarps; ++w) {
                total += next[w][threadIdx.x];
            }
            inclusive = total;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const unsigned o = __shfl_up_sync(fb::kFullMask, inclusive, off);
                inclusive += lane >= off ? o : 0;
            }
            if (lane == 31) {
                warp_totals[warp] = inclusive;
            }
        }
        __syncthreads();
        if (threadIdx.x < kDigits) {
            unsigned position = inclusive - total;
            for (int w = 0; w < warp; ++w) {
                position += warp_totals[w];
            }
            for (int w = 0; w < kPrepareWarps; ++w) {
                const unsigned c = next[w][threadIdx.x];
                next[w][threadIdx.x] = position;
                position += c;
            }
        }
        __syncthreads();
#pragma unroll
        for (int step = 0; step < kSortSteps; ++step) {
            if (step < steps) {
                const bool live = first + step * 32 < p.rows;
                const unsigned digit = live ? (held[step] >> shift) & (kDigits - 1) : kNoDigit;
                const unsigned peers = __match_any_sync(fb::kFullMask, digit);
                if (live) {
                    const unsigned at = next[warp][digit] + __popc(peers & ((1u << lane) - 1u));
                    keys[at] = held[step];
                }
                __syncwarp();
                if (live && rank_leader(peers, lane)) {
                    next[warp][digit] += __popc(peers);
                }
                __syncwarp();
            }
        }
        __syncthreads();
    }
    if (threadIdx.x < 3) {
        warp_totals[threadIdx.x] = 0;
    }
    __syncthreads();
    for (unsigned i = threadIdx.x; i < p.rows; i += kPrepareThreads) {
        p.sorted_tokens[i] = static_cast<uint16_t>(keys[i] >> 16);
        p.sorted_rows[i] = keys[i] & 0xffffu;
        list_head(p.lists, warp_totals, i, p.rows,
                  [&](size_t k) -> unsigned { return keys[k] >> 16; });
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        p.lists.counts[threadIdx.x] = warp_totals[threadIdx.x];
    }
}

__device__ __forceinline__ void comp_add4(Comp (&a)[4], const float4& v) {
    fb::comp_add(a[0], v.x);
    fb::comp_add(a[1], v.y);
    fb::comp_add(a[2], v.z);
    fb::comp_add(a[3], v.w);
}

__device__ __forceinline__ float4 add4(const float4& a, const float4& b) {
    return make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z),
                       __fadd_rn(a.w, b.w));
}

// The column-sum scheme for a single chunk (at most 256 sequences), four columns a thread:
// a stream's rows are a row stride apart, so the first rows of all eight streams are asked
// for together. The second pass over one chunk merges it with nothing, which leaves value
// and bits as they are: it is done here.
__device__ void position_columns(const PrepareParams& p, size_t quad) {
    float4 head[kLaneRows];
#pragma unroll
    for (int y = 0; y < kLaneRows; ++y) {
        head[y] = y < static_cast<int>(p.sequences) ? p.dx[y * p.position_quads + quad]
                                                    : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    Comp total[4];
#pragma unroll
    for (int y = 0; y < kLaneRows; ++y) {
        Comp acc[4];
        if (y < static_cast<int>(p.sequences)) {
            comp_add4(acc, head[y]);
        }
#pragma unroll 4
        for (unsigned r = y + kLaneRows; r < p.sequences; r += kLaneRows) {
            comp_add4(acc, p.dx[r * p.position_quads + quad]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (y == 0) {
                total[j] = acc[j];
            } else {
                fb::comp_merge(total[j], acc[j].s, acc[j].e);
            }
        }
    }
    p.partial[quad] = make_float4(total[0].s, total[1].s, total[2].s, total[3].s);
    p.partial[p.position_quads + quad] =
        make_float4(total[0].e, total[1].e, total[2].e, total[3].e);
    Comp last[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        fb::comp_merge(last[j], total[j].s, total[j].e);
    }
    float4 r = make_float4(fb::comp_value(last[0]), fb::comp_value(last[1]),
                           fb::comp_value(last[2]), fb::comp_value(last[3]));
    if (p.accumulate_wpe) {
        r = add4(p.dwpe[quad], r);
    }
    p.dwpe[quad] = r;
}

__global__ void __launch_bounds__(kPrepareThreads, 2)
    fb_embedding_prepare(const __grid_constant__ PrepareParams p) {
    extern __shared__ unsigned sort_keys[];   // [rows], sorting CTA only
    __shared__ unsigned next[kPrepareWarps][kDigits];
    __shared__ unsigned warp_totals[kDigits / 32];
    fb::dependency_wait();
    fb::dependency_release();
    unsigned block = blockIdx.x;
    if (block < p.sort_blocks) {
        sort_tokens(p, sort_keys, next, warp_totals);
        return;
    }
    block -= p.sort_blocks;
    if (block < p.position_blocks) {
        const size_t quad = size_t{block} * kPrepareThreads + threadIdx.x;
        if (quad < p.position_quads) {
            position_columns(p, quad);
        }
        return;
    }
    block -= p.position_blocks;
    const size_t base = size_t{block} * kZeroQuads + threadIdx.x;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const size_t at = base + size_t(i) * kPrepareThreads;
        if (at < p.word_quads) {
            __stcs(p.dwte + at, make_float4(0.0f, 0.0f, 0.0f, 0.0f));  // dx stays in L2
        }
    }
}

// The words in use, a slice of 128 columns at a time: each run's rows of dx are added in
// ascending row order with a compensated sum. That order is a chain of additions, so what
// bounds a run is how many of its rows are on their way at once. Long runs (a handful of
// words, first) take a CTA: all its threads fetch rows into a ring in shared memory, 96
// ahead, and a thread per column adds them. Middling runs take a warp, which asks for
// sixteen rows at a time; short ones a warp for all their columns. The last blocks fill
// `offsets`.
constexpr int kWordThreads = 256;
constexpr int kWordWarps = kWordThreads / 32;
constexpr int kWordStages = 4;
constexpr int kStageRows = 32;
constexpr int kSliceColumns = 128;
constexpr int kWordSmem = kWordStages * kStageRows * kSliceColumns * 4;

struct WordParams {
    float4* dwte;
    const float4* dx;
    const uint16_t* sorted_tokens;
    const unsigned* sorted_rows;
    RunLists lists;
    unsigned* offsets;
    unsigned rows, vocab, quads, slices, word_blocks;
    bool accumulate;
};

// One long run's slice, by the whole CTA. Row numbers are read a stage before the copies
// that need them, so that no stage waits for one load after another.
__device__ void add_long_run(const WordParams& p, size_t head, unsigned slice, float* ring) {
    const unsigned token = p.sorted_tokens[head];
    const int lane = threadIdx.x % 32;
    const int warp = threadIdx.x / 32;
    const unsigned quad = slice * 32 + lane;
    const unsigned column = slice * kSliceColumns + threadIdx.x;
    const uint32_t ring_at = shared_address(ring);
    // A stage's 32 sorted positions, one a lane: the token there (none past the end) and its row.
    unsigned at_token = 0;
    unsigned at_row = 0;
    auto look_up = [&](int stage) {
        const size_t k = head + size_t(stage) * kStageRows + lane;
        at_token = k < p.rows ? p.sorted_tokens[k] : 0x10000u;
        at_row = k < p.rows ? p.sorted_rows[k] : 0;
    };
    // Warp w fetches rows w, w + 8, ... of a stage; returns how many of the stage's rows belong
    // to the run (sorted: they come first), and looks the next stage up.
    auto fetch = [&](int stage) {
        const int count = __popc(__ballot_sync(fb::kFullMask, at_token == token));
#pragma unroll
        for (int j = 0; j < kStageRows / kWordWarps; ++j) {
            const int row = warp + j * kWordWarps;
            const unsigned from = __shfl_sync(fb::kFullMask, at_row, row);
            if (quad < p.quads && row < count) {
                const uint32_t dst =
                    ring_at + ((stage % kWordStages) * kStageRows + row) * (kSliceColumns * 4) + lane * 16;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst),
                             "l"(p.dx + size_t{from} * p.quads + quad)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        look_up(stage + 1);
        return count;
    };
    int counts[kWordStages];
    look_up(0);
#pragma unroll
    for (int stage = 0; stage < kWordStages - 1; ++stage) {
        counts[stage] = fetch(stage);
    }
    Comp acc;
    for (int stage = 0;; stage += kWordStages) {
        bool done = false;
#pragma unroll
        for (int i = 0; i < kWordStages && !done; ++i) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kWordStages - 2) : "memory");
            __syncthreads();   // the stage has landed, and everyone is done with the one before it
            counts[(i + kWordStages - 1) % kWordStages] = fetch(stage + i + kWordStages - 1);
            const int count = counts[i];
            if (threadIdx.x < kSliceColumns) {
                const float* from = ring + i * kStageRows * kSliceColumns + threadIdx.x;
                if (count == kStageRows) {
                    float v[kStageRows];
#pragma unroll
                    for (int row = 0; row < kStageRows; ++row) {
                        v[row] = from[row * kSliceColumns];
                    }
#pragma unroll
                    for (int row = 0; row < kStageRows; ++row) {
                        fb::comp_add(acc, v[row]);
                    }
                } else {
                    for (int row = 0; row < count; ++row) {
                        fb::comp_add(acc, from[row * kSliceColumns]);
                    }
                }
            }
            done = count < kStageRows;
        }
        if (done) {
            break;
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();       // the ring is free for the next run
    if (threadIdx.x < kSliceColumns && column < p.quads * 4) {
        float* out = reinterpret_cast<float*>(p.dwte) + size_t{token} * p.quads * 4 + column;
        const float r = fb::comp_value(acc);
        *out = p.accumulate ? __fadd_rn(*out, r) : r;
    }
}

// kSlices slices of a run from `slice` on, by a warp, kRows rows at a time.
template <int kSlices, int kRows>
__device__ __forceinline__ void add_slices(const WordParams& p, size_t head, unsigned token,
                                           unsigned slice) {
    const int lane = threadIdx.x % 32;
    Comp acc[kSlices][4];
    for (size_t base = head;; base += 32) {
        const size_t k = base + lane;
        const unsigned at_token = k < p.rows ? p.sorted_tokens[k] : 0x10000u;
        const unsigned row = k < p.rows ? p.sorted_rows[k] : 0;
        // Sorted: the run's lanes come first.
        const int count = __popc(__ballot_sync(fb::kFullMask, at_token == token));
        for (int part = 0; part < count; part += kRows) {
            float4 d[kSlices][kRows];
#pragma unroll
            for (int j = 0; j < kRows; ++j) {
                // Past the run's end the last row is read again, and not added.
                const size_t r = __shfl_sync(fb::kFullMask, row, min(part + j, count - 1));
#pragma unroll
                for (int i = 0; i < kSlices; ++i) {
                    const unsigned quad = (slice + i) * 32 + lane;
                    d[i][j] = p.dx[r * p.quads + (quad < p.quads ? quad : 0)];
                }
            }
#pragma unroll
            for (int j = 0; j < kRows; ++j) {
                if (part + j < count) {
#pragma unroll
                    for (int i = 0; i < kSlices; ++i) {
                        comp_add4(acc[i], d[i][j]);
                    }
                }
            }
        }
        if (count < 32) {
            break;
        }
    }
#pragma unroll
    for (int i = 0; i < kSlices; ++i) {
        const unsigned quad = (slice + i) * 32 + lane;
        if (quad >= p.quads) {
            continue;
        }
        float4* out = p.dwte + size_t{token} * p.quads + quad;
        const float4 r = make_float4(fb::comp_value(acc[i][0]), fb::comp_value(acc[i][1]),
                                     fb::comp_value(acc[i][2]), fb::comp_value(acc[i][3]));
        *out = p.accumulate ? add4(*out, r) : r;
    }
}

__global__ void __launch_bounds__(kWordThreads)
    fb_word_gradient(const __grid_constant__ WordParams p) {
    extern __shared__ float word_ring[];
    fb::dependency_wait();
    fb::dependency_release();
    if (blockIdx.x >= p.word_blocks) {
        // offsets[v] = number of sorted tokens below v, for v = 0..vocab (binary search).
        const unsigned v = (blockIdx.x - p.word_blocks) * kWordThreads + threadIdx.x;
        if (v > p.vocab) {
            return;
        }
        unsigned lo = 0;
        unsigned hi = p.rows;
        while (lo < hi) {
            const unsigned mid = lo + (hi - lo) / 2;
            if (p.sorted_tokens[mid] < v) {
                lo = mid + 1;
            } else {
                hi = mid;
            }
        }
        p.offsets[v] = lo;
        return;
    }
    const size_t longs = size_t{p.lists.counts[2]} * p.slices;
    for (size_t task = blockIdx.x; task < longs; task += p.word_blocks) {
        const size_t head = p.lists.heads[p.rows - 1 - task / p.slices];
        if (p.sorted_tokens[head] < p.vocab) {
            add_long_run(p, head, static_cast<unsigned>(task % p.slices), word_ring);
        }
    }
    // The others from the last block backwards: the first ones may still hold a long run.
    const size_t first = size_t{p.word_blocks - 1 - blockIdx.x} * kWordWarps + threadIdx.x / 32;
    const size_t stride = size_t{p.word_blocks} * kWordWarps;
    const size_t middles = size_t{p.lists.counts[1]} * p.slices;
    const size_t tasks = middles + p.lists.counts[0];
    for (size_t task = first; task < tasks; task += stride) {
        const bool middle = task < middles;
        const size_t head = middle ? p.lists.middle[task / p.slices] : p.lists.heads[task - middles];
        const unsigned token = p.sorted_tokens[head];
        if (token >= p.vocab) {
            continue;
        }
        if (middle) {
            add_slices<1, 16>(p, head, token, static_cast<unsigned>(task % p.slices));
        } else {
            for (unsigned slice = 0; slice < p.slices; slice += 6) {
                add_slices<6, 2>(p, head, token, slice);
            }
        }
    }
}

flint_status check_column_dims(const char* name, size_t rows, size_t cols, bool allow_zero_cols,
                               size_t max_rows) {
    if ((cols == 0 && !allow_zero_cols) || cols % 8 != 0 || cols > kMaxCols) {
        if (allow_zero_cols) {
            return fb::fail(FLINT_ERROR_INVALID_ARGUMENT,
                            "%s: cols (%zu) must be a multiple of 8 up to %zu", name, cols,
                            kMaxCols);
        }
        return fb::fail(FLINT_ERROR_INVALID_ARGUMENT,
                        "%s: cols (%zu) must be a multiple of 8 from 8 to %zu", name, cols,
                        kMaxCols);
    }
    if (rows == 0 || rows > max_rows) {
        return fb::fail(FLINT_ERROR_INVALID_ARGUMENT, "%s: rows (%zu) must be from 1 to %zu", name,
                        rows, max_rows);
    }
    return FLINT_OK;
}

flint_status check_embedding_dims(const char* name, size_t sequences, size_t length, size_t vocab,
                                  size_t width) {
    constexpr size_t kMaxVocab = size_t{1} << 16;
    constexpr size_t kMaxSortRows = 0xffffffffu;
    if (width == 0 || width % 8 != 0 || width > kMaxCols) {
        return fb::fail(FLINT_ERROR_INVALID_ARGUMENT,
                        "%s: width (%zu) must be a multiple of 8 from 8 to %zu", name, width,
                        kMaxCols);
    }
    if (vocab == 0 || vocab > kMaxVocab) {
        return fb::fail(FLINT_ERROR_INVALID_ARGUMENT, "%s: vocab (%zu) must be from 1 to %zu",
                        name, vocab, kMaxVocab);
    }
    if (length == 0 || length > kMaxCols / width) {
        return fb::fail(FLINT_ERROR_INVALID_ARGUMENT,
                        "%s: length (%zu) must be from 1 to %zu, so that length x width (%zu) "
                        "is at most %zu",
                        name, length, kMaxCols / width, width, kMaxCols);
    }
    if (sequences == 0 || sequences > kMaxSortRows / length) {
        return fb::fail(FLINT_ERROR_INVALID_ARGUMENT,
                        "%s: sequences (%zu) must be from 1 to %zu, so that sequences x length "
                        "is at most %zu rows",
                        name, sequences, kMaxSortRows / length, kMaxSortRows);
    }
    return FLINT_OK;
}

}  // namespace

namespace fb {

cudaError_t reductions_error_flag(int* value, bool reset) {
    cudaError_t e = cudaMemcpyFromSymbol(value, g_reduction_error, sizeof(int));
    if (e == cudaSuccess && reset && *value != 0) {
        const int zero = 0;
        e = cudaMemcpyToSymbol(g_reduction_error, &zero, sizeof(int));
    }
    return e;
}

// Internal launchers, also used by the model assembly.
size_t column_partial_bytes(size_t rows, size_t cols) { return column_sum_workspace(rows, cols); }

cudaError_t launch_column_finishes(const ColumnFinishList& list, size_t rows, cudaStream_t stream) {
    if (list.count == 0) {
        return cudaSuccess;
    }
    FinishJobs jobs = {};
    jobs.count = list.count;
    int blocks = 0;
    for (int j = 0; j < list.count; ++j) {
        const ColumnFinishList::Job& job = list.jobs[j];
        jobs.out[j] = static_cast<float4*>(job.out);
        jobs.partial[j] = static_cast<const float4*>(job.partial);
        jobs.quads[j] = static_cast<int>(job.cols / 4);
        jobs.first_block[j] = blocks;
        jobs.accumulate |= job.accumulate ? 1u << j : 0u;
        blocks += (jobs.quads[j] + kFinishWarps - 1) / kFinishWarps;
    }
    jobs.first_block[list.count] = blocks;
    const size_t chunks = (rows + kChunkRows - 1) / kChunkRows;
    return fb::launch_dependent(fb_column_finish_many, dim3(static_cast<unsigned>(blocks)),
                                dim3(32 * kFinishWarps), 0, stream, jobs, chunks);
}

namespace {
// The second pass now, or noted for launch_column_finishes.
cudaError_t finish_or_defer(void* out, const void* workspace, size_t rows, size_t cols,
                            bool accumulate, cudaStream_t stream, ColumnFinishList* later) {
    if (later == nullptr) {
        return launch_finish(out, workspace, rows, cols, accumulate, stream);
    }
    return later->add(out, workspace, cols, accumulate) ? cudaSuccess : cudaErrorInvalidValue;
}
}  // namespace

cudaError_t launch_bias_gradient(void* dbias, const void* dy, size_t rows, size_t cols,
                                 bool accumulate, void* workspace, cudaStream_t stream,
                                 bool plain, ColumnFinishList* later) {
    cudaError_t e =
        plain ? launch_partials<Source::kHalf, true>(workspace, dy, nullptr, nullptr, nullptr, rows,
                                                     cols, stream)
              : launch_partials<Source::kHalf>(workspace, dy, nullptr, nullptr, nullptr, rows, cols,
                                               stream);
    if (e != cudaSuccess) {
        return e;
    }
    return finish_or_defer(dbias, workspace, rows, cols, accumulate, stream, later);
}

cudaError_t launch_layernorm_backward(void* dx, void* dgamma, void* dbeta, const void* dy,
                                      const void* x, const void* mean, const void* rstd,
                                      const void* gamma, size_t rows, size_t cols,
                                      bool accumulate_dx, bool accumulate_params, void* workspace,
                                      cudaStream_t stream, void* dx_half, bool plain,
                                      ColumnFinishList* later) {
    // dgamma's partial sums fill the workspace. dbeta's follow them (plain: the caller provides
    // twice the public workspace size), or else lie at the end of dx, whose last rows are then
    // written after the second pass. Where dx holds something that is added to, or has less room
    // (a single row), dbeta takes a pass of its own, before dgamma's partial sums reuse the workspace
    // (stream order), and dx comes last.
    const size_t partial_bytes = column_sum_workspace(rows, cols);
    const bool apart = rows >= (size_t{1} << 31) || (!plain && (accumulate_dx || rows * cols * 4 < partial_bytes));
    cudaError_t e = cudaSuccess;
    if (apart) {
        e = launch_bias_gradient(dbeta, dy, rows, cols, accumulate_params, workspace, stream, plain);
        if (e == cudaSuccess) {
            e = plain ? launch_partials<Source::kHalfTimesXhat, true, false>(workspace, dy, x, mean, rstd, rows,
                                                                             cols, stream)
                      : launch_partials<Source::kHalfTimesXhat, false, false>(workspace, dy, x, mean, rstd,
                                                                              rows, cols, stream);
        }
        if (e == cudaSuccess) {
            e = launch_finish(dgamma, workspace, rows, cols, accumulate_params, stream);
        }
        return e == cudaSuccess ? launch_dx(dx, dy, x, mean, rstd, gamma, 0, rows, cols, accumulate_dx, dx_half, stream)
                                : e;
    }
    // The rows of dx that are free: all, or those before the partial sums at its end.
    const size_t lent = plain ? 0 : (partial_bytes + cols * 4 - 1) / (cols * 4);
    const size_t dx_rows = rows - lent;
    void* second = plain ? static_cast<unsigned char*>(workspace) + partial_bytes
                         : static_cast<unsigned char*>(dx) + dx_rows * cols * 4;
    // (Beyond 768 columns dx's warps hold so many registers that one CTA of a common launch is left to an
    // SM: 8,192 x 1,024 33.7 us apart, 47.8 together, 4,096 x 1,280 26.0 and 31.8.)
    const bool together = cols <= 768;
    if (together) {
        e = plain ? launch_both<true>(dx, dy, x, mean, rstd, gamma, rows, cols, accumulate_dx, workspace, second,
                                      dx_rows, dx_half, stream)
                  : launch_both<false>(dx, dy, x, mean, rstd, gamma, rows, cols, false, workspace, second, dx_rows,
                                       dx_half, stream);
    } else {
        e = plain ? launch_partials<Source::kHalfTimesXhat, true>(workspace, dy, x, mean, rstd, rows, cols, stream,
                                                                  second)
                  : launch_partials<Source::kHalfTimesXhat>(workspace, dy, x, mean, rstd, rows, cols, stream, second);
    }
    if (e != cudaSuccess) {
        return e;
    }
    ColumnFinishList here;
    ColumnFinishList* list = plain && later != nullptr ? later : &here;
    if (!list->add(dgamma, workspace, cols, accumulate_params) || !list->add(dbeta, second, cols, accumulate_params)) {
        return cudaErrorInvalidValue;
    }
    if (list == &here) {
        e = launch_column_finishes(here, rows, stream);
    }
    const size_t done = together ? dx_rows : 0;
    if (e == cudaSuccess && done < rows) {
        e = launch_dx(dx, dy, x, mean, rstd, gamma, done, rows, cols, accumulate_dx, dx_half, stream);
    }
    return e;
}

namespace {
// The sort for more rows than one CTA holds.
cudaError_t sort_by_launches(uint16_t* sorted_tokens, unsigned* sorted_rows, uint16_t* pass_tokens,
                             unsigned* pass_rows, unsigned* counts, const uint16_t* in_tokens,
                             size_t rows, cudaStream_t stream) {
    const unsigned tiles = static_cast<unsigned>((rows + kSortTileRows - 1) / kSortTileRows);
    const size_t entries = size_t{tiles} * kDigits;
    for (int pass = 0; pass < 2; ++pass) {
        const int shift = 8 * pass;
        const uint16_t* from_tokens = pass == 0 ? in_tokens : pass_tokens;
        const unsigned* from_rows = pass == 0 ? nullptr : pass_rows;
        uint16_t* to_tokens = pass == 0 ? pass_tokens : sorted_tokens;
        unsigned* to_rows = pass == 0 ? pass_rows : sorted_rows;
        fb_sort_count<<<tiles, kSortThreads, 0, stream>>>(counts, from_tokens, rows, shift);
        cudaError_t e = fb::after_launch();
        if (e != cudaSuccess) {
            return e;
        }
        fb_sort_scan<<<1, 1024, 0, stream>>>(counts, entries);
        e = fb::after_launch();
        if (e != cudaSuccess) {
            return e;
        }
        fb_sort_scatter<<<tiles, kSortThreads, 0, stream>>>(to_tokens, to_rows, from_tokens,
                                                            from_rows, counts, rows, shift);
        e = fb::after_launch();
        if (e != cudaSuccess) {
            return e;
        }
    }
    // The first pass's arrays and the counters have served: they carry the lists of runs.
    const cudaError_t e = cudaMemsetAsync(counts, 0, 12, stream);
    if (e != cudaSuccess) {
        return e;
    }
    fb_list_heads<<<static_cast<unsigned>((rows + 255) / 256), 256, 0, stream>>>(
        RunLists{pass_rows, reinterpret_cast<unsigned*>(pass_tokens), counts}, sorted_tokens, rows);
    return fb::after_launch();
}
}  // namespace

cudaError_t launch_embedding_backward(void* dwte, void* dwpe, const void* dx, const void* tokens,
                                      size_t sequences, size_t length, size_t vocab, size_t width,
                                      bool accumulate_wte, bool accumulate_wpe, void* workspace,
                                      cudaStream_t stream) {
    const size_t rows = sequences * length;
    const EmbeddingLayout l = embedding_layout(sequences, length, vocab, width);
    auto* base = static_cast<unsigned char*>(workspace);
    auto* sorted_tokens = reinterpret_cast<uint16_t*>(base + l.sorted_tokens);
    auto* sorted_rows = reinterpret_cast<unsigned*>(base + l.sorted_rows);
    auto* offsets = reinterpret_cast<unsigned*>(base + l.offsets);
    auto* pass_tokens = reinterpret_cast<uint16_t*>(base + l.pass_tokens);
    auto* pass_rows = reinterpret_cast<unsigned*>(base + l.pass_rows);
    auto* counts = reinterpret_cast<unsigned*>(base + l.counts);
    const auto* in_tokens = static_cast<const uint16_t*>(tokens);

    const bool one_cta = rows <= kOneCtaRows;
    if (!one_cta) {
        const cudaError_t e = sort_by_launches(sorted_tokens, sorted_rows, pass_tokens, pass_rows,
                                               counts, in_tokens, rows, stream);
        if (e != cudaSuccess) {
            return e;
        }
    }
    const unsigned quads = static_cast<unsigned>(width / 4);
    const bool table_here = sequences <= kChunkRows;   // one chunk of the column-sum scheme
    PrepareParams p{};
    p.dwte = static_cast<float4*>(dwte);
    p.dwpe = static_cast<float4*>(dwpe);
    p.partial = reinterpret_cast<float4*>(base);
    p.dx = static_cast<const float4*>(dx);
    p.tokens = in_tokens;
    p.sorted_tokens = sorted_tokens;
    p.sorted_rows = sorted_rows;
    p.lists = RunLists{pass_rows, reinterpret_cast<unsigned*>(pass_tokens), counts};
    p.rows = static_cast<unsigned>(rows);
    p.sequences = static_cast<unsigned>(sequences);
    p.sort_blocks = one_cta ? 1 : 0;
    p.position_quads = length * quads;
    p.position_blocks = table_here ? static_cast<unsigned>((p.position_quads + kPrepareThreads - 1) /
                                                           kPrepareThreads)
                                   : 0;
    p.word_quads = accumulate_wte ? 0 : vocab * quads;
    p.accumulate_wpe = accumulate_wpe;
    const unsigned zero_blocks = static_cast<unsigned>((p.word_quads + kZeroQuads - 1) / kZeroQuads);
    const unsigned blocks = p.sort_blocks + p.position_blocks + zero_blocks;
    cudaError_t e = cudaSuccess;
    if (blocks > 0) {
        const int smem = one_cta ? static_cast<int>(align16(rows * 4)) : 0;
        static std::atomic<bool> configured[64] = {};
        e = fb::allow_shared_memory(fb_embedding_prepare, static_cast<int>(kOneCtaRows) * 4, configured);
        if (e == cudaSuccess) {
            e = fb::launch_dependent(fb_embedding_prepare, dim3(blocks), dim3(kPrepareThreads),
                                     static_cast<size_t>(smem), stream, p);
        }
        if (e != cudaSuccess) {
            return e;
        }
    }
    int sms = 0;
    e = fb::sm_count(&sms);
    if (e != cudaSuccess) {
        return e;
    }
    static std::atomic<bool> words_configured[64] = {};
    e = fb::allow_shared_memory(fb_word_gradient, kWordSmem, words_configured);
    if (e != cudaSuccess) {
        return e;
    }
    WordParams q{};
    q.dwte = p.dwte;
    q.dx = p.dx;
    q.sorted_tokens = sorted_tokens;
    q.sorted_rows = sorted_rows;
    q.lists = p.lists;
    q.offsets = offsets;
    q.rows = p.rows;
    q.vocab = static_cast<unsigned>(vocab);
    q.quads = quads;
    q.slices = (quads + 31) / 32;
    // Two CTAs per SM (64 KB of shared memory and 127 registers a thread each).
    q.word_blocks = static_cast<unsigned>(2 * sms);
    q.accumulate = accumulate_wte;
    const unsigned offset_blocks = static_cast<unsigned>((vocab + kWordThreads) / kWordThreads);
    e = fb::launch_dependent(fb_word_gradient, dim3(q.word_blocks + offset_blocks), dim3(kWordThreads),
                             kWordSmem, stream, q);
    if (e != cudaSuccess || table_here) {
        return e;
    }
    // The position table: dx viewed as sequences x (length * width), FP32.
    const size_t cols = length * width;
    e = launch_partials<Source::kFloat>(base, dx, nullptr, nullptr, nullptr, sequences, cols,
                                        stream);
    if (e != cudaSuccess) {
        return e;
    }
    return launch_finish(dwpe, base, sequences, cols, accumulate_wpe, stream);
}

}  // namespace fb

namespace {
// ---- a bias gradient that needs no workspace from the caller -------------------------------
//
// Some hosts cannot hand this library a workspace: a plug-in living inside an
// application that owns every byte of device memory and gives none away after
// start-up, or a serving loop whose latency budget rules out cudaMalloc (it
// synchronises the whole device). For them the partial sums of the first pass go
// into this fixed array, which is part of the library's image: every GPU that
// loads the library carries these 4 MiB until the process exits.
constexpr size_t kStaticScratchBytes = size_t{4} << 20;
static __device__ __align__(256) unsigned char g_bias_gradient_scratch[kStaticScratchBytes];

// In host code the array's name is only a handle for the runtime, not an address
// a kernel can use; the device address comes from cudaGetSymbolAddress, asked
// once per device while that device is current.
// Host threads may make their first calls at the same time: the cache slots are
// atomics, and two threads that both miss simply store the same address.
cudaError_t static_scratch(void** pointer) {
    constexpr int kMaxDevices = 64;
    static std::atomic<void*> cached[kMaxDevices] = {};
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) {
        return e;
    }
    const bool slot = device >= 0 && device < kMaxDevices;
    if (slot) {
        void* known = cached[device].load(std::memory_order_relaxed);
        if (known != nullptr) {
            *pointer = known;
            return cudaSuccess;
        }
    }
    void* address = nullptr;
    e = cudaGetSymbolAddress(&address, g_bias_gradient_scratch);
    if (e != cudaSuccess) {
        return e;
    }
    if (slot) {
        cached[device].store(address, std::memory_order_relaxed);
    }
    *pointer = address;
    return cudaSuccess;
}

}  // namespace

extern "C" {

flint_status flint_bias_gradient_workspace(size_t rows, size_t cols, size_t* bytes) {
    constexpr const char* name = "flint_bias_gradient_workspace";
    if (bytes == nullptr) {
        return fb::fail(FLINT_ERROR_INVALID_ARGUMENT, "%s: bytes is null", name);
    }
    FB_TRY(check_column_dims(name, rows, cols, true, kMaxBiasRows));
    *bytes = column_sum_workspace(rows, cols);
    return FLINT_OK;
}

flint_status flint_bias_gradient(void* dbias, const void* dy, size_t rows, size_t cols,
                                 int accumulate, void* workspace, size_t workspace_bytes,
                                 flint_stream stream) {
    constexpr const char* name = "flint_bias_gradient";
    FB_TRY(check_column_dims(name, rows, cols, true, kMaxBiasRows));
    if (cols == 0) {
        return FLINT_OK;
    }
    const size_t needed = column_sum_workspace(rows, cols);
    if (workspace_bytes < needed) {
        return fb::fail(FLINT_ERROR_INVALID_ARGUMENT,
                        "%s: needs %zu bytes of workspace, given %zu", name, needed,
                        workspace_bytes);
    }
    const fb::Span spans[] = {
        {"dbias", dbias, cols * 4},
        {"workspace", workspace, needed},
        {"dy", dy, rows * cols * 2},
    };
    FB_TRY(fb::check_spans(name, spans, 2));
    FB_CUDA(fb::launch_bias_gradient(dbias, dy, rows, cols, accumulate != 0, workspace, stream,
                                     false));
    return FLINT_OK;
}

flint_status flint_b200_bias_gradient_static(void* dbias, const void* dy, size_t rows, size_t cols,
                                             int accumulate, flint_stream stream) {
    constexpr const char* name = "flint_b200_bias_gradient_static";
    FB_TRY(check_column_dims(name, rows, cols, true, kMaxBiasRows));
    if (cols == 0) {
        return FLINT_OK;
    }
    const size_t needed = column_sum_workspace(rows, cols);
    if (needed > kStaticScratchBytes) {
        return fb::fail(FLINT_ERROR_INVALID_ARGUMENT,
                        "%s: rows (%zu) x cols (%zu) needs %zu bytes of scratch, and the built-in "
                        "scratch holds %zu; use flint_bias_gradient with a workspace",
                        name, rows, cols, needed, kStaticScratchBytes);
    }
    // Arguments are judged before any CUDA call, like everywhere else in the library.
    const fb::Span spans[] = {
        {"dbias", dbias, cols * 4},
        {"dy", dy, rows * cols * 2},
    };
    FB_TRY(fb::check_spans(name, spans, 1));
    void* scratch = nullptr;
    FB_CUDA(static_scratch(&scratch));
    // The first pass overwrites every partial sum the second pass reads, so what an
    // earlier call left in the array never matters and nothing needs clearing.
    FB_CUDA(fb::launch_bias_gradient(dbias, dy, rows, cols, accumulate != 0, scratch, stream,
                                     false));
    return FLINT_OK;
}

flint_status flint_layernorm_backward_workspace(size_t rows, size_t cols, size_t* bytes) {
    constexpr const char* name = "flint_layernorm_backward_workspace";
    if (bytes == nullptr) {
        return fb::fail(FLINT_ERROR_INVALID_ARGUMENT, "%s: bytes is null", name);
    }
    FB_TRY(check_column_dims(name, rows, cols, false, kMaxRows8));
    *bytes = column_sum_workspace(rows, cols);
    return FLINT_OK;
}

flint_status flint_layernorm_backward(void* dx, void* dgamma, void* dbeta, const void* dy,
                                      const void* x, const void* mean, const void* rstd,
                                      const void* gamma, size_t rows, size_t cols,
                                      int accumulate_dx, int accumulate_params, void* workspace,
                                      size_t workspace_bytes, flint_stream stream) {
    constexpr const char* name = "flint_layernorm_backward";
    FB_TRY(check_column_dims(name, rows, cols, false, kMaxRows8));
    const size_t needed = column_sum_workspace(rows, cols);
    if (workspace_bytes < needed) {
        return fb::fail(FLINT_ERROR_INVALID_ARGUMENT,
                        "%s: needs %zu bytes of workspace, given %zu", name, needed,
                        workspace_bytes);
    }
    const fb::Span spans[] = {
        {"dx", dx, rows * cols * 4},       {"dgamma", dgamma, cols * 4},
        {"dbeta", dbeta, cols * 4},        {"workspace", workspace, needed},
        {"dy", dy, rows * cols * 2},       {"x", x, rows * cols * 4},
        {"mean", mean, rows * 4},          {"rstd", rstd, rows * 4},
        {"gamma", gamma, cols * 4},
    };
    FB_TRY(fb::check_spans(name, spans, 4));
    FB_CUDA(fb::launch_layernorm_backward(dx, dgamma, dbeta, dy, x, mean, rstd, gamma, rows, cols,
                                          accumulate_dx != 0, accumulate_params != 0, workspace,
                                          stream, nullptr, false));
    return FLINT_OK;
}

flint_status flint_embedding_backward_workspace(size_t sequences, size_t length, size_t vocab,
                                                size_t width, size_t* bytes) {
    constexpr const char* name = "flint_embedding_backward_workspace";
    if (bytes == nullptr) {
        return fb::fail(FLINT_ERROR_INVALID_ARGUMENT, "%s: bytes is null", name);
    }
    FB_TRY(check_embedding_dims(name, sequences, length, vocab, width));
    *bytes = embedding_layout(sequences, length, vocab, width).bytes;
    return FLINT_OK;
}

flint_status flint_embedding_backward(void* dwte, void* dwpe, const void* dx, const void* tokens,
                                      size_t sequences, size_t length, size_t vocab, size_t width,
                                      int accumulate_wte, int accumulate_wpe, void* workspace,
                                      size_t workspace_bytes, flint_stream stream) {
    constexpr const char* name = "flint_embedding_backward";
    FB_TRY(check_embedding_dims(name, sequences, length, vocab, width));
    const size_t needed = embedding_layout(sequences, length, vocab, width).bytes;
    if (workspace_bytes < needed) {
        return fb::fail(FLINT_ERROR_INVALID_ARGUMENT,
                        "%s: needs %zu bytes of workspace, given %zu", name, needed,
                        workspace_bytes);
    }
    const size_t rows = sequences * length;
    const fb::Span spans[] = {
        {"dwte", dwte, vocab * width * 4},   {"dwpe", dwpe, length * width * 4},
        {"workspace", workspace, needed},    {"dx", dx, rows * width * 4},
        {"tokens", tokens, rows * 2},
    };
    FB_TRY(fb::check_spans(name, spans, 3));
    FB_CUDA(fb::launch_embedding_backward(dwte, dwpe, dx, tokens, sequences, length, vocab, width,
                                          accumulate_wte != 0, accumulate_wpe != 0, workspace,
                                          stream));
    return FLINT_OK;
}

}  // extern "C"

// FP16 x FP16 -> FP32-accumulate GEMMs on the 5th-generation tensor cores:
// flint_gemm_nt / _nt_bias / _nt_bias_gelu / _nt_bias_residual / _nn / _nn_dgelu /
// _tn (+ workspace query) and the three batched forms.
//
// One persistent, warp-specialised kernel template serves every layout and
// epilogue:
//   warp 0      TMA producer: 128-byte-swizzled operand tiles into a shared
//               memory ring, one mbarrier per stage
//   warp 1      MMA issuer: one thread issues tcgen05.mma (M=128, N=BN, K=16)
//               from shared-memory descriptors into a tensor-memory accumulator;
//               tcgen05.commit releases ring stages and publishes accumulators
//   warps 2-9   epilogue: tcgen05.ld of the FP32 accumulators, the fused
//               epilogue in registers, predicated global stores
// Tensor memory holds two accumulators, so the epilogue of tile i overlaps the
// main loop of tile i+1. Every k-block is 64 wide for every layout, so all
// variants of a shape add their products in the same order and the batched
// forms reproduce the plain ones bit for bit. (Small outputs with a long k take their
// sums in two or four parts, by a rule on the shape alone, the number of rows included.) Large problems run on
// CTA pairs (fb_gemm_pair), those of a single round on fb_gemm_once.
//
// Operand layouts map onto UMMA "major-ness" instead of register transposes:
// NT reads both operands K-major, NN reads w (k x n) MN-major, TN reads both x
// (k x m) and w (k x n) MN-major. Ragged edges come from TMA's zero fill.
//
// Reference behaviour: src/kernels/gemm.cu:419-587 (main loop and epilogues),
// :733-784 (split rule) and src/api/gemm.cpp:27-454 (checks and messages).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>

#include <cuda.h>
#include <cuda_fp16.h>

#include "common.h"
#include "device_utils.cuh"
#include "gemm.h"
#include "sm100.cuh"

namespace fb {
namespace {

constexpr int kBM = 128;
constexpr int kBK = 64;
constexpr int kEpilogueWarps = 8;  // two per TMEM lane quadrant, alternating 32-column chunks
constexpr int kThreads = 64 + 32 * kEpilogueWarps;
constexpr int kRingBytes = 192 * 1024;
constexpr int kGroupM = 8;  // rows of tiles handed out together, for L2 reuse

// Set by a kernel whose bounded wait ran out; read by flint_b200_gemm_error().
__device__ int g_gemm_error = 0;

struct GemmParams {
    CUtensorMap map_a;
    CUtensorMap map_b;
    CUtensorMap map_y;    // FP16 outputs leave through TMA stores
    CUtensorMap map_pre;  // bias+GELU: the pre-activation output; residual boxes: the residual
    int tma_out;          // the two maps above are valid
    void* y;
    void* aux_out;        // bias+GELU: the pre-activation output
    const void* aux_in;   // dGELU: pre-activations; residual: the FP32 residual
    const float* bias;
    float* partials;      // split TN: [split][m][n] FP32
    int m, n, k;
    int batches;          // 1 for the plain forms
    int splits;           // TN only
    int split_len;        // k per split, a multiple of 64
    int tiles_m, tiles_n;
    long long tiles_total;
    float scale;
    int accumulate;
    int batched;
    // Parts of a sum over k, each in order, then added in order (kernels for parts only). Last, where it moves no other
    // member: behind `batches` it did, and single rounds on fb_gemm_tc took 0.1 us more (NN 4,096 x 512 x 512 5.54 -> 5.70).
    int parts;
};

// ---- epilogue math ----------------------------------------------------------------

// 2^x on the special-function unit (relative error about 2^-22; flushes denormals).
__device__ __forceinline__ float exp2_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float rcp_fast(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// GPT-2's tanh GELU written as x * sigmoid(2u), u = sqrt(2/pi) (x + 0.044715 x^3):
// the same function without the cancellation of 1 + tanh(u) for negative x.
// e = exp(-2u) is taken as 2^(-2u log2 e) in one special-function instruction:
// its error (a few FP32 ulps) is three orders below the FP16 result's rounding.
// Two values at a time on the packed FP32 instructions; the scalar forms below
// run the same instructions, so every path gives the same bits.
__device__ __forceinline__ fb::F2 gelu_tanh2(fb::F2 x) {
    constexpr float kScale = -2.302208198144325f;  // -2 sqrt(2/pi) log2(e)
    const fb::F2 one = fb::f2_pack(1.0f, 1.0f);
    const fb::F2 t = fb::f2_fma(fb::f2_pack(0.044715f, 0.044715f), fb::f2_mul(x, x), one);
    const fb::F2 arg = fb::f2_mul(fb::f2_mul(fb::f2_pack(kScale, kScale), x), t);
    float a0, a1;
    fb::f2_unpack(arg, a0, a1);
    const fb::F2 d = fb::f2_add(fb::f2_pack(exp2_fast(a0), exp2_fast(a1)), one);
    float d0, d1;
    fb::f2_unpack(d, d0, d1);
    return fb::f2_mul(x, fb::f2_pack(rcp_fast(d0), rcp_fast(d1)));
}

__device__ __forceinline__ float gelu_tanh(float x) {
    float lo, hi;
    fb::f2_unpack(gelu_tanh2(fb::f2_pack(x, x)), lo, hi);
    return lo;
}

// d/dx of the above: s + x s (1 - s) * 2u', s = sigmoid(2u). For x >= 0,
// 1 - s is computed as e * s to keep its relative accuracy near s = 1.
__device__ __forceinline__ fb::F2 gelu_tanh_grad2(fb::F2 x) {
    constexpr float kScale = -2.302208198144325f;
    constexpr float k2Rt2OverPi = 1.5957691216057308f;
    constexpr float k6KappaRt2OverPi = 0.21406444946504453f;  // 2 sqrt(2/pi) * 3 * 0.044715
    const fb::F2 one = fb::f2_pack(1.0f, 1.0f);
    const fb::F2 x2 = fb::f2_mul(x, x);
    const fb::F2 t = fb::f2_fma(fb::f2_pack(0.044715f, 0.044715f), x2, one);
    const fb::F2 arg = fb::f2_mul(fb::f2_mul(fb::f2_pack(kScale, kScale), x), t);
    float a0, a1, x0, x1;
    fb::f2_unpack(arg, a0, a1);
    fb::f2_unpack(x, x0, x1);
    const fb::F2 e = fb::f2_pack(exp2_fast(a0), exp2_fast(a1));
    float d0, d1;
    fb::f2_unpack(fb::f2_add(e, one), d0, d1);
    const fb::F2 s = fb::f2_pack(rcp_fast(d0), rcp_fast(d1));
    float n0, n1, p0, p1;
    fb::f2_unpack(fb::f2_sub(one, s), n0, n1);  // 1 - s, accurate for x < 0
    fb::f2_unpack(fb::f2_mul(e, s), p0, p1);    // e s,   accurate for x >= 0
    const fb::F2 one_minus_s = fb::f2_pack(x0 < 0.0f ? n0 : p0, x1 < 0.0f ? n1 : p1);
    const fb::F2 slope = fb::f2_fma(fb::f2_pack(k6KappaRt2OverPi, k6KappaRt2OverPi), x2,
                                    fb::f2_pack(k2Rt2OverPi, k2Rt2OverPi));
    const fb::F2 q = fb::f2_mul(fb::f2_mul(x, one_minus_s), slope);
    float g0, g1;
    fb::f2_unpack(fb::f2_fma(s, q, s), g0, g1);
    g0 = isinf(x0) ? (x0 > 0.0f ? 1.0f : 0.0f) : g0;
    g1 = isinf(x1) ? (x1 > 0.0f ? 1.0f : 0.0f) : g1;
    return fb::f2_pack(g0, g1);
}

__device__ __forceinline__ float gelu_tanh_grad(float x) {
    float lo, hi;
    fb::f2_unpack(gelu_tanh_grad2(fb::f2_pack(x, x)), lo, hi);
    return lo;
}

__device__ __forceinline__ float half_bits_to_float(unsigned short h) {
    return __half2float(__ushort_as_half(h));
}

// One output row segment: 32 consecutive columns starting at `col` of row
// `row`, FP32 accumulators in acc. `valid` = how many of the 32 columns lie
// inside the matrix.
template <Epilogue E>
__device__ __forceinline__ void store_segment(const GemmParams& p, size_t batch_offset,
                                              long long split, size_t row, int col,
                                              float (&acc)[32], int valid) {
    const size_t n = static_cast<size_t>(p.n);
    const size_t at = batch_offset + row * n + col;
    if constexpr (E == Epilogue::kBias || E == Epilogue::kBiasGelu ||
                  E == Epilogue::kBiasResidual) {
        const float* bias = p.bias + col;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            if (j < valid) {
                acc[j] = __fadd_rn(acc[j], bias[j]);
            }
        }
    }
    if constexpr (E == Epilogue::kScale) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            acc[j] = __fmul_rn(acc[j], p.scale);
        }
    }
    if constexpr (E == Epilogue::kDGelu) {
        const __half* pre = static_cast<const __half*>(p.aux_in) + at;
        // NN's n is a multiple of 8, so 8-column groups are whole and 16-byte aligned.
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            if (g * 8 < valid) {
                const uint4 q = *reinterpret_cast<const uint4*>(pre + g * 8);
                const unsigned w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float lo = half_bits_to_float(static_cast<unsigned short>(w[j]));
                    const float hi = half_bits_to_float(static_cast<unsigned short>(w[j] >> 16));
                    acc[g * 8 + 2 * j] = __fmul_rn(acc[g * 8 + 2 * j], gelu_tanh_grad(lo));
                    acc[g * 8 + 2 * j + 1] = __fmul_rn(acc[g * 8 + 2 * j + 1], gelu_tanh_grad(hi));
                }
            }
        }
    }

    if constexpr (E == Epilogue::kBiasResidual || E == Epilogue::kTnStore ||
                  E == Epilogue::kTnPartial) {
        // FP32 outputs.
        float* out;
        if constexpr (E == Epilogue::kTnPartial) {
            out = p.partials + static_cast<size_t>(split) * p.m * n + row * n + col;
        } else {
            out = static_cast<float*>(p.y) + at;
        }
        const float* res = E == Epilogue::kBiasResidual
                               ? static_cast<const float*>(p.aux_in) + at
                               : out;
        const bool add = E == Epilogue::kBiasResidual || (E == Epilogue::kTnStore && p.accumulate);
        if (p.n % 4 == 0) {
#pragma unroll
            for (int g = 0; g < 8; ++g) {
                if (g * 4 < valid) {
                    float4 v = make_float4(acc[4 * g], acc[4 * g + 1], acc[4 * g + 2],
                                           acc[4 * g + 3]);
                    if (add) {
                        const float4 o = *reinterpret_cast<const float4*>(res + 4 * g);
                        v = make_float4(__fadd_rn(o.x, v.x), __fadd_rn(o.y, v.y),
                                        __fadd_rn(o.z, v.z), __fadd_rn(o.w, v.w));
                    }
                    *reinterpret_cast<float4*>(out + 4 * g) = v;
                }
            }
        } else {
            // n even (the residual form's only requirement): 8-byte pairs.
#pragma unroll
            for (int g = 0; g < 16; ++g) {
                if (g * 2 < valid) {
                    float2 v = make_float2(acc[2 * g], acc[2 * g + 1]);
                    if (add) {
                        const float2 o = *reinterpret_cast<const float2*>(res + 2 * g);
                        v = make_float2(__fadd_rn(o.x, v.x), __fadd_rn(o.y, v.y));
                    }
                    *reinterpret_cast<float2*>(out + 2 * g) = v;
                }
            }
        }
        return;
    } else {
        // FP16 outputs; the GELU form writes the pre-activation too.
        __half* out = static_cast<__half*>(p.y) + at;
        __half* pre_out = nullptr;
        if constexpr (E == Epilogue::kBiasGelu) {
            pre_out = static_cast<__half*>(p.aux_out) + at;
        }
        if (p.n % 8 == 0) {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                if (g * 8 < valid) {
                    uint4 q;
                    unsigned* w = reinterpret_cast<unsigned*>(&q);
                    if constexpr (E == Epilogue::kBiasGelu) {
                        uint4 qp;
                        unsigned* wp = reinterpret_cast<unsigned*>(&qp);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float a = acc[g * 8 + 2 * j];
                            const float b = acc[g * 8 + 2 * j + 1];
                            const __half2 hp = __floats2half2_rn(a, b);
                            const __half2 hy = __floats2half2_rn(gelu_tanh(a), gelu_tanh(b));
                            wp[j] = *reinterpret_cast<const unsigned*>(&hp);
                            w[j] = *reinterpret_cast<const unsigned*>(&hy);
                        }
                        *reinterpret_cast<uint4*>(pre_out + g * 8) = qp;
                    } else {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const __half2 h =
                                __floats2half2_rn(acc[g * 8 + 2 * j], acc[g * 8 + 2 * j + 1]);
                            w[j] = *reinterpret_cast<const unsigned*>(&h);
                        }
                    }
                    *reinterpret_cast<uint4*>(out + g * 8) = q;
                }
            }
        } else {
            // Any n (NT allows odd n): rows are only 2-byte aligned.
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                if (j < valid) {
                    if constexpr (E == Epilogue::kBiasGelu) {
                        pre_out[j] = __float2half_rn(acc[j]);
                        out[j] = __float2half_rn(gelu_tanh(acc[j]));
                    } else {
                        out[j] = __float2half_rn(acc[j]);
                    }
                }
            }
        }
    }
}

// ---- coalesced epilogue ------------------------------------------------------------------
//
// After tcgen05.ld each lane holds 32 consecutive columns of its own row, so a
// direct store touches 32 rows per instruction. Instead the warp stages its
// 32 x 32 chunk in a private 4 KB shared-memory buffer (16-byte slots, swizzled
// in groups of 8 so both directions are conflict-free) and reads it back so
// that consecutive lanes hold consecutive 16-byte pieces of a row: every global
// access then covers whole 64- or 128-byte row segments. Second operands (the
// saved pre-activation, the residual, the old value when accumulating) are
// fetched in the same coalesced layout.

__device__ __forceinline__ uint32_t stage_slot(uint32_t base, int logical) {
    return base + static_cast<uint32_t>(((logical & ~7) | ((logical & 7) ^ ((logical >> 3) & 7)))
                                        << 4);
}

__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint4 v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y),
                 "r"(v.z), "r"(v.w)
                 : "memory");
}

__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(addr)
                 : "memory");
    return v;
}

__device__ __forceinline__ uint4 pack_half8(const float* v) {
    uint4 q;
    unsigned* w = reinterpret_cast<unsigned*>(&q);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const __half2 h = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
        w[j] = *reinterpret_cast<const unsigned*>(&h);
    }
    return q;
}

// FP16 chunks that leave by a TMA store are staged row-major, 64 bytes per row, in
// the tensor map's 64-byte swizzle (16-byte piece c of row r at c ^ ((r >> 1) & 3)):
// lane = row stores are conflict-free and the copy engine undoes the swizzle. The
// store is asynchronous: the warp goes on to its next chunk and only waits, before it
// overwrites the slot, for the engine to have read it.
__device__ __forceinline__ void stage_row_for_store(uint32_t slot, int row, const float* v) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        st_shared_v4(slot + row * 64 + ((c ^ ((row >> 1) & 3)) << 4), pack_half8(v + 8 * c));
    }
}

__device__ __forceinline__ void store_wait_slots_read() {
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

__device__ __forceinline__ void store_wait_all() {
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// One lane: the staged 32 x 32 chunk to rows [row, row + 32), columns [col, col + 32);
// parts outside the matrix are clipped by the copy engine.
__device__ __forceinline__ void store_chunk_async(const CUtensorMap* map, uint32_t slot, int col,
                                                  int row) {
    asm volatile(
        "cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
        ::"l"(reinterpret_cast<uint64_t>(map)), "r"(slot), "r"(col), "r"(row)
        : "memory");
}

__device__ __forceinline__ void store_chunk_async(const CUtensorMap* map, uint32_t slot, int col,
                                                  int row, int batch) {
    asm volatile(
        "cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
        ::"l"(reinterpret_cast<uint64_t>(map)), "r"(slot), "r"(col), "r"(row), "r"(batch)
        : "memory");
}

// Moves the warp's staged FP16 chunk (4 slots per row) to `out` (row-major, ld = n).
__device__ __forceinline__ void flush_half_chunk(uint32_t stage, __half* out_chunk, size_t n,
                                                 int rows_left, int valid, int lane) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int logical = lane + 32 * i;
        const int r = logical >> 2;
        const int c = logical & 3;
        if (r < rows_left && c * 8 < valid) {
            *reinterpret_cast<uint4*>(out_chunk + static_cast<size_t>(r) * n + c * 8) =
                ld_shared_v4(stage_slot(stage, logical));
        }
    }
}

// Second operands of a chunk, fetched in the coalesced layout before the
// accumulators are needed: the residual (bias+residual), the old value (TN
// store with accumulate) or the saved pre-activation (dGELU). The loads are
// issued a chunk ahead of their use, so their latency hides behind the previous
// chunk's work instead of stalling every store.
template <Epilogue E>
__host__ __device__ constexpr int aux_slots() {
    return (E == Epilogue::kBiasResidual || E == Epilogue::kTnStore) ? 8
           : E == Epilogue::kDGelu                                   ? 4
                                                                      : 1;
}

template <Epilogue E>
struct Aux {
    uint4 q[aux_slots<E>()];
};

template <Epilogue E>
__device__ __forceinline__ void load_aux(Aux<E>& aux, const GemmParams& p, size_t batch_offset,
                                         size_t row0, int col, int valid, int lane) {
    const size_t n = static_cast<size_t>(p.n);
    const size_t at0 = batch_offset + row0 * n + col;
    const long long rows_long = static_cast<long long>(p.m) - static_cast<long long>(row0);
    const int rows_left = rows_long > 32 ? 32 : static_cast<int>(rows_long);
    if constexpr (E == Epilogue::kBiasResidual || E == Epilogue::kTnStore) {
        const bool add = E == Epilogue::kBiasResidual || p.accumulate;
        const float* old = E == Epilogue::kBiasResidual
                               ? static_cast<const float*>(p.aux_in) + at0
                               : static_cast<const float*>(p.y) + at0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int logical = lane + 32 * i;
            const int r = logical >> 3;
            const int c = logical & 7;
            aux.q[i] = make_uint4(0u, 0u, 0u, 0u);
            if (add && r < rows_left && c * 4 < valid) {
                aux.q[i] = *reinterpret_cast<const uint4*>(old + static_cast<size_t>(r) * n + c * 4);
            }
        }
    } else if constexpr (E == Epilogue::kDGelu) {
        // Each lane fetches its own row's 64 bytes (two whole sectors), so the saved
        // pre-activations need no trip through shared memory.
        const __half* pre = static_cast<const __half*>(p.aux_in) + at0 + static_cast<size_t>(lane) * n;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            aux.q[i] = make_uint4(0u, 0u, 0u, 0u);
            if (lane < rows_left && i * 8 < valid) {
                aux.q[i] = *reinterpret_cast<const uint4*>(pre + i * 8);
            }
        }
    }
}

// This lane's bias value for a chunk starting at column `col` (0 for the other
// epilogues and past the last column).
template <Epilogue E>
__device__ __forceinline__ float load_bias_lane(const GemmParams& p, int col, int lane) {
    if constexpr (E == Epilogue::kBias || E == Epilogue::kBiasGelu ||
                  E == Epilogue::kBiasResidual) {
        return col + lane < p.n ? p.bias[col + lane] : 0.0f;
    } else {
        return 0.0f;
    }
}

// The whole warp calls this for one 32 x 32 chunk whose top-left element is
// (row0, col). acc holds this lane's row. Requires n % 8 == 0 (FP16 outputs) or
// n % 4 == 0 (FP32 outputs).
template <Epilogue E>
__device__ __forceinline__ void store_chunk(const GemmParams& p, uint32_t stage,
                                            size_t batch_offset, long long split, size_t row0,
                                            int col, float (&acc)[32], int valid, int lane,
                                            const Aux<E>& aux, float bias_lane) {
    const size_t n = static_cast<size_t>(p.n);
    const size_t at0 = batch_offset + row0 * n + col;  // the chunk's first element
    const long long rows_long = static_cast<long long>(p.m) - static_cast<long long>(row0);
    const int rows_left = rows_long > 32 ? 32 : static_cast<int>(rows_long);

    if constexpr (E == Epilogue::kBias || E == Epilogue::kBiasGelu ||
                  E == Epilogue::kBiasResidual) {
        // Lane j holds bias[col + j] (fetched by the caller a chunk ahead, zero past the
        // matrix's edge); every lane needs all 32, so they are passed round by shuffles
        // instead of each lane waiting on its own loads.
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            acc[j] = __fadd_rn(acc[j], __shfl_sync(0xffffffffu, bias_lane, j));
        }
    }
    if constexpr (E == Epilogue::kScale) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            acc[j] = __fmul_rn(acc[j], p.scale);
        }
    }

    if constexpr (E == Epilogue::kBiasResidual || E == Epilogue::kTnStore ||
                  E == Epilogue::kTnPartial) {
        // FP32 output: 8 slots per row.
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            st_shared_v4(stage_slot(stage, lane * 8 + c),
                         make_uint4(__float_as_uint(acc[4 * c]), __float_as_uint(acc[4 * c + 1]),
                                    __float_as_uint(acc[4 * c + 2]),
                                    __float_as_uint(acc[4 * c + 3])));
        }
        __syncwarp();
        float* out;
        if constexpr (E == Epilogue::kTnPartial) {
            out = p.partials + static_cast<size_t>(split) * p.m * n + row0 * n + col;
        } else {
            out = static_cast<float*>(p.y) + at0;
        }
        bool add = false;
        if constexpr (E == Epilogue::kBiasResidual || E == Epilogue::kTnStore) {
            add = E == Epilogue::kBiasResidual || p.accumulate;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int logical = lane + 32 * i;
            const int r = logical >> 3;
            const int c = logical & 7;
            if (r < rows_left && c * 4 < valid) {
                const uint4 q = ld_shared_v4(stage_slot(stage, logical));
                float4 v = make_float4(__uint_as_float(q.x), __uint_as_float(q.y),
                                       __uint_as_float(q.z), __uint_as_float(q.w));
                const size_t off = static_cast<size_t>(r) * n + c * 4;
                if constexpr (E == Epilogue::kBiasResidual || E == Epilogue::kTnStore) {
                    if (add) {
                        const uint4 o = aux.q[i];
                        v = make_float4(__fadd_rn(__uint_as_float(o.x), v.x),
                                        __fadd_rn(__uint_as_float(o.y), v.y),
                                        __fadd_rn(__uint_as_float(o.z), v.z),
                                        __fadd_rn(__uint_as_float(o.w), v.w));
                    }
                }
                *reinterpret_cast<float4*>(out + off) = v;
            }
        }
        __syncwarp();
        return;
    } else {
        __half* out = static_cast<__half*>(p.y) + at0;
        if constexpr (E == Epilogue::kDGelu) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const uint4 q = aux.q[c];
                const unsigned w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float lo = half_bits_to_float(static_cast<unsigned short>(w[j]));
                    const float hi = half_bits_to_float(static_cast<unsigned short>(w[j] >> 16));
                    float g0, g1;
                    fb::f2_unpack(gelu_tanh_grad2(fb::f2_pack(lo, hi)), g0, g1);
                    acc[c * 8 + 2 * j] = __fmul_rn(acc[c * 8 + 2 * j], g0);
                    acc[c * 8 + 2 * j + 1] = __fmul_rn(acc[c * 8 + 2 * j + 1], g1);
                }
            }
        }
        if (p.tma_out != 0) {
            // Asynchronous stores: wait until the copy engine has read what this slot held.
            if (lane == 0) {
                store_wait_slots_read();
            }
            __syncwarp();
            if constexpr (E == Epilogue::kBiasGelu) {
                stage_row_for_store(stage, lane, acc);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    fb::f2_unpack(gelu_tanh2(fb::f2_pack(acc[2 * j], acc[2 * j + 1])), acc[2 * j],
                                  acc[2 * j + 1]);
                }
                stage_row_for_store(stage + 2048u, lane, acc);
            } else {
                stage_row_for_store(stage, lane, acc);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                if constexpr (E == Epilogue::kBiasGelu) {
                    store_chunk_async(&p.map_pre, stage, col, static_cast<int>(row0));
                    store_chunk_async(&p.map_y, stage + 2048u, col, static_cast<int>(row0));
                } else if (p.batched) {
                    store_chunk_async(&p.map_y, stage, col, static_cast<int>(row0),
                                      static_cast<int>(split));
                } else {
                    store_chunk_async(&p.map_y, stage, col, static_cast<int>(row0));
                }
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            return;
        }
        if constexpr (E == Epilogue::kBiasGelu) {
            // The pre-activation goes to the slot's first half, GELU of the unrounded
            // sums to the second; one trip through shared memory serves both outputs.
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                st_shared_v4(stage_slot(stage, lane * 4 + c), pack_half8(acc + 8 * c));
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                fb::f2_unpack(gelu_tanh2(fb::f2_pack(acc[2 * j], acc[2 * j + 1])), acc[2 * j],
                              acc[2 * j + 1]);
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                st_shared_v4(stage_slot(stage + 2048u, lane * 4 + c), pack_half8(acc + 8 * c));
            }
            __syncwarp();
            flush_half_chunk(stage, static_cast<__half*>(p.aux_out) + at0, n, rows_left, valid,
                             lane);
            flush_half_chunk(stage + 2048u, out, n, rows_left, valid, lane);
            __syncwarp();
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                st_shared_v4(stage_slot(stage, lane * 4 + c), pack_half8(acc + 8 * c));
            }
            __syncwarp();
            flush_half_chunk(stage, out, n, rows_left, valid, lane);
            __syncwarp();
        }
    }
}

template <Epilogue E>
__device__ __forceinline__ bool chunk_path_ok(const GemmParams& p) {
    if constexpr (E == Epilogue::kBiasResidual || E == Epilogue::kTnStore ||
                  E == Epilogue::kTnPartial) {
        return p.n % 4 == 0;
    } else {
        return p.n % 8 == 0;
    }
}

// ---- the tensor-core kernel --------------------------------------------------------------

template <int BN>
struct Ring {
    static constexpr int kStageA = kBM * kBK * 2;
    static constexpr int kStageB = BN * kBK * 2;
    static constexpr int kStage = kStageA + kStageB;
    static constexpr int kStages = kRingBytes / kStage;
    // ring + epilogue staging (4 KB per epilogue warp) + barriers + alignment slack
    static constexpr int kSmemBytes = kStages * kStage + kEpilogueWarps * 4096 + 1024 + 256;
};

struct TileCoord {
    long long z;  // batch (batched forms) or split (TN)
    int tm, tn;
};

__device__ __forceinline__ TileCoord decode_tile(const GemmParams& p, long long id) {
    const long long per = static_cast<long long>(p.tiles_m) * p.tiles_n;
    TileCoord c;
    c.z = id / per;
    const long long r = id - c.z * per;
    const long long group_span = static_cast<long long>(kGroupM) * p.tiles_n;
    const long long g = r / group_span;
    const int first_m = static_cast<int>(g) * kGroupM;
    const int rows_here = min(kGroupM, p.tiles_m - first_m);
    const long long in_group = r - g * group_span;
    c.tm = first_m + static_cast<int>(in_group % rows_here);
    c.tn = static_cast<int>(in_group / rows_here);
    return c;
}

// The blocks of 64 of k that part `part` of `parts` (2 or 4) takes begin here, and end where the next
// part's begin. (A division here was 0.1 us per part between two issues of products.)
__device__ __forceinline__ int part_begin(int blocks, int part, int parts) {
    return blocks * part >> (parts / 2);
}

// A tile's epilogue where its sums over k are taken in parts (p.parts): each part has an accumulator to
// itself, in turn, and a warp keeps the running sums of all its chunks in registers, so that the next
// part's products (of this tile or the next) are on their way meanwhile. `columns` of tensor memory
// per accumulator, the warp's first chunk at `at` in the first of them; `full` names an accumulator's
// barrier and `hand_back` returns it. False if a wait gave up.
// A part costs 0.2 us between the products of two accumulators, which four accumulators instead of two
// do not change. Batches on these kernels with whole sums -> on fb_gemm_once in parts, which does not
// overlap its epilogues -> here: 96 x 512 x 256 x 1,024 33.3 -> 63 -> 35 us, 24 x 768 x 768 x 2,048 49.8 -> 82 -> 51,
// 48 x 512 x 512 x 1,536 38.1 -> 70 -> 40; of one round, 12 x 256 x 256 x 1,024 7.0 -> 8.1 -> 7.6.
template <Epilogue E, int kChunks, int kStep, typename Full, typename HandBack>
__device__ __forceinline__ bool finish_parts(const GemmParams& p, uint32_t at, int columns, int& acc,
                                             uint32_t& acc_phase, Full full, HandBack hand_back,
                                             volatile int* abort, uint32_t stage, size_t batch_offset,
                                             long long z, size_t row, int col, int lane) {
    float sums[kChunks][32];
#pragma unroll
    for (int i = 0; i < kChunks; ++i) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            sums[i][j] = -0.0f;   // what a sum begins with: -0 + x is x
        }
    }
    auto add_chunk = [&](int i) {
#pragma unroll
        for (int h = 0; h < 32; h += 16) {
            uint32_t raw[16];
            sm100::tmem_ld_32x16(at + static_cast<uint32_t>(acc * columns + i * kStep + h), raw);
            sm100::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; j += 8) {   // (nothing that reads them moves above the wait)
                asm volatile(""
                             : "+r"(raw[j]), "+r"(raw[j + 1]), "+r"(raw[j + 2]), "+r"(raw[j + 3]),
                               "+r"(raw[j + 4]), "+r"(raw[j + 5]), "+r"(raw[j + 6]), "+r"(raw[j + 7]));
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                sums[i][h + j] = __fadd_rn(sums[i][h + j], __uint_as_float(raw[j]));
            }
        }
    };
    auto done_with_accumulator = [&]() {
        sm100::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
            hand_back(acc);
        }
        acc ^= 1;
        if (acc == 0) {
            acc_phase ^= 1u;
        }
    };
#pragma unroll 1
    for (int part = 1; part < p.parts; ++part) {
        if (!sm100::mbar_wait_warp(full(acc), acc_phase, abort)) {
            return false;
        }
        sm100::tc_fence_after_sync();
#pragma unroll
        for (int i = 0; i < kChunks; ++i) {
            add_chunk(i);
        }
        done_with_accumulator();
    }
    if (!sm100::mbar_wait_warp(full(acc), acc_phase, abort)) {
        return false;
    }
    sm100::tc_fence_after_sync();
    const bool coalesced = chunk_path_ok<E>(p);
#pragma unroll
    for (int i = 0; i < kChunks; ++i) {
        add_chunk(i);
        if (i + 1 == kChunks) {
            done_with_accumulator();
        }
        const int valid = min(32, p.n - (col + i * kStep));  // warp-uniform
        if (valid <= 0) {
            continue;
        }
        if (coalesced) {
            store_chunk<E>(p, stage, batch_offset, z, row - lane, col + i * kStep, sums[i], valid, lane,
                           Aux<E>{}, 0.0f);
        } else if (row < static_cast<size_t>(p.m)) {
            store_segment<E>(p, batch_offset, z, row, col + i * kStep, sums[i], valid);
        }
    }
    return true;
}

// kParted: sums over k in p.parts parts (batches of products whose shape takes them so).
template <Layout L, Epilogue E, int BN, bool kParted = false>
__global__ void __launch_bounds__(kThreads, 1)
    fb_gemm_tc(const __grid_constant__ GemmParams p) {
    using R = Ring<BN>;
    constexpr bool kAMn = L == Layout::kTN;
    constexpr bool kBMn = L != Layout::kNT;
    constexpr bool kIsTn = L == Layout::kTN;
    constexpr uint32_t kIdesc = sm100::instr_desc_f16(kBM, BN, kAMn, kBMn);
    constexpr uint32_t kTmemCols = 2 * BN < 32 ? 32 : 2 * BN;

    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem_base = (sm100::smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t staging = smem_base + R::kStages * R::kStage;
    const uint32_t bars = staging + kEpilogueWarps * 4096;
    // barrier slots (8 bytes each): full[kStages], empty[kStages], acc_full[2], acc_empty[2]
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (R::kStages + s); };
    auto acc_full_bar = [&](int a) { return bars + 8u * (2 * R::kStages + a); };
    auto acc_empty_bar = [&](int a) { return bars + 8u * (2 * R::kStages + 2 + a); };
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < R::kStages; ++s) {
            sm100::mbar_init(full_bar(s), 1);
            sm100::mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            sm100::mbar_init(acc_full_bar(a), 1);
            sm100::mbar_init(acc_empty_bar(a), kEpilogueWarps);
        }
        sm100::mbar_fence_init();
        sm100::tma_prefetch_descriptor(&p.map_a);
        sm100::tma_prefetch_descriptor(&p.map_b);
    }
    if (warp == 1) {
        sm100::tmem_alloc(sm100::smem_u32(&tmem_base_slot), kTmemCols);
    }
    sm100::tc_fence_before_sync();
    __syncthreads();
    sm100::tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_slot;
    volatile int* abort = &abort_flag;
    // Everything above ran while the previous kernel in the stream may still have been
    // finishing; global memory is touched only from here on.
    fb::dependency_wait();
    if (threadIdx.x == 0) {
        fb::dependency_release();
    }

    if (warp == 0) {
        // ---- TMA producer ----
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (long long id = blockIdx.x; ok && id < p.tiles_total; id += gridDim.x) {
                const TileCoord t = decode_tile(p, id);
                const bool split_k = kIsTn && !p.batched;
                const int k0 = split_k ? static_cast<int>(t.z) * p.split_len : 0;
                const int k1 = split_k ? min(p.k, k0 + p.split_len) : p.k;
                const int batch = p.batched ? static_cast<int>(t.z) : 0;
                const int row_a = t.tm * kBM;
                const int row_b = t.tn * BN;
                for (int kk = k0; kk < k1; kk += kBK) {
                    if (!sm100::mbar_wait(empty_bar(stage), phase ^ 1u, abort)) {
                        ok = false;
                        break;
                    }
                    const uint32_t a_dst = smem_base + stage * R::kStage;
                    const uint32_t b_dst = a_dst + R::kStageA;
                    const uint32_t bar = full_bar(stage);
                    sm100::mbar_expect_tx(bar, R::kStage);
                    if constexpr (!kAMn) {
                        if (p.batched) {
                            sm100::tma_load_3d(a_dst, &p.map_a, bar, kk, row_a, batch);
                        } else {
                            sm100::tma_load_2d(a_dst, &p.map_a, bar, kk, row_a);
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < kBM / 64; ++j) {
                            if (p.batched) {
                                sm100::tma_load_3d(a_dst + j * 8192, &p.map_a, bar, row_a + 64 * j,
                                                   kk, batch);
                            } else {
                                sm100::tma_load_2d(a_dst + j * 8192, &p.map_a, bar, row_a + 64 * j,
                                                   kk);
                            }
                        }
                    }
                    if constexpr (!kBMn) {
                        if (p.batched) {
                            sm100::tma_load_3d(b_dst, &p.map_b, bar, kk, row_b, batch);
                        } else {
                            sm100::tma_load_2d(b_dst, &p.map_b, bar, kk, row_b);
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < BN / 64; ++j) {
                            if (p.batched) {
                                sm100::tma_load_3d(b_dst + j * 8192, &p.map_b, bar, row_b + 64 * j,
                                                   kk, batch);
                            } else {
                                sm100::tma_load_2d(b_dst + j * 8192, &p.map_b, bar, row_b + 64 * j,
                                                   kk);
                            }
                        }
                    }
                    if (++stage == R::kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer ----
        // The whole warp runs the loop, so that its state stays warp-uniform; one elected
        // lane waits and issues (with the loop inside `lane == 0`, every MMA paid moves into uniform
        // registers: a k-block of a 64-column tile took 0.27 us instead of 0.24). If its wait
        // gives up it stays in the loop, whose elections need every lane, and issues nothing more.
        {
            int stage = 0;
            uint32_t phase = 0;
            int acc = 0;
            uint32_t acc_phase = 0;
            bool alive = true;   // the elected lane's: its waits have not given up
            for (long long id = blockIdx.x; id < p.tiles_total; id += gridDim.x) {
                const TileCoord t = decode_tile(p, id);
                const bool split_k = kIsTn && !p.batched;
                const int k0 = split_k ? static_cast<int>(t.z) * p.split_len : 0;
                const int k1 = split_k ? min(p.k, k0 + p.split_len) : p.k;
                for (int part = 0; part < (kParted ? p.parts : 1); ++part) {
                    const int blocks = (p.k + kBK - 1) / kBK;
                    const int from = kParted ? part_begin(blocks, part, p.parts) * kBK : k0;
                    const int to = kParted ? part_begin(blocks, part + 1, p.parts) * kBK : k1;
                    if (sm100::elect_one()) {
                        alive = alive && sm100::mbar_wait(acc_empty_bar(acc), acc_phase ^ 1u, abort);
                    }
                    const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
                    uint32_t accumulate = 0;
                    for (int kk = from; kk < to; kk += kBK) {
                        const uint32_t a_addr = smem_base + stage * R::kStage;
                        const uint32_t b_addr = a_addr + R::kStageA;
                        const uint64_t a_desc = kAMn ? sm100::smem_desc_sw128(a_addr, 8192, 1024)
                                                     : sm100::smem_desc_sw128(a_addr, 16, 1024);
                        const uint64_t b_desc = kBMn ? sm100::smem_desc_sw128(b_addr, 8192, 1024)
                                                     : sm100::smem_desc_sw128(b_addr, 16, 1024);
                        if (sm100::elect_one()) {
                            alive = alive && sm100::mbar_wait(full_bar(stage), phase, abort);
                            if (alive) {
                                sm100::tc_fence_after_sync();
#pragma unroll
                                for (int ks = 0; ks < kBK / 16; ++ks) {
                                    if (ks == 0) {
                                        sm100::mma_f16_ss_at<-1>(d_tmem, a_desc, 0, b_desc, 0, kIdesc, accumulate);
                                    } else {
                                        sm100::mma_f16_ss_at<1>(d_tmem, a_desc, ks * (kAMn ? 128 : 2), b_desc,
                                                                ks * (kBMn ? 128 : 2), kIdesc);
                                    }
                                }
                                sm100::mma_commit(empty_bar(stage));
                            }
                        }
                        accumulate = 1;
                        if (++stage == R::kStages) {
                            stage = 0;
                            phase ^= 1u;
                        }
                    }
                    if (sm100::elect_one() && alive) {
                        sm100::mma_commit(acc_full_bar(acc));
                    }
                    acc ^= 1;
                    if (acc == 0) {
                        acc_phase ^= 1u;
                    }
                }
            }
        }
    } else {
        // ---- epilogue warps ----
        const int quadrant = warp % 4;      // the TMEM lanes this warp may read
        const int column_half = (warp - 2) / 4;  // which of the alternating 32-column chunks
        const bool coalesced = chunk_path_ok<E>(p);
        const bool prefetch = coalesced && aux_slots<E>() > 1;
        const uint32_t stage = staging + static_cast<uint32_t>(warp - 2) * 4096u;
        int acc = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        for (long long id = blockIdx.x; ok && id < p.tiles_total; id += gridDim.x) {
            const TileCoord t = decode_tile(p, id);
            const size_t row = static_cast<size_t>(t.tm) * kBM + quadrant * 32 + lane;
            const bool row_ok = row < static_cast<size_t>(p.m);
            const int col0 = t.tn * BN;
            const size_t batch_offset =
                p.batched ? static_cast<size_t>(t.z) * p.m * static_cast<size_t>(p.n) : 0;
            if constexpr (kParted) {
                ok = finish_parts<E, BN / 64, 64>(
                    p, tmem_base + (static_cast<uint32_t>(quadrant * 32) << 16) + column_half * 32, BN, acc, acc_phase,
                    acc_full_bar, [&](int a) { sm100::mbar_arrive(acc_empty_bar(a)); }, abort, stage, batch_offset, t.z,
                    row, col0 + column_half * 32, lane);
                continue;
            }
            // The first chunk's second operands are requested before the accumulator is
            // awaited, each later chunk's while the one before it is processed.
            Aux<E> aux;
            if (prefetch && p.n - (col0 + column_half * 32) > 0) {
                load_aux<E>(aux, p, batch_offset, row - lane, col0 + column_half * 32,
                            min(32, p.n - (col0 + column_half * 32)), lane);
            }
            if (!sm100::mbar_wait_warp(acc_full_bar(acc), acc_phase, abort)) {
                ok = false;
                break;
            }
            sm100::tc_fence_after_sync();
            const uint32_t t_addr = tmem_base + static_cast<uint32_t>(acc * BN) +
                                    (static_cast<uint32_t>(quadrant * 32) << 16);
#pragma unroll 1
            for (int c = column_half * 32; c < BN; c += 64) {
                const bool last = c + 64 >= BN;
                const int col = col0 + c;
                const int valid = min(32, p.n - col);  // warp-uniform
                Aux<E> next = aux;
                if (prefetch && !last && p.n - (col + 64) > 0) {
                    load_aux<E>(next, p, batch_offset, row - lane, col + 64,
                                min(32, p.n - (col + 64)), lane);
                }
                const float bias_lane = load_bias_lane<E>(p, col, lane);
                uint32_t raw[32];
                if (valid > 0) {
                    sm100::tmem_ld_32x32(t_addr + c, raw);
                    sm100::tmem_ld_wait();
                }
                if (last) {
                    // This warp's reads of the accumulator are complete: hand it back.
                    sm100::tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) {
                        sm100::mbar_arrive(acc_empty_bar(acc));
                    }
                }
                if (valid > 0) {
                    float v[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        v[j] = __uint_as_float(raw[j]);
                    }
                    if (coalesced) {
                        store_chunk<E>(p, stage, batch_offset, t.z, row - lane, col, v, valid,
                                       lane, aux, bias_lane);
                    } else if (row_ok) {
                        store_segment<E>(p, batch_offset, t.z, row, col, v, valid);
                    }
                }
                aux = next;
            }
            acc ^= 1;
            if (acc == 0) {
                acc_phase ^= 1u;
            }
        }
        // Asynchronous output stores must have landed before the kernel is over.
        if (p.tma_out != 0 && lane == 0) {
            store_wait_all();
        }
    }

    // ---- teardown ----
    __syncthreads();
    if (abort_flag != 0) {
        if (threadIdx.x == 0) {
            atomicExch(&g_gemm_error, 1);
        }
        // Let any TMA copy still in flight land before shared memory is released.
        const long long start = clock64();
        while (clock64() - start < 2000000LL) {
        }
        __syncthreads();
    }
    if (warp == 1) {
        sm100::tc_fence_after_sync();
        sm100::tmem_dealloc(tmem_base, kTmemCols);
    }
}

// ---- one tile per CTA, k over a cluster -------------------------------------------------------
//
// For problems whose tiles all run at once. Nothing overlaps such a launch's last epilogue, and
// a tile's k loop is the launch's time: 0.235 us per 64 of k for 64 columns, 0.265 / 0.305 /
// 0.345 for 128 / 192 / 256, i.e. 58 to 76 bytes per clock into one SM, whatever the ring's
// depth from three stages on and however many blocks an issue round takes; so this kernel
//   - divides k over the 1, 2 or 4 CTAs of a cluster that share a tile. Each forms a partial
//     tile and sends CTA r rows [128 r / c, 128 (r + 1) / c) of it, FP32, through distributed
//     shared memory; CTA r adds them in cluster order, whoever came first, so a tile's bits
//     do not depend on timing. (st.async into a box of its own, counted by an mbarrier, was
//     0.4 us faster than staging and bulk copies; either moves about 20 bytes per clock.)
//     NN 256 x 768 x 3,072: 13.7 -> 7.9 us, 64 x 1,600 x 6,400: 25.1 -> 10.9,
//     1,000 x 768 x 3,072: 14.7 -> 11.5;
//   - has sixteen epilogue warps, four per scheduler: with eight, a tile's last chunks of 32
//     columns cost 1.4 us each in a biased or element-wise epilogue, mostly latency
//     (bias+GELU 1,000 x 3,072 x 768: 12.4 -> 10.1 us, with 192 columns a tile);
//   - stores its rows straight from registers (see store_row): NN 256 x 768 x 768, 64 columns,
//     5.64 -> 5.54 us, in clusters of two 5.65 -> 5.25.
// The accumulator is not double-buffered. A batch of products whose shape takes its sums in parts
// (see sum_parts) but which does not fit the GPU at once runs on the persistent kernels, which
// then form the same partial sums in one accumulator after the other (see finish_parts).

constexpr int kOnceWarps = 16;   // warp 0 loads and warp 1 issues MMAs before their share of the epilogue
constexpr int kOnceThreads = 32 * kOnceWarps;
constexpr int kOnceMostStages = 8;

// Shared memory: the ring, whose memory is later the staging of sums and outputs, then what the
// other CTAs of the cluster send, then the barriers.
template <int BN>
struct OnceRing {
    static constexpr int kStageA = kBM * kBK * 2;
    static constexpr int kStageB = BN * kBK * 2;
    static constexpr int kStage = kStageA + kStageB;
    // 32 x 32 chunks of 4 KB: those of the CTA's own rows, and those that a CTA sends or gets.
    static constexpr int own(int cluster) { return BN / 32 * 4 / cluster; }
    static constexpr int received(int cluster) { return own(cluster) * (cluster - 1); }
    static constexpr int stages(int cluster) {
        const int fit = (216 * 1024 - received(cluster) * 4096) / kStage;
        return fit < kOnceMostStages ? fit : kOnceMostStages;
    }
    static constexpr int bytes(int cluster) {
        return stages(cluster) * kStage + received(cluster) * 4096 + 1024 + 256;
    }
};

// 16 bytes to another CTA of the cluster, whose mbarrier counts them as they arrive.
__device__ __forceinline__ void send_to_cta(uint32_t cluster_dst, const uint32_t* v,
                                            uint32_t cluster_bar) {
    asm volatile(
        "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
        ::"r"(cluster_dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(cluster_bar)
        : "memory");
}

// ---- output rows straight from registers ----
//
// A lane's 32 columns of its row are 64 bytes (FP16) or 128 (FP32): whole sectors, so they
// need no trip through shared memory. Where nothing overlaps the epilogue that trip's fence,
// copy and wait cost more than the scattered rows do.

template <int W>
__device__ __forceinline__ void store_words(void* at, const uint32_t* w) {
    if constexpr (W == 8) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(at), "r"(w[0]),
                     "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                     : "memory");
    } else {
        *reinterpret_cast<uint4*>(at) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// `bytes_valid` of the row's 64 or 128 bytes are inside the matrix (a multiple of 16).
template <int kWords>
__device__ __forceinline__ void store_row(void* at, const uint32_t (&w)[kWords], int bytes_valid,
                                          bool wide) {
    unsigned char* out = static_cast<unsigned char*>(at);
    if (wide) {
#pragma unroll
        for (int i = 0; i < kWords; i += 8) {
            if (i * 4 < bytes_valid) {
                store_words<8>(out + i * 4, w + i);
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < kWords; i += 4) {
            if (i * 4 < bytes_valid) {
                store_words<4>(out + i * 4, w + i);
            }
        }
    }
}

// The second operand of a lane's row segment: the residual, the old value or the saved
// pre-activation (see Aux), in row order.
template <Epilogue E>
__device__ __forceinline__ void load_row_aux(Aux<E>& aux, const GemmParams& p, size_t at, int valid) {
    if constexpr (E == Epilogue::kBiasResidual || E == Epilogue::kTnStore) {
        const float* old = E == Epilogue::kBiasResidual ? static_cast<const float*>(p.aux_in) + at
                                                        : static_cast<const float*>(p.y) + at;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            aux.q[i] = i * 4 < valid ? *reinterpret_cast<const uint4*>(old + i * 4)
                                     : make_uint4(0u, 0u, 0u, 0u);
        }
    } else if constexpr (E == Epilogue::kDGelu) {
        const __half* pre = static_cast<const __half*>(p.aux_in) + at;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            aux.q[i] = i * 8 < valid ? *reinterpret_cast<const uint4*>(pre + i * 8)
                                     : make_uint4(0u, 0u, 0u, 0u);
        }
    }
}

// The epilogue of a lane's row segment: 32 sums from column `col` on, `at` its first element.
// The arithmetic is store_chunk's.
template <Epilogue E>
__device__ __forceinline__ void finish_row(const GemmParams& p, bool wide, size_t at, float (&acc)[32], int valid,
                                           bool inside, const Aux<E>& aux, float bias_lane) {
    if constexpr (E == Epilogue::kBias || E == Epilogue::kBiasGelu || E == Epilogue::kBiasResidual) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            acc[j] = __fadd_rn(acc[j], __shfl_sync(0xffffffffu, bias_lane, j));
        }
    }
    if (!inside) {
        return;
    }
    if constexpr (E == Epilogue::kScale) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            acc[j] = __fmul_rn(acc[j], p.scale);
        }
    }
    if constexpr (E == Epilogue::kBiasResidual || E == Epilogue::kTnStore) {
        if (E == Epilogue::kBiasResidual || p.accumulate) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                acc[4 * i] = __fadd_rn(__uint_as_float(aux.q[i].x), acc[4 * i]);
                acc[4 * i + 1] = __fadd_rn(__uint_as_float(aux.q[i].y), acc[4 * i + 1]);
                acc[4 * i + 2] = __fadd_rn(__uint_as_float(aux.q[i].z), acc[4 * i + 2]);
                acc[4 * i + 3] = __fadd_rn(__uint_as_float(aux.q[i].w), acc[4 * i + 3]);
            }
        }
        uint32_t words[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            words[j] = __float_as_uint(acc[j]);
        }
        store_row(static_cast<float*>(p.y) + at, words, valid * 4, wide);
    } else {
        if constexpr (E == Epilogue::kDGelu) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const unsigned w[4] = {aux.q[c].x, aux.q[c].y, aux.q[c].z, aux.q[c].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float lo = half_bits_to_float(static_cast<unsigned short>(w[j]));
                    const float hi = half_bits_to_float(static_cast<unsigned short>(w[j] >> 16));
                    float g0, g1;
                    fb::f2_unpack(gelu_tanh_grad2(fb::f2_pack(lo, hi)), g0, g1);
                    acc[c * 8 + 2 * j] = __fmul_rn(acc[c * 8 + 2 * j], g0);
                    acc[c * 8 + 2 * j + 1] = __fmul_rn(acc[c * 8 + 2 * j + 1], g1);
                }
            }
        }
        uint32_t words[16];
        auto pack = [&]() {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const __half2 h = __floats2half2_rn(acc[2 * j], acc[2 * j + 1]);
                words[j] = *reinterpret_cast<const unsigned*>(&h);
            }
        };
        pack();
        if constexpr (E == Epilogue::kBiasGelu) {
            store_row(static_cast<__half*>(p.aux_out) + at, words, valid * 2, wide);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                fb::f2_unpack(gelu_tanh2(fb::f2_pack(acc[2 * j], acc[2 * j + 1])), acc[2 * j],
                              acc[2 * j + 1]);
            }
            pack();
        }
        store_row(static_cast<__half*>(p.y) + at, words, valid * 2, wide);
    }
}

struct OnceParams {
    GemmParams gemm;
    int cluster;    // CTAs that share a tile and divide its k
    int stages;     // of the operand ring
    int wide_out;   // every row segment of the output is 32-byte aligned
    int steady_b;   // B was written before the kernel before this one began: see fetch below
};

// kParted: k is divided over a cluster.
template <Layout L, Epilogue E, int BN, bool kParted>
__global__ void __launch_bounds__(kOnceThreads, 1)
    fb_gemm_once(const __grid_constant__ OnceParams once) {
    const GemmParams& p = once.gemm;
    using R = OnceRing<BN>;
    constexpr bool kAMn = L == Layout::kTN;
    constexpr bool kBMn = L != Layout::kNT;
    constexpr uint32_t kIdesc = sm100::instr_desc_f16(kBM, BN, kAMn, kBMn);
    constexpr int kChunks = BN / 32;   // per 32 rows

    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem_base = (sm100::smem_u32(smem_raw) + 1023u) & ~1023u;
    const int cluster = kParted ? once.cluster : 1;
    const int rank = cluster > 1 ? static_cast<int>(sm100::cluster_cta_rank()) : 0;
    const int quadrants = 4 / cluster;          // of 32 rows that this CTA finishes
    const int total = quadrants * kChunks;      // their chunks
    const int stages = once.stages;
    constexpr uint32_t kTmemCols = BN <= 64 ? 64 : BN <= 128 ? 128 : 256;
    const uint32_t inbox = smem_base + static_cast<uint32_t>(stages) * R::kStage;
    const uint32_t bars = inbox + static_cast<uint32_t>(total * (cluster - 1)) * 4096u;
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (kOnceMostStages + s); };
    const uint32_t acc_full_bar = bars + 16u * kOnceMostStages;
    const uint32_t inbox_bar = acc_full_bar + 8u;
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < stages; ++s) {
            sm100::mbar_init(full_bar(s), 1);
            sm100::mbar_init(empty_bar(s), 1);
        }
        sm100::mbar_init(acc_full_bar, 1);
        sm100::mbar_init(inbox_bar, 1);
        sm100::mbar_fence_init();
        sm100::tma_prefetch_descriptor(&p.map_a);
        sm100::tma_prefetch_descriptor(&p.map_b);
    }
    if (warp == 1) {
        sm100::tmem_alloc(sm100::smem_u32(&tmem_base_slot), kTmemCols);
    }
    sm100::tc_fence_before_sync();
    __syncthreads();
    if (cluster > 1) {
        // Every CTA's barriers exist before another one signals them.
        if (threadIdx.x == 0) {
            sm100::mbar_expect_tx(inbox_bar, static_cast<uint32_t>(total * (cluster - 1)) * 4096u);
        }
        sm100::cluster_sync_all();
    }
    sm100::tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_slot;
    volatile int* abort = &abort_flag;

    const TileCoord t = decode_tile(p, blockIdx.x / cluster);
    // This CTA's share of the blocks of k.
    const int all_blocks = (p.k + kBK - 1) / kBK;
    const int block0 = all_blocks * rank / cluster;
    const int blocks = all_blocks * (rank + 1) / cluster - block0;
    const int k0 = block0 * kBK;

    const int batch = p.batched ? static_cast<int>(t.z) : 0;
    const int row_a = t.tm * kBM;
    const int row_b = t.tn * BN;
    auto fetch_b = [&](uint32_t b_dst, uint32_t bar, int kk) {
        if constexpr (!kBMn) {
            if (p.batched) {
                sm100::tma_load_3d(b_dst, &p.map_b, bar, kk, row_b, batch);
            } else {
                sm100::tma_load_2d(b_dst, &p.map_b, bar, kk, row_b);
            }
        } else {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j) {
                if (p.batched) {
                    sm100::tma_load_3d(b_dst + j * 8192, &p.map_b, bar, row_b + 64 * j, kk, batch);
                } else {
                    sm100::tma_load_2d(b_dst + j * 8192, &p.map_b, bar, row_b + 64 * j, kk);
                }
            }
        }
    };
    // Weights that no running kernel writes fill the ring's half of the first stages already.
    const int early = once.steady_b != 0 ? min(stages, blocks) : 0;
    if (threadIdx.x == 0) {
        for (int i = 0; i < early; ++i) {
            sm100::mbar_expect_tx(full_bar(i), R::kStage);
            fetch_b(smem_base + i * R::kStage + R::kStageA, full_bar(i), k0 + i * kBK);
        }
    }

    // Everything above ran while the previous kernel in the stream may still have been
    // finishing; what that kernel may have written is touched only from here on.
    fb::dependency_wait();
    if (threadIdx.x == 0) {
        fb::dependency_release();
    }

    if (warp == 0) {
        // ---- TMA producer ----
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            for (int i = 0; i < blocks; ++i) {
                const int kk = k0 + i * kBK;
                if (!sm100::mbar_wait(empty_bar(stage), phase ^ 1u, abort)) {
                    break;
                }
                const uint32_t a_dst = smem_base + stage * R::kStage;
                const uint32_t bar = full_bar(stage);
                if (i >= early) {
                    sm100::mbar_expect_tx(bar, R::kStage);
                    fetch_b(a_dst + R::kStageA, bar, kk);
                }
                if constexpr (!kAMn) {
                    if (p.batched) {
                        sm100::tma_load_3d(a_dst, &p.map_a, bar, kk, row_a, batch);
                    } else {
                        sm100::tma_load_2d(a_dst, &p.map_a, bar, kk, row_a);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < kBM / 64; ++j) {
                        if (p.batched) {
                            sm100::tma_load_3d(a_dst + j * 8192, &p.map_a, bar, row_a + 64 * j, kk,
                                               batch);
                        } else {
                            sm100::tma_load_2d(a_dst + j * 8192, &p.map_a, bar, row_a + 64 * j, kk);
                        }
                    }
                }
                if (++stage == stages) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer: warp-uniform, one elected lane issues (see fb_gemm_tc) ----
        int stage = 0;
        uint32_t phase = 0;
        bool alive = true;   // the elected lane's: its waits have not given up
        uint32_t accumulate = 0;
        for (int i = 0; i < blocks; ++i) {
            const uint32_t a_addr = smem_base + stage * R::kStage;
            const uint32_t b_addr = a_addr + R::kStageA;
            const uint64_t a_desc = kAMn ? sm100::smem_desc_sw128(a_addr, 8192, 1024)
                                         : sm100::smem_desc_sw128(a_addr, 16, 1024);
            const uint64_t b_desc = kBMn ? sm100::smem_desc_sw128(b_addr, 8192, 1024)
                                         : sm100::smem_desc_sw128(b_addr, 16, 1024);
            if (sm100::elect_one()) {
                alive = alive && sm100::mbar_wait(full_bar(stage), phase, abort);
                if (alive) {
                    sm100::tc_fence_after_sync();
                    sm100::mma_f16_ss_at<-1>(tmem_base, a_desc, 0, b_desc, 0, kIdesc, accumulate);
#pragma unroll
                    for (int ks = 1; ks < kBK / 16; ++ks) {
                        sm100::mma_f16_ss_at<1>(tmem_base, a_desc, ks * (kAMn ? 128 : 2), b_desc,
                                                ks * (kBMn ? 128 : 2), kIdesc);
                    }
                    sm100::mma_commit(empty_bar(stage));
                    if (i + 1 == blocks) {
                        sm100::mma_commit(acc_full_bar);
                    }
                }
            }
            accumulate = 1;
            if (++stage == stages) {
                stage = 0;
                phase ^= 1u;
            }
        }
    }
    __syncwarp();
    // ---- epilogue, by every warp ----
    {
        const int quadrant = warp % 4;   // the TMEM lanes this warp may read
        const int part = warp / 4;       // which of every four chunks of the quadrant's rows
        const int row_tile = t.tm * kBM;
        const int col0 = t.tn * BN;
        const size_t batch_offset =
            p.batched ? static_cast<size_t>(t.z) * p.m * static_cast<size_t>(p.n) : 0;
        const bool coalesced = chunk_path_ok<E>(p);
        // The chunks this warp finishes: chunk `work` of the CTA's rows, then every sixteenth.
        // With one CTA to a tile a warp has its own quadrant's, so that they come straight from
        // tensor memory; from shared memory any warp may take any.
        auto chunk_at = [&](int work, int& row, int& column) {
            if (cluster == 1) {
                row = quadrant;
                column = work / 4;       // work = 4 * column + quadrant's place
            } else {
                row = rank * quadrants + work / kChunks;
                column = work % kChunks;
            }
        };
        const int first = warp;
        Aux<E> aux;
        float bias_lane = 0.0f;
        // A chunk's second operands, asked for ahead of its sums.
        auto request = [&](int work) {
            int row, column;
            chunk_at(work, row, column);
            const int col = col0 + column * 32;
            const size_t mine = static_cast<size_t>(row_tile) + row * 32 + lane;
            if (p.n - col > 0) {
                if (aux_slots<E>() > 1 && coalesced && mine < static_cast<size_t>(p.m) &&
                    (E != Epilogue::kTnStore || p.accumulate)) {
                    load_row_aux<E>(aux, p, batch_offset + mine * p.n + col, min(32, p.n - col));
                }
                bias_lane = load_bias_lane<E>(p, col, lane);
            }
        };
        if (first < total) {
            request(first);
        }
        bool there = sm100::mbar_wait_warp(acc_full_bar, 0, abort);
        sm100::tc_fence_after_sync();
        const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(quadrant * 32) << 16);
        if (cluster > 1) {
            // All 128 rows' chunks go to their owners; this CTA's own to the ring's memory. (The
            // MMAs have read their operands, and no more are on the way.)
            const int owner = quadrant / quadrants;
            const int place = quadrant % quadrants * kChunks;   // of the quadrant, among its owner's
            if (there) {
#pragma unroll 1
                for (int c = part; c < kChunks; c += 4) {
                    uint32_t raw[32];
                    sm100::tmem_ld_32x32(t_addr + c * 32, raw);
                    sm100::tmem_ld_wait();
                    const uint32_t offset = static_cast<uint32_t>(place + c) * 4096u + lane * 16u;
                    if (owner == rank) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            st_shared_v4(smem_base + offset + j * 512u,
                                         make_uint4(raw[4 * j], raw[4 * j + 1], raw[4 * j + 2], raw[4 * j + 3]));
                        }
                    } else {
                        const uint32_t slot = static_cast<uint32_t>((rank - (rank > owner ? 1 : 0)) * total) * 4096u;
                        const uint32_t to = sm100::map_to_cta(inbox + slot + offset, static_cast<uint32_t>(owner));
                        const uint32_t bar = sm100::map_to_cta(inbox_bar, static_cast<uint32_t>(owner));
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            send_to_cta(to + j * 512u, raw + 4 * j, bar);
                        }
                    }
                }
            }
            // The CTA's own chunks are there for any warp to read; so are, then, the others'.
            __syncthreads();
            there = sm100::mbar_wait_warp(inbox_bar, 0, abort) && there;
        }
        if (there) {
#pragma unroll 1
            for (int work = first; work < total; work += kOnceWarps) {
                int row32, column;
                chunk_at(work, row32, column);
                const int col = col0 + column * 32;
                const int valid = min(32, p.n - col);
                if (work != first) {
                    request(work);
                }
                float v[32];
                if constexpr (!kParted) {
                    uint32_t raw[32];
                    sm100::tmem_ld_32x32(t_addr + column * 32, raw);
                    sm100::tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        v[j] = __uint_as_float(raw[j]);
                    }
                } else {
                    // The partial sums in the order of k.
#pragma unroll 1
                    for (int r = 0; r < cluster; ++r) {
                        uint32_t raw[32];
                        const int place = r == rank ? work : (r - (r > rank ? 1 : 0)) * total + work;
                        const uint32_t from =
                            (r == rank ? smem_base : inbox) + static_cast<uint32_t>(place) * 4096u + lane * 16u;
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const uint4 q = ld_shared_v4(from + j * 512u);
                            raw[4 * j] = q.x;
                            raw[4 * j + 1] = q.y;
                            raw[4 * j + 2] = q.z;
                            raw[4 * j + 3] = q.w;
                        }
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            const float sum = __uint_as_float(raw[j]);
                            v[j] = r == 0 ? sum : __fadd_rn(v[j], sum);
                        }
                    }
                }
                const size_t row = static_cast<size_t>(row_tile) + row32 * 32 + lane;
                if (valid > 0) {
                    const bool inside = row < static_cast<size_t>(p.m);
                    if (coalesced) {
                        finish_row<E>(p, once.wide_out != 0, batch_offset + row * p.n + col, v, valid, inside, aux, bias_lane);
                    } else if (inside) {
                        store_segment<E>(p, batch_offset, t.z, row, col, v, valid);
                    }
                }
            }
        }
    }

    // ---- teardown: no CTA leaves while another may still write to its shared memory ----
    __syncthreads();
    if (cluster > 1) {
        sm100::cluster_sync_all();
    }
    if (abort_flag != 0) {
        if (threadIdx.x == 0) {
            atomicExch(&g_gemm_error, 1);
        }
        // Let any copy still in flight land before shared memory is released.
        const long long start = clock64();
        while (clock64() - start < 2000000LL) {
        }
        __syncthreads();
    }
    if (warp == 1) {
        sm100::tc_fence_after_sync();
        sm100::tmem_dealloc(tmem_base, kTmemCols);
    }
}

// ---- the CTA-pair kernel: 256 x 256 tiles --------------------------------------------------
//
// Two CTAs of a cluster work on one 256 x 256 output tile with
// tcgen05.mma.cta_group::2 (M = 256, N = 256): CTA r of the pair loads rows
// [128 r, 128 r + 128) of the A tile and the same range of the B tile (its half
// of N), so each SM moves 32 KB per k-block instead of the 48 KB of a 128 x 256
// single-CTA tile, and its tensor memory receives its own 128 rows of D. The
// leader (rank 0) issues every MMA; commits reach both CTAs' barriers; the
// peer's TMA transactions and epilogue arrivals are counted on the leader's
// barriers. Roles per CTA are those of fb_gemm_tc.

constexpr int kPairBN = 256;
constexpr int kPairStageA = kBM * kBK * 2;          // 16 KB
constexpr int kPairStageB = 128 * kBK * 2;          // 16 KB: half of the 256 B rows
constexpr int kPairStage = kPairStageA + kPairStageB;
constexpr int kPairGroupM = 4;  // rows of 256-row tiles handed out together

__device__ __forceinline__ TileCoord decode_pair_tile(const GemmParams& p, long long id) {
    const long long per = static_cast<long long>(p.tiles_m) * p.tiles_n;
    TileCoord c;
    c.z = id / per;
    const long long r = id - c.z * per;
    const long long group_span = static_cast<long long>(kPairGroupM) * p.tiles_n;
    const long long g = r / group_span;
    const int first_m = static_cast<int>(g) * kPairGroupM;
    const int rows_here = min(kPairGroupM, p.tiles_m - first_m);
    const long long in_group = r - g * group_span;
    c.tm = first_m + static_cast<int>(in_group % rows_here);
    c.tn = static_cast<int>(in_group / rows_here);
    return c;
}

// Epilogue warps per CTA of the pair kernel, with 4 KB of staging each: two per TMEM lane
// quadrant, and four for bias+GELU over a short k in more than one round. Those warps mostly wait (with
// eight, 28 % of the issue slots and 30 % of the special-function unit are in use), and at k = 768 a tile's
// epilogue outlasts its k loop: 8,192 x 3,072 x 768 44.8 -> 42.5 us, 16,384 rows 94.2 -> 85.0, for a stage
// of the ring. With a longer k the loop counts for more: 8,192 x 4,096 and 16,384 x 3,072 gain 2 % at k = 896
// and lose 5 and 7 % at 1,024 (2,048 x 3,072 gains 4 %, 8,192 x 1,024 loses 11). In a single round there is
// nothing to gain (1,000 x 4,104 x 768 12.5 -> 13.1).
// (Four for dGELU 51.4 -> 59 us, which then has no registers to ask for its pre-activations a chunk ahead;
// for bias+residual 42 -> 45.) The scaled batched product of k = 64, attention's scores, is epilogue alone:
// 24 x 1,024 x 1,024 15.0 -> 13.2 us, 48 x 512 x 512 9.9 -> 8.7.
// Rows that are no multiples of 32 bytes share sectors, and where the outputs outgrow two thirds of the L2,
// sixteen warps lose by it: scores of 48 x 904 x 904 24.3 -> 23.2 us but 48 x 1,000 x 1,000 x 128 28.9 -> 32.0,
// 96 x 904 x 904 44.8 -> 51.5 (96 x 992 x 992 44.3 -> 40.2); bias+GELU 8,192 x 2,312 x 512 34.3 -> 31.0 but 8,192 x 4,104 x 768 63.0 -> 65.5.
constexpr int kManyWarps = 16;
constexpr size_t kManyWarpsMostK = 960;
constexpr size_t kManyWarpsMostScaledK = 128;
constexpr size_t kManyWarpsMostRaggedBytes = size_t{84} << 20;

// Residual boxes (kBoxes): with rows of 16-byte multiples and a short k the FP32 residual comes, and
// the FP32 output leaves, by tensor copies of boxes of 128 rows x 32 columns through a ring in shared
// memory, loaded ahead by a warp of their own; the epilogue adds to a box in place. (A warp that
// fetches its own second operands a chunk ahead has 4 KB on their way, an SM 32 KB, which at a loaded
// memory's latency is 2.5 TB/s.) 768 x 768: 16,384 rows 36.1 -> 29.4 us, 8,192 24.0 -> 20.7, 4,096 13.7 -> 11.4. With a long k
// the two stages that the boxes cost the operand ring count for more: 8,192 x 768 x 3,072 41.7 -> 46.4.
constexpr int kBoxBytes = kBM * 32 * 4;
constexpr int kBoxSlots = 6;
constexpr size_t kBoxesMostK = 1024;

__host__ __device__ constexpr int pair_threads(int epilogue_warps, bool boxes) {
    return 64 + 32 * epilogue_warps + (boxes ? 32 : 0);
}
__host__ __device__ constexpr int pair_stages(int epilogue_warps, bool boxes) {
    return boxes ? 4 : epilogue_warps == 8 ? 6 : 5;
}
__host__ __device__ constexpr int pair_smem_bytes(int epilogue_warps, bool boxes) {
    return pair_stages(epilogue_warps, boxes) * kPairStage +
           (boxes ? kBoxSlots * kBoxBytes : epilogue_warps * 4096) + 1024 + 256;
}

template <Layout L, Epilogue E, int kEpi, bool kBoxes = false, bool kParted = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(pair_threads(kEpi, kBoxes), 1)
    fb_gemm_pair(const __grid_constant__ GemmParams p) {
    constexpr int kStages = pair_stages(kEpi, kBoxes);
    constexpr int kColumnStep = 32 * (kEpi / 4);            // between a warp's chunks
    constexpr uint32_t kSlotBytes = 4096;
    constexpr bool kAMn = L == Layout::kTN;
    constexpr bool kBMn = L != Layout::kNT;
    constexpr bool kIsTn = L == Layout::kTN;
    constexpr uint32_t kIdesc = sm100::instr_desc_f16(256, kPairBN, kAMn, kBMn);
    constexpr uint32_t kTmemCols = 512;

    extern __shared__ unsigned char smem_raw[];
    const uint32_t smem_base = (sm100::smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t staging = smem_base + kStages * kPairStage;
    const uint32_t bars = staging + (kBoxes ? kBoxSlots * kBoxBytes : kEpi * 4096);
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (kStages + s); };
    auto acc_full_bar = [&](int a) { return bars + 8u * (2 * kStages + a); };
    auto acc_empty_bar = [&](int a) { return bars + 8u * (2 * kStages + 2 + a); };
    auto box_full_bar = [&](int s) { return bars + 8u * (2 * kStages + 4 + s); };
    auto box_empty_bar = [&](int s) { return bars + 8u * (2 * kStages + 4 + kBoxSlots + s); };
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    const uint32_t rank = sm100::cluster_cta_rank();
    const bool leader = rank == 0;
    const long long pair = blockIdx.x / 2;
    const long long pairs = gridDim.x / 2;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < kStages; ++s) {
            sm100::mbar_init(full_bar(s), 1);
            sm100::mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            sm100::mbar_init(acc_full_bar(a), 1);
            sm100::mbar_init(acc_empty_bar(a), 2 * kEpi);
        }
        if (kBoxes) {
            for (int s = 0; s < kBoxSlots; ++s) {
                sm100::mbar_init(box_full_bar(s), 1);
                sm100::mbar_init(box_empty_bar(s), 4);   // a warp per quadrant
            }
        }
        sm100::mbar_fence_init();
        sm100::tma_prefetch_descriptor(&p.map_a);
        sm100::tma_prefetch_descriptor(&p.map_b);
    }
    if (warp == 1) {
        sm100::tmem_alloc_pair(sm100::smem_u32(&tmem_base_slot), kTmemCols);
    }
    sm100::tc_fence_before_sync();
    __syncthreads();
    // Both CTAs' barriers exist before either touches the other's.
    sm100::cluster_sync_all();
    sm100::tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_slot;
    volatile int* abort = &abort_flag;
    // Everything above ran while the previous kernel in the stream may still have been
    // finishing; global memory is touched only from here on.
    fb::dependency_wait();
    if (threadIdx.x == 0) {
        fb::dependency_release();
    }

    if (warp == 0) {
        // ---- TMA producer (both CTAs) ----
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (long long id = pair; ok && id < p.tiles_total; id += pairs) {
                const TileCoord t = decode_pair_tile(p, id);
                const bool split_k = kIsTn && !p.batched;
                const int k0 = split_k ? static_cast<int>(t.z) * p.split_len : 0;
                const int k1 = split_k ? min(p.k, k0 + p.split_len) : p.k;
                const int batch = p.batched ? static_cast<int>(t.z) : 0;
                const int row_a = t.tm * 256 + static_cast<int>(rank) * 128;
                const int row_b = t.tn * kPairBN + static_cast<int>(rank) * 128;
                for (int kk = k0; kk < k1; kk += kBK) {
                    if (!sm100::mbar_wait(empty_bar(stage), phase ^ 1u, abort)) {
                        ok = false;
                        break;
                    }
                    const uint32_t a_dst = smem_base + stage * kPairStage;
                    const uint32_t b_dst = a_dst + kPairStageA;
                    if (leader) {
                        // The leader's barrier counts both CTAs' bytes.
                        sm100::mbar_expect_tx(full_bar(stage), 2 * kPairStage);
                    }
                    const uint32_t bar = sm100::map_to_cta(full_bar(stage), 0);
                    if constexpr (!kAMn) {
                        if (p.batched) {
                            sm100::tma_load_3d_pair(a_dst, &p.map_a, bar, kk, row_a, batch);
                        } else {
                            sm100::tma_load_2d_pair(a_dst, &p.map_a, bar, kk, row_a);
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            if (p.batched) {
                                sm100::tma_load_3d_pair(a_dst + j * 8192, &p.map_a, bar,
                                                        row_a + 64 * j, kk, batch);
                            } else {
                                sm100::tma_load_2d_pair(a_dst + j * 8192, &p.map_a, bar,
                                                        row_a + 64 * j, kk);
                            }
                        }
                    }
                    if constexpr (!kBMn) {
                        if (p.batched) {
                            sm100::tma_load_3d_pair(b_dst, &p.map_b, bar, kk, row_b, batch);
                        } else {
                            sm100::tma_load_2d_pair(b_dst, &p.map_b, bar, kk, row_b);
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            if (p.batched) {
                                sm100::tma_load_3d_pair(b_dst + j * 8192, &p.map_b, bar,
                                                        row_b + 64 * j, kk, batch);
                            } else {
                                sm100::tma_load_2d_pair(b_dst + j * 8192, &p.map_b, bar,
                                                        row_b + 64 * j, kk);
                            }
                        }
                    }
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer (leader only) ----
        if (leader) {
            int stage = 0;
            uint32_t phase = 0;
            int acc = 0;
            uint32_t acc_phase = 0;
            bool alive = true;   // the elected lane's: its waits have not given up
            for (long long id = pair; id < p.tiles_total; id += pairs) {
                const TileCoord t = decode_pair_tile(p, id);
                const bool split_k = kIsTn && !p.batched;
                const int k0 = split_k ? static_cast<int>(t.z) * p.split_len : 0;
                const int k1 = split_k ? min(p.k, k0 + p.split_len) : p.k;
                for (int part = 0; part < (kParted ? p.parts : 1); ++part) {
                    const int blocks = (p.k + kBK - 1) / kBK;
                    const int from = kParted ? part_begin(blocks, part, p.parts) * kBK : k0;
                    const int to = kParted ? part_begin(blocks, part + 1, p.parts) * kBK : k1;
                    if (sm100::elect_one()) {
                        alive = alive && sm100::mbar_wait(acc_empty_bar(acc), acc_phase ^ 1u, abort);
                    }
                    const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * kPairBN);
                    uint32_t accumulate = 0;
                    for (int kk = from; kk < to; kk += kBK) {
                        const uint32_t a_addr = smem_base + stage * kPairStage;
                        const uint32_t b_addr = a_addr + kPairStageA;
                        const uint64_t a_desc = kAMn ? sm100::smem_desc_sw128(a_addr, 8192, 1024)
                                                     : sm100::smem_desc_sw128(a_addr, 16, 1024);
                        const uint64_t b_desc = kBMn ? sm100::smem_desc_sw128(b_addr, 8192, 1024)
                                                     : sm100::smem_desc_sw128(b_addr, 16, 1024);
                        if (sm100::elect_one()) {
                            alive = alive && sm100::mbar_wait(full_bar(stage), phase, abort);
                            if (alive) {
                                sm100::tc_fence_after_sync();
#pragma unroll
                                for (int ks = 0; ks < kBK / 16; ++ks) {
                                    sm100::mma_f16_ss_pair(d_tmem, a_desc + ks * (kAMn ? 128 : 2),
                                                           b_desc + ks * (kBMn ? 128 : 2), kIdesc,
                                                           ks == 0 ? accumulate : 1u);
                                }
                                sm100::mma_commit_pair(empty_bar(stage), 3);
                            }
                        }
                        accumulate = 1;
                        if (++stage == kStages) {
                            stage = 0;
                            phase ^= 1u;
                        }
                    }
                    if (sm100::elect_one() && alive) {
                        sm100::mma_commit_pair(acc_full_bar(acc), 3);
                    }
                    acc ^= 1;
                    if (acc == 0) {
                        acc_phase ^= 1u;
                    }
                }
            }
        }
    } else if (kBoxes && warp == 2 + kEpi) {
        // ---- residual producer (both CTAs): a tile's eight boxes in column order ----
        if (lane == 0) {
            uint32_t sequence = 0;
            bool ok = true;
            for (long long id = pair; ok && id < p.tiles_total; id += pairs) {
                const TileCoord t = decode_pair_tile(p, id);
                const int row = t.tm * 256 + static_cast<int>(rank) * 128;
                for (int box = 0; box < kPairBN / 32; ++box, ++sequence) {
                    const int slot = sequence % kBoxSlots;
                    if (!sm100::mbar_wait(box_empty_bar(slot), ((sequence / kBoxSlots) & 1u) ^ 1u, abort)) {
                        ok = false;
                        break;
                    }
                    sm100::mbar_expect_tx(box_full_bar(slot), kBoxBytes);
                    sm100::tma_load_2d(staging + slot * kBoxBytes, &p.map_pre, box_full_bar(slot),
                                       t.tn * kPairBN + box * 32, row);
                }
            }
        }
    } else if (kBoxes) {
        // ---- epilogue warps (both CTAs): a quadrant's 32 rows of every other box ----
        const int quadrant = warp % 4;
        const int column_part = (warp - 2) / 4;
        const int row_in_box = quadrant * 32 + lane;
        int acc = 0;
        uint32_t acc_phase = 0;
        uint32_t boxes = 0;          // of earlier tiles
        int held = -1;               // the slot whose store may still be read
        bool ok = true;
        for (long long id = pair; ok && id < p.tiles_total; id += pairs, boxes += kPairBN / 32) {
            const TileCoord t = decode_pair_tile(p, id);
            const int row = t.tm * 256 + static_cast<int>(rank) * 128 + quadrant * 32;
            const int col0 = t.tn * kPairBN;
            float bias_next = load_bias_lane<E>(p, col0 + column_part * 32, lane);
            if (!sm100::mbar_wait_warp(acc_full_bar(acc), acc_phase, abort)) {
                ok = false;
                break;
            }
            sm100::tc_fence_after_sync();
            const uint32_t t_addr = tmem_base + static_cast<uint32_t>(acc * kPairBN) +
                                    (static_cast<uint32_t>(quadrant * 32) << 16);
            const uint32_t leader_empty = sm100::map_to_cta(acc_empty_bar(acc), 0);
#pragma unroll 1
            for (int box = column_part; box < kPairBN / 32; box += 2) {
                const bool last = box + 2 >= kPairBN / 32;
                const int col = col0 + box * 32;
                const float bias_lane = bias_next;
                if (!last) {
                    bias_next = load_bias_lane<E>(p, col + 64, lane);
                }
                const uint32_t sequence = boxes + box;
                const int slot = sequence % kBoxSlots;
                uint32_t raw[32];
                sm100::tmem_ld_32x32(t_addr + box * 32, raw);
                if (!sm100::mbar_wait_warp(box_full_bar(slot), (sequence / kBoxSlots) & 1u, abort)) {
                    sm100::tmem_ld_wait();
                    ok = false;
                    break;
                }
                sm100::tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; j += 8) {
                    asm volatile(""
                                 : "+r"(raw[j]), "+r"(raw[j + 1]), "+r"(raw[j + 2]), "+r"(raw[j + 3]),
                                   "+r"(raw[j + 4]), "+r"(raw[j + 5]), "+r"(raw[j + 6]), "+r"(raw[j + 7]));
                }
                if (last) {
                    // This warp's reads of the accumulator are complete: hand it back.
                    sm100::tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) {
                        sm100::mbar_arrive_cluster(leader_empty);
                    }
                }
                // 16-byte piece c of row r lies at c ^ (r & 7) (the tensor map's 128-byte swizzle).
                const uint32_t at = staging + slot * kBoxBytes + row_in_box * 128;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint32_t piece = at + ((c ^ (row_in_box & 7)) << 4);
                    const uint4 old = ld_shared_v4(piece);
                    const uint32_t was[4] = {old.x, old.y, old.z, old.w};
                    uint32_t now[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float sum = __fadd_rn(__uint_as_float(raw[4 * c + j]),
                                                    __shfl_sync(0xffffffffu, bias_lane, 4 * c + j));
                        now[j] = __float_as_uint(__fadd_rn(__uint_as_float(was[j]), sum));
                    }
                    st_shared_v4(piece, make_uint4(now[0], now[1], now[2], now[3]));
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    if (col < p.n) {
                        store_chunk_async(&p.map_y, staging + slot * kBoxBytes + quadrant * 4096, col, row);
                    }
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    // The box before this one has been read by its store: its slot is free.
                    asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    if (held >= 0) {
                        sm100::mbar_arrive(box_empty_bar(held));
                    }
                }
                held = slot;
            }
            acc ^= 1;
            if (acc == 0) {
                acc_phase ^= 1u;
            }
        }
        // Asynchronous output stores must have landed before the kernel is over.
        if (lane == 0) {
            store_wait_all();
        }
    } else {
        // ---- epilogue warps (both CTAs) ----
        const int quadrant = warp % 4;
        const int column_part = (warp - 2) / 4;
        const bool coalesced = chunk_path_ok<E>(p);
        const bool prefetch = coalesced && aux_slots<E>() > 1;
        constexpr bool kAhead = kEpi == 8;  // room to keep the next chunk's operands too
        const uint32_t stage = staging + static_cast<uint32_t>(warp - 2) * kSlotBytes;
        int acc = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        // A chunk's second operands (residual, pre-activations) are requested while the
        // chunk before it is processed. For the dGELU epilogue the first chunk of a tile
        // counts as following the last chunk of the tile before, so only this CTA's very
        // first chunk waits for its operands with nothing else to do; the others request
        // a tile's first operands before they wait for its accumulator.
        Aux<E> aux;
        bool aux_requested = false;
        for (long long id = pair; ok && id < p.tiles_total; id += pairs) {
            const TileCoord t = decode_pair_tile(p, id);
            const size_t row = static_cast<size_t>(t.tm) * 256 + rank * 128 + quadrant * 32 + lane;
            const bool row_ok = row < static_cast<size_t>(p.m);
            const int col0 = t.tn * kPairBN;
            const size_t batch_offset =
                p.batched ? static_cast<size_t>(t.z) * p.m * static_cast<size_t>(p.n) : 0;
            if constexpr (kParted) {
                ok = finish_parts<E, kPairBN / kColumnStep, kColumnStep>(
                    p, tmem_base + (static_cast<uint32_t>(quadrant * 32) << 16) + column_part * 32, kPairBN, acc,
                    acc_phase, acc_full_bar,
                    [&](int a) { sm100::mbar_arrive_cluster(sm100::map_to_cta(acc_empty_bar(a), 0)); }, abort, stage,
                    batch_offset, t.z, row, col0 + column_part * 32, lane);
                continue;
            }
            if (prefetch && !aux_requested && p.n - (col0 + column_part * 32) > 0) {
                load_aux<E>(aux, p, batch_offset, row - lane, col0 + column_part * 32,
                            min(32, p.n - (col0 + column_part * 32)), lane);
            }
            aux_requested = false;
            float bias_next = load_bias_lane<E>(p, col0 + column_part * 32, lane);
            if (!sm100::mbar_wait_warp(acc_full_bar(acc), acc_phase, abort)) {
                ok = false;
                break;
            }
            sm100::tc_fence_after_sync();
            const uint32_t t_addr = tmem_base + static_cast<uint32_t>(acc * kPairBN) +
                                    (static_cast<uint32_t>(quadrant * 32) << 16);
            const uint32_t leader_empty = sm100::map_to_cta(acc_empty_bar(acc), 0);
            // The warp's chunks, software-pipelined: chunk i+1's accumulators are being
            // read from tensor memory into the other register set while chunk i is
            // worked on.
            constexpr int kChunks = kPairBN / kColumnStep;
            // The epilogues with second operands already hold a chunk of those ahead; a
            // second accumulator set in flight as well would not fit in registers.
            constexpr bool kPipelined =
                !(E == Epilogue::kBiasResidual || kEpi == kManyWarps || E == Epilogue::kTnStore ||
                  E == Epilogue::kTnPartial || E == Epilogue::kDGelu);
            uint32_t raw[2][32];
            auto chunk_column = [&](int i) { return column_part * 32 + i * kColumnStep; };
            auto chunk_valid = [&](int i) { return min(32, p.n - (col0 + chunk_column(i))); };
            if (kPipelined && chunk_valid(0) > 0) {
                sm100::tmem_ld_32x32(t_addr + chunk_column(0), raw[0]);
            }
            auto work = [&](int i) {
                const bool last = i + 1 == kChunks;
                const int c = chunk_column(i);
                const int col = col0 + c;
                const int valid = chunk_valid(i);
                const float bias_lane = bias_next;
                if (!last) {
                    bias_next = load_bias_lane<E>(p, col + kColumnStep, lane);
                }
                Aux<E> next = aux;
                if (kAhead && prefetch && !last && chunk_valid(i + 1) > 0) {
                    load_aux<E>(next, p, batch_offset, row - lane, col + kColumnStep,
                                chunk_valid(i + 1), lane);
                }
                // (Only where the operands are few registers: with the FP32 residual's 32
                // registers held through the last chunk as well, the kernel was slower.)
                if (E == Epilogue::kDGelu && kAhead && prefetch && last &&
                    id + pairs < p.tiles_total) {
                    // The next tile's first chunk.
                    const TileCoord t2 = decode_pair_tile(p, id + pairs);
                    const size_t row2 =
                        static_cast<size_t>(t2.tm) * 256 + rank * 128 + quadrant * 32;
                    const int col2 = t2.tn * kPairBN + column_part * 32;
                    const size_t offset2 =
                        p.batched ? static_cast<size_t>(t2.z) * p.m * static_cast<size_t>(p.n) : 0;
                    if (p.n - col2 > 0) {
                        load_aux<E>(next, p, offset2, row2, col2, min(32, p.n - col2), lane);
                        aux_requested = true;
                    }
                }
                const int kSet = kPipelined ? (i & 1) : 0;  // static once unrolled
                if (!kPipelined && valid > 0) {
                    sm100::tmem_ld_32x32(t_addr + c, raw[0]);
                }
                sm100::tmem_ld_wait();
                // The loaded registers are "rewritten" by empty volatile statements so
                // that nothing reading them can be scheduled above the wait.
#pragma unroll
                for (int j = 0; j < 32; j += 8) {
                    asm volatile(""
                                 : "+r"(raw[kSet][j]), "+r"(raw[kSet][j + 1]),
                                   "+r"(raw[kSet][j + 2]), "+r"(raw[kSet][j + 3]),
                                   "+r"(raw[kSet][j + 4]), "+r"(raw[kSet][j + 5]),
                                   "+r"(raw[kSet][j + 6]), "+r"(raw[kSet][j + 7]));
                }
                if (kPipelined && !last && chunk_valid(i + 1) > 0) {
                    sm100::tmem_ld_32x32(t_addr + chunk_column(i + 1), raw[(i + 1) & 1]);
                }
                if (last) {
                    // Every read of this accumulator has completed: hand it back.
                    sm100::tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) {
                        sm100::mbar_arrive_cluster(leader_empty);
                    }
                }
                if (valid > 0) {
                    float v[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        v[j] = __uint_as_float(raw[kSet][j]);
                    }
                    if (coalesced) {
                        store_chunk<E>(p, stage, batch_offset, t.z, row - lane, col, v, valid,
                                       lane, aux, bias_lane);
                    } else if (row_ok) {
                        store_segment<E>(p, batch_offset, t.z, row, col, v, valid);
                    }
                }
                if (kAhead) {
                    aux = next;
                } else if (prefetch && !last && chunk_valid(i + 1) > 0) {
                    load_aux<E>(aux, p, batch_offset, row - lane, col + kColumnStep,
                                chunk_valid(i + 1), lane);
                }
            };
            // (Unrolled by a count instead, dGELU spilled: 8,192 x 3,072 x 768 51.2 us -> 54.3.)
            if constexpr (kEpi == kManyWarps) {
#pragma unroll 1
                for (int i = 0; i < kChunks; ++i) {
                    work(i);
                }
            } else {
#pragma unroll
                for (int i = 0; i < kChunks; ++i) {
                    work(i);
                }
            }
            acc ^= 1;
            if (acc == 0) {
                acc_phase ^= 1u;
            }
        }
        // Asynchronous output stores must have landed before the kernel is over.
        if (p.tma_out != 0 && lane == 0) {
            store_wait_all();
        }
    }

    // ---- teardown: neither CTA leaves while the other may still signal it ----
    __syncthreads();
    if (abort_flag != 0) {
        if (threadIdx.x == 0) {
            atomicExch(&g_gemm_error, 1);
        }
        const long long start = clock64();
        while (clock64() - start < 2000000LL) {
        }
        __syncthreads();
    }
    sm100::tc_fence_before_sync();
    sm100::cluster_sync_all();
    if (warp == 1) {
        sm100::tc_fence_after_sync();
        sm100::tmem_dealloc_pair(tmem_base, kTmemCols);
    }
}

// ---- plain CUDA-core kernel, for debugging the pipeline only -------------------------
//
// Selected with FLINT_B200_GEMM=simt in the environment; never the default.

template <Layout L, Epilogue E>
__global__ void __launch_bounds__(256)
    fb_gemm_simt(GemmParams p, const __half* __restrict__ x, const __half* __restrict__ w) {
    const long long total = static_cast<long long>(p.batches) * p.m * p.n;
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
        const long long b = i / (static_cast<long long>(p.m) * p.n);
        const long long r = i - b * p.m * p.n;
        const int row = static_cast<int>(r / p.n);
        const int col = static_cast<int>(r % p.n);
        const __half* xb = x + b * p.m * p.k;
        const __half* wb = w + b * p.n * p.k;
        float acc = 0.0f;
        for (int kk = 0; kk < p.k; ++kk) {
            float a;
            float c;
            if (L == Layout::kTN) {
                a = __half2float(xb[static_cast<size_t>(kk) * p.m + row]);
            } else {
                a = __half2float(xb[static_cast<size_t>(row) * p.k + kk]);
            }
            if (L == Layout::kNT) {
                c = __half2float(wb[static_cast<size_t>(col) * p.k + kk]);
            } else {
                c = __half2float(wb[static_cast<size_t>(kk) * p.n + col]);
            }
            acc = fmaf(a, c, acc);
        }
        const size_t at = static_cast<size_t>(b) * p.m * p.n + static_cast<size_t>(row) * p.n + col;
        if (E == Epilogue::kBias || E == Epilogue::kBiasGelu || E == Epilogue::kBiasResidual) {
            acc = __fadd_rn(acc, p.bias[col]);
        }
        if (E == Epilogue::kScale) {
            acc = __fmul_rn(acc, p.scale);
        }
        if (E == Epilogue::kDGelu) {
            acc = __fmul_rn(acc, gelu_tanh_grad(__half2float(static_cast<const __half*>(p.aux_in)[at])));
        }
        if (E == Epilogue::kBiasResidual) {
            static_cast<float*>(p.y)[at] = __fadd_rn(static_cast<const float*>(p.aux_in)[at], acc);
        } else if (E == Epilogue::kTnStore) {
            float* out = static_cast<float*>(p.y) + at;
            *out = p.accumulate ? __fadd_rn(*out, acc) : acc;
        } else if (E == Epilogue::kBiasGelu) {
            static_cast<__half*>(p.aux_out)[at] = __float2half_rn(acc);
            static_cast<__half*>(p.y)[at] = __float2half_rn(gelu_tanh(acc));
        } else {
            static_cast<__half*>(p.y)[at] = __float2half_rn(acc);
        }
    }
}

// y = (old +) p0 + p1 + ... in split order.
__global__ void __launch_bounds__(256)
    fb_gemm_tn_reduce(float4* __restrict__ y, const float4* __restrict__ partials, size_t quads,
                      int splits, int accumulate) {
    fb::dependency_wait();
    fb::dependency_release();
    partials = fb::after_wait(partials);
    for (size_t i = size_t{blockIdx.x} * 256 + threadIdx.x; i < quads;
         i += size_t{gridDim.x} * 256) {
        float4 s = partials[i];
        for (int k = 1; k < splits; ++k) {
            const float4 v = partials[static_cast<size_t>(k) * quads + i];
            s = make_float4(__fadd_rn(s.x, v.x), __fadd_rn(s.y, v.y), __fadd_rn(s.z, v.z),
                            __fadd_rn(s.w, v.w));
        }
        if (accumulate) {
            const float4 o = y[i];
            s = make_float4(__fadd_rn(o.x, s.x), __fadd_rn(o.y, s.y), __fadd_rn(o.z, s.z),
                            __fadd_rn(o.w, s.w));
        }
        y[i] = s;
    }
}

// ---- host side ----------------------------------------------------------------------------

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                 const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

cudaError_t encode_fn(EncodeTiled* out) {
    static EncodeTiled cached = nullptr;
    if (cached == nullptr) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult status;
        const cudaError_t e =
            cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &status);
        if (e != cudaSuccess) {
            return e;
        }
        if (status != cudaDriverEntryPointSuccess || fn == nullptr) {
            return cudaErrorNotSupported;
        }
        cached = reinterpret_cast<EncodeTiled>(fn);
    }
    *out = cached;
    return cudaSuccess;
}

// A row-major FP16 matrix [outer][inner] (inner contiguous), optionally
// repeated `batches` times back to back; boxes are 64 inner elements (one
// 128-byte swizzle row) by box_outer rows.
cudaError_t make_map(CUtensorMap* map, const void* base, size_t inner, size_t outer,
                     size_t batches, bool batched, int box_outer) {
    EncodeTiled encode = nullptr;
    cudaError_t e = encode_fn(&encode);
    if (e != cudaSuccess) {
        return e;
    }
    const cuuint64_t dims[3] = {inner, outer, batches};
    const cuuint64_t strides[2] = {inner * 2, inner * outer * 2};
    const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box_outer), 1};
    const cuuint32_t elem[3] = {1, 1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, batched ? 3 : 2,
                              const_cast<void*>(base), dims, strides, box, elem,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// FP16 outputs leave through TMA stores when the rows are 16-byte multiples (the tensor map's
// requirement; the same rule as the coalesced path). Batches are a third dimension, so that
// a ragged last tile is clipped at its own batch's edge.
template <Epilogue E>
cudaError_t make_store_maps(GemmParams& p) {
    constexpr bool kHalfOut = E == Epilogue::kNone || E == Epilogue::kBias ||
                              E == Epilogue::kBiasGelu || E == Epilogue::kDGelu ||
                              E == Epilogue::kScale;
    p.tma_out = 0;
    if (!kHalfOut || p.n % 8 != 0) {
        return cudaSuccess;
    }
    EncodeTiled encode = nullptr;
    cudaError_t e = encode_fn(&encode);
    if (e != cudaSuccess) {
        return e;
    }
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(p.n), static_cast<cuuint64_t>(p.m),
                                static_cast<cuuint64_t>(p.batches)};
    const cuuint64_t strides[2] = {dims[0] * 2, dims[0] * dims[1] * 2};
    const cuuint32_t box[3] = {32, 32, 1};
    const cuuint32_t elem[3] = {1, 1, 1};
    auto make = [&](CUtensorMap* map, void* base) {
        return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, p.batched ? 3 : 2, base, dims, strides,
                      box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    if (!make(&p.map_y, p.y) || (E == Epilogue::kBiasGelu && !make(&p.map_pre, p.aux_out))) {
        return cudaErrorInvalidValue;
    }
    p.tma_out = 1;
    return cudaSuccess;
}

bool use_simt() {
    static int cached = -1;
    if (cached < 0) {
        const char* v = std::getenv("FLINT_B200_GEMM");
        cached = (v != nullptr && std::strcmp(v, "simt") == 0) ? 1 : 0;
    }
    return cached == 1;
}

bool pair_disabled() {
    static int cached = -1;
    if (cached < 0) {
        const char* v = std::getenv("FLINT_B200_GEMM");
        cached = (v != nullptr && std::strcmp(v, "single") == 0) ? 1 : 0;
    }
    return cached == 1;
}

// ---- which kernel and tile a problem gets ----------------------------------------------------
//
// The pair kernel's 256 x 256 tiles move the fewest bytes per FLOP and win wherever they fill
// the GPU more than twice. Below that a problem is a few rounds of tiles at most, and its
// time is what one SM spends: the k loop of a tile, which costs about the same per 64 of k
// for every width up to 128, and the epilogue, which grows with the tile's columns. So small
// problems take the narrowest tile that still fits one round, on fb_gemm_once, and divide long
// k loops over clusters. The estimates below reproduce the measured times of 64 to 8,192 rows (widths
// 256 to 1,600; 1,900 timings of fb_gemm_once) to about 15 %; against the best of all tiles, the choice
// lost 5 % or less nearly everywhere.

enum class Tile { k64, k128, k256, kPair, kOnce64, kOnce128, kOnce192 };

struct Plan {
    Tile tile;
    int cluster;   // CTAs over which fb_gemm_once divides k
    int parts;     // of a sum over k, on the persistent kernels
    int splits;    // TN: pieces of k with partial sums in the workspace
};

int tile_columns(Tile t) {
    constexpr int kColumns[] = {64, 128, 256, 256, 64, 128, 192};
    return kColumns[static_cast<int>(t)];
}

constexpr Tile kOnceTiles[] = {Tile::kOnce64, Tile::kOnce128, Tile::kOnce192};

// Microseconds that all tiles have alike, and per 32-column chunk of an epilogue warp: when
// it is the last thing a launch does, and when it runs beside the next tile's k loop (the
// pair kernel stores asynchronously and reads the accumulators a chunk ahead).
constexpr double kTileFixed = 2.7;
struct ChunkTime {
    double last, steady_pair, steady_single;
};
constexpr ChunkTime chunk_time(Epilogue e, size_t k) {
    switch (e) {
    case Epilogue::kNone:
    case Epilogue::kScale:
        return {0.4, 0.5, 0.6};
    case Epilogue::kBias:
        return {0.7, 0.9, 1.2};
    case Epilogue::kTnStore:
    case Epilogue::kTnPartial:
        return {1.1, 1.3, 1.5};
    case Epilogue::kBiasResidual:
        return {1.4, k <= kBoxesMostK ? 2.2 : 2.3, 3.9};
    case Epilogue::kDGelu:
        return {1.5, 1.7, 2.7};
    default:
        return {1.4, 1.4, 2.6};
    }
}

double tile_time(Tile t, Layout l, Epilogue e, long long tiles, size_t k, int sms) {
    constexpr double kBlock[2][4] = {{0.24, 0.26, 0.34, 0.28}, {0.28, 0.34, 0.37, 0.33}};
    const double loop = kBlock[l == Layout::kTN][static_cast<int>(t)] * static_cast<double>((k + kBK - 1) / kBK);
    const long long slots = t == Tile::kPair ? std::max(1, sms / 2) : sms;
    const double more = static_cast<double>((tiles + slots - 1) / slots - 1);
    const int chunks = tile_columns(t) / 64;   // per epilogue warp
    const ChunkTime c = chunk_time(e, k);
    return kTileFixed + loop + chunks * c.last + more * std::max(1.2 * loop, chunks * (t == Tile::kPair ? c.steady_pair : c.steady_single));
}

long long tile_count(Tile t, size_t m, size_t n) {
    const size_t rows = t == Tile::kPair ? 256 : kBM;
    const size_t columns = tile_columns(t);
    return static_cast<long long>((m + rows - 1) / rows) * static_cast<long long>((n + columns - 1) / columns);
}

// Whether a shape can use a tile at all: no tile whose last 64 (of 256: 128) columns would be empty.
bool tile_fits(Tile t, size_t m, size_t n) {
    switch (t) {
    case Tile::k64:
    case Tile::kOnce64:
        return true;
    case Tile::k128:
    case Tile::kOnce128:
        return n > 64;
    case Tile::kPair:
        return !pair_disabled() && m > 128 && n > 128;
    default:
        return n > 128;
    }
}

// fb_gemm_once: microseconds, or 0 where the CTAs would not run at once or the tile cannot be used. Of
// clusters of four, 33 fit this GPU's 148 SMs: a processing cluster of SMs holds whole ones only.
double once_time(Tile t, Layout l, Epilogue e, size_t m, size_t n, size_t k, long long batches,
                 int cluster, int sms) {
    const int i = static_cast<int>(t) - static_cast<int>(Tile::kOnce64);
    const size_t blocks = (k + kBK - 1) / kBK;
    const long long ctas = tile_count(t, m, n) * batches * cluster;
    if (!tile_fits(t, m, n) || ctas > (cluster == 4 ? sms * 8 / 9 : sms)) {
        return 0.0;
    }
    constexpr double kBlock[2][3] = {{0.235, 0.265, 0.305}, {0.285, 0.335, 0.37}};
    // Everything but the k loop, with up to half of the SMs and with more of them at work.
    const int busy = ctas > sms / 2;
    constexpr double kNone[3][2] = {{2.3, 3.0}, {2.9, 3.8}, {3.9, 4.6}}, kBias[3][2] = {{2.6, 3.0}, {3.1, 3.9}, {3.9, 4.6}},
                     kGelu[3][2] = {{3.3, 3.8}, {4.1, 5.3}, {5.4, 6.2}}, kDGelu[3][2] = {{3.4, 3.8}, {4.6, 5.1}, {6.9, 7.7}},
                     kResidual[3][2] = {{3.3, 4.0}, {4.5, 5.4}, {6.7, 8.9}}, kTn[3][2] = {{3.5, 4.1}, {3.9, 4.2}, {4.6, 5.4}};
    const double(*rest)[2] = kNone;
    double more = 0.0;   // than a plain epilogue takes in a cluster, where no warp finishes two chunks
    switch (e) {
    case Epilogue::kBias:
        rest = kBias;
        more = 0.1;
        break;
    case Epilogue::kBiasGelu:
        rest = kGelu;
        more = 0.5;
        break;
    case Epilogue::kDGelu:
        rest = kDGelu;
        more = 0.7;
        break;
    case Epilogue::kBiasResidual:
        rest = kResidual;
        more = 0.3;
        break;
    case Epilogue::kTnStore:
    case Epilogue::kTnPartial:
        rest = kTn;   // (clusters of two at 0.2 more gave up splits in memory: 1,024 x 1,024 x 3,072 13.7 -> 14.9 us)
        more = cluster == 2 && busy != 0 ? 1.2 : 0.2;
        break;
    default:
        break;
    }
    // The same in clusters of two and four, the exchange of partial sums included.
    constexpr double kCluster[2][3][2] = {{{4.0, 5.0}, {4.8, 6.1}, {5.7, 7.0}}, {{4.4, 5.5}, {5.2, 6.5}, {6.3, 7.8}}};
    const double block = l == Layout::kTN && cluster > 1 && i == 2 ? 0.42 : kBlock[l == Layout::kTN][i];
    return (cluster > 1 ? kCluster[cluster / 4][i][busy] + more : rest[i][busy]) +
           block * static_cast<double>((blocks + cluster - 1) / cluster);
}

// What whole sums on fb_gemm_once's 64-column tile take beyond that: past the ring's first rounds its loads
// are slower where most SMs load, or rows are many, and always for TN. (Without this fb_gemm_tc's tile
// was given up for a loss: 2,048 x 512 x 2,048 10.6 -> 11.1 us, with the residual 10.9 -> 11.8, TN 2,048 x 512 x 768
// 6.7 -> 7.2. sum_parts does without: bits change with it.)
double late_blocks(Tile t, Layout l, size_t m, size_t n, size_t k, long long batches, int sms) {
    const double blocks = static_cast<double>((k + kBK - 1) / kBK);
    const long long ctas = tile_count(t, m, n) * batches;
    if (t != Tile::kOnce64) {
        return 0.0;
    }
    if (l == Layout::kTN) {
        return std::max(0.0, 0.08 * (blocks - 8.0));
    }
    const bool many = ctas > sms / 2 && (m > 2 * kBM || (m > kBM && ctas * 4 > sms * 3));
    return many ? std::max(0.0, 0.04 * (blocks - 10.0)) : 0.0;
}

// How often TN may split k with tile `t`: into pieces of at least 1,024, and not at all where
// whole tiles keep three quarters of the CTAs (or pairs) busy.
int most_splits(Tile t, size_t m, size_t n, size_t k, int sms) {
    const long long tiles = tile_count(t, m, n);
    const long long slots = t == Tile::kPair ? std::max(1, sms / 2) : sms;
    const long long waves = (tiles + slots - 1) / slots;
    if (4 * tiles >= 3 * waves * slots) {
        return 1;
    }
    return static_cast<int>(std::min<size_t>(16, std::max<size_t>(1, k / 1024)));
}

// In how many parts an output's sum over k is taken, each part's sum in order and then the parts'
// sums in order. A function of the shape alone, so that every form of a product (NT, NN, TN without a
// workspace, biased, batched) rounds the same sums: what suits the plain NT product. Products a head
// wide are left whole, because those come in batches that fill the GPU by themselves.
int sum_parts(size_t m, size_t n, size_t k, int sms) {
    if (n < 256 || k < 512) {
        return 1;
    }
    double best = 0.0;
    for (Tile t : {Tile::kPair, Tile::k256, Tile::k128, Tile::k64}) {
        if (tile_fits(t, m, n)) {
            const double time = tile_time(t, Layout::kNT, Epilogue::kNone, tile_count(t, m, n), k, sms);
            best = best == 0.0 ? time : std::min(best, time);
        }
    }
    int parts = 1;
    for (int cluster : {1, 2, 4}) {
        for (Tile t : kOnceTiles) {
            const double time = once_time(t, Layout::kNT, Epilogue::kNone, m, n, k, 1, cluster, sms);
            if (time != 0.0 && time < (parts < cluster ? 0.95 : 1.0) * best) {
                best = time;
                parts = cluster;
            }
        }
    }
    return parts;
}

// The kernel for `batches` problems of one shape. With `may_split` (TN) k may also be split with
// partial sums in a workspace, which cost a second launch that reads and adds them.
Plan pick_plan(Layout l, Epilogue e, size_t m, size_t n, size_t k, long long batches, int sms,
               bool may_split) {
    Plan plan = {Tile::k64, 1, 1, 1};
    double best = 0.0;
    // A wider tile, or fewer splits, are given up for a gain of a twentieth, no less; a cluster for
    // splits in memory more easily (TN 2,304 x 768 x 8,192: 30.1 us in splits, 33.4 over clusters).
    auto consider = [&](double time, const Plan& p) {
        if (time != 0.0 && (best == 0.0 || time < (plan.cluster > 1 ? 0.98 : 0.95) * best)) {
            best = time;
            plan = p;
        }
    };
    const int parts = sum_parts(m, n, k, sms);
    if (parts > 1) {
        for (Tile t : kOnceTiles) {
            consider(once_time(t, l, e, m, n, k, batches, parts, sms), Plan{t, parts, 1, 1});
        }
    }
    for (Tile t : {Tile::kPair, Tile::k256, Tile::k128, Tile::k64}) {
        if (!tile_fits(t, m, n)) {
            continue;
        }
        const int most = may_split ? most_splits(t, m, n, k, sms) : 1;
        // (One product that is taken in parts runs on clusters: sum_parts has seen that they fit.)
        for (int s = parts > 1 && batches == 1 ? 2 : 1; s <= most; ++s) {
            double time = tile_time(t, l, e, tile_count(t, m, n) * batches * s, (k + s - 1) / s, sms);
            if (s > 1) {
                time += 1.0 + static_cast<double>(s + 1) * static_cast<double>(m) * static_cast<double>(n) * 4.0 / 16e6;
            }
            consider(time, Plan{t, 1, batches > 1 ? parts : 1, s});
        }
        if (t == Tile::kPair && tile_count(t, m, n) * batches > static_cast<long long>(sms)) {
            return plan;  // more than two rounds of pairs
        }
    }
    if (parts == 1) {
        for (Tile t : kOnceTiles) {
            double time = once_time(t, l, e, m, n, k, batches, 1, sms);
            if (time != 0.0) {
                time += late_blocks(t, l, m, n, k, batches, sms);
            }
            if (time != 0.0 && time < best) {
                best = time;
                plan = Plan{t, 1, 1, 1};
            }
        }
    }
    return plan;
}

// Tensor maps of the FP32 residual, loaded in boxes of 128 rows, and of the FP32 output, stored in
// boxes of 32.
cudaError_t make_box_maps(GemmParams& p) {
    EncodeTiled encode = nullptr;
    const cudaError_t e = encode_fn(&encode);
    if (e != cudaSuccess) {
        return e;
    }
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(p.n), static_cast<cuuint64_t>(p.m)};
    const cuuint64_t strides[1] = {dims[0] * 4};
    const cuuint32_t elem[2] = {1, 1};
    auto make = [&](CUtensorMap* map, const void* base, cuuint32_t rows) {
        const cuuint32_t box[2] = {32, rows};
        return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box,
                      elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    return make(&p.map_pre, p.aux_in, kBM) && make(&p.map_y, p.y, 32) ? cudaSuccess : cudaErrorInvalidValue;
}

// Tensor maps of both operands, B in boxes of `columns` rows (or 64-column panels of it).
template <Layout L>
cudaError_t make_operand_maps(GemmParams& p, const void* x, const void* w, int columns) {
    const bool batched = p.batched != 0;
    const cudaError_t e =
        L == Layout::kTN ? make_map(&p.map_a, x, p.m, p.k, p.batches, batched, kBK)
                         : make_map(&p.map_a, x, p.k, p.m, p.batches, batched, kBM);
    if (e != cudaSuccess) {
        return e;
    }
    return L != Layout::kNT ? make_map(&p.map_b, w, p.n, p.k, p.batches, batched, kBK)
                            : make_map(&p.map_b, w, p.k, p.n, p.batches, batched, columns);
}

// The forms that gemm_batched launches.
template <Layout L, Epilogue E>
constexpr bool batched_form() {
    return E == (L == Layout::kNT ? Epilogue::kScale : Epilogue::kNone);
}

template <Layout L, Epilogue E, int BN>
cudaError_t launch_tc(GemmParams& p, const void* x, const void* w, int sms, cudaStream_t stream) {
    using R = Ring<BN>;
    const bool batched = p.batched != 0;
    cudaError_t e = make_operand_maps<L>(p, x, w, BN);
    if (e != cudaSuccess) {
        return e;
    }
    e = make_store_maps<E>(p);
    if (e != cudaSuccess) {
        return e;
    }
    p.tiles_m = (p.m + kBM - 1) / kBM;
    p.tiles_n = (p.n + BN - 1) / BN;
    const long long z = L == Layout::kTN && !batched ? p.splits : p.batches;
    p.tiles_total = static_cast<long long>(p.tiles_m) * p.tiles_n * z;

    auto launch = [&](auto kernel, std::atomic<bool> (&configured)[64]) {
        const cudaError_t error = fb::allow_shared_memory(kernel, R::kSmemBytes, configured);
        if (error != cudaSuccess) {
            return error;
        }
        const unsigned grid = static_cast<unsigned>(std::min<long long>(p.tiles_total, sms));
        return fb::launch_dependent(kernel, dim3(grid), dim3(kThreads), R::kSmemBytes, stream, p);
    };
    static std::atomic<bool> configured[2][64] = {};
    if constexpr (batched_form<L, E>()) {
        if (p.parts > 1) {
            return launch(fb_gemm_tc<L, E, BN, true>, configured[1]);
        }
    }
    return launch(fb_gemm_tc<L, E, BN>, configured[0]);
}

template <Layout L, Epilogue E>
cudaError_t launch_pair(GemmParams& p, const void* x, const void* w, int sms, cudaStream_t stream) {
    const bool batched = p.batched != 0;
    cudaError_t e = make_operand_maps<L>(p, x, w, 128);
    if (e != cudaSuccess) {
        return e;
    }
    e = make_store_maps<E>(p);
    if (e != cudaSuccess) {
        return e;
    }
    p.tiles_m = (p.m + 255) / 256;
    p.tiles_n = (p.n + kPairBN - 1) / kPairBN;
    const long long z = L == Layout::kTN && !batched ? p.splits : p.batches;
    p.tiles_total = static_cast<long long>(p.tiles_m) * p.tiles_n * z;

    const long long pairs = std::min<long long>(p.tiles_total, sms / 2);
    auto launch = [&](auto kernel, int epilogue_warps, bool boxes, std::atomic<bool> (&configured)[64]) {
        const int smem = pair_smem_bytes(epilogue_warps, boxes);
        const cudaError_t error = fb::allow_shared_memory(kernel, smem, configured);
        if (error != cudaSuccess) {
            return error;
        }
        return fb::launch_dependent(kernel, dim3(static_cast<unsigned>(2 * pairs)),
                                    dim3(static_cast<unsigned>(pair_threads(epilogue_warps, boxes))),
                                    static_cast<size_t>(smem), stream, p);
    };
    static std::atomic<bool> configured[3][64] = {};
    if constexpr (batched_form<L, E>()) {
        if (p.parts > 1) {
            return launch(fb_gemm_pair<L, E, kEpilogueWarps, false, true>, kEpilogueWarps, false, configured[2]);
        }
    }
    if constexpr (E == Epilogue::kBiasResidual) {
        if (p.n % 4 == 0 && static_cast<size_t>(p.k) <= kBoxesMostK) {
            e = make_box_maps(p);
            return e != cudaSuccess ? e
                                    : launch(fb_gemm_pair<L, E, kEpilogueWarps, true>, kEpilogueWarps, true, configured[1]);
        }
    }
    if constexpr (E == Epilogue::kBiasGelu || E == Epilogue::kScale) {
        constexpr bool kScores = E == Epilogue::kScale;
        const size_t bytes = static_cast<size_t>(p.batches) * p.m * p.n * (kScores ? 2 : 4);   // of all outputs
        if (static_cast<size_t>(p.k) <= (kScores ? kManyWarpsMostScaledK : kManyWarpsMostK) &&
            (p.n % 16 == 0 || bytes <= kManyWarpsMostRaggedBytes) && (kScores || p.tiles_total > pairs)) {
            return launch(fb_gemm_pair<L, E, kManyWarps>, kManyWarps, false, configured[1]);
        }
    }
    return launch(fb_gemm_pair<L, E, kEpilogueWarps>, kEpilogueWarps, false, configured[0]);
}

template <Layout L, Epilogue E, int BN>
cudaError_t launch_once(GemmParams& p, const void* x, const void* w, const Plan& plan, bool steady_w,
                        cudaStream_t stream) {
    const int cluster = plan.cluster;
    using R = OnceRing<BN>;
    cudaError_t e = make_operand_maps<L>(p, x, w, BN);
    if (e != cudaSuccess) {
        return e;
    }
    constexpr bool kFloatOut = E == Epilogue::kBiasResidual || E == Epilogue::kTnStore;
    auto wide = [](const void* at) { return reinterpret_cast<uintptr_t>(at) % 32 == 0; };
    OnceParams once;
    once.steady_b = steady_w ? 1 : 0;
    once.wide_out = p.n % (kFloatOut ? 8 : 16) == 0 && wide(p.y) && wide(p.aux_out);
    once.cluster = cluster;
    p.tiles_m = (p.m + kBM - 1) / kBM;
    p.tiles_n = (p.n + BN - 1) / BN;
    p.tiles_total = static_cast<long long>(p.tiles_m) * p.tiles_n * p.batches;

    once.stages = R::stages(cluster);
    once.gemm = p;
    auto launch = [&](auto kernel, std::atomic<bool> (&configured)[64]) {
        const cudaError_t error = fb::allow_shared_memory(kernel, 220 * 1024, configured);
        if (error != cudaSuccess) {
            return error;
        }
        return fb::launch_dependent_cluster(kernel, dim3(static_cast<unsigned>(p.tiles_total * cluster)),
                                            dim3(kOnceThreads), static_cast<unsigned>(cluster),
                                            R::bytes(cluster), stream, once);
    };
    static std::atomic<bool> configured[2][64] = {};
    return cluster > 1 ? launch(fb_gemm_once<L, E, BN, true>, configured[1])
                                    : launch(fb_gemm_once<L, E, BN, false>, configured[0]);
}

template <Layout L, Epilogue E>
cudaError_t launch_any(GemmParams& p, const void* x, const void* w, cudaStream_t stream,
                       const Plan* given = nullptr, bool steady_w = false) {
    int sms = 0;
    cudaError_t e = sm_count(&sms);
    if (e != cudaSuccess) {
        return e;
    }
    if (use_simt()) {
        const long long total = static_cast<long long>(p.batches) * p.m * p.n;
        const unsigned grid =
            static_cast<unsigned>(std::min<long long>((total + 255) / 256, sms * 32LL));
        fb_gemm_simt<L, E><<<grid, 256, 0, stream>>>(p, static_cast<const __half*>(x),
                                                     static_cast<const __half*>(w));
        return fb::after_launch();
    }
    const Plan plan = given != nullptr ? *given : pick_plan(L, E, p.m, p.n, p.k, p.batches, sms, false);
    if constexpr (E != Epilogue::kTnPartial) {
        switch (plan.tile) {
        case Tile::kOnce192:
            return launch_once<L, E, 192>(p, x, w, plan, steady_w, stream);
        case Tile::kOnce128:
            return launch_once<L, E, 128>(p, x, w, plan, steady_w, stream);
        case Tile::kOnce64:
            return launch_once<L, E, 64>(p, x, w, plan, steady_w, stream);
        default:
            break;
        }
    }
    p.parts = plan.parts;
    switch (plan.tile) {
    case Tile::kPair:
        return launch_pair<L, E>(p, x, w, sms, stream);
    case Tile::k256:
        return launch_tc<L, E, 256>(p, x, w, sms, stream);
    case Tile::k128:
        return launch_tc<L, E, 128>(p, x, w, sms, stream);
    default:
        return launch_tc<L, E, 64>(p, x, w, sms, stream);
    }
}

GemmParams base_params(void* y, size_t m, size_t n, size_t k, size_t batches, bool batched) {
    GemmParams p;
    std::memset(&p, 0, sizeof p);
    p.y = y;
    p.m = static_cast<int>(m);
    p.n = static_cast<int>(n);
    p.k = static_cast<int>(k);
    p.batches = static_cast<int>(batches);
    p.batched = batched ? 1 : 0;
    p.parts = 1;
    p.splits = 1;
    p.split_len = static_cast<int>((k + kBK - 1) / kBK * kBK);
    p.scale = 1.0f;
    return p;
}

}  // namespace

// ---- internal launchers (declared in gemm.h) --------------------------------------------

namespace {
// (kTnPartial's and kTnStore's chunks cost the same, so both see one plan.)
Plan tn_plan(size_t m, size_t n, size_t k, int sms, TnSplit* split) {
    const Plan plan = pick_plan(Layout::kTN, Epilogue::kTnStore, m, n, k, 1, sms, true);
    const size_t per = (k + plan.splits - 1) / plan.splits;
    split->len = static_cast<int>((per + kBK - 1) / kBK * kBK);
    split->count = static_cast<int>((k + split->len - 1) / split->len);
    return plan;
}
}  // namespace

TnSplit tn_split(size_t m, size_t n, size_t k, int sms) {
    TnSplit split;
    tn_plan(m, n, k, sms, &split);
    return split;
}

cudaError_t gemm_nt(Epilogue e, void* y, void* pre, const void* x, const void* w,
                    const void* bias, const void* residual, size_t m, size_t n, size_t k,
                    cudaStream_t stream, bool steady_w) {
    GemmParams p = base_params(y, m, n, k, 1, false);
    p.bias = static_cast<const float*>(bias);
    p.aux_out = pre;
    p.aux_in = residual;
    switch (e) {
    case Epilogue::kNone:
        return launch_any<Layout::kNT, Epilogue::kNone>(p, x, w, stream);
    case Epilogue::kBias:
        return launch_any<Layout::kNT, Epilogue::kBias>(p, x, w, stream, nullptr, steady_w);
    case Epilogue::kBiasGelu:
        return launch_any<Layout::kNT, Epilogue::kBiasGelu>(p, x, w, stream, nullptr, steady_w);
    case Epilogue::kBiasResidual:
        return launch_any<Layout::kNT, Epilogue::kBiasResidual>(p, x, w, stream, nullptr, steady_w);
    default:
        return cudaErrorInvalidValue;
    }
}

cudaError_t gemm_nn(Epilogue e, void* y, const void* x, const void* w, const void* pre, size_t m,
                    size_t n, size_t k, cudaStream_t stream) {
    GemmParams p = base_params(y, m, n, k, 1, false);
    p.aux_in = pre;
    if (e == Epilogue::kDGelu) {
        return launch_any<Layout::kNN, Epilogue::kDGelu>(p, x, w, stream);
    }
    return launch_any<Layout::kNN, Epilogue::kNone>(p, x, w, stream);
}

cudaError_t gemm_tn(void* y, const void* x, const void* w, size_t m, size_t n, size_t k,
                    bool accumulate, void* workspace, cudaStream_t stream) {
    int sms = 0;
    cudaError_t e = sm_count(&sms);
    if (e != cudaSuccess) {
        return e;
    }
    GemmParams p = base_params(y, m, n, k, 1, false);
    p.accumulate = accumulate ? 1 : 0;
    TnSplit s{1, p.split_len};
    Plan plan{Tile::k64, 1, 1, 1};
    if (!use_simt()) {
        plan = tn_plan(m, n, k, sms, &s);
    }
    if (s.count == 1) {
        return launch_any<Layout::kTN, Epilogue::kTnStore>(p, x, w, stream, &plan);
    }
    p.splits = s.count;
    p.split_len = s.len;
    p.partials = static_cast<float*>(workspace);
    e = launch_any<Layout::kTN, Epilogue::kTnPartial>(p, x, w, stream, &plan);
    if (e != cudaSuccess) {
        return e;
    }
    const size_t quads = m * n / 4;
    const unsigned grid =
        static_cast<unsigned>(std::min<size_t>((quads + 255) / 256, static_cast<size_t>(sms) * 8));
    return fb::launch_dependent(fb_gemm_tn_reduce, dim3(grid), dim3(256), 0, stream,
                                static_cast<float4*>(y), static_cast<const float4*>(workspace),
                                quads, s.count, p.accumulate);
}

cudaError_t gemm_batched(Layout l, void* y, const void* x, const void* w, size_t batches,
                         size_t m, size_t n, size_t k, float scale, cudaStream_t stream) {
    GemmParams p = base_params(y, m, n, k, batches, true);
    p.scale = scale;
    switch (l) {
    case Layout::kNT:
        return launch_any<Layout::kNT, Epilogue::kScale>(p, x, w, stream);
    case Layout::kNN:
        return launch_any<Layout::kNN, Epilogue::kNone>(p, x, w, stream);
    default:
        return launch_any<Layout::kTN, Epilogue::kNone>(p, x, w, stream);
    }
}

cudaError_t gemm_error_flag(int* value, bool reset) {
    cudaError_t e = cudaMemcpyFromSymbol(value, g_gemm_error, sizeof(int));
    if (e == cudaSuccess && reset && *value != 0) {
        const int zero = 0;
        e = cudaMemcpyToSymbol(g_gemm_error, &zero, sizeof(int));
    }
    return e;
}

}  // namespace fb

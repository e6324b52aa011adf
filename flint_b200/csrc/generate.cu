// Autoregressive decoding for a GPT-2 model's weights: a KV cache, single-query
// (decode) attention, and weight-only int8 linear layers (extension; the reference
// lists this as its inference milestone in README.md:148 and has no code for it).
// The oracle is the reference's PyTorch model run on the whole sequence
// (scripts/gpt2_torch.py:52-131): the logits at each position must agree.
//
// Two regimes:
//   prefill   the prompt's rows go through the library's tensor-core GEMMs and the
//             fused causal attention kernel, exactly as in the training forward pass,
//             and their keys and values are copied into the cache
//   decode    one new token per sequence, five kernels per layer. At this size no single
//             kernel is long enough to be bound by HBM; a step is a chain of dependent
//             kernels, so what counts is how little each does after the one before it has
//             finished. Every kernel is launched to start early (programmatic dependent
//             launch), fetches what does not depend on the step into registers (its weights,
//             the cache's older keys and values), and only then waits for its predecessor.
//             Products run on mma.sync with the sequences as the 16 rows of A and eight
//             output features as the columns of B, so up to 16 sequences cost one MMA per
//             16 weights of a feature.
//             (Many rows of a wide FP16 model take the prompt's GEMMs: tensor_core_step().)
//             Positions live in device memory, so a step's launches do not change from
//             token to token and are captured once into a CUDA graph.
//
// Cache layout: [layer][K or V][sequence][head][position][64] FP16. A position's key is
// 128 contiguous bytes and a head's positions are contiguous, so decode attention
// reads whole cache lines in order.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <memory>
#include <new>
#include <vector>

#include <cuda_fp16.h>

#include "attention.h"
#include "common.h"
#include "device_utils.cuh"
#include "flint/flint_b200.h"
#include "gemm.h"
#include "gpt2.h"

namespace {

constexpr flint_status kInvalid = FLINT_ERROR_INVALID_ARGUMENT;
constexpr int kHeadWidth = 64;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kEps = 1e-5f;

enum class Act { kNone, kGelu, kResidual };

struct Matrix {
    const __half* half = nullptr;   // [n, k] FP16 (the model's compute copy)
    int8_t* q = nullptr;            // [n, k] int8 (generator-owned) or null
    float* scale = nullptr;         // [n] FP32: w[n, :] ~ q[n, :] * scale[n]
    const float* bias = nullptr;    // [n] FP32 or null
    size_t n = 0, k = 0;
};

struct Layer {
    const float *ln1_w, *ln1_b, *ln2_w, *ln2_b;
    Matrix attn, proj, fc, fcproj;
};

__device__ __forceinline__ float gelu_tanh(float x) {
    const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
    return 0.5f * x * (1.0f + tanhf(u));
}

// ---- per-row int8 quantisation -----------------------------------------------------------------

// One warp per row: scale = max|w| / 127, q = round(w / scale).
__global__ void __launch_bounds__(256)
    fb_quantize_rows(int8_t* __restrict__ q, float* __restrict__ scale,
                     const __half* __restrict__ w, size_t rows, size_t cols) {
    const size_t row = blockIdx.x * 8ull + threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    if (row >= rows) {
        return;
    }
    const __half* src = w + row * cols;
    float top = 0.0f;
    for (size_t c = lane; c < cols; c += 32) {
        top = fmaxf(top, fabsf(__half2float(src[c])));
    }
    top = fb::warp_max(top);
    const float s = top > 0.0f ? top / 127.0f : 1.0f;
    const float inv = 1.0f / s;
    for (size_t c = lane; c < cols; c += 32) {
        const float v = rintf(__half2float(src[c]) * inv);
        q[row * cols + c] = static_cast<int8_t>(fminf(fmaxf(v, -127.0f), 127.0f));
    }
    if (lane == 0) {
        scale[row] = s;
    }
}

// The int8 matrices of a layer back to FP16, for a prompt's GEMMs: 16 values a thread, one launch.
// (A launch per matrix and a value per thread: 48 launches of 5.6 us in a prompt of GPT-2 124M.)
struct DequantizeArgs {
    static constexpr int kMatrices = 4;
    const int8_t* q[kMatrices];
    const float* scale[kMatrices];
    unsigned cols[kMatrices];     // multiples of 128
    unsigned end[kMatrices];      // 16-value pieces up to this matrix's end
    __half* out;                  // the matrices one after the other
};

__global__ void __launch_bounds__(256) fb_dequantize_layer(const DequantizeArgs p) {
    fb::dependency_wait();        // the GEMMs that read the layer before have finished
    fb::dependency_release();
    const unsigned total = p.end[DequantizeArgs::kMatrices - 1];
    for (unsigned i = blockIdx.x * 256u + threadIdx.x; i < total; i += gridDim.x * 256u) {
        int m = 0;
        while (i >= p.end[m]) {
            ++m;
        }
        const unsigned piece = i - (m > 0 ? p.end[m - 1] : 0u);
        const float scale = p.scale[m][piece / (p.cols[m] / 16)];
        const uint4 raw = reinterpret_cast<const uint4*>(p.q[m])[piece];
        const unsigned words[4] = {raw.x, raw.y, raw.z, raw.w};
        unsigned halves[8];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float lo = static_cast<float>(static_cast<int8_t>(words[w] >> (16 * h)));
                const float hi = static_cast<float>(static_cast<int8_t>(words[w] >> (16 * h + 8)));
                halves[2 * w + h] = fb::pack2(lo * scale, hi * scale);
            }
        }
        uint4* out = reinterpret_cast<uint4*>(p.out) + 2 * static_cast<size_t>(i);
        out[0] = make_uint4(halves[0], halves[1], halves[2], halves[3]);
        out[1] = make_uint4(halves[4], halves[5], halves[6], halves[7]);
    }
}

// ---- linear layers of a decode step -----------------------------------------------------------
//
// y[b, n] = act(sum_k x[b, k] w[n, k] (* scale[n]) + bias[n]) for one row b per sequence.
// A dot product does not care in which order k is taken, so a lane's share of an MMA is
// chosen to be contiguous: lane (g, t) = (lane / 4, lane % 4) loads 16 bytes of feature g's
// weights and the matching activations of rows g and g + 8, and each group of four values
// becomes the four k positions that lane holds in one m16n8k16. Weights need no shuffling,
// no shared memory and no conversion (int8 becomes FP16 exactly: all 256 values are FP16
// integers), and come straight into registers before the kernel waits for its predecessor.

constexpr int kWarps = 8;
constexpr int kThreads = 32 * kWarps;

// 16 bytes that will not be read again: bypass L1.
__device__ __forceinline__ uint4 load_streaming(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

// 16 bytes that an earlier kernel of the step wrote while this one was already resident:
// volatile, so after the wait it stands behind, and from L2.
__device__ __forceinline__ uint4 load_fresh(const void* p) {
    uint4 v;
    asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}

__device__ __forceinline__ float load_fresh_float(const float* p) {
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}

// 16 products per element, added by the tensor core; never onto an earlier sum. (It cuts sums
// off where FP32 additions round them, and over a chain of MMAs the cuts add up. Relative error
// of dot products of 3,072 values, signed and all positive: FP32 FMAs and a butterfly 1.7e-7
// and 0.5e-7, MMA chains 2.7e-7 and 8.6e-7, one MMA at a time with FP32 additions 1.0e-7 and
// 0.7e-7; of 768: 1.0e-7 and 0.5e-7, 1.2e-7 and 1.7e-7, 0.9e-7 and 0.7e-7.)
__device__ __forceinline__ void mma_16x8x16(float (&d)[4], unsigned a0, unsigned a1, unsigned a2,
                                            unsigned a3, unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}

// Four int8 values as two FP16 pairs: the byte with its sign bit flipped is v + 128, under
// 0x64 the FP16 number 1024 + (v + 128), from which 1152 is subtracted exactly.
__device__ __forceinline__ void int8_to_half(unsigned word, unsigned& lo, unsigned& hi) {
    const unsigned biased = word ^ 0x80808080u;
    const __half2 offset = __half2half2(__ushort_as_half(0x6480));  // 1152
    unsigned l = __byte_perm(biased, 0x64646464u, 0x4140);
    unsigned h = __byte_perm(biased, 0x64646464u, 0x4342);
    const __half2 l2 = __hsub2(*reinterpret_cast<const __half2*>(&l), offset);
    const __half2 h2 = __hsub2(*reinterpret_cast<const __half2*>(&h), offset);
    lo = *reinterpret_cast<const unsigned*>(&l2);
    hi = *reinterpret_cast<const unsigned*>(&h2);
}

// A lane's 16 weight bytes of one step: kStepK values of k per warp and step, kValues of them
// this lane's, in kPieces groups of eight activations.
template <typename W>
struct Step;
template <>
struct Step<__half> {
    static constexpr int kStepK = 32, kValues = 8, kPieces = 1;
    static __device__ __forceinline__ void weights(const uint4& raw, int i, unsigned& b0,
                                                   unsigned& b1) {
        b0 = i == 0 ? raw.x : raw.z;
        b1 = i == 0 ? raw.y : raw.w;
    }
};
template <>
struct Step<int8_t> {
    static constexpr int kStepK = 64, kValues = 16, kPieces = 2;
    static __device__ __forceinline__ void weights(const uint4& raw, int i, unsigned& b0,
                                                   unsigned& b1) {
        const unsigned word = i == 0 ? raw.x : i == 1 ? raw.y : i == 2 ? raw.z : raw.w;
        int8_to_half(word, b0, b1);
    }
};

// One step of NT feature tiles: x(block, piece) gives this lane's eight activations of row
// 8 * block + g. RB: blocks of eight rows (1, or an even number).
template <typename W, int RB, int NT, typename X>
__device__ __forceinline__ void multiply(float (&acc)[(RB + 1) / 2][NT][4], const uint4 (&raw)[NT], X x) {
#pragma unroll
    for (int piece = 0; piece < Step<W>::kPieces; ++piece) {
#pragma unroll
        for (int m = 0; m < (RB + 1) / 2; ++m) {
            const uint4 xa = x(2 * m, piece);
            const uint4 xb = RB > 1 ? x(2 * m + 1, piece) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                unsigned b0, b1;
                float first[4];
                float second[4];
                Step<W>::weights(raw[nt], 2 * piece, b0, b1);
                mma_16x8x16(first, xa.x, xb.x, xa.y, xb.y, b0, b1);
                Step<W>::weights(raw[nt], 2 * piece + 1, b0, b1);
                mma_16x8x16(second, xa.z, xb.z, xa.w, xb.w, b0, b1);
#pragma unroll
                for (int i = 0; i < (RB == 1 ? 2 : 4); ++i) {
                    acc[m][nt][i] += first[i] + second[i];
                }
            }
        }
    }
}

template <int N>
__device__ __forceinline__ float add_pairwise(float (&part)[N]) {
#pragma unroll
    for (int stride = 1; stride < N; stride *= 2) {
#pragma unroll
        for (int i = 0; i + stride < N; i += 2 * stride) {
            part[i] += part[i + stride];
        }
    }
    return part[0];
}

// LayerNorm of `rows` FP32 rows into FP16 rows of k + 8 values in shared memory (the 16 bytes
// between rows keep eight rows' 16-byte reads off each other's banks): a warp per row, the
// row in registers, QN float4s a lane. Each lane takes its own values' mean and centred
// squares; one butterfly merges both (Chan, Golub and LeVeque's update for equal counts: k is
// a multiple of 128, so every lane has k / 32 values).
// Precision: a lane's few values are added pairwise, the merges of the squares keep their
// rounding errors (TwoSum), and 1 / sqrt is rsqrtf() with a Newton-Raphson step behind it. A
// row before its rounding to FP16 is then as close to the exact one as
// flint_layernorm_forward's compensated sums bring it (relative error, emulated on rows of
// normal values: 5.4e-8 against 5.9e-8 for 256 columns, 5.7e-8 against 6.0e-8 for 768; with outlier
// channels 5.7e-8 against 5.8e-8); with plain merges and rsqrtf() alone it was 1.0e-7. That
// function's own sums, or sums in 64 bits, made a step 9 to 36 % longer here, these 2 %.
template <int QN>
__device__ __forceinline__ void normalise_rows(__half* h, const float* x, const float* gain,
                                               const float* shift, int rows, int k) {
    const int lane = threadIdx.x % 32;
    const float inverse = 32.0f / static_cast<float>(k);   // of a lane's count
    for (int row = threadIdx.x / 32; row < rows; row += kWarps) {
        const float4* src = reinterpret_cast<const float4*>(x + static_cast<size_t>(row) * k);
        float4 v[QN];
#pragma unroll
        for (int i = 0; i < QN; ++i) {
            v[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (128 * i < k) {
                const uint4 raw = load_fresh(src + lane + 32 * i);
                v[i] = make_float4(__uint_as_float(raw.x), __uint_as_float(raw.y),
                                   __uint_as_float(raw.z), __uint_as_float(raw.w));
            }
        }
        // (Absent float4s are zeros: they change neither sum.)
        float part[QN];
#pragma unroll
        for (int i = 0; i < QN; ++i) {
            part[i] = (v[i].x + v[i].y) + (v[i].z + v[i].w);
        }
        float mean = add_pairwise(part) * inverse;
#pragma unroll
        for (int i = 0; i < QN; ++i) {
            part[i] = 0.0f;
            if (128 * i < k) {
                const float4 d = make_float4(v[i].x - mean, v[i].y - mean, v[i].z - mean, v[i].w - mean);
                part[i] = fmaf(d.x, d.x, d.y * d.y) + fmaf(d.z, d.z, d.w * d.w);
            }
        }
        float centred = add_pairwise(part);
        float lost = 0.0f;                                  // what the merges of `centred` left over
        float half_count = static_cast<float>(k) / 64.0f;   // half of what each side has
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const float other = __shfl_xor_sync(fb::kFullMask, mean, off);
            const float theirs = __shfl_xor_sync(fb::kFullMask, centred, off);
            const float their_loss = __shfl_xor_sync(fb::kFullMask, lost, off);
            const float apart = other - mean;
            mean = 0.5f * (mean + other);
            const float both = __fadd_rn(centred, theirs);
            const float added = __fsub_rn(both, centred);
            const float error = __fadd_rn(__fsub_rn(centred, __fsub_rn(both, added)),
                                          __fsub_rn(theirs, added));
            centred = both;
            lost = (lost + their_loss) + fmaf(apart * apart, half_count, error);
            half_count *= 2.0f;
        }
        const float variance = fmaf(centred + lost, 1.0f / static_cast<float>(k), kEps);
        const float guess = rsqrtf(variance);
        const float rstd = fmaf(0.5f * guess, fmaf(-(variance * guess), guess, 1.0f), guess);
#pragma unroll
        for (int i = 0; i < QN; ++i) {
            const int q = lane + 32 * i;
            if (128 * i < k) {
                const float4 g = reinterpret_cast<const float4*>(gain)[q];
                const float4 b = reinterpret_cast<const float4*>(shift)[q];
                uint2 packed;
                packed.x = fb::pack2((v[i].x - mean) * rstd * g.x + b.x, (v[i].y - mean) * rstd * g.y + b.y);
                packed.y = fb::pack2((v[i].z - mean) * rstd * g.z + b.z, (v[i].w - mean) * rstd * g.w + b.w);
                reinterpret_cast<uint2*>(h + static_cast<size_t>(row) * (k + 8))[q] = packed;
            }
        }
    }
}

struct LinearArgs {
    void* out;
    const void* w;
    const float* scale;     // int8: one per feature
    const float* bias;
    const void* x;          // FP16 rows, or FP32 rows to normalise first
    const float* gain;
    const float* shift;
    const float* residual;
    int rows, n, k;
};

// Shared memory of a kernel that normalises: gain, shift and the FP16 rows.
__host__ __device__ constexpr int norm_bytes(int rows, int k) { return 8 * k + rows * (k + 8) * 2; }

// Shared memory of a linear kernel: the above, then the warps' sums (of 64 rows they do not
// fit beside 64 wide rows; they then take the rows' place once those have been used).
__host__ __device__ constexpr int sums_bytes(int rb, int nt) { return kWarps * 8 * rb * 8 * nt * 4; }
__host__ __device__ constexpr int linear_bytes(bool norm, int rb, int nt, int rows, int k) {
    const int first = norm ? norm_bytes(rows, k) : 0;
    return rb < 8 ? first + sums_bytes(rb, nt)
                  : (first > sums_bytes(rb, nt) ? first : sums_bytes(rb, nt));
}

// CTAs per SM that registers must leave room for. Kernels of a step are resident several deep,
// so a few registers decide what fits beside what: with 42 instead of 40 for the small int8
// projection four sequences took 189 us a step instead of 171, and one CTA per SM in place of
// two for the widest FP16 one made a step of one sequence 1,536 wide 378 us instead of 349.
constexpr int linear_blocks(bool norm, int rb, int steps) {
    return rb == 8                       ? 1
           : norm || steps > 3 || rb > 2 ? (rb == 4 && steps > 12 ? 1 : 2)
           : rb == 2                     ? 4
           : steps == 3                  ? 5
                                         : 6;
}

// A CTA owns 8 NT features, its warps a share of k each; the warps' sums meet in shared
// memory and are added in warp order. kSteps: the steps a warp's share can have.
template <typename W, Act A, bool kNorm, int RB, int NT, int kSteps, int QN>
__global__ void __launch_bounds__(kThreads, linear_blocks(kNorm, RB, kSteps))
    fb_decode_linear(const LinearArgs p) {
    using S = Step<W>;
    constexpr int kColumns = 8 * NT;
    extern __shared__ __align__(16) unsigned char decode_smem[];
    using Sums = float[8 * RB][kColumns];
    Sums* sums = reinterpret_cast<Sums*>(decode_smem +
                                         (kNorm && RB < 8 ? norm_bytes(p.rows, p.k) : 0));
    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    const int g = lane / 4;
    const int t = lane % 4;
    const int first = blockIdx.x * kColumns;
    const int steps = p.k / S::kStepK;
    const int share = (steps + kWarps - 1) / kWarps;
    const int begin = warp * share;
    const int mine = min(share, steps - begin);   // may be none
    uint4 raw[kSteps][NT];
#pragma unroll
    for (int j = 0; j < kSteps; ++j) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            raw[j][nt] = make_uint4(0u, 0u, 0u, 0u);
            if (j < mine) {
                raw[j][nt] = load_streaming(static_cast<const W*>(p.w) +
                                            static_cast<size_t>(first + 8 * nt + g) * p.k +
                                            (begin + j) * S::kStepK + t * S::kValues);
            }
        }
    }
    const int feature = first + static_cast<int>(threadIdx.x) % kColumns;
    const float scale = p.scale != nullptr ? p.scale[feature] : 1.0f;
    const float bias = p.bias[feature];
    float* gain = reinterpret_cast<float*>(decode_smem);
    float* shift = gain + p.k;
    __half* rows = reinterpret_cast<__half*>(shift + p.k);
    if constexpr (kNorm) {
        for (int i = threadIdx.x; i < p.k / 4; i += kThreads) {
            reinterpret_cast<float4*>(gain)[i] = reinterpret_cast<const float4*>(p.gain)[i];
            reinterpret_cast<float4*>(shift)[i] = reinterpret_cast<const float4*>(p.shift)[i];
        }
        __syncthreads();
    }
    // Nothing above depends on the step's kernels.
    fb::dependency_wait();
    fb::dependency_release();
    const size_t out_at = static_cast<size_t>(threadIdx.x / kColumns) * p.n + feature;
    float residual = 0.0f;
    if (A == Act::kResidual && static_cast<int>(threadIdx.x) / kColumns < p.rows) {
        residual = load_fresh_float(p.residual + out_at);
    }
    const __half* x = static_cast<const __half*>(p.x);
    int stride = p.k;
    if constexpr (kNorm) {
        normalise_rows<QN>(rows, static_cast<const float*>(p.x), gain, shift, p.rows, p.k);
        __syncthreads();
        x = rows;
        stride = p.k + 8;
    }
    // Activations of a chunk of steps are all asked for before the first product needs one.
    constexpr int MB = (RB + 1) / 2;
    constexpr int kRoom = RB == 1 ? 12 : RB == 2 ? 6 : 2;          // steps' worth of registers
    constexpr int kChunk = kSteps * S::kPieces <= kRoom ? kSteps : (kRoom + S::kPieces - 1) / S::kPieces;
    float acc[MB][NT][4] = {};
#pragma unroll
    for (int from = 0; from < kSteps; from += kChunk) {
        if (from >= mine) {
            break;
        }
        uint4 values[kChunk][RB][S::kPieces];
#pragma unroll
        for (int j = 0; j < kChunk; ++j) {
            const int step = min(from + j, mine - 1);
#pragma unroll
            for (int block = 0; block < RB; ++block) {
                // (Rows past the last one repeat it: an MMA's rows do not meet, and theirs go
                // nowhere. A load without a condition costs no branch.)
                const int row = min(8 * block + g, p.rows - 1);
                const __half* at = x + static_cast<size_t>(row) * stride + (begin + step) * S::kStepK +
                                   t * S::kValues;
#pragma unroll
                for (int piece = 0; piece < S::kPieces; ++piece) {
                    values[j][block][piece] = kNorm ? *reinterpret_cast<const uint4*>(at + 8 * piece)
                                                    : load_fresh(at + 8 * piece);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < kChunk; ++j) {
            if (from + j < kSteps && from + j < mine) {
                multiply<W, RB, NT>(acc, raw[from + j < kSteps ? from + j : 0],
                                    [&](int block, int piece) { return values[j][block][piece]; });
            }
        }
    }
    if (kNorm && RB == 8) {
        __syncthreads();   // the rows' place is free
    }
#pragma unroll
    for (int m = 0; m < MB; ++m) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
            for (int i = 0; i < (RB == 1 ? 2 : 4); ++i) {
                sums[warp][16 * m + 8 * (i / 2) + g][8 * nt + 2 * t + i % 2] = acc[m][nt][i];
            }
        }
    }
    __syncthreads();
    // kThreads is a multiple of kColumns: a thread keeps its feature from row to row.
    for (int row = threadIdx.x / kColumns; row < p.rows; row += kThreads / kColumns) {
        float of_warp[kWarps];
#pragma unroll
        for (int other = 0; other < kWarps; ++other) {
            of_warp[other] = sums[other][row][threadIdx.x % kColumns];
        }
        float v = add_pairwise(of_warp);
        if (sizeof(W) == 1) {
            v *= scale;
        }
        v += bias;
        const size_t at = static_cast<size_t>(row) * p.n + feature;
        if constexpr (A == Act::kResidual) {
            static_cast<float*>(p.out)[at] = (at == out_at ? residual : load_fresh_float(p.residual + at)) + v;
        } else if constexpr (A == Act::kGelu) {
            static_cast<__half*>(p.out)[at] = __float2half_rn(gelu_tanh(v));
        } else {
            static_cast<__half*>(p.out)[at] = __float2half_rn(v);
        }
    }
}

// ---- final LayerNorm, output layer and greedy choice ---------------------------------------------
//
// The one kernel of a step whose weights are many (77 MB in FP16): two CTAs per SM stream
// them, a warp per eight features, the next twelve steps' weights on their way while twelve
// are used (eight with more than 16 rows, whose sums need the registers: 64 rows of 768, FP16,
// 872 -> 852 us a step). Every lane remembers the largest logit it saw; a sequence's best candidates meet
// in a 64-bit maximum of (ordered logit, inverted index), and the last CTA writes the tokens,
// advances the position and leaves the scratch as it found it.

struct HeadArgs {
    float* logits;
    const void* w;
    const float* scale;
    const float* x;
    const float* gain;
    const float* shift;
    unsigned long long* best;
    unsigned* ticket;
    uint16_t* next;
    int* position;
    int rows, n, k, vocab, advance;
};

__device__ __forceinline__ unsigned long long candidate(float value, int index) {
    const unsigned bits = __float_as_uint(value + 0.0f);   // -0 counts as +0
    const unsigned ordered = (bits & 0x80000000u) != 0 ? ~bits : bits | 0x80000000u;
    return (static_cast<unsigned long long>(ordered) << 32) | (0xffffffffu - static_cast<unsigned>(index));
}

template <typename W, int RB, int QN>
__global__ void __launch_bounds__(kThreads, 2) fb_decode_head(const HeadArgs p) {
    using S = Step<W>;
    constexpr int MB = (RB + 1) / 2;
    constexpr int kHalves = RB == 1 ? 1 : 2;
    constexpr int kAhead = (RB < 4 ? 12 : 8) / S::kPieces;   // steps per batch of loads
    extern __shared__ __align__(16) unsigned char decode_smem[];
    __shared__ unsigned long long chosen[kWarps][8 * RB];
    __shared__ bool last_cta;
    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    const int g = lane / 4;
    const int t = lane % 4;
    const int steps = p.k / S::kStepK;
    const int batches = (steps + kAhead - 1) / kAhead;
    const int tiles = (p.n + 7) / 8;
    const int stride_tiles = gridDim.x * kWarps;
    auto load = [&](uint4 (&raw)[kAhead], int tile, int batch) {
        const W* row = static_cast<const W*>(p.w) +
                       static_cast<size_t>(min(8 * tile + g, p.n - 1)) * p.k + t * S::kValues;
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
            const int step = batch * kAhead + j;
            raw[j] = make_uint4(0u, 0u, 0u, 0u);
            if (tile < tiles && step < steps) {
                raw[j] = load_streaming(row + step * S::kStepK);
            }
        }
    };
    int tile = blockIdx.x * kWarps + warp;
    int batch = 0;
    uint4 raw[kAhead];
    load(raw, tile, batch);
    float* gain = reinterpret_cast<float*>(decode_smem);
    float* shift = gain + p.k;
    __half* rows = reinterpret_cast<__half*>(shift + p.k);
    for (int i = threadIdx.x; i < p.k / 4; i += kThreads) {
        reinterpret_cast<float4*>(gain)[i] = reinterpret_cast<const float4*>(p.gain)[i];
        reinterpret_cast<float4*>(shift)[i] = reinterpret_cast<const float4*>(p.shift)[i];
    }
    __syncthreads();
    fb::dependency_wait();
    fb::dependency_release();
    normalise_rows<QN>(rows, p.x, gain, shift, p.rows, p.k);
    __syncthreads();
    float best_value[MB][2];
    int best_index[MB][2];
#pragma unroll
    for (int m = 0; m < MB; ++m) {
        best_value[m][0] = best_value[m][1] = -INFINITY;
        best_index[m][0] = best_index[m][1] = 0;
    }
    float acc[MB][1][4] = {};
    while (tile < tiles) {
        const bool done = batch + 1 == batches;
        const int next_tile = done ? tile + stride_tiles : tile;
        const int next_batch = done ? 0 : batch + 1;
        uint4 ahead[kAhead];
        load(ahead, next_tile, next_batch);
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
            const int step = batch * kAhead + j;
            if (step < steps) {
                const __half* at = rows + step * S::kStepK + t * S::kValues;
                const uint4 one[1] = {raw[j]};
                multiply<W, RB, 1>(acc, one, [&](int block, int piece) {
                    return *reinterpret_cast<const uint4*>(at + min(8 * block + g, p.rows - 1) * (p.k + 8) +
                                                           8 * piece);
                });
            }
        }
        if (done) {
            const int column = 8 * tile + 2 * t;    // n is a multiple of 8
            float s0 = 1.0f;
            float s1 = 1.0f;
            if (sizeof(W) == 1) {
                s0 = p.scale[column];
                s1 = p.scale[column + 1];
            }
#pragma unroll
            for (int m = 0; m < MB; ++m) {
#pragma unroll
                for (int half = 0; half < kHalves; ++half) {
                    const int row = 16 * m + 8 * half + g;
                    const float v0 = acc[m][0][2 * half] * s0;
                    const float v1 = acc[m][0][2 * half + 1] * s1;
                    if (row < p.rows) {
                        *reinterpret_cast<float2*>(p.logits + static_cast<size_t>(row) * p.n + column) =
                            make_float2(v0, v1);
                    }
                    if (column < p.vocab && v0 > best_value[m][half]) {
                        best_value[m][half] = v0;
                        best_index[m][half] = column;
                    }
                    if (column + 1 < p.vocab && v1 > best_value[m][half]) {
                        best_value[m][half] = v1;
                        best_index[m][half] = column + 1;
                    }
                    acc[m][0][2 * half] = 0.0f;
                    acc[m][0][2 * half + 1] = 0.0f;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < kAhead; ++j) {
            raw[j] = ahead[j];
        }
        tile = next_tile;
        batch = next_batch;
    }
    // The lowest index of the largest logit: over the row's four lanes, the warps, the CTAs.
#pragma unroll
    for (int m = 0; m < MB; ++m) {
#pragma unroll
        for (int half = 0; half < kHalves; ++half) {
            unsigned long long key = candidate(best_value[m][half], best_index[m][half]);
#pragma unroll
            for (int off = 1; off < 4; off <<= 1) {
                const unsigned long long other = __shfl_xor_sync(fb::kFullMask, key, off);
                key = other > key ? other : key;
            }
            if (t == 0) {
                chosen[warp][16 * m + 8 * half + g] = key;
            }
        }
    }
    __syncthreads();
    for (int row = threadIdx.x; row < p.rows; row += kThreads) {
        unsigned long long key = chosen[0][row];
        for (int w2 = 1; w2 < kWarps; ++w2) {
            key = chosen[w2][row] > key ? chosen[w2][row] : key;
        }
        atomicMax(&p.best[row], key);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        last_cta = atomicAdd(p.ticket, 1u) + 1 == gridDim.x;
    }
    __syncthreads();
    if (!last_cta) {
        return;
    }
    __threadfence();
    for (int row = threadIdx.x; row < p.rows; row += kThreads) {
        const unsigned long long key = atomicExch(&p.best[row], 0ull);
        p.next[row] = static_cast<uint16_t>(0xffffffffu - static_cast<unsigned>(key));
    }
    if (threadIdx.x == 0) {
        *p.ticket = 0;
        *p.position += p.advance;
    }
}

// ---- decode-side element kernels ------------------------------------------------------------------

// x[b, :] = wte[tokens[b], :] + wpe[position, :] for one new token per sequence.
__global__ void __launch_bounds__(256)
    fb_decode_embed(float* __restrict__ x, const uint16_t* __restrict__ tokens,
                    const float* __restrict__ wte, const float* __restrict__ wpe,
                    const int* __restrict__ position, int width, int vocab_rows) {
    const int b = blockIdx.x;
    const int token = min(static_cast<int>(tokens[b]), vocab_rows - 1);
    const int pos = *position;
    for (int c = threadIdx.x; c < width; c += blockDim.x) {
        x[static_cast<size_t>(b) * width + c] =
            wte[static_cast<size_t>(token) * width + c] + wpe[static_cast<size_t>(pos) * width + c];
    }
}

// Prefill: copies the keys and values of `count` consecutive positions per sequence from
// packed qkv rows [sequences * count, 3 width] into the cache, starting at position `first`.
__global__ void __launch_bounds__(256)
    fb_cache_store(__half* __restrict__ cache_k, __half* __restrict__ cache_v,
                   const __half* __restrict__ qkv, int first, int count, int heads,
                   int max_length) {
    fb::dependency_wait();
    fb::dependency_release();
    qkv = fb::after_wait(qkv);
    const int width = heads * kHeadWidth;
    const int row = blockIdx.x;            // sequence * count + offset
    const int sequence = row / count;
    const int t = first + row % count;
    const uint4* src = reinterpret_cast<const uint4*>(qkv + static_cast<size_t>(row) * 3 * width);
    const int pieces = width / 8;          // 16-byte pieces per K (or V) row
    for (int i = threadIdx.x; i < 2 * pieces; i += blockDim.x) {
        const int which = i / pieces;      // 0: K, 1: V
        const int piece = i % pieces;
        const int head = piece / (kHeadWidth / 8);
        const int inner = piece % (kHeadWidth / 8);
        __half* dst = (which == 0 ? cache_k : cache_v) +
                      ((static_cast<size_t>(sequence) * heads + head) * max_length + t) * kHeadWidth;
        reinterpret_cast<uint4*>(dst)[inner] = src[(1 + which) * pieces + piece];
    }
}

// One query per (sequence, head) against the cache's positions 0 .. *position, a CTA each. A
// warp takes 16 positions at a time, the CTA 256.
//   scores   K times q on mma.sync: the 16 positions are A's rows, q is column 0 of B (the
//            other seven are zeros). As in the linear layers a lane's 16 contiguous bytes of
//            a key are the k positions it holds; lane 4g gets positions g and g + 8. (With
//            FP32 FMAs on unpacked halves the conversions alone made this kernel issue-bound:
//            1,800 clocks per 256 positions.)
//   values   in FP32: eight lanes per position, 16 bytes each, probabilities as FP32 numbers
//            passed round by shuffles.
// A warp keeps one running maximum. Before it waits for the new token's qkv row, a thread
// copies its share of up to 512 older positions into its own slots of shared memory (which
// cost the neighbouring kernels no registers). The warps' (maximum, sum, weighted values)
// meet at the end. The new token's own key and value come from its row, and are stored in the
// cache for the steps to come (nothing else reads that position during this launch).
// (A cluster of up to eight CTAs per head was tried: its two barriers cost 1,900 clocks, more
// than eight times the positions do.)
constexpr int kAttentionThreads = 512;
constexpr int kAttentionWarps = kAttentionThreads / 32;
constexpr int kBatchPositions = 16 * kAttentionWarps;
constexpr int kMostStaged = 2;         // batches in shared memory

constexpr int attention_bytes(int batches) { return batches * kBatchPositions * 2 * kHeadWidth * 2; }

// The weight of a set of positions whose largest score is m (-inf: no positions).
__device__ __forceinline__ float merge_weight(float m, float top) {
    return m == -INFINITY ? 0.0f : exp2f(m - top);
}

// A thread's share of 16 positions: of positions g and g + 8, pieces t and t + 4 of the key
// (i = 0..3: position half i / 2, piece half i % 2); of positions 4 i + lane / 8, piece
// lane % 8 of the value.
__device__ __forceinline__ int key_position(int lane, int i) { return lane / 4 + 8 * (i / 2); }
__device__ __forceinline__ int key_piece(int lane, int i) { return lane % 4 + 4 * (i % 2); }

__global__ void __launch_bounds__(kAttentionThreads)
    fb_decode_attention(__half* out, const __half* qkv, __half* cache_k, __half* cache_v,
                        const int* position, int heads, int max_length, int staged, float scale) {
    extern __shared__ __align__(16) unsigned char attention_smem[];
    __shared__ float partial[kAttentionWarps][kHeadWidth];
    __shared__ float partial_m[kAttentionWarps];
    __shared__ float partial_l[kAttentionWarps];
    static_assert(kAttentionWarps == 16, "half a warp holds the warps' maxima");
    const int head = blockIdx.x % heads;
    const int sequence = blockIdx.x / heads;
    const int width = heads * kHeadWidth;
    const int tid = threadIdx.x;
    const int lane = tid % 32;
    const int warp = tid / 32;
    // The position and every older row were written before this step's first kernel began.
    const int newest = *position;
    const size_t base = (static_cast<size_t>(sequence) * heads + head) * max_length * kHeadWidth;
    const uint4* keys = reinterpret_cast<const uint4*>(cache_k + base);
    const uint4* values = reinterpret_cast<const uint4*>(cache_v + base);
    uint4* slots = reinterpret_cast<uint4*>(attention_smem) + tid;   // [batch][K 0-3, V 0-3][thread]
    const uint32_t slots_at = static_cast<uint32_t>(__cvta_generic_to_shared(slots));
    for (int batch = 0; batch < staged; ++batch) {
        const int first = batch * kBatchPositions + 16 * warp;
        if (first >= newest) {
            break;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k_at = first + key_position(lane, i);
            const int v_at = first + 4 * i + lane / 8;
            const uint32_t dst = slots_at + (batch * 8 + i) * (kAttentionThreads * 16);
            if (k_at < newest) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst),
                             "l"(keys + static_cast<size_t>(k_at) * (kHeadWidth / 8) + key_piece(lane, i))
                             : "memory");
            }
            if (v_at < newest) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                 dst + 4 * kAttentionThreads * 16),
                             "l"(values + static_cast<size_t>(v_at) * (kHeadWidth / 8) + lane % 8)
                             : "memory");
            }
        }
    }
    fb::dependency_wait();
    fb::dependency_release();
    const uint4* row = reinterpret_cast<const uint4*>(qkv + static_cast<size_t>(sequence) * 3 * width +
                                                      head * kHeadWidth);
    // B's column 0 (lanes 0-3): this lane's pieces of q.
    uint4 q0 = load_fresh(row + lane % 4);
    uint4 q1 = load_fresh(row + lane % 4 + 4);
    uint4 new_q = make_uint4(0u, 0u, 0u, 0u);
    uint4 new_k = new_q;
    uint4 new_v = new_q;
    if (warp == 0) {
        new_q = load_fresh(row + lane % 8);
        new_k = load_fresh(row + width / 8 + lane % 8);
        new_v = load_fresh(row + 2 * (width / 8) + lane % 8);
    }
    if (lane >= 4) {
        q0 = q1 = make_uint4(0u, 0u, 0u, 0u);
    }
    const float to_base2 = scale * kLog2e;
    float m = -INFINITY;
    float l = 0.0f;          // lanes 4g: over their own positions
    float acc[8] = {};       // this lane's positions, columns 8 (lane % 8) ...
    asm volatile("cp.async.wait_all;" ::: "memory");   // (a thread reads its own slots only)
    for (int batch = 0; batch * kBatchPositions + 16 * warp < newest; ++batch) {
        const int first = batch * kBatchPositions + 16 * warp;
        uint4 k[4];
        uint4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k_at = first + key_position(lane, i);
            const int v_at = first + 4 * i + lane / 8;
            k[i] = v[i] = make_uint4(0u, 0u, 0u, 0u);
            if (batch < staged) {
                const uint4* slot = slots + (batch * 8 + i) * kAttentionThreads;
                if (k_at < newest) {
                    k[i] = slot[0];
                }
                if (v_at < newest) {
                    v[i] = slot[4 * kAttentionThreads];
                }
            } else {
                if (k_at < newest) {
                    k[i] = load_streaming(keys + static_cast<size_t>(k_at) * (kHeadWidth / 8) +
                                          key_piece(lane, i));
                }
                if (v_at < newest) {
                    v[i] = load_streaming(values + static_cast<size_t>(v_at) * (kHeadWidth / 8) + lane % 8);
                }
            }
        }
        float s0;
        float s1;
        {
            float a[4];
            float b[4];
            mma_16x8x16(a, k[0].x, k[2].x, k[0].y, k[2].y, q0.x, q0.y);
            mma_16x8x16(b, k[0].z, k[2].z, k[0].w, k[2].w, q0.z, q0.w);
            s0 = a[0] + b[0];
            s1 = a[2] + b[2];
            mma_16x8x16(a, k[1].x, k[3].x, k[1].y, k[3].y, q1.x, q1.y);
            mma_16x8x16(b, k[1].z, k[3].z, k[1].w, k[3].w, q1.z, q1.w);
            s0 += a[0] + b[0];
            s1 += a[2] + b[2];
        }
        // Positions g and g + 8, in lanes 4g (column 0).
        const bool holds = lane % 4 == 0;
        s0 = holds && first + lane / 4 < newest ? s0 * to_base2 : -INFINITY;
        s1 = holds && first + lane / 4 + 8 < newest ? s1 * to_base2 : -INFINITY;
        float top = fmaxf(s0, s1);
        top = fmaxf(top, __shfl_xor_sync(fb::kFullMask, top, 4));
        top = fmaxf(top, __shfl_xor_sync(fb::kFullMask, top, 8));
        top = fmaxf(top, __shfl_xor_sync(fb::kFullMask, top, 16));
        top = fmaxf(m, __shfl_sync(fb::kFullMask, top, 0));
        const float keep = merge_weight(m, top);
        m = top;
        s0 = s0 == -INFINITY ? 0.0f : exp2f(s0 - m);
        s1 = s1 == -INFINITY ? 0.0f : exp2f(s1 - m);
        l = l * keep + (s0 + s1);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            acc[j] *= keep;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            // Position 4 i + lane / 8: half i / 2, g = 4 (i % 2) + lane / 8, in lane 4 g.
            const float p = __shfl_sync(fb::kFullMask, i < 2 ? s0 : s1, 16 * (i % 2) + lane / 8 * 4);
            float vv[8];
            fb::unpack8(vv, v[i]);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                acc[j] = fmaf(p, vv[j], acc[j]);
            }
        }
    }
    if (warp == 0) {
        float qv[8];
        float kv[8];
        float vv[8];
        fb::unpack8(qv, new_q);
        fb::unpack8(kv, new_k);
        fb::unpack8(vv, new_v);
        float s = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            s = fmaf(kv[j], qv[j], s);
        }
        s += __shfl_xor_sync(fb::kFullMask, s, 1);
        s += __shfl_xor_sync(fb::kFullMask, s, 2);
        s += __shfl_xor_sync(fb::kFullMask, s, 4);
        s *= to_base2;
        const float top = fmaxf(m, s);
        const float keep = merge_weight(m, top);
        const float p = s == -INFINITY ? 0.0f : exp2f(s - top);
        m = top;
        l = l * keep + (lane == 0 ? p : 0.0f);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            acc[j] = acc[j] * keep + (lane < 8 ? p * vv[j] : 0.0f);
        }
        if (lane < 8) {
            reinterpret_cast<uint4*>(cache_k + base + static_cast<size_t>(newest) * kHeadWidth)[lane] = new_k;
            reinterpret_cast<uint4*>(cache_v + base + static_cast<size_t>(newest) * kHeadWidth)[lane] = new_v;
        }
    }
    // The warp: l over lanes 4g, the values over lanes with the same columns.
    l += __shfl_xor_sync(fb::kFullMask, l, 4);
#pragma unroll
    for (int off = 8; off < 32; off <<= 1) {
        l += __shfl_xor_sync(fb::kFullMask, l, off);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            acc[j] += __shfl_xor_sync(fb::kFullMask, acc[j], off);
        }
    }
    if (lane < 8) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            partial[warp][8 * lane + j] = acc[j];
        }
        if (lane == 0) {
            partial_m[warp] = m;
            partial_l[warp] = l;
        }
    }
    __syncthreads();
    if (tid < kHeadWidth) {
        // Lane w (and w + 16) weighs warp w's share; the weights go round by shuffles.
        const float mine = partial_m[lane % 16];
        float top = mine;
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) {
            top = fmaxf(top, __shfl_xor_sync(fb::kFullMask, top, off));
        }
        const float weight = merge_weight(mine, top);
        float sum = weight * partial_l[lane % 16];
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) {
            sum += __shfl_xor_sync(fb::kFullMask, sum, off);
        }
        float even = 0.0f;
        float odd = 0.0f;
#pragma unroll
        for (int w = 0; w < kAttentionWarps; w += 2) {
            even = fmaf(__shfl_sync(fb::kFullMask, weight, w), partial[w][tid], even);
            odd = fmaf(__shfl_sync(fb::kFullMask, weight, w + 1), partial[w + 1][tid], odd);
        }
        out[static_cast<size_t>(sequence) * width + head * kHeadWidth + tid] =
            __float2half_rn((even + odd) / sum);
    }
}

// The last position's row of each sequence, [sequences * length, width] -> [sequences, width], of the
// residual stream (FP32) and of the attention output (FP16).
__global__ void __launch_bounds__(256)
    fb_take_last_rows(float* __restrict__ out, __half* __restrict__ attn_out, const float* __restrict__ x,
                      const __half* __restrict__ attn, int length, int width) {
    const int b = blockIdx.x;
    const size_t from = (static_cast<size_t>(b) * length + length - 1) * width;
    for (int c = threadIdx.x; c < width; c += blockDim.x) {
        out[static_cast<size_t>(b) * width + c] = x[from + c];
        attn_out[static_cast<size_t>(b) * width + c] = attn[from + c];
    }
}

}  // namespace

struct flint_b200_generator {
    const flint_gpt2* model = nullptr;
    size_t sequences = 0, max_length = 0;
    size_t layers = 0, heads = 0, width = 0, vocab = 0, padded_vocab = 0;
    bool int8 = false;
    std::vector<Layer> blocks;
    Matrix head;                       // the tied output layer (wte)
    const float *wte = nullptr, *wpe = nullptr, *lnf_w = nullptr, *lnf_b = nullptr;
    size_t host_position = 0;          // tokens held per sequence (mirror of *position)
    // device
    int* position = nullptr;
    __half* cache = nullptr;           // [layers][2][sequences][heads][max_length][64]
    float *x_a = nullptr, *x_b = nullptr, *last = nullptr;
    __half *h = nullptr, *qkv = nullptr, *attn = nullptr, *act = nullptr, *pre = nullptr;
    float *mean = nullptr, *rstd = nullptr, *lse = nullptr, *logits = nullptr;
    uint16_t* next = nullptr;
    unsigned long long* best = nullptr;  // greedy choice in progress, per sequence
    unsigned* ticket = nullptr;
    __half* dequantized = nullptr;     // int8: a layer's matrices in FP16
    std::vector<void*> owned;
    cudaGraphExec_t step_graph = nullptr;
    const void* graph_tokens = nullptr;
    void* graph_next = nullptr;

    ~flint_b200_generator() {
        if (step_graph != nullptr) {
            cudaGraphExecDestroy(step_graph);
        }
        for (void* p : owned) {
            cudaFree(p);
        }
        cudaGetLastError();
    }
    size_t cache_stride() const { return sequences * heads * max_length * kHeadWidth; }
    __half* keys(size_t layer) const { return cache + (2 * layer) * cache_stride(); }
    __half* values(size_t layer) const { return cache + (2 * layer + 1) * cache_stride(); }
};

namespace {

template <typename T>
flint_status allocate(flint_b200_generator& g, T** out, size_t count) {
    void* p = nullptr;
    FB_CUDA(cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T)));
    g.owned.push_back(p);
    *out = static_cast<T*>(p);
    return FLINT_OK;
}

Matrix matrix_of(const fb::Tensor* weight, const fb::Tensor* bias) {
    Matrix m;
    m.half = static_cast<const __half*>(weight->half);
    m.bias = bias == nullptr ? nullptr : static_cast<const float*>(bias->data);
    m.n = weight->rows;
    m.k = weight->cols;
    return m;
}

flint_status quantize(flint_b200_generator& g, Matrix& m, cudaStream_t stream) {
    if (m.q == nullptr) {
        FB_TRY(allocate(g, &m.q, m.n * m.k));
        FB_TRY(allocate(g, &m.scale, m.n));
    }
    fb_quantize_rows<<<static_cast<unsigned>((m.n + 7) / 8), 256, 0, stream>>>(m.q, m.scale, m.half,
                                                                                m.n, m.k);
    FB_CUDA(fb::after_launch());
    return FLINT_OK;
}

template <typename W, Act A, bool kNorm, int RB, int NT, int kSteps, int QN>
flint_status launch_linear(const LinearArgs& args, cudaStream_t stream) {
    auto kernel = fb_decode_linear<W, A, kNorm, RB, NT, kSteps, QN>;
    const int smem = linear_bytes(kNorm, RB, NT, args.rows, args.k);
    static std::atomic<bool> configured[64] = {};
    FB_CUDA(fb::allow_shared_memory(kernel, linear_bytes(kNorm, RB, NT, 8 * RB, 128 * QN), configured));
    FB_CUDA(fb::launch_dependent(kernel, dim3(static_cast<unsigned>(args.n / (8 * NT))), dim3(kThreads),
                                 static_cast<size_t>(smem), stream, args));
    return FLINT_OK;
}

// The step counts and register rows follow from k: the layers' k is the width (at most 768,
// or at most 1,536) or, behind the GELU, four times that. A normalising kernel takes 16
// features per CTA (its CTAs each normalise every row, so there should not be many), the
// others 8 (so that 768 of them spread over 96 CTAs).
template <typename W, Act A, int RB>
flint_status linear_for(const LinearArgs& args, cudaStream_t stream) {
    constexpr bool kNorm = A != Act::kResidual;
    constexpr int kPer = Step<W>::kPieces;   // int8 takes twice the k per step
    if constexpr (kNorm) {
        return args.k <= 768 ? launch_linear<W, A, true, RB, 2, (3 + kPer - 1) / kPer, 6>(args, stream)
                             : launch_linear<W, A, true, RB, 2, 6 / kPer, 12>(args, stream);
    } else {
        if (args.k <= 768) {
            return launch_linear<W, A, false, RB, 1, (3 + kPer - 1) / kPer, 1>(args, stream);
        }
        if (args.k <= 3072) {
            return launch_linear<W, A, false, RB, 1, 12 / kPer, 1>(args, stream);
        }
        return launch_linear<W, A, false, RB, 1, 24 / kPer, 1>(args, stream);
    }
}

template <typename W, Act A>
flint_status linear_rows(const LinearArgs& args, cudaStream_t stream) {
    return args.rows <= 8    ? linear_for<W, A, 1>(args, stream)
           : args.rows <= 16 ? linear_for<W, A, 2>(args, stream)
           : args.rows <= 32 ? linear_for<W, A, 4>(args, stream)
                             : linear_for<W, A, 8>(args, stream);
}

// One decode linear layer. kNone and kGelu normalise x (FP32 rows) first.
template <Act A>
flint_status decode_linear(const flint_b200_generator& g, const Matrix& m, void* out, const void* x,
                           const float* gain, const float* shift, const float* residual,
                           cudaStream_t stream) {
    const LinearArgs args{out,  g.int8 ? static_cast<const void*>(m.q) : m.half,
                          m.scale, m.bias, x, gain, shift, residual,
                          static_cast<int>(g.sequences), static_cast<int>(m.n), static_cast<int>(m.k)};
    return g.int8 ? linear_rows<int8_t, A>(args, stream) : linear_rows<__half, A>(args, stream);
}

template <typename W, int RB, int QN>
flint_status launch_head(const HeadArgs& args, cudaStream_t stream) {
    auto kernel = fb_decode_head<W, RB, QN>;
    static std::atomic<bool> configured[64] = {};
    FB_CUDA(fb::allow_shared_memory(kernel, norm_bytes(8 * RB, 128 * QN), configured));
    int sms = 0;
    FB_CUDA(fb::sm_count(&sms));
    const int tiles = (args.n + 8 * kWarps - 1) / (8 * kWarps);
    FB_CUDA(fb::launch_dependent(kernel, dim3(static_cast<unsigned>(std::min(2 * sms, tiles))),
                                 dim3(kThreads), static_cast<size_t>(norm_bytes(args.rows, args.k)),
                                 stream, args));
    return FLINT_OK;
}

template <typename W, int RB>
flint_status head_width(const HeadArgs& args, cudaStream_t stream) {
    return args.k <= 768 ? launch_head<W, RB, 6>(args, stream) : launch_head<W, RB, 12>(args, stream);
}

template <typename W>
flint_status head_for(const HeadArgs& args, cudaStream_t stream) {
    return args.rows <= 8    ? head_width<W, 1>(args, stream)
           : args.rows <= 16 ? head_width<W, 2>(args, stream)
           : args.rows <= 32 ? head_width<W, 4>(args, stream)
                             : head_width<W, 8>(args, stream);
}

// The FP16 weights of a layer that the tensor-core GEMMs read: the model's copies, or the int8
// weights expanded into the scratch memory (of the last layer only the first matrix: run_last_rows reads
// the others as they are. Two layers of 768 columns, 4 x 256 tokens: 128 us with all, 122; one of 1,536,
// 64 x 8: 190 and 174).
struct DenseLayer {
    const __half *attn, *proj, *fc, *fcproj;
};

flint_status dense_weights(const flint_b200_generator& g, size_t layer, DenseLayer* dense, cudaStream_t stream) {
    const Layer& l = g.blocks[layer];
    *dense = DenseLayer{l.attn.half, l.proj.half, l.fc.half, l.fcproj.half};
    if (!g.int8) {
        return FLINT_OK;
    }
    const Matrix* matrices[DequantizeArgs::kMatrices] = {&l.attn, &l.proj, &l.fc, &l.fcproj};
    const __half** out[DequantizeArgs::kMatrices] = {&dense->attn, &dense->proj, &dense->fc, &dense->fcproj};
    DequantizeArgs args;
    args.out = g.dequantized;
    unsigned pieces = 0;
    const int wanted = layer + 1 < g.layers ? DequantizeArgs::kMatrices : 1;
    for (int i = 0; i < DequantizeArgs::kMatrices; ++i) {
        if (i >= wanted) {      // none of it: the matrix ends where it begins
            *out[i] = nullptr;
            args.q[i] = nullptr;
            args.scale[i] = nullptr;
            args.cols[i] = 16;
            args.end[i] = pieces;
            continue;
        }
        *out[i] = g.dequantized + static_cast<size_t>(pieces) * 16;
        args.q[i] = matrices[i]->q;
        args.scale[i] = matrices[i]->scale;
        args.cols[i] = static_cast<unsigned>(matrices[i]->k);
        pieces += static_cast<unsigned>(matrices[i]->n * matrices[i]->k / 16);
        args.end[i] = pieces;
    }
    FB_CUDA(fb::launch_dependent(fb_dequantize_layer, dim3(std::min((pieces + 255) / 256, 1184u)), dim3(256), 0,
                                 stream, args));
    return FLINT_OK;
}

// y = act(x w^T + bias) for a prompt's rows. kNone/kGelu: FP16 out; kResidual: FP32 out =
// residual + (x w^T + bias).
template <Act A>
flint_status linear(const flint_b200_generator& g, const Matrix& m, const __half* w, void* out, const __half* x,
                    const float* residual, size_t rows, cudaStream_t stream) {
    if constexpr (A == Act::kNone) {
        FB_CUDA(fb::gemm_nt(fb::Epilogue::kBias, out, nullptr, x, w, m.bias, nullptr, rows, m.n, m.k,
                            stream, true));
    } else if constexpr (A == Act::kGelu) {
        FB_CUDA(fb::gemm_nt(fb::Epilogue::kBiasGelu, out, g.pre, x, w, m.bias, nullptr, rows, m.n,
                            m.k, stream, true));
    } else {
        FB_CUDA(fb::gemm_nt(fb::Epilogue::kBiasResidual, out, nullptr, x, w, m.bias, residual, rows,
                            m.n, m.k, stream, true));
    }
    return FLINT_OK;
}

flint_status layernorm(const flint_b200_generator& g, const float* gain, const float* bias,
                       const float* x, size_t rows, cudaStream_t stream) {
    return flint_layernorm_forward(g.h, g.mean, g.rstd, x, gain, bias, rows, g.width, kEps, stream);
}

float attention_scale() { return 1.0f / std::sqrt(static_cast<float>(kHeadWidth)); }

// The transformer over a prompt of `count` positions per sequence, up to the last block's attention
// output: beyond that only the prompt's last position matters (see run_last_rows). The stream of
// rows is in x_a: every block but the last moves it to x_b and back.
flint_status run_prompt(flint_b200_generator& g, size_t count, cudaStream_t stream) {
    const size_t rows = g.sequences * count;
    for (size_t i = 0; i < g.layers; ++i) {
        const Layer& l = g.blocks[i];
        DenseLayer dense;
        // (Ahead of the LayerNorm: the GEMM behind it fetches weights before its wait, see common.h.)
        FB_TRY(dense_weights(g, i, &dense, stream));
        FB_TRY(layernorm(g, l.ln1_w, l.ln1_b, g.x_a, rows, stream));
        FB_TRY(linear<Act::kNone>(g, l.attn, dense.attn, g.qkv, g.h, nullptr, rows, stream));
        FB_CUDA(fb::launch_dependent(
            fb_cache_store, dim3(static_cast<unsigned>(rows)), dim3(256), 0, stream, g.keys(i), g.values(i),
            static_cast<const __half*>(g.qkv), static_cast<int>(g.host_position), static_cast<int>(count),
            static_cast<int>(g.heads), static_cast<int>(g.max_length)));
        const size_t w3 = 3 * g.width;
        auto view = [&](const void* base, size_t first, size_t row_width) {
            return fb::AttentionView{static_cast<const __half*>(base) + first,
                                     static_cast<long long>(row_width), kHeadWidth,
                                     static_cast<long long>(count * row_width)};
        };
        FB_CUDA(fb::attention_forward(view(g.attn, 0, g.width), g.lse, view(g.qkv, 0, w3),
                                      view(g.qkv, g.width, w3), view(g.qkv, 2 * g.width, w3),
                                      fb::AttentionShape{g.sequences, g.heads, count},
                                      attention_scale(), stream));
        if (i + 1 == g.layers) {
            break;
        }
        FB_TRY(linear<Act::kResidual>(g, l.proj, dense.proj, g.x_b, g.attn, g.x_a, rows, stream));
        FB_TRY(layernorm(g, l.ln2_w, l.ln2_b, g.x_b, rows, stream));
        FB_TRY(linear<Act::kGelu>(g, l.fc, dense.fc, g.act, g.h, nullptr, rows, stream));
        FB_TRY(linear<Act::kResidual>(g, l.fcproj, dense.fcproj, g.x_a, g.act, g.x_b, rows, stream));
    }
    return FLINT_OK;
}

// Whether a step's linear layers run on the prompt's GEMMs (FP16 weights only: int8 ones would be
// expanded on every step). The step's own kernels read every row in every CTA, which grows with
// rows times width and passes what 128-row tensor-core tiles waste at about 33 rows of 1,280, 41
// of 1,024 or 47 of 896; models up to 768 wide never get there. us per step of 12 layers, own
// kernels -> GEMMs: 33 x 1,280 1,298 -> 1,074, 33 x 1,536 1,463 -> 1,274, 48 x 1,024 1,059 -> 1,015,
// 64 x 896 1,170 -> 1,013, 64 x 1,536 2,127 -> 1,498; but 33 x 896 810 -> 848, 33 x 1,024 864 -> 908,
// 40 x 1,024 941 -> 959, 64 x 768 852 -> 886, 32 x 1,536 1,209 -> 1,251.
bool tensor_core_step(const flint_b200_generator& g) {
    return !g.int8 && g.sequences > 32 && g.width > 768 && g.sequences * g.width >= 42000;
}

// The rest of the last block for one row per sequence, on what a step would use: the residual stream in
// g.last, the attention output in g.h; the block's output in g.last. (For all rows of a 4 x 256
// prompt it took 32 us. FP16, 64 sequences of 8 tokens at 1,536 columns, one layer: 164 us with all 512
// rows on the GEMMs, 173 with the last 64 on the decode kernels, 131 with those on the GEMMs.)
flint_status run_last_rows(flint_b200_generator& g, cudaStream_t stream) {
    const Layer& l = g.blocks.back();
    if (tensor_core_step(g)) {
        const size_t rows = g.sequences;
        FB_TRY(linear<Act::kResidual>(g, l.proj, l.proj.half, g.x_b, g.h, g.last, rows, stream));
        FB_TRY(layernorm(g, l.ln2_w, l.ln2_b, g.x_b, rows, stream));
        FB_TRY(linear<Act::kGelu>(g, l.fc, l.fc.half, g.act, g.h, nullptr, rows, stream));
        return linear<Act::kResidual>(g, l.fcproj, l.fcproj.half, g.last, g.act, g.x_b, rows, stream);
    }
    FB_TRY(decode_linear<Act::kResidual>(g, l.proj, g.x_b, g.h, nullptr, nullptr, g.last, stream));
    FB_TRY(decode_linear<Act::kGelu>(g, l.fc, g.act, g.x_b, l.ln2_w, l.ln2_b, nullptr, stream));
    return decode_linear<Act::kResidual>(g, l.fcproj, g.last, g.act, nullptr, nullptr, g.x_b, stream);
}

// The transformer over one new position per sequence.
flint_status run_token(flint_b200_generator& g, cudaStream_t stream) {
    // Shared memory for as many positions as there can be, within what one CTA per SM may have,
    // or two where there are more CTAs than SMs.
    int sms = 0;
    FB_CUDA(fb::sm_count(&sms));
    const size_t pairs = g.sequences * g.heads;
    const size_t batches = std::min<size_t>(pairs <= static_cast<size_t>(sms) ? kMostStaged : 1,
                                            (g.max_length + kBatchPositions - 1) / kBatchPositions);
    static std::atomic<bool> configured[64] = {};
    FB_CUDA(fb::allow_shared_memory(fb_decode_attention, attention_bytes(kMostStaged), configured));
    const bool dense = tensor_core_step(g);
    const size_t rows = g.sequences;
    for (size_t i = 0; i < g.layers; ++i) {
        const Layer& l = g.blocks[i];
        if (dense) {
            FB_TRY(layernorm(g, l.ln1_w, l.ln1_b, g.x_a, rows, stream));
            FB_TRY(linear<Act::kNone>(g, l.attn, l.attn.half, g.qkv, g.h, nullptr, rows, stream));
        } else {
            FB_TRY(decode_linear<Act::kNone>(g, l.attn, g.qkv, g.x_a, l.ln1_w, l.ln1_b, nullptr, stream));
        }
        FB_CUDA(fb::launch_dependent(
            fb_decode_attention, dim3(static_cast<unsigned>(pairs)), dim3(kAttentionThreads),
            static_cast<size_t>(attention_bytes(static_cast<int>(batches))),
            stream, g.attn, g.qkv, g.keys(i), g.values(i), g.position, static_cast<int>(g.heads),
            static_cast<int>(g.max_length), static_cast<int>(batches), attention_scale()));
        if (dense) {
            FB_TRY(linear<Act::kResidual>(g, l.proj, l.proj.half, g.x_b, g.attn, g.x_a, rows, stream));
            FB_TRY(layernorm(g, l.ln2_w, l.ln2_b, g.x_b, rows, stream));
            FB_TRY(linear<Act::kGelu>(g, l.fc, l.fc.half, g.act, g.h, nullptr, rows, stream));
            FB_TRY(linear<Act::kResidual>(g, l.fcproj, l.fcproj.half, g.x_a, g.act, g.x_b, rows, stream));
        } else {
            FB_TRY(decode_linear<Act::kResidual>(g, l.proj, g.x_b, g.attn, nullptr, nullptr, g.x_a, stream));
            FB_TRY(decode_linear<Act::kGelu>(g, l.fc, g.act, g.x_b, l.ln2_w, l.ln2_b, nullptr, stream));
            FB_TRY(decode_linear<Act::kResidual>(g, l.fcproj, g.x_a, g.act, nullptr, nullptr, g.x_b, stream));
        }
    }
    return FLINT_OK;
}

// Final LayerNorm, output layer and greedy choice over the `sequences` rows at `x`; the
// position moves on by `advance`.
flint_status run_head(flint_b200_generator& g, const float* x, void* next_tokens, int advance,
                      cudaStream_t stream) {
    const HeadArgs args{g.logits, g.int8 ? static_cast<const void*>(g.head.q) : g.head.half,
                        g.head.scale, x, g.lnf_w, g.lnf_b, g.best, g.ticket,
                        next_tokens != nullptr ? static_cast<uint16_t*>(next_tokens) : g.next,
                        g.position, static_cast<int>(g.sequences), static_cast<int>(g.head.n),
                        static_cast<int>(g.head.k), static_cast<int>(g.vocab), advance};
    return g.int8 ? head_for<int8_t>(args, stream) : head_for<__half>(args, stream);
}

flint_status enqueue_step(flint_b200_generator& g, const void* tokens, void* next_tokens,
                          cudaStream_t stream) {
    // Launched the ordinary way: it begins when everything before the step has finished, and
    // so do the step's other kernels, which read weights and older cache rows ahead of time.
    fb_decode_embed<<<static_cast<unsigned>(g.sequences), 256, 0, stream>>>(
        g.x_a, static_cast<const uint16_t*>(tokens), g.wte, g.wpe, g.position,
        static_cast<int>(g.width), static_cast<int>(g.padded_vocab));
    FB_CUDA(fb::after_launch());
    FB_TRY(run_token(g, stream));
    return run_head(g, g.x_a, next_tokens, 1, stream);
}

flint_status build(flint_b200_generator& g, cudaStream_t stream) {
    const flint_gpt2& m = *g.model;
    const flint_gpt2_config& c = m.config;
    g.layers = c.layers;
    g.heads = c.heads;
    g.width = c.width;
    g.vocab = c.vocab;
    g.padded_vocab = c.padded_vocab;
    g.wte = static_cast<const float*>(m.wte->data);
    g.wpe = static_cast<const float*>(m.wpe->data);
    g.lnf_w = static_cast<const float*>(m.lnf_w->data);
    g.lnf_b = static_cast<const float*>(m.lnf_b->data);
    g.head = matrix_of(m.wte, nullptr);
    for (size_t i = 0; i < c.layers; ++i) {
        const fb::BlockWeights& w = m.weights[i];
        Layer l;
        l.ln1_w = static_cast<const float*>(w.ln1_w->data);
        l.ln1_b = static_cast<const float*>(w.ln1_b->data);
        l.ln2_w = static_cast<const float*>(w.ln2_w->data);
        l.ln2_b = static_cast<const float*>(w.ln2_b->data);
        l.attn = matrix_of(w.attn_w, w.attn_b);
        l.proj = matrix_of(w.proj_w, w.proj_b);
        l.fc = matrix_of(w.fc_w, w.fc_b);
        l.fcproj = matrix_of(w.fcproj_w, w.fcproj_b);
        g.blocks.push_back(l);
    }
    const size_t rows = g.sequences * g.max_length;
    const size_t w = g.width;
    FB_TRY(allocate(g, &g.position, 4));
    FB_CUDA(cudaMemsetAsync(g.position, 0, 16, stream));
    FB_TRY(allocate(g, &g.cache, 2 * g.layers * g.cache_stride()));
    FB_TRY(allocate(g, &g.x_a, rows * w));
    FB_TRY(allocate(g, &g.x_b, rows * w));
    FB_TRY(allocate(g, &g.last, g.sequences * w));
    FB_TRY(allocate(g, &g.h, rows * w));
    FB_TRY(allocate(g, &g.qkv, rows * 3 * w));
    FB_TRY(allocate(g, &g.attn, rows * w));
    FB_TRY(allocate(g, &g.act, rows * 4 * w));
    FB_TRY(allocate(g, &g.pre, rows * 4 * w));
    FB_TRY(allocate(g, &g.mean, rows));
    FB_TRY(allocate(g, &g.rstd, rows));
    FB_TRY(allocate(g, &g.lse, g.sequences * g.heads * g.max_length));
    FB_TRY(allocate(g, &g.logits, g.sequences * g.padded_vocab));
    FB_TRY(allocate(g, &g.next, g.sequences));
    FB_TRY(allocate(g, &g.best, g.sequences));
    FB_TRY(allocate(g, &g.ticket, 1));
    FB_CUDA(cudaMemsetAsync(g.best, 0, g.sequences * sizeof(*g.best), stream));
    FB_CUDA(cudaMemsetAsync(g.ticket, 0, sizeof(*g.ticket), stream));
    if (g.int8) {
        FB_TRY(allocate(g, &g.dequantized, 12 * w * w));
    }
    return FLINT_OK;
}

}  // namespace

extern "C" {

flint_status flint_b200_generator_create(const flint_gpt2* model, size_t sequences,
                                         size_t max_length, int int8_weights,
                                         flint_b200_generator** generator) {
    constexpr const char* name = "flint_b200_generator_create";
    if (generator == nullptr) {
        return fb::fail(kInvalid, "%s: generator is null", name);
    }
    *generator = nullptr;
    if (model == nullptr) {
        return fb::fail(kInvalid, "%s: model is null", name);
    }
    const flint_gpt2_config& c = model->config;
    if (c.width / c.heads != kHeadWidth || c.width % 128 != 0 || c.width > 1600) {
        return fb::fail(kInvalid, "%s: needs heads of width 64 and a width (%zu) that is a "
                        "multiple of 128 up to 1600", name, c.width);
    }
    if (model->tensors.empty() || model->wte->half == nullptr) {
        return fb::fail(kInvalid, "%s: the model has no FP16 weight copies", name);
    }
    if (sequences < 1 || sequences > 64) {
        return fb::fail(kInvalid, "%s: sequences (%zu) must be from 1 to 64", name, sequences);
    }
    if (max_length < 8 || max_length % 8 != 0 || max_length > c.block_size || max_length > 1024) {
        return fb::fail(kInvalid, "%s: max_length (%zu) must be a multiple of 8 from 8 to "
                        "min(block_size (%zu), 1024)", name, max_length, c.block_size);
    }
    std::unique_ptr<flint_b200_generator> g(new (std::nothrow) flint_b200_generator);
    if (!g) {
        return fb::fail(FLINT_ERROR_CUDA, "%s: out of host memory", name);
    }
    g->model = model;
    g->sequences = sequences;
    g->max_length = max_length;
    g->int8 = int8_weights != 0;
    try {
        FB_TRY(build(*g, nullptr));
        FB_TRY(flint_b200_generator_refresh(g.get(), nullptr));
    } catch (const std::bad_alloc&) {
        return fb::fail(FLINT_ERROR_CUDA, "%s: out of host memory", name);
    }
    FB_CUDA(cudaDeviceSynchronize());
    *generator = g.release();
    return FLINT_OK;
}

void flint_b200_generator_destroy(flint_b200_generator* generator) { delete generator; }

flint_status flint_b200_generator_refresh(flint_b200_generator* generator, flint_stream stream) {
    if (generator == nullptr) {
        return fb::fail(kInvalid, "flint_b200_generator_refresh: generator is null");
    }
    flint_b200_generator& g = *generator;
    if (g.int8) {
        for (Layer& l : g.blocks) {
            FB_TRY(quantize(g, l.attn, stream));
            FB_TRY(quantize(g, l.proj, stream));
            FB_TRY(quantize(g, l.fc, stream));
            FB_TRY(quantize(g, l.fcproj, stream));
        }
        FB_TRY(quantize(g, g.head, stream));
    }
    return FLINT_OK;
}

flint_status flint_b200_generator_prefill(flint_b200_generator* generator, const void* tokens,
                                          size_t length, flint_stream stream) {
    constexpr const char* name = "flint_b200_generator_prefill";
    if (generator == nullptr) {
        return fb::fail(kInvalid, "%s: generator is null", name);
    }
    flint_b200_generator& g = *generator;
    if (length < 8 || length % 8 != 0 || length > g.max_length) {
        return fb::fail(kInvalid, "%s: length (%zu) must be a multiple of 8 from 8 to max_length "
                        "(%zu)", name, length, g.max_length);
    }
    const size_t rows = g.sequences * length;
    const fb::Span spans[] = {{"tokens", tokens, rows * 2}};
    FB_TRY(fb::check_spans(name, spans, 0));
    g.host_position = 0;
    FB_CUDA(cudaMemsetAsync(g.position, 0, 4, stream));
    FB_TRY(flint_embedding_forward(g.x_a, tokens, g.wte, g.wpe, g.sequences, length, g.padded_vocab,
                                   g.width, stream));
    FB_TRY(run_prompt(g, length, stream));
    // Launched the ordinary way: the kernel behind it reads weights before its wait.
    fb_take_last_rows<<<static_cast<unsigned>(g.sequences), 256, 0, stream>>>(
        g.last, g.h, g.x_a, g.attn, static_cast<int>(length), static_cast<int>(g.width));
    FB_CUDA(fb::after_launch());
    FB_TRY(run_last_rows(g, stream));
    FB_TRY(run_head(g, g.last, nullptr, static_cast<int>(length), stream));
    g.host_position = length;
    return FLINT_OK;
}

flint_status flint_b200_generator_step(flint_b200_generator* generator, const void* tokens,
                                       void* next_tokens, int use_graph, flint_stream stream) {
    constexpr const char* name = "flint_b200_generator_step";
    if (generator == nullptr) {
        return fb::fail(kInvalid, "%s: generator is null", name);
    }
    flint_b200_generator& g = *generator;
    if (g.host_position >= g.max_length) {
        return fb::fail(kInvalid, "%s: the cache is full (%zu positions)", name, g.max_length);
    }
    const fb::Span spans[] = {{"tokens", tokens, g.sequences * 2}};
    FB_TRY(fb::check_spans(name, spans, 0));
    if (use_graph == 0) {
        FB_TRY(enqueue_step(g, tokens, next_tokens, stream));
        g.host_position += 1;
        return FLINT_OK;
    }
    // The step's launches depend on the position only through device memory, so one
    // captured graph serves every token as long as the caller's buffers stay the same.
    if (g.step_graph != nullptr && (g.graph_tokens != tokens || g.graph_next != next_tokens)) {
        cudaGraphExecDestroy(g.step_graph);
        g.step_graph = nullptr;
    }
    if (g.step_graph == nullptr) {
        cudaStream_t capture = nullptr;
        FB_CUDA(cudaStreamCreateWithFlags(&capture, cudaStreamNonBlocking));
        cudaGraph_t graph = nullptr;
        cudaError_t e = cudaStreamBeginCapture(capture, cudaStreamCaptureModeThreadLocal);
        flint_status status = FLINT_OK;
        if (e == cudaSuccess) {
            status = enqueue_step(g, tokens, next_tokens, capture);
            e = cudaStreamEndCapture(capture, &graph);
        }
        if (e == cudaSuccess && status == FLINT_OK) {
            e = cudaGraphInstantiate(&g.step_graph, graph, 0);
        }
        if (graph != nullptr) {
            cudaGraphDestroy(graph);
        }
        cudaStreamDestroy(capture);
        if (status != FLINT_OK) {
            return status;
        }
        FB_CUDA(e);
        g.graph_tokens = tokens;
        g.graph_next = next_tokens;
    }
    FB_CUDA(cudaGraphLaunch(g.step_graph, stream));
    g.host_position += 1;
    return FLINT_OK;
}

flint_status flint_b200_generator_logits(const flint_b200_generator* generator,
                                         const void** logits, size_t* position) {
    if (generator == nullptr) {
        return fb::fail(kInvalid, "flint_b200_generator_logits: generator is null");
    }
    if (logits != nullptr) {
        *logits = generator->logits;
    }
    if (position != nullptr) {
        *position = generator->host_position;
    }
    return FLINT_OK;
}

flint_status flint_b200_generator_bytes_per_step(const flint_b200_generator* generator,
                                                 size_t* weight_bytes, size_t* cache_bytes) {
    if (generator == nullptr) {
        return fb::fail(kInvalid, "flint_b200_generator_bytes_per_step: generator is null");
    }
    const flint_b200_generator& g = *generator;
    const size_t element = g.int8 ? 1 : 2;
    size_t weights = g.head.n * g.head.k * element;
    for (const Layer& l : g.blocks) {
        for (const Matrix* m : {&l.attn, &l.proj, &l.fc, &l.fcproj}) {
            weights += m->n * m->k * element;
        }
    }
    if (weight_bytes != nullptr) {
        *weight_bytes = weights;
    }
    if (cache_bytes != nullptr) {
        *cache_bytes = 2 * g.layers * g.sequences * g.heads * (g.host_position + 1) * kHeadWidth * 2;
    }
    return FLINT_OK;
}

}  // extern "C"

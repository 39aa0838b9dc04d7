// Linear of at most 16 rows (the time, label and resnet embeddings of a UNet step): activations quantised, multiplied
// and finished in one launch.
//
// What bounds it: latency. The weights of such a projection are 0.4 to 4 MB, under a microsecond of memory time,
// while the tensor-memory GEMM issues one MMA chain over all of K behind a quantiser launch (a 128-row MMA per
// 32 bytes of K, whatever the row count). Here a block owns 8 x kGroups output columns and its 16 warps split K,
// so most loads of the problem are in flight at once; the partial products meet in shared memory, added in warp order.
// Measured on B200 in a stream of calls: FP8 [2, 1280], K = 320 with SiLU 8.9 us in three launches, now 3.8; INT8
// [16, 1280], K = 2816, rotated 13.6 us, now 8.2, half of it the rotating quantiser.
//
// The warp-wide MMA m16n8k16 (k32 for INT8) sums over k in any order, as long as both operands agree on it: lane
// (g = lane / 4, t = lane % 4) takes 16 consecutive values of K, 64 c + 16 t .. + 15 of chunk c, for rows g and g + 8 of X
// and for row g of the weights' group, so both operands come straight from global memory with 16-byte loads and no
// exchange. FP8 values enter the FP16 MMA (exact) and are summed in FP32.
//
// FP16 input of an FP8 or unrotated INT8 projection: a block's warps read all of X between them, so each block
// finds the maximum (of the tensor, of each row) and casts its values in registers, with the arithmetic of the
// stand-alone quantisers.

#include "internal.cuh"
#include "quantize.cuh"
#include "fp8_math.cuh"
#include "int8_math.cuh"

namespace sdxlq {

struct SkinnyParams {
    const void* a;               // [M, K] FP16 (kFromHalf, and always for FP16 weights) or quantised values
    const void* b;               // [N, K] weights
    EpilogueParams ep;
};

namespace {

constexpr uint32_t kWarps = 16;
constexpr uint32_t kRows = 16;
constexpr uint32_t kChunk = 64;                          // values of K per warp step

enum : int { SKINNY_I8 = 0, SKINNY_E4M3 = 1, SKINNY_E5M2 = 2, SKINNY_F16 = 3 };

__device__ __forceinline__ uint4 load16(const void* base, size_t byte, bool inside) {
    return inside ? __ldg(reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(base) + byte)) : make_uint4(0u, 0u, 0u, 0u);
}

// two FP8 values (low half of `pair`) -> two FP16 values, exact
template <int kKind>
__device__ __forceinline__ uint32_t widen_fp8(uint32_t pair) {
    const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(pair & 0xFFFFu),
                                                     kKind == SKINNY_E4M3 ? __NV_E4M3 : __NV_E5M2);
    return static_cast<uint32_t>(h.x) | (static_cast<uint32_t>(h.y) << 16);
}

// 16 consecutive values of K as the MMA takes them: eight words of FP16 pairs, or (INT8) four words of bytes.
template <int kKind> struct Fragment { uint32_t word[8]; };
template <> struct Fragment<SKINNY_I8> { uint32_t word[4]; };

// Stored values (weights, quantised activations) of row `row`, values k .. k + 15, zero past the matrix.
template <int kKind>
__device__ __forceinline__ Fragment<kKind> load_stored(const void* base, uint32_t row, uint32_t rows, uint32_t k, uint32_t width) {
    Fragment<kKind> f;
    if constexpr (kKind == SKINNY_F16) {
        const size_t at = (static_cast<size_t>(row) * width + k) * 2;
        const uint4 lo = load16(base, at, row < rows && k < width), hi = load16(base, at + 16, row < rows && k + 8 < width);
        f.word[0] = lo.x; f.word[1] = lo.y; f.word[2] = lo.z; f.word[3] = lo.w;
        f.word[4] = hi.x; f.word[5] = hi.y; f.word[6] = hi.z; f.word[7] = hi.w;
    } else {
        const uint4 raw = load16(base, static_cast<size_t>(row) * width + k, row < rows && k < width);
        const uint32_t words[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if constexpr (kKind == SKINNY_I8) {
                f.word[i] = words[i];
            } else {
                f.word[2 * i] = widen_fp8<kKind>(words[i]);
                f.word[2 * i + 1] = widen_fp8<kKind>(words[i] >> 16);
            }
        }
    }
    return f;
}

// FP16 activations cast as the stand-alone quantisers do (FP8: x * inverse saturated; INT8: rn(x * inverse) clamped).
template <int kKind>
__device__ __forceinline__ Fragment<kKind> quantise(const Fragment<SKINNY_F16>& x, float inverse) {
    Fragment<kKind> f;
    if constexpr (kKind == SKINNY_I8) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t lo = x.word[2 * i], hi = x.word[2 * i + 1];
            f.word[i] = pack_bytes(quantize_s8(__fmul_rn(half_lo(lo), inverse)), quantize_s8(__fmul_rn(half_hi(lo), inverse)),
                                   quantize_s8(__fmul_rn(half_lo(hi), inverse)), quantize_s8(__fmul_rn(half_hi(hi), inverse)));
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            f.word[i] = widen_fp8<kKind>(encode_fp8x2(__fmul_rn(half_lo(x.word[i]), inverse), __fmul_rn(half_hi(x.word[i]), inverse),
                                                      kKind == SKINNY_E4M3 ? 0u : 1u));
        }
    }
    return f;
}

// Accumulators as 32-bit words: FP32, or INT32 for INT8. top: row g, low: row g + 8 of X.
template <int kKind>
__device__ __forceinline__ void multiply(uint32_t (&acc)[4], const Fragment<kKind>& top, const Fragment<kKind>& low, const Fragment<kKind>& b) {
    if constexpr (kKind == SKINNY_I8) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                : "+r"(acc[0]), "+r"(acc[1]), "+r"(acc[2]), "+r"(acc[3])
                : "r"(top.word[2 * j]), "r"(low.word[2 * j]), "r"(top.word[2 * j + 1]), "r"(low.word[2 * j + 1]), "r"(b.word[2 * j]),
                  "r"(b.word[2 * j + 1]));
        }
    } else {
        float c[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) c[i] = __uint_as_float(acc[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                : "r"(top.word[2 * j]), "r"(low.word[2 * j]), "r"(top.word[2 * j + 1]), "r"(low.word[2 * j + 1]), "r"(b.word[2 * j]),
                  "r"(b.word[2 * j + 1]));
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] = __float_as_uint(c[i]);
    }
}

// Largest magnitude of the fragment's halves, in half precision (exact; NaN never wins).
__device__ __forceinline__ __half2 widest(const Fragment<SKINNY_F16>& x, __half2 largest) {
#pragma unroll
    for (int i = 0; i < 8; ++i) largest = __hmax2(largest, __habs2(as_half2(x.word[i])));
    return largest;
}

// The same over finite values only, as the INT8 scale wants it.
__device__ __forceinline__ float widest_finite(const Fragment<SKINNY_F16>& x, float largest) {
    largest = finite_max(make_uint4(x.word[0], x.word[1], x.word[2], x.word[3]), largest);
    return finite_max(make_uint4(x.word[4], x.word[5], x.word[6], x.word[7]), largest);
}

// The larger of the two magnitudes as FP16 bits, which order like integers. The argument holds no NaN.
__device__ __forceinline__ uint32_t magnitude_bits(__half2 maximum) {
    return max(static_cast<uint32_t>(__half_as_ushort(__low2half(maximum))), static_cast<uint32_t>(__half_as_ushort(__high2half(maximum))));
}

// Maximum over the block; `words`: a word of shared memory per warp.
__device__ __forceinline__ uint32_t block_maximum(uint32_t value, uint32_t* words) {
    value = __reduce_max_sync(0xffffffffu, value);
    if ((threadIdx.x & 31u) == 0) words[threadIdx.x >> 5] = value;
    __syncthreads();
    value = 0;
#pragma unroll
    for (uint32_t w = 0; w < kWarps; ++w) value = max(value, words[w]);
    return value;
}

}  // namespace

// kGroups: groups of eight output columns per block; with GEGLU the second half of them are gate columns.
template <int kKind, bool kFromHalf, int kGroups>
__global__ void __launch_bounds__(32 * kWarps)
sdxlq_skinny_linear_kernel(const __grid_constant__ SkinnyParams p) {
    __shared__ uint32_t partial[kWarps][kGroups][4][32];
    __shared__ uint32_t warp_maximum[kWarps][kRows];
    __shared__ float row_scale[kRows];
    wait_for_prior_kernels_then_release_next();
    const EpilogueParams& ep = p.ep;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint32_t k_width = ep.k, m = ep.m;
    const uint32_t chunks = (k_width + kChunk - 1) / kChunk;
    const bool geglu = ep.activation == ACT_GEGLU;
    const uint32_t out_groups = geglu ? kGroups / 2 : kGroups;
    const uint32_t first_column = blockIdx.x * out_groups * 8u;
    // the lane's weight row in a group; columns past the matrix get a row that loads zeros
    const auto weight_row = [&](uint32_t group) {
        const bool gate = geglu && group >= out_groups;
        const uint32_t column = first_column + (gate ? group - out_groups : group) * 8u + g;
        if (column >= ep.n_out) return ep.n;
        return gate ? ep.n_out + column : column;
    };

    // the weights of the warp's first chunk travel while the maximum is found
    Fragment<kKind> ahead[kGroups];
#pragma unroll
    for (int group = 0; group < kGroups; ++group) {
        ahead[group] = load_stored<kKind>(p.b, weight_row(group), ep.n, warp < chunks ? warp * kChunk + t * 16u : k_width, k_width);
    }

    float inverse_top = 1.0f, inverse_low = 1.0f;
    if constexpr (kFromHalf) {
        if constexpr (kKind == SKINNY_I8) {
            float top = 0.0f, low = 0.0f;
            for (uint32_t c = warp; c < chunks; c += kWarps) {
                top = widest_finite(load_stored<SKINNY_F16>(p.a, g, m, c * kChunk + t * 16u, k_width), top);
                low = widest_finite(load_stored<SKINNY_F16>(p.a, g + 8u, m, c * kChunk + t * 16u, k_width), low);
            }
#pragma unroll
            for (int offset = 1; offset < 4; offset <<= 1) {
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, offset));
                low = fmaxf(low, __shfl_xor_sync(0xffffffffu, low, offset));
            }
            if (t == 0) {
                warp_maximum[warp][g] = __float_as_uint(top);
                warp_maximum[warp][g + 8u] = __float_as_uint(low);
            }
            __syncthreads();
            if (threadIdx.x < kRows) {
                uint32_t bits = 0;
                for (uint32_t w = 0; w < kWarps; ++w) bits = max(bits, warp_maximum[w][threadIdx.x]);
                row_scale[threadIdx.x] = scale_from_amax(__uint_as_float(bits));
            }
            __syncthreads();
            inverse_top = __fdiv_rn(1.0f, row_scale[g]);
            inverse_low = __fdiv_rn(1.0f, row_scale[g + 8u]);
        } else {
            __half2 largest = __float2half2_rn(0.0f);
            for (uint32_t c = warp; c < chunks; c += kWarps) {
                largest = widest(load_stored<SKINNY_F16>(p.a, g, m, c * kChunk + t * 16u, k_width), largest);
                largest = widest(load_stored<SKINNY_F16>(p.a, g + 8u, m, c * kChunk + t * 16u, k_width), largest);
            }
            const uint32_t bits = block_maximum(magnitude_bits(largest), &warp_maximum[0][0]);
            const float maximum = __half2float(__ushort_as_half(static_cast<unsigned short>(bits)));
            const float scale = fp8_scale_from_amax(maximum, kKind == SKINNY_E4M3 ? 0u : 1u);
            inverse_top = inverse_low = __fdiv_rn(1.0f, scale);
            if (threadIdx.x < kRows) row_scale[threadIdx.x] = scale;
        }
    } else if (kKind != SKINNY_F16) {
        if (threadIdx.x < kRows) row_scale[threadIdx.x] = kKind == SKINNY_I8 ? (threadIdx.x < m ? ep.a_scales[threadIdx.x] : 0.0f) : ep.a_scales[0];
    }

    uint32_t acc[kGroups][4] = {};
    for (uint32_t c = warp; c < chunks; c += kWarps) {
        const uint32_t k = c * kChunk + t * 16u;
        Fragment<kKind> top, low, b[kGroups];
        if constexpr (kFromHalf && kKind != SKINNY_F16) {
            top = quantise<kKind>(load_stored<SKINNY_F16>(p.a, g, m, k, k_width), inverse_top);
            low = quantise<kKind>(load_stored<SKINNY_F16>(p.a, g + 8u, m, k, k_width), inverse_low);
        } else {
            top = load_stored<kKind>(p.a, g, m, k, k_width);
            low = load_stored<kKind>(p.a, g + 8u, m, k, k_width);
        }
#pragma unroll
        for (int group = 0; group < kGroups; ++group) {
            b[group] = ahead[group];
            ahead[group] = load_stored<kKind>(p.b, weight_row(group), ep.n, c + kWarps < chunks ? k + kWarps * kChunk : k_width, k_width);
        }
#pragma unroll
        for (int group = 0; group < kGroups; ++group) multiply<kKind>(acc[group], top, low, b[group]);
    }
#pragma unroll
    for (int group = 0; group < kGroups; ++group) {
#pragma unroll
        for (int i = 0; i < 4; ++i) partial[warp][group][i][lane] = acc[group][i];
    }
    __syncthreads();

    // Accumulator i of lane (g, t) belongs to row g + 8 (i / 2), column 2 t + i % 2 of its group. Warps without a chunk
    // left zeros.
    const auto total = [&](uint32_t group, uint32_t row, uint32_t column) {
        const uint32_t i = (row >> 3) * 2u + (column & 1u), from = (row & 7u) * 4u + (column >> 1);
        uint32_t sum = partial[0][group][i][from];
#pragma unroll
        for (uint32_t w = 1; w < kWarps; ++w) {
            const uint32_t next = partial[w][group][i][from];
            sum = kKind == SKINNY_I8 ? sum + next : __float_as_uint(__uint_as_float(sum) + __uint_as_float(next));
        }
        return sum;
    };
    float maximum = 0.0f;
    for (uint32_t item = threadIdx.x; item < out_groups * 8u * m; item += 32u * kWarps) {
        const uint32_t row = item / (out_groups * 8u), local = item % (out_groups * 8u);
        const uint32_t column = first_column + local, group = local >> 3;
        if (column >= ep.n_out) continue;
        const bool scaled = kKind != SKINNY_F16, has_bias = ep.bias != nullptr;
        const float a_scale = scaled ? row_scale[row] : 1.0f;
        const auto project = [&](uint32_t in_group, uint32_t weight) {
            const uint32_t bits = total(in_group, row, local & 7u);
            if (ep.acc_out != nullptr) ep.acc_out[static_cast<size_t>(row) * ep.n + weight] = static_cast<int32_t>(bits);
            return project_to_half(bits, ep.kind, a_scale, scaled ? ep.w_scales[ep.w_scale_per_channel ? weight : 0u] : 1.0f);
        };
        __half result;
        if (geglu) {
            const __half value = project(group, column), gate = project(out_groups + group, ep.n_out + column);
            result = finish_geglu(value, ep.bias[column], gate, ep.bias[ep.n_out + column]);
        } else {
            result = finish_scalar(project(group, column), has_bias, has_bias ? ep.bias[column] : __half(0), ep.activation);
            if (ep.residual != nullptr) result = __hadd(result, ep.residual[static_cast<size_t>(row) * ep.n_out + column]);
        }
        ep.y[static_cast<size_t>(row) * ep.n_out + column] = result;
        maximum = fmaxf(maximum, fabsf(__half2float(result)));
    }
    if (ep.y_amax != nullptr) {
        __syncwarp();
        const uint32_t bits = __reduce_max_sync(0xffffffffu, __float_as_uint(maximum));
        if (lane == 0 && bits != 0) atomicMax(ep.y_amax, bits);
    }
}

namespace {

template <int kKind, bool kFromHalf>
cudaError_t launch_groups(const SkinnyParams& params, uint32_t sm_count, cudaStream_t stream, bool early_launch) {
    // As few columns per block as keep the grid within two blocks per SM, which fit with one or two groups (at most 58
    // registers; with four, 102 registers leave room for one block, 64 in INT8 for two). Every block reads all of X.
    const uint32_t halves = params.ep.activation == ACT_GEGLU ? 2 : 1;          // value and gate columns
    const uint32_t column_groups = (params.ep.n_out + 7) / 8;
    uint32_t out_groups = 1;
    while (out_groups * halves < 4 && (column_groups + out_groups - 1) / out_groups > 2 * sm_count) out_groups *= 2;
    const uint32_t blocks = (column_groups + out_groups - 1) / out_groups;
    const auto run = [&](auto kernel) { return launch_behind(kernel, blocks, 32 * kWarps, 0, stream, early_launch, params); };
    if (out_groups * halves == 1) return run(sdxlq_skinny_linear_kernel<kKind, kFromHalf, 1>);
    if (out_groups * halves == 2) return run(sdxlq_skinny_linear_kernel<kKind, kFromHalf, 2>);
    return run(sdxlq_skinny_linear_kernel<kKind, kFromHalf, 4>);
}

}  // namespace

// `from_half`: `a` holds FP16 activations that the kernel quantises itself (FP8 and unrotated INT8 weights).
cudaError_t launch_skinny_linear(const void* a, const void* b, const EpilogueParams& ep, bool from_half, uint32_t sm_count,
                                 cudaStream_t stream, bool early_launch) {
    const SkinnyParams params{a, b, ep};
    switch (ep.kind) {
    case KIND_I8: return from_half ? launch_groups<SKINNY_I8, true>(params, sm_count, stream, early_launch)
                                   : launch_groups<SKINNY_I8, false>(params, sm_count, stream, early_launch);
    case KIND_E4M3: return from_half ? launch_groups<SKINNY_E4M3, true>(params, sm_count, stream, early_launch)
                                     : launch_groups<SKINNY_E4M3, false>(params, sm_count, stream, early_launch);
    case KIND_E5M2: return from_half ? launch_groups<SKINNY_E5M2, true>(params, sm_count, stream, early_launch)
                                     : launch_groups<SKINNY_E5M2, false>(params, sm_count, stream, early_launch);
    default: return launch_groups<SKINNY_F16, false>(params, sm_count, stream, early_launch);
    }
}

}  // namespace sdxlq

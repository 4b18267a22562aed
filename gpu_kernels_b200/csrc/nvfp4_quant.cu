// NVFP4 quantise / pack and dequantise kernels for sm_100a.
//
// quantise: x[rows, K] (bf16 / fp16 / fp32) -> packed E2M1 [rows, K/2] plus one
// UE4M3 scale per 16 values, written directly in the 128-row x 4-block scale
// atoms that cuBLASLt's VEC16 mode and the tcgen05 block-scaled MMA read.
// Arithmetic follows the reference's PyTorch quantiser step by step
// (reference/python/nvfp4.py:30-37 and :6-14): amax -> IEEE divide by 6 ->
// clamp [2^-9, 448] -> E4M3 nearest-even -> IEEE divide -> E2M1 nearest-even
// with sign bit (q < 0), bit for bit. The kernel is HBM-bound: 2 B read (bf16) and 0.5625 B
// written per value; a CTA owns a 128-row x 256-column tile so that each scale
// atom (512 B) and each packed row segment (128 B) leaves in full lines.
#include "nvfp4_internal.h"
#include "ptx.cuh"
#include "quant_device.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

namespace nvfp4_b200 {
namespace {

constexpr int Q_ROWS = 128;      // rows per CTA tile = rows of one scale atom
constexpr int Q_THREADS = 256;
constexpr int MAX_GRID_Y = 32768;  // row tiles per layer of the grid

template <typename T> struct PairFormat { using type = void; };
template <> struct PairFormat<__nv_bfloat16> { using type = Bf16Pairs; };
template <> struct PairFormat<__half> { using type = Fp16Pairs; };

// One block of 16 values, as loaded, to its scale byte and packed codes. SCALED: every value times inv_global, in
// FP32, first (the product is no longer a 16-bit value, so it takes the FP32 routine whatever the input type).
template <typename T, bool SCALED>
__device__ __forceinline__ uint32_t quantise_raw(const uint4 (&raw)[sizeof(T)], float inv_global, uint2& out) {
    if constexpr (sizeof(T) == 2 && !SCALED) {
        const uint32_t w[8] = {raw[0].x, raw[0].y, raw[0].z, raw[0].w, raw[1].x, raw[1].y, raw[1].z, raw[1].w};
        return quantise_block_pairs<typename PairFormat<T>::type>(w, out);
    } else {
        float v[16];
        #pragma unroll
        for (int i = 0; i < int(sizeof(T)); ++i) {
            const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
            #pragma unroll
            for (int j = 0; j < 4; ++j) {
                if constexpr (sizeof(T) == 4) {
                    v[4 * i + j] = __uint_as_float(w[j]);
                } else {
                    v[8 * i + 2 * j] = PairFormat<T>::type::widen(w[j] & 0xFFFFu);
                    v[8 * i + 2 * j + 1] = PairFormat<T>::type::widen(w[j] >> 16);
                }
            }
        }
        if constexpr (SCALED) {
            #pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = __fmul_rn(v[i], inv_global);
        }
        return quantise_block(v, out);
    }
}

// Four CTAs per SM: the register cap this implies (64) keeps 32 warps resident, which together with the loads
// kept ahead is what it takes to cover the memory latency (measured on 8192 x 8192 bf16: 3 CTAs 37.3 us,
// 4 CTAs 34.9 us, 5 CTAs, which leaves no registers for the loads ahead, 39.1 us).
// COLS: K values per CTA tile (256 = four scale atoms, or 128 = two). The narrower tile gives twice the CTAs,
// which evens out the last wave of a grid that is only a few waves long.
// TAIL: the instance for a tensor whose last row tile is partial (rows % 128 != 0): rows the tensor does not have are
// read as zeros, which gives them the scale byte of a zero block (0x01) in the atom and no packed bytes. One launch for
// all row tiles: the last one as a launch of its own cost 1000 x 8192 bf16 another 4 us behind the 7 us of the others.
// SCALED (two-level scaling): the values are first multiplied by the reciprocal of a per-tensor scale; the GEMM undoes
// the tensor scales through its alpha.
// EARLY: the kernel behind this one may start while it runs (see quantise() in nvfp4_internal.h).
template <typename T, int COLS, bool TAIL, bool SCALED, bool EARLY>
__global__ void __launch_bounds__(Q_THREADS, 4)
quantise_kernel(const T* __restrict__ x, uint8_t* __restrict__ packed, uint8_t* __restrict__ scales,
                int rows, int K, float inv_global) {
    // Launched through launch_chained(): the launch itself overlaps the tail of the kernel in front. The wait comes first:
    // a product behind this kernel requests its weights before its own wait, and an earlier kernel may have written them.
    ptx::grid_dependency_wait();
    if constexpr (EARLY) ptx::grid_launch_dependents();
    constexpr int BLOCKS = COLS / 16;                           // 16-value blocks across the tile
    constexpr int ROWS_PER_PASS = Q_THREADS / BLOCKS;
    constexpr int PASSES = Q_ROWS / ROWS_PER_PASS;
    constexpr int ATOMS = COLS / 64;
    __shared__ __align__(16) uint8_t sf_tile[ATOMS * 512];
    const int kb = threadIdx.x % BLOCKS;                        // 16-value block inside the tile
    const int row_in_pass = threadIdx.x / BLOCKS;
    const int col0 = blockIdx.x * COLS;
    const int row_tile = int(blockIdx.z) * MAX_GRID_Y + int(blockIdx.y);
    if (row_tile * Q_ROWS >= rows) return;                     // (the last layer of a grid with several)
    const int row_base = row_tile * Q_ROWS;
    const int k = col0 + kb * 16;
    const bool live = k < K;                                    // K is a multiple of 64, the tile of COLS
    auto emit = [&](int r, uint32_t sbyte, const uint2& out) {
        if (!TAIL || row_base + r < rows)
            *reinterpret_cast<uint2*>(packed + size_t(row_base + r) * (K / 2) + k / 2) = out;
        sf_tile[(kb >> 2) * 512 + (r & 31) * 16 + (r >> 5) * 4 + (kb & 3)] = static_cast<uint8_t>(sbyte);
    };
    // The loads of the next passes are kept in flight ahead of the arithmetic, so that a warp waits for memory once per
    // tile rather than once per pass: two passes for 16-bit inputs (32 bytes per thread and pass), one for FP32 (64).
    constexpr int WORDS = int(sizeof(T)), AHEAD = sizeof(T) == 2 ? 2 : 1;
    uint4 raw[AHEAD][WORDS];
    auto fetch = [&](int pass, uint4 (&to)[WORDS]) {
        const int r = pass * ROWS_PER_PASS + row_in_pass;
        const uint4* p = reinterpret_cast<const uint4*>(x + size_t(row_base + r) * K + k);
        const bool there = !TAIL || row_base + r < rows;
        #pragma unroll
        for (int i = 0; i < WORDS; ++i) to[i] = there ? __ldg(p + i) : make_uint4(0u, 0u, 0u, 0u);
    };
    if (live) {
        #pragma unroll
        for (int i = 0; i < AHEAD; ++i) fetch(i, raw[i]);
        #pragma unroll
        for (int pass = 0; pass < PASSES; ++pass) {
            uint4 now[WORDS];
            #pragma unroll
            for (int i = 0; i < WORDS; ++i) now[i] = raw[pass % AHEAD][i];
            if (pass + AHEAD < PASSES) fetch(pass + AHEAD, raw[pass % AHEAD]);
            uint2 out;
            const uint32_t sbyte = quantise_raw<T, SCALED>(now, inv_global, out);
            emit(pass * ROWS_PER_PASS + row_in_pass, sbyte, out);
        }
    }
    __syncthreads();
    // The tile's atoms are consecutive in the VEC16 layout: one 16-byte store per thread.
    const int atoms = min(ATOMS, (K - col0) / 64);
    if (int(threadIdx.x) < atoms * 32) {
        const size_t first_atom = size_t(row_tile) * (K / 64) + size_t(blockIdx.x) * ATOMS;
        reinterpret_cast<uint4*>(scales + first_atom * 512)[threadIdx.x] =
            reinterpret_cast<const uint4*>(sf_tile)[threadIdx.x];
    }
}

// packed + scales -> FP32 [rows, K]; one thread per 16-value block
// (reference/python/nvfp4.py:40-47).
__global__ void __launch_bounds__(256)
dequantise_kernel(const uint8_t* __restrict__ packed, const uint8_t* __restrict__ scales,
                  float* __restrict__ out, int rows, int K) {
    const size_t idx = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int blocks_per_row = K / 16;
    if (idx >= size_t(rows) * blocks_per_row) return;
    const int r = static_cast<int>(idx / blocks_per_row), b = static_cast<int>(idx % blocks_per_row);
    const size_t off = (size_t(r / 128) * (K / 64) + b / 4) * 512 + (r % 32) * 16 + ((r % 128) / 32) * 4 + b % 4;
    const uint32_t sb = scales[off];
    // 0x7F / 0xFF are NaN in E4M3 (finite-only format); the quantiser never sets the sign bit.
    float s = (sb & 0x7Fu) == 0x7Fu ? __uint_as_float(0x7FC00000u) : ue4m3_to_float(sb & 0x7Fu);
    if (sb & 0x80u) s = -s;
    const uint2 p = __ldg(reinterpret_cast<const uint2*>(packed + size_t(r) * (K / 2) + b * 8));
    const uint32_t w[2] = {p.x, p.y};
    float4* dst = reinterpret_cast<float4*>(out + size_t(r) * K + b * 16);
    #pragma unroll
    for (int h = 0; h < 2; ++h) {
        float f[8];
        #pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t c = (w[h] >> (4 * i)) & 15u;
            const uint32_t m = c & 7u;
            // levels 0, .5, 1, 1.5, 2, 3, 4, 6
            const float level = m < 2u ? 0.5f * m : __uint_as_float(((126u + (m >> 1)) << 23) | ((m & 1u) << 22));
            f[i] = level * (1.0f - 2.0f * static_cast<float>(c >> 3)) * s;
        }
        dst[2 * h] = make_float4(f[0], f[1], f[2], f[3]);
        dst[2 * h + 1] = make_float4(f[4], f[5], f[6], f[7]);
    }
}

// ---- MXFP4 (OCP microscaling): E2M1 values, one UE8M0 power-of-two scale per 32 values ------------------------
// Per block: e = floor(log2(amax)) - 2 (2 = the largest exponent of E2M1), clamped to [-127, 127]; scale byte
// e + 127; q = x * 2^-e (exact but for underflow) encoded as E2M1 with the quantiser's rounding and sign rule.
// An all-zero block takes e = -127; a block with a NaN or an infinity takes the NaN scale 0xFF and the codes of
// the NVFP4 NaN block. The scale bytes go to cuBLASLt's VEC32 order: the VEC16 atoms with K/32 blocks per row.
// A CTA owns one scale atom, 128 rows x 128 columns: two blocks of 32 per thread, the second's loads in flight during the
// first's arithmetic, the atom's bytes gathered in shared memory and written as one run. Against one thread per block with
// each scale byte stored by itself: 8192 x 8192 bf16 39.4 -> 32.5 us (5.3 TB/s), 2048 x 2048 f16 4.8 -> 4.0 us; what
// bounds it is HBM and the fixed cost of a launch, as for the NVFP4 kernel.
template <typename T>
__global__ void __launch_bounds__(Q_THREADS, sizeof(T) == 2 ? 4 : 3)
quantise_mx_kernel(const T* __restrict__ x, uint8_t* __restrict__ packed, uint8_t* __restrict__ scales, int rows, int K) {
    ptx::grid_dependency_wait();
    constexpr int WORDS = 2 * int(sizeof(T));                  // 16-byte words of a block
    __shared__ __align__(16) uint8_t sf_tile[512];
    const int kb = threadIdx.x & 3, row_in_pass = threadIdx.x >> 2, row_base = int(blockIdx.x / unsigned(K / 128)) * Q_ROWS;
    const size_t k = size_t(blockIdx.x % unsigned(K / 128)) * 128 + kb * 32;
    uint4 raw[2][WORDS];
    #pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
        const int row = row_base + pass * 64 + row_in_pass;
        const uint4* p = reinterpret_cast<const uint4*>(x + size_t(row) * K + k);
        #pragma unroll
        for (int i = 0; i < WORDS; ++i) raw[pass][i] = row < rows ? __ldg(p + i) : make_uint4(0u, 0u, 0u, 0u);
    }
    #pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
        const int r = pass * 64 + row_in_pass;
        float v[32];
        #pragma unroll
        for (int i = 0; i < WORDS; ++i) {
            const uint32_t w[4] = {raw[pass][i].x, raw[pass][i].y, raw[pass][i].z, raw[pass][i].w};
            #pragma unroll
            for (int j = 0; j < 4; ++j) {
                if constexpr (sizeof(T) == 4) {
                    v[4 * i + j] = __uint_as_float(w[j]);
                } else {
                    v[8 * i + 2 * j] = PairFormat<T>::type::widen(w[j] & 0xFFFFu);
                    v[8 * i + 2 * j + 1] = PairFormat<T>::type::widen(w[j] >> 16);
                }
            }
        }
        uint32_t mx = 0;
        #pragma unroll
        for (int i = 0; i < 32; ++i) mx = max(mx, __float_as_uint(v[i]) & 0x7FFFFFFFu);
        uint32_t words[4] = {0x77777777u, 0x77777777u, 0x77777777u, 0x77777777u}, sbyte = 0xFFu;
        if (mx < 0x7F800000u) {
            // floor(log2(amax)) is the exponent field; zero and subnormal maxima end at the clamp either way
            const int e = max(int(mx >> 23) - 129, -127);
            const float inv = __uint_as_float(uint32_t(127 - e) << 23);
            #pragma unroll
            for (int h = 0; h < 4; ++h) {
                float q[8];
                uint32_t signs = 0;
                #pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float t = __fmul_rn(v[8 * h + i], inv);
                    q[i] = fabsf(t);
                    signs |= t < 0.0f ? (8u << (4 * i)) : 0u;
                }
                words[h] = e2m1x8_from_quotients(q) | signs;
            }
            sbyte = uint32_t(e + 127);
        }
        if (row_base + r < rows)
            *reinterpret_cast<uint4*>(packed + size_t(row_base + r) * (K / 2) + k / 2) = make_uint4(words[0], words[1], words[2], words[3]);
        sf_tile[(r & 31) * 16 + (r >> 5) * 4 + kb] = static_cast<uint8_t>(sbyte);     // a row the tensor does not have: a zero block's 0
    }
    __syncthreads();
    if (threadIdx.x < 32)
        reinterpret_cast<uint4*>(scales + size_t(blockIdx.x) * 512)[threadIdx.x] =
            reinterpret_cast<const uint4*>(sf_tile)[threadIdx.x];
}

// MXFP4 bytes -> FP32 [rows, K]; one thread per block of 32 (the check path).
__global__ void __launch_bounds__(256)
dequantise_mx_kernel(const uint8_t* __restrict__ packed, const uint8_t* __restrict__ scales, float* __restrict__ out,
                     int rows, int K) {
    const size_t idx = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int blocks_per_row = K / 32;
    if (idx >= size_t(rows) * blocks_per_row) return;
    const int r = int(idx / blocks_per_row), b = int(idx % blocks_per_row);
    const uint32_t sb = scales[scale_byte_offset(r, b, K / 2)];
    const float s = sb == 0xFFu ? __uint_as_float(0x7FC00000u) : scalbnf(1.0f, int(sb) - 127);
    const uint4 p = __ldg(reinterpret_cast<const uint4*>(packed + size_t(r) * (K / 2) + size_t(b) * 16));
    const uint32_t w[4] = {p.x, p.y, p.z, p.w};
    float* dst = out + size_t(r) * K + size_t(b) * 32;
    #pragma unroll
    for (int h = 0; h < 4; ++h)
        #pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t c = (w[h] >> (4 * i)) & 15u, m = c & 7u;
            const float level = m < 2u ? 0.5f * m : __uint_as_float(((126u + (m >> 1)) << 23) | ((m & 1u) << 22));
            dst[8 * h + i] = level * (1.0f - 2.0f * static_cast<float>(c >> 3)) * s;
        }
}

}  // namespace

void check_quant_shape(int rows, int K) {
    if (rows <= 0 || K <= 0) throw std::invalid_argument("nvfp4 quantise: rows and K must be positive");
    if (K % 64 != 0) throw std::invalid_argument("nvfp4 quantise: K must be a multiple of 64");
}

namespace {

template <bool SCALED, bool EARLY>
void launch_quantise(const void* x, int dtype, float inv_global, uint8_t* packed, uint8_t* scales, int rows, int K,
                     cudaStream_t stream) {
    // 256-column tiles; 128-column ones when the grid would otherwise be less than two waves of resident CTAs
    // (four per SM). Measured, 128 / 256 columns: 4096 x 4096 bf16 12.3 / 14.4 us, 8192 x 8192 36.9 / 34.0 us.
    int device = 0, sms = 0;
    cuda_check(cudaGetDevice(&device));
    cuda_check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    const long long wide_ctas = (long long)((K + 255) / 256) * (rows / Q_ROWS);
    const bool narrow = K % 128 == 0 && wide_ctas < 2LL * 4 * sms;
    auto launch = [&](auto tag) {
        using T = decltype(tag);
        const int cols = narrow ? 128 : 256;
        const int row_tiles = (rows + Q_ROWS - 1) / Q_ROWS;
        const dim3 grid((K + cols - 1) / cols, std::min(row_tiles, MAX_GRID_Y), (row_tiles + MAX_GRID_Y - 1) / MAX_GRID_Y);
        auto go = [&](auto kernel) {
            launch_chained(kernel, grid, dim3(Q_THREADS), size_t(0), stream, static_cast<const T*>(x), packed, scales, rows, K, inv_global);
        };
        const bool tail = rows % Q_ROWS != 0;
        if (narrow) tail ? go(quantise_kernel<T, 128, true, SCALED, EARLY>) : go(quantise_kernel<T, 128, false, SCALED, EARLY>);
        else tail ? go(quantise_kernel<T, 256, true, SCALED, EARLY>) : go(quantise_kernel<T, 256, false, SCALED, EARLY>);
    };
    switch (dtype) {
        case DTYPE_BF16: launch(__nv_bfloat16{}); break;
        case DTYPE_F16: launch(__half{}); break;
        case DTYPE_F32: launch(float{}); break;
        default:
            throw std::invalid_argument("nvfp4 quantise: dtype must be 0 (bf16), 1 (fp16) or 2 (fp32)");
    }
    cuda_check(cudaGetLastError());
}

void check_quant_pointers(const void* x, const uint8_t* packed, const uint8_t* scales) {
    if (!x || !packed || !scales) throw std::invalid_argument("nvfp4 quantise: null pointer");
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(packed) | reinterpret_cast<uintptr_t>(scales)) & 15)
        throw std::invalid_argument("nvfp4 quantise: pointers must be 16-byte aligned");
}

}  // namespace

void quantise(const void* x, int dtype, uint8_t* packed, uint8_t* scales, int rows, int K, cudaStream_t stream, bool early) {
    check_quant_shape(rows, K);
    check_quant_pointers(x, packed, scales);
    if (early) launch_quantise<false, true>(x, dtype, 1.0f, packed, scales, rows, K, stream);
    else launch_quantise<false, false>(x, dtype, 1.0f, packed, scales, rows, K, stream);
}

void quantise_scaled(const void* x, int dtype, float inv_global, uint8_t* packed, uint8_t* scales, int rows, int K,
                     cudaStream_t stream) {
    check_quant_shape(rows, K);
    check_quant_pointers(x, packed, scales);
    if (!(inv_global > 0.0f) || !(inv_global < 3.0e38f)) throw std::invalid_argument("nvfp4 quantise: the tensor scale must be positive and finite");
    launch_quantise<true, false>(x, dtype, inv_global, packed, scales, rows, K, stream);
}

void check_mx_shape(int rows, int K) {
    if (rows <= 0 || K <= 0) throw std::invalid_argument("mxfp4: rows and K must be positive");
    if (K % 128 != 0) throw std::invalid_argument("mxfp4: K must be a multiple of 128 (one scale atom covers 4 blocks of 32)");
}

void quantise_mx(const void* x, int dtype, uint8_t* packed, uint8_t* scales, int rows, int K, cudaStream_t stream) {
    check_mx_shape(rows, K);
    if (!x || !packed || !scales) throw std::invalid_argument("mxfp4 quantise: null pointer");
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(packed) | reinterpret_cast<uintptr_t>(scales)) & 15)
        throw std::invalid_argument("mxfp4 quantise: pointers must be 16-byte aligned");
    const dim3 grid(unsigned(K / 128) * unsigned((rows + Q_ROWS - 1) / Q_ROWS));
    auto launch = [&](auto tag) {
        using T = decltype(tag);
        launch_chained(quantise_mx_kernel<T>, grid, dim3(Q_THREADS), size_t(0), stream, static_cast<const T*>(x), packed, scales, rows, K);
    };
    switch (dtype) {
        case DTYPE_BF16: launch(__nv_bfloat16{}); break;
        case DTYPE_F16: launch(__half{}); break;
        case DTYPE_F32: launch(float{}); break;
        default: throw std::invalid_argument("mxfp4 quantise: dtype must be 0 (bf16), 1 (fp16) or 2 (fp32)");
    }
    cuda_check(cudaGetLastError());
}

void dequantise_mx(const uint8_t* packed, const uint8_t* scales, float* out, int rows, int K, cudaStream_t stream) {
    check_mx_shape(rows, K);
    if (!packed || !scales || !out) throw std::invalid_argument("mxfp4 dequantise: null pointer");
    const size_t blocks = size_t(rows) * (K / 32);
    dequantise_mx_kernel<<<static_cast<unsigned>((blocks + 255) / 256), 256, 0, stream>>>(packed, scales, out, rows, K);
    cuda_check(cudaGetLastError());
}

void dequantise(const uint8_t* packed, const uint8_t* scales, float* out, int rows, int K, cudaStream_t stream) {
    check_quant_shape(rows, K);
    if (!packed || !scales || !out) throw std::invalid_argument("nvfp4 dequantise: null pointer");
    const size_t blocks = size_t(rows) * (K / 16);
    dequantise_kernel<<<static_cast<unsigned>((blocks + 255) / 256), 256, 0, stream>>>(packed, scales, out, rows, K);
    cuda_check(cudaGetLastError());
}

}  // namespace nvfp4_b200

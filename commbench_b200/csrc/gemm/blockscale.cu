// Block-scaled fp8 (e4m3) operands: activations carry one fp32 scale per 1 x 128 block
// along K, weights one per 128 x 128 block.  These kernels expand them to bf16 so that the
// bf16 tcgen05 GEMMs (plain and fused) consume them: fp8 halves the bytes that are stored and
// moved, the tensor cores run in bf16.  (The reference's fp8 GEMMs are unscaled:
// datasets/example052_thunderkitten_ag_gemm_fp8_easy/nv/empty_thunderkitten_ag_gemm_fp8.cu:92-122.)
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../prim/pdl.cuh"

namespace cb {
void set_last_error(const std::string& s);

// x [rows, K] e4m3; scale [rows / rb, K / 128] with rb = 1 (activations) or 128 (weights).
__global__ void dequant_blockscaled_kernel(const uint8_t* __restrict__ x,
                                           const float* __restrict__ scale,
                                           __nv_bfloat16* __restrict__ out, long long rows, int K,
                                           int rb) {
  const long long vec_per_row = K / 8;
  const long long total = rows * vec_per_row;
  const int kblocks = K / 128;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = idx / vec_per_row;
    const int v = static_cast<int>(idx % vec_per_row);
    const float s = scale[(r / rb) * kblocks + v / 16];
    const uint2 raw = *reinterpret_cast<const uint2*>(x + r * K + v * 8);
    const __nv_fp8x2_storage_t* p8 = reinterpret_cast<const __nv_fp8x2_storage_t*>(&raw);
    uint4 o;
    __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2(p8[i], __NV_E4M3);
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hr));
      ob[i] = __floats2bfloat162_rn(f.x * s, f.y * s);
    }
    *reinterpret_cast<uint4*>(out + r * K + v * 8) = o;
  }
}

// Biased exponent of the smallest power of two >= s (clamped to the normal range): bump the
// exponent when any mantissa bit is set.
__device__ __forceinline__ uint32_t pow2_ceil_exponent(float s) {
  const uint32_t bits = __float_as_uint(s);
  uint32_t e = (bits >> 23) & 0xffu;
  if ((bits & 0x7fffffu) != 0u) ++e;
  if (e < 1u) e = 1u;
  if (e > 254u) e = 254u;
  return e;
}

// bf16 [rows, K] -> e4m3 + scales (rb = 1: one scale per row and 128 columns; rb = 128: one
// per 128 x 128 block).  One warp per (row block, k block).
//
// pow2 != 0: the scale is rounded UP to a power of two (so that it is exactly representable as an
// 8-bit exponent, "UE8M0", the scale format the tensor cores apply in hardware) and, when
// `sf_bytes` is given, its exponent byte is also written there in the packed layout of the
// block-scaled GEMM: byte (kb % 4) of the 32-bit word [kb / 4][row], `sf_ld` = rows per K group.
// For rb = 128 the byte is replicated to every row of the block (one byte per output column
// of a GEMM and K block).
__global__ void quant_blockscaled_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q,
                                         float* __restrict__ scale, long long rows, int K, int rb,
                                         int pow2, uint8_t* __restrict__ sf_bytes, int sf_ld) {
  const int kblocks = K / 128;
  const long long nblocks = ((rows + rb - 1) / rb) * kblocks;
  const long long w = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= nblocks) return;
  const long long br = w / kblocks;
  const int kb = static_cast<int>(w % kblocks);
  const long long r0 = br * rb;
  const long long r1 = r0 + rb < rows ? r0 + rb : rows;
  float amax = 0.f;
  for (long long r = r0; r < r1; ++r) {
    const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(x + r * K + kb * 128 + lane * 4);
    const __nv_bfloat162 h2 =
        *reinterpret_cast<const __nv_bfloat162*>(x + r * K + kb * 128 + lane * 4 + 2);
    const float2 a = __bfloat1622float2(h), b = __bfloat1622float2(h2);
    amax = fmaxf(amax, fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(b.x), fabsf(b.y))));
  }
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  float s = amax > 0.f ? amax / 448.f : 1.f;
  if (pow2) {
    const uint32_t e = pow2_ceil_exponent(s);
    s = __uint_as_float(e << 23);
    if (sf_bytes != nullptr)
      for (long long r = r0 + lane; r < r1; r += 32)
        sf_bytes[(static_cast<long long>(kb >> 2) * sf_ld + r) * 4 + (kb & 3)] =
            static_cast<uint8_t>(e);
  }
  const float inv = 1.f / s;
  if (lane == 0) scale[br * kblocks + kb] = s;
  for (long long r = r0; r < r1; ++r) {
    const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(x + r * K + kb * 128 + lane * 4);
    const __nv_bfloat162 h2 =
        *reinterpret_cast<const __nv_bfloat162*>(x + r * K + kb * 128 + lane * 4 + 2);
    const float2 a = __bfloat1622float2(h), b = __bfloat1622float2(h2);
    const __nv_fp8x2_storage_t lo =
        __nv_cvt_float2_to_fp8x2(make_float2(a.x * inv, a.y * inv), __NV_SATFINITE, __NV_E4M3);
    const __nv_fp8x2_storage_t hi =
        __nv_cvt_float2_to_fp8x2(make_float2(b.x * inv, b.y * inv), __NV_SATFINITE, __NV_E4M3);
    *reinterpret_cast<uint32_t*>(q + r * K + kb * 128 + lane * 4) =
        static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
  }
}

// Row-block-1 form (activations), bound by memory: x is read once (2 bytes an element), q written
// once (1).  A warp takes kQuantRows rows x 512 columns: 16 lanes of 8 elements hold one 128-column
// block, so the absolute maximum is a four-step shuffle, the row stays in registers between the
// maximum and the conversion, and 2 x kQuantRows 16-byte loads per lane are in flight.  512 columns
// are also the four blocks of one packed scale word, so the word is written whole - missing blocks
// of a ragged K as 127 = 1.0 - instead of byte by byte into a pre-filled array.
// With every lane dividing for its own block the kernel was bound by issue slots (58 us at
// 8192 x 8192): each lane now divides for ONE of the warp's 16 blocks and the factors are
// shuffled back, and the maximum is taken on packed bf16 pairs (exact).  The arithmetic is that of
// quant_blockscaled_kernel, bit for bit.
// Measured at 8192 x 8192 (201 MB): 196 us with one warp per block, 58 us, now 30-34 us (6.0-6.7 TB/s).
static constexpr int kQuantRows = 4;
__global__ void __launch_bounds__(256)
    quant_rows_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q,
                      float* __restrict__ scale, long long rows, int K, int pow2,
                      uint32_t* __restrict__ sf_words, int sf_ld) {
  pdl_launch_dependents();   // the product's set-up overlaps this kernel; it waits for its end
  const int kblocks = K / 128;
  const int kgroups = (kblocks + 3) / 4;
  const long long w = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long long r0 = w / kgroups * kQuantRows;
  const int kg = static_cast<int>(w % kgroups);
  if (r0 >= rows) return;
  // half-warp h holds block 2 i + h of the group in raw[.][i]
  uint4 raw[kQuantRows][2];
#pragma unroll
  for (int u = 0; u < kQuantRows; ++u)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int col = kg * 512 + i * 256 + lane * 8;
      raw[u][i] = (r0 + u < rows && col < K)
                      ? __ldg(reinterpret_cast<const uint4*>(x + (r0 + u) * K + col))
                      : make_uint4(0, 0, 0, 0);
    }
  // lane l of a half keeps the maximum of row (l & 7) / 2, load l & 1
  const int mine = lane & 7;
  __nv_bfloat162 keep = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
  for (int u = 0; u < kQuantRows; ++u)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[u][i]);
      __nv_bfloat162 m = __hmax2(__hmax2(__habs2(h[0]), __habs2(h[1])),
                                 __hmax2(__habs2(h[2]), __habs2(h[3])));
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) m = __hmax2(m, __shfl_xor_sync(0xffffffffu, m, o));
      if (mine == 2 * u + i) keep = m;
    }
  const float2 mf = __bfloat1622float2(keep);
  const float amax = fmaxf(fmaxf(0.f, mf.x), mf.y);
  float s = amax > 0.f ? amax / 448.f : 1.f;
  if (pow2) {
    const uint32_t e = pow2_ceil_exponent(s);
    s = __uint_as_float(e << 23);
    // lane u collects the four exponents of row u: blocks 0 and 2 sit in the lower half
    const int u = lane & 3;
    const uint32_t e0 = __shfl_sync(0xffffffffu, e, 2 * u);
    const uint32_t e1 = __shfl_sync(0xffffffffu, e, 16 + 2 * u);
    const uint32_t e2 = __shfl_sync(0xffffffffu, e, 2 * u + 1);
    const uint32_t e3 = __shfl_sync(0xffffffffu, e, 16 + 2 * u + 1);
    if (sf_words != nullptr && lane < kQuantRows && r0 + u < rows) {
      const int left = kblocks - kg * 4;
      sf_words[static_cast<long long>(kg) * sf_ld + r0 + u] =
          e0 | ((left > 1 ? e1 : 127u) << 8) | ((left > 2 ? e2 : 127u) << 16) |
          ((left > 3 ? e3 : 127u) << 24);
    }
  }
  const float inv = 1.f / s;
  {
    const long long row = r0 + (mine >> 1);
    const int kb = kg * 4 + 2 * (mine & 1) + (lane >> 4);
    if ((lane & 8) == 0 && row < rows && kb < kblocks) scale[row * kblocks + kb] = s;
  }
#pragma unroll
  for (int u = 0; u < kQuantRows; ++u)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int col = kg * 512 + i * 256 + lane * 8;
      const float f = __shfl_sync(0xffffffffu, inv, (lane & 16) + 2 * u + i);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[u][i]);
      uint32_t b[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float2 v0 = __bfloat1622float2(h[2 * j]), v1 = __bfloat1622float2(h[2 * j + 1]);
        const __nv_fp8x2_storage_t lo =
            __nv_cvt_float2_to_fp8x2(make_float2(v0.x * f, v0.y * f), __NV_SATFINITE, __NV_E4M3);
        const __nv_fp8x2_storage_t hi =
            __nv_cvt_float2_to_fp8x2(make_float2(v1.x * f, v1.y * f), __NV_SATFINITE, __NV_E4M3);
        b[j] = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
      }
      if (r0 + u < rows && col < K)
        *reinterpret_cast<uint2*>(q + (r0 + u) * K + col) = make_uint2(b[0], b[1]);
    }
}

// Row-block-1 launches whose pointers allow 16-byte loads and 8-byte stores go to
// quant_rows_kernel; 128 x 128 blocks and other alignments to quant_blockscaled_kernel.
static int launch_quant(const void* x, void* q, void* scale, long long rows, int K, int row_block,
                        int pow2, void* sf_words, int sf_ld, cudaStream_t st) {
  const int threads = 256;
  const bool wide = (reinterpret_cast<uintptr_t>(x) & 15u) == 0 &&
                    (reinterpret_cast<uintptr_t>(q) & 7u) == 0;
  const long long warps =
      row_block == 1 && wide
          ? ((rows + kQuantRows - 1) / kQuantRows) * ((K / 128 + 3) / 4)
          : ((rows + row_block - 1) / row_block) * (K / 128);
  const unsigned blocks = static_cast<unsigned>((warps * 32 + threads - 1) / threads);
  const __nv_bfloat16* xb = static_cast<const __nv_bfloat16*>(x);
  uint8_t* qb = static_cast<uint8_t*>(q);
  float* sb = static_cast<float*>(scale);
  if (row_block == 1 && wide)
    quant_rows_kernel<<<blocks, threads, 0, st>>>(xb, qb, sb, rows, K, pow2,
                                                  static_cast<uint32_t*>(sf_words), sf_ld);
  else
    quant_blockscaled_kernel<<<blocks, threads, 0, st>>>(xb, qb, sb, rows, K, row_block, pow2,
                                                         static_cast<uint8_t*>(sf_words), sf_ld);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace cb

using namespace cb;

extern "C" {

int cb_dequant_blockscaled(const void* x, const void* scale, void* out, long long rows, int K,
                           int row_block, void* stream) {
  if (K % 128 != 0 || (row_block != 1 && row_block != 128)) {
    set_last_error("block scales: K must be a multiple of 128 and row_block 1 or 128");
    return -1;
  }
  dequant_blockscaled_kernel<<<1184, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint8_t*>(x), static_cast<const float*>(scale),
      static_cast<__nv_bfloat16*>(out), rows, K, row_block);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int cb_quant_blockscaled(const void* x, void* q, void* scale, long long rows, int K, int row_block,
                         void* stream) {
  if (K % 128 != 0 || (row_block != 1 && row_block != 128)) {
    set_last_error("block scales: K must be a multiple of 128 and row_block 1 or 128");
    return -1;
  }
  return launch_quant(x, q, scale, rows, K, row_block, 0, nullptr, 0,
                      static_cast<cudaStream_t>(stream));
}

// Same with power-of-two scales; `sf_words` = ceil(K / 512) x sf_rows 32-bit words (sf_rows >=
// rows; pre-filled with 0x7f7f7f7f = 1.0 by the caller) receives the packed exponent bytes (see
// the kernel).  Feeds cb_gemm_fp8_mx.
int cb_quant_blockscaled_pow2(const void* x, void* q, void* scale, void* sf_words, int sf_rows,
                              long long rows, int K, int row_block, void* stream) {
  if (K % 128 != 0 || (row_block != 1 && row_block != 128) || sf_rows < rows) {
    set_last_error("block scales: K % 128 == 0, row_block 1 or 128, sf_rows >= rows");
    return -1;
  }
  return launch_quant(x, q, scale, rows, K, row_block, 1, sf_words, sf_rows,
                      static_cast<cudaStream_t>(stream));
}

}  // extern "C"

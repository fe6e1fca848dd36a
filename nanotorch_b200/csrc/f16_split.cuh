// Operand planes of the fp16 product (gemm_f16.cu): an fp32 matrix as two fp16 numbers per value.
//
// A block of 64 x 64 values has one power-of-two factor 2^e that brings its largest magnitude into [2^14, 2^15), and a value
// y = 2^e x is held as  hi = fp16(y)  and  lo = fp16(2^12 (y - hi)).  fp16 has the significand of TF32, so where hi is a
// normal number (|y| >= 2^-14, down to 2^-28 of the block's largest) hi + 2^-12 lo is y to 2^-22 relative at least, the split
// of tf32_split.cuh; the two 5-bit exponents are what the factor and the 2^12 are for.  Below, the remainder loses a bit per
// factor of two.  Such values are rare -- one in 10^8 of normally distributed ones -- and a block may hold them as long as
// they are not what a row or column is made of: not more than 3 threads' worth (a row of the block is 16 threads, a column
// 8), none below 2^-20 (2^-34 of the largest; its relative error 2^-17).  A block that holds more, that does not come into
// range by a factor of 2^+-60, or that holds an infinity or NaN is `wide`; a matrix with one wide block says so in its
// header, and its products go through TF32 planes (gemm_tc.cu).
//
// Memory: header, then a float 2^-e per block [batch][ceil(R / 64)][Cp / 64], then the planes [hi | lo][batch][R][Cp], Cp = C
// rounded up to 64, padded with zeros.
#pragma once

#include <cuda_fp16.h>

#include <cstdint>

#include "launch.cuh"

namespace ntb {

struct F16Header {
  int wide;          // of the split that finished last
  unsigned int done; // CTAs of a split in progress; zero between them, like `any`
  int any;
};

// Where the parts of a plane set lie.
struct F16Planes {
  F16Header *header;
  float *scale;
  __half *planes; // lo: batch * R * Cp values behind hi
  int64_t RB, CB; // blocks
  int64_t Cp;
  size_t bytes;
};
inline F16Planes f16_planes_at(void *base, int64_t batch, int64_t R, int64_t C) {
  F16Planes p;
  p.RB = ceil_div(R, 64);
  p.CB = ceil_div(C, 64);
  p.Cp = p.CB * 64;
  const size_t scale_bytes = size_t(ceil_div(batch * p.RB * p.CB * 4, 256)) * 256;
  char *b = static_cast<char *>(base);
  p.header = reinterpret_cast<F16Header *>(b);
  p.scale = reinterpret_cast<float *>(b + 256);
  p.planes = reinterpret_cast<__half *>(b + 256 + scale_bytes);
  p.bytes = 256 + scale_bytes + size_t(2 * batch * R * p.Cp) * 2;
  return p;
}

struct F16SplitArgs {
  const float *a, *b; // operands of the op; the split of a matrix that is in memory has `a` alone
  float *out;         // the op's result, dense [R][C]
  __half *hi, *lo;
  float *scale;
  F16Header *header;
  int64_t R, C, Cp, s_r, s_b; // rows, columns, and the row and batch strides of `a` (and of `b`)
  int vec;                    // rows may be read 128 bits at a time
};
struct SplitScaledF { // the matrix itself, or its product with a factor that waits to be applied
  float factor;
  __device__ __forceinline__ float operator()(float x) const { return factor * x; }
};

// f(a) or f(a, b) of a 64 x 128 piece (two blocks) per CTA, written to `out` if OUT, and its planes.  Bound by HBM: 4 bytes
// read and 4 written per value for a split.  A thread has 8 rows of 4 columns, all loads issued before the first use; 16
// lanes share a block's row, so both planes leave in whole 128-byte lines.
template <class F, int NIN, bool OUT> __global__ void __launch_bounds__(256) f16_planes_kernel(F f, F16SplitArgs g) {
  pdl_trigger();
  pdl_wait();
  __shared__ uint32_t top[8][2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, side = lane >> 4;
  const int64_t c = int64_t(blockIdx.x) * 128 + 4 * lane, r0 = int64_t(blockIdx.y) * 64 + warp;
  const bool inside = c < g.Cp; // Cp is a multiple of 64: a group of 4 is inside or outside
  const float *a = g.a + int64_t(blockIdx.z) * g.s_b, *b = NIN == 2 ? g.b + int64_t(blockIdx.z) * g.s_b : nullptr;
  float4 x[8], y[NIN == 2 ? 8 : 1];
  auto load = [&](const float *p) {
    if (g.vec && c + 3 < g.C) return __ldcs(reinterpret_cast<const float4 *>(p));
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c + 0 < g.C) v.x = p[0];
    if (c + 1 < g.C) v.y = p[1];
    if (c + 2 < g.C) v.z = p[2];
    if (c + 3 < g.C) v.w = p[3];
    return v;
  };
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t r = r0 + 8 * i;
    x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (NIN == 2) y[i] = x[i];
    if (r < g.R && inside) {
      x[i] = load(a + r * g.s_r + c);
      if constexpr (NIN == 2) y[i] = load(b + r * g.s_r + c);
    }
  }
  uint32_t m = 0; // largest magnitude, as its bits
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t r = r0 + 8 * i;
    if (r < g.R && inside) {
      if constexpr (NIN == 1) x[i] = make_float4(f(x[i].x), f(x[i].y), f(x[i].z), f(x[i].w));
      else x[i] = make_float4(f(x[i].x, y[i].x), f(x[i].y, y[i].y), f(x[i].z, y[i].z), f(x[i].w, y[i].w));
      if constexpr (OUT) *reinterpret_cast<float4 *>(g.out + r * g.C + c) = x[i]; // dense, aligned, C a multiple of 64
      if constexpr (!OUT) { // what the op makes of the padding
        if (c + 0 >= g.C) x[i].x = 0.f;
        if (c + 1 >= g.C) x[i].y = 0.f;
        if (c + 2 >= g.C) x[i].z = 0.f;
        if (c + 3 >= g.C) x[i].w = 0.f;
      }
      m = max(max(m, max(__float_as_uint(x[i].x) & 0x7fffffffu, __float_as_uint(x[i].y) & 0x7fffffffu)),
              max(__float_as_uint(x[i].z) & 0x7fffffffu, __float_as_uint(x[i].w) & 0x7fffffffu));
    }
  }
#pragma unroll
  for (int s = 8; s > 0; s >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, s));
  if ((lane & 15) == 0) top[warp][side] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) m = max(m, top[w][side]);
  const int wanted = m ? 141 - int(m >> 23) : 0; // 14 - (exponent of the largest)
  const int e = min(max(wanted, -60), 60);
  const float up = __uint_as_float(uint32_t(127 + e) << 23);
  bool wide = m >= 0x7f800000u || wanted < -60, faint = false;
  const int64_t plane = int64_t(blockIdx.z) * g.R * g.Cp;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t r = r0 + 8 * i;
    if (r < g.R && inside) {
      const float v[4] = {x[i].x * up, x[i].y * up, x[i].z * up, x[i].w * up};
      __half h[4], l[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        h[k] = __float2half_rn(v[k]);
        l[k] = __float2half_rn((v[k] - __half2float(h[k])) * 4096.0f);
        const float size = fabsf(v[k]);
        if (size < 0x1p-14f && size != 0.0f) {
          faint = true;
          if (size < 0x1p-20f) wide = true;
        }
      }
      const int64_t at = plane + r * g.Cp + c;
      *reinterpret_cast<uint2 *>(g.hi + at) = make_uint2(uint32_t(__half_as_ushort(h[0])) | uint32_t(__half_as_ushort(h[1])) << 16,
                                                         uint32_t(__half_as_ushort(h[2])) | uint32_t(__half_as_ushort(h[3])) << 16);
      *reinterpret_cast<uint2 *>(g.lo + at) = make_uint2(uint32_t(__half_as_ushort(l[0])) | uint32_t(__half_as_ushort(l[1])) << 16,
                                                         uint32_t(__half_as_ushort(l[2])) | uint32_t(__half_as_ushort(l[3])) << 16);
    }
  }
  if (warp == 0 && (lane & 15) == 0 && inside)
    g.scale[(int64_t(blockIdx.z) * gridDim.y + blockIdx.y) * (g.Cp >> 6) + blockIdx.x * 2 + side] = __uint_as_float(uint32_t(127 - e) << 23);
  const int many = __syncthreads_count(faint);
  const int any = __syncthreads_or(wide) || many > 3;
  if (threadIdx.x == 0) { // the CTA that is last says what the matrix is, and leaves the counters at zero
    if (any) atomicOr(&g.header->any, 1);
    __threadfence();
    if (atomicAdd(&g.header->done, 1u) == gridDim.x * gridDim.y * gridDim.z - 1) {
      g.header->wide = atomicExch(&g.header->any, 0);
      g.header->done = 0;
    }
  }
}

// One launch over the matrix or matrices that `g` describes.
template <class F, int NIN, bool OUT> void launch_f16_planes(F f, const F16SplitArgs &g, int64_t batch) {
  const dim3 grid{unsigned(ceil_div(g.Cp, 128)), unsigned(ceil_div(g.R, 64)), unsigned(batch)};
  launch(f16_planes_kernel<F, NIN, OUT>, grid, 256, 0, f, g);
  check_launch("f16_planes_kernel");
}

} // namespace ntb

// The fp16 product over operand planes (gemm_f16.cu) as the code that owns the planes (gemm_tc.cu) sees it.
#pragma once

#include "f16_split.cuh"
#include "gemm_tf32.cuh"

namespace ntb {

// Factors of an operand's blocks: count_mn blocks along m (or n), s_k elements from one chain of k to the next.
struct F16Scales {
  const float *p;
  int64_t s_batch, s_mn, s_k;
  int count_mn;
  __device__ __forceinline__ const float *at(int batch, int mn, int chain) const {
    return p + batch * s_batch + min(mn, count_mn - 1) * s_mn + chain * s_k;
  }
};
struct F16Operand {
  F16Planes p;
  int64_t R, C; // rows and columns of the planes
  bool mn;      // the columns are m (or n), k goes down the rows
};
inline F16Scales f16_scales(const F16Operand &o) {
  F16Scales s;
  s.p = o.p.scale;
  s.s_batch = o.p.RB * o.p.CB;
  s.s_mn = o.mn ? 1 : o.p.CB;
  s.s_k = o.mn ? o.p.CB : 1;
  s.count_mn = int(o.mn ? o.p.CB : o.p.RB);
  return s;
}
// What the kernel does instead where a header says wide, which only the device knows: every CTA splits its share of both
// operands into TF32 planes, all wait for one another, and the product goes over those.
struct F16Fallback {
  CUtensorMap map_a, map_b; // of the TF32 planes
  TileArgs t;
  NatSplitArgs a, b;
  unsigned int *arrived; // CTAs at the wait; zero between launches
};
// C = A B (+ bias) over planes; `t` as for the kernel over TF32 planes, num_kb aside.
void gemm_f16_launch(const F16Operand &a, const F16Operand &b, TileArgs t, int64_t K, const F16Fallback &f);

} // namespace ntb

// Exact FP32 products on the CUDA cores: three kernels over strided operands, each output accumulated in ascending k
// with one rounding per multiply-add (FUSED) or a rounded product and a rounded sum (the reference's CPU loop).
//
//   sgemm_small<T>  T x T output tiles (T = 64, 32 or 16; 4 x 4, 4 x 2 or 2 x 2 outputs per thread), cp.async into a
//                   4-stage ring of 32-deep k-slices.  What bounds a small product is not arithmetic but how many SMs take part and the
//                   chain of loads each CTA waits for: 256 x 256 x 10 through one 128-wide tile per CTA used 2 SMs
//                   and took 42 us.  With `splits` > 1 a cluster of CTAs shares a tile, each over its own k-range; the
//                   partial tiles meet in distributed shared memory and are added in rank order, so the result
//                   does not depend on timing (one launch, no workspace).
//   sgemm_thin      at most 8 rows: a column per lane, see there.
//   sgemm_large     128 x 256 tiles, 8 x 16 outputs per thread as packed pairs: fma.rn.f32x2 does two IEEE fused
//                   multiply-adds per instruction, which leaves issue slots for loads and moves (a scalar FFMA takes
//                   every slot of its scheduler).  8 x 16 because shared memory feeds registers at 128 bytes a clock:
//                   8 x 8 outputs need 64 bytes per 64 multiply-adds and tie with the arithmetic, 8 x 16 need 96 per 128.
#pragma once

#include <cooperative_groups.h>

#include "cp_async.cuh"
#include "launch.cuh"
#include "nt_core.cuh"

namespace ntb {

struct BatchIndex {
  int ndim;
  int64_t shape[NT_MAX_DIMS];
  int64_t a_strides[NT_MAX_DIMS];
  int64_t b_strides[NT_MAX_DIMS];
};

struct GemmArgs {
  const float *A, *B;
  float *C;
  const float *bias;   // C[m][n] = fl(fl(sum) + bias[n * bias_stride]) when non-null
  int64_t bias_stride;
  int64_t M, N, K;
  int64_t a_sm, a_sk, b_sk, b_sn;
  BatchIndex batch;
  int a_vec, b_vec;    // 16-byte loads along the unit-stride dim are aligned and whole
  int c_vec;           // C rows may be written 128 bits at a time
  int splits;          // small kernel: CTAs of a cluster along k
  int64_t k_per_split;
};

__device__ __forceinline__ void gemm_batch_base(const GemmArgs &g, int64_t lin, const float *&A, const float *&B) {
  for (int d = g.batch.ndim - 1; d >= 0; --d) {
    const int64_t q = lin / g.batch.shape[d];
    const int64_t r = lin - q * g.batch.shape[d];
    lin = q;
    A += r * g.batch.a_strides[d];
    B += r * g.batch.b_strides[d];
  }
}

template <bool FUSED> __device__ __forceinline__ float mad(float a, float b, float c) {
  if constexpr (FUSED) return fmaf(a, b, c);
  else return __fadd_rn(c, __fmul_rn(a, b));
}

// ---------------------------------------------------------------------------------------------
// Small products.  A_K / B_K: the operand's unit-stride dim is k (shared tile [row][k]); otherwise rows run along the
// unit stride (shared tile [k][row]).  A thread owns RM x RN outputs: rows RM ty + i where the tile is [k][row], so that
// one load covers them, and ty + GM i where it is [row][k], so that the 128-bit loads along k of neighbouring threads fall
// into different banks; columns likewise.  What bounds a CTA that has its SM for itself is the shared-memory pipe -- a
// 128-bit load fills 512 bytes of registers, four clocks, also when lanes share the address -- against the latency that
// few warps leave open: per 32-deep slice the 32-wide tile took 1600 clocks with 2 warps of 4 x 4 outputs, 1190 with 4 of
// 4 x 2 and 1000 with 8 of 2 x 2, but the last is 15 % slower once the SMs are full.  So: 64 x 64 with 4 x 4, 32 x 32 with
// 4 x 2, and 16 x 16 with 2 x 2 for products whose chain is all that counts.
constexpr int SG_BK = 32, SG_STAGES = 4;
template <int T, bool K_MAJOR> constexpr int sg_tile_floats = K_MAJOR ? T * (SG_BK + 4) : SG_BK * (T + 4);
template <int T, bool A_K, bool B_K> // the ring; a partial tile of T x T is smaller
constexpr int sg_smem_bytes = SG_STAGES * (sg_tile_floats<T, A_K> + sg_tile_floats<T, B_K>) * 4;
template <int T> constexpr int sg_rm = T == 16 ? 2 : 4; // outputs of a thread: sg_rm x sg_rn
template <int T> constexpr int sg_rn = T == 64 ? 4 : 2;
template <int T> constexpr int sg_threads = (T / sg_rm<T>) * (T / sg_rn<T>);

// R values of an operand at each of 4 k, as v[row][k]
template <int R, int G, int PITCH, bool KM> __device__ __forceinline__ void sg_operands(const float *st, int t, int k, float (&v)[R][4]) {
  if constexpr (KM) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const float4 x = *reinterpret_cast<const float4 *>(st + (t + G * i) * PITCH + k);
      v[i][0] = x.x, v[i][1] = x.y, v[i][2] = x.z, v[i][3] = x.w;
    }
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float *q = st + (k + e) * PITCH + R * t;
      if constexpr (R == 4) {
        const float4 x = *reinterpret_cast<const float4 *>(q);
        v[0][e] = x.x, v[1][e] = x.y, v[2][e] = x.z, v[3][e] = x.w;
      } else {
        const float2 x = *reinterpret_cast<const float2 *>(q);
        v[0][e] = x.x, v[1][e] = x.y;
      }
    }
  }
}

// One thread's copies of an operand's [T rows][SG_BK of k] slices: a first address, uniform steps between the copies of a
// slice, and one between slices.  What lies outside the operand becomes zero.
template <int T, int NT, bool KM> struct SgLoad {
  static constexpr int NV = T * SG_BK / 4 / NT, NS = T * SG_BK / NT; // 16-byte and 4-byte copies per slice
  const float *p, *safe;
  int64_t step;      // between this thread's copies
  int64_t next;      // to the next slice
  int k, k_step;     // k of the first copy inside a slice, and of each further one (0 along rows)
  unsigned rows;     // bit i: copy i's row exists
  int dst, dst_step; // floats
  bool vec;

  __device__ __forceinline__ void init(const float *base, int64_t r0, int64_t R, int64_t s_r, int64_t s_k, bool v, int64_t k0) {
    const int tid = threadIdx.x;
    vec = v;
    safe = base;
    next = SG_BK * s_k;
    const int W = v ? 4 : 1; // values per copy
    int r, r_step;
    if constexpr (KM) {
      r = tid / (SG_BK / W);
      k = (tid % (SG_BK / W)) * W;
      r_step = NT / (SG_BK / W);
      k_step = 0;
      dst = r * (SG_BK + 4) + k;
      dst_step = r_step * (SG_BK + 4);
      step = r_step * s_r;
    } else {
      r = (tid % (T / W)) * W;
      k = tid / (T / W);
      r_step = 0;
      k_step = NT / (T / W);
      dst = k * (T + 4) + r;
      dst_step = k_step * (T + 4);
      step = k_step * s_k;
    }
    rows = 0;
#pragma unroll
    for (int i = 0; i < NS; ++i)
      if (r0 + r + i * r_step < R) rows |= 1u << i;
    p = base + (r0 + r) * s_r + (k0 + k) * s_k;
  }
  __device__ __forceinline__ void fetch(float *st, int left) { // left: values of k that remain, counted from this slice
    const float *q = p;
    float *d = st + dst;
    if (vec) { // the unit-stride extent is a multiple of 4: a group is inside or outside as a whole
#pragma unroll
      for (int i = 0; i < NV; ++i, q += step, d += dst_step) {
        const bool live = (rows >> i & 1) && k + i * k_step < left;
        cp_async16(d, live ? q : safe, live);
      }
    } else {
#pragma unroll 4
      for (int i = 0; i < NS; ++i, q += step, d += dst_step) {
        const bool live = (rows >> i & 1) && k + i * k_step < left;
        cp_async4(d, live ? q : safe, live);
      }
    }
    p += next;
  }
};

template <int T, bool A_K, bool B_K, bool FUSED> __global__ void __launch_bounds__(sg_threads<T>) sgemm_small(GemmArgs g) {
  constexpr int RM = sg_rm<T>, RN = sg_rn<T>, GM = T / RM, GN = T / RN, NT = GM * GN;
  constexpr int AF = sg_tile_floats<T, A_K>, BF = sg_tile_floats<T, B_K>;
  extern __shared__ __align__(16) float sg_smem[];
  const int tid = threadIdx.x, tx = tid % GN, ty = tid / GN;
  const int split = blockIdx.x % g.splits;
  const int64_t n0 = int64_t(blockIdx.x / g.splits) * T, m0 = int64_t(blockIdx.y) * T;
  const float *A = g.A, *B = g.B;
  gemm_batch_base(g, blockIdx.z, A, B);
  const int64_t k_lo = split * g.k_per_split, k_hi = min(g.K, k_lo + g.k_per_split);
  const int depth = k_hi > k_lo ? int(k_hi - k_lo) : 0, steps = (depth + SG_BK - 1) / SG_BK;

  SgLoad<T, NT, A_K> la;
  SgLoad<T, NT, B_K> lb;
  la.init(A, m0, g.M, g.a_sm, g.a_sk, g.a_vec, k_lo);
  lb.init(B, n0, g.N, g.b_sn, g.b_sk, g.b_vec, k_lo);
  auto fetch = [&](int step) {
    if (step < steps) {
      float *st = sg_smem + (step % SG_STAGES) * (AF + BF);
      la.fetch(st, depth - step * SG_BK);
      lb.fetch(st + AF, depth - step * SG_BK);
    }
    cp_async_commit();
  };

  float acc[RM][RN];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < RN; ++j) acc[i][j] = 0.0f;

#pragma unroll
  for (int s = 0; s < SG_STAGES - 1; ++s) fetch(s);
  for (int s = 0; s < steps; ++s) {
    cp_async_wait<SG_STAGES - 2>();
    __syncthreads(); // slice s has landed for everyone, and slice s - 1 has been read by everyone
    fetch(s + SG_STAGES - 1);
    const float *as = sg_smem + (s % SG_STAGES) * (AF + BF), *bs = as + AF;
#pragma unroll
    for (int k = 0; k < SG_BK; k += 4) {
      float a[RM][4], b[RN][4];
      sg_operands<RM, GM, A_K ? SG_BK + 4 : T + 4, A_K>(as, ty, k, a);
      sg_operands<RN, GN, B_K ? SG_BK + 4 : T + 4, B_K>(bs, tx, k, b);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
          for (int j = 0; j < RN; ++j) acc[i][j] = mad<FUSED>(a[i][kk], b[j][kk], acc[i][j]);
    }
  }

  float *C = g.C + int64_t(blockIdx.z) * g.M * g.N;
  auto row = [&](int i) { return A_K ? ty + GM * i : RM * ty + i; };
  auto col = [&](int j) { return B_K ? tx + GN * j : RN * tx + j; };
  if (g.splits == 1) {
#pragma unroll
    for (int i = 0; i < RM; ++i) {
      const int64_t m = m0 + row(i);
      if (m >= g.M) continue;
      if constexpr (!B_K && RN == 4) {
        if (g.c_vec && !g.bias && n0 + 4 * tx < g.N) {
          *reinterpret_cast<float4 *>(C + m * g.N + n0 + 4 * tx) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
          continue;
        }
      }
#pragma unroll
      for (int j = 0; j < RN; ++j) {
        const int64_t n = n0 + col(j);
        if (n < g.N) C[m * g.N + n] = g.bias ? acc[i][j] + __ldg(g.bias + n * g.bias_stride) : acc[i][j];
      }
    }
    return;
  }
  // the cluster's partial tiles, added in rank order; each CTA finishes its share of the tile
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __syncthreads(); // the ring is free
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < RN; ++j) sg_smem[row(i) * T + col(j)] = acc[i][j];
  cluster.sync();
  const float *part[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) part[r] = cluster.map_shared_rank(sg_smem, r < g.splits ? r : 0);
  for (int e = split * NT + tid; e < T * T; e += NT * g.splits) {
    const int64_t m = m0 + e / T, n = n0 + e % T;
    if (m >= g.M || n >= g.N) continue;
    float v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = r < g.splits ? part[r][e] : 0.0f;
    float sum = v[0];
#pragma unroll
    for (int r = 1; r < 8; ++r)
      if (r < g.splits) sum += v[r];
    C[m * g.N + n] = g.bias ? sum + __ldg(g.bias + n * g.bias_stride) : sum;
  }
  cluster.sync(); // nobody leaves while its tile is being read
}

// ---------------------------------------------------------------------------------------------
// A few rows (M <= 8) times a row-major matrix: a prediction for one sample or a handful.  A CTA owns 32 columns and
// keeps up to TH_STAGES slices of 64 k on their way; warp w multiplies rows w and w + 4, a column per lane: a chain of
// one multiply-add per k and row, which is what bounds it.  (The 32 x 32 tiles spend 31 of 32 rows on nothing.)  Four warps
// of their own start the copies: by the multiplying warps, the copies of a slice, some 30 instructions with their addresses,
// came between its multiply-adds (1 x 4096 x 512 28.9 us, now 22.6; 1 x 784 x 256 7.0 / 6.5; 8 x 2000 x 100 21.2 / 17.3).
constexpr int TH_M = 8, TH_N = 32, TH_BK = 64, TH_STAGES = 10, TH_NT = 256, TH_COPY = 128;
constexpr int TH_STAGE = TH_BK * (TH_N + TH_M); // floats: [k][32] of B, then [row][64] of A
constexpr int TH_SMEM = TH_STAGES * TH_STAGE * 4;

// FOUR: M <= 4
template <bool FUSED, bool FOUR> __global__ void __launch_bounds__(TH_NT) sgemm_thin(GemmArgs g) {
  pdl_wait();
  extern __shared__ __align__(16) float th_smem[];
  const bool copies = threadIdx.x >= TH_NT - TH_COPY;
  const int tid = threadIdx.x % TH_COPY, lane = tid & 31, warp = tid >> 5;
  const int64_t n0 = int64_t(blockIdx.x) * TH_N;
  const float *A = g.A, *B = g.B;
  gemm_batch_base(g, blockIdx.z, A, B);
  const int steps = int((g.K + TH_BK - 1) / TH_BK);
  // copies of B: rows kb, kb + kb_step, ... of a slice, 16 bytes (or single values) each; of A: k = tid % 64 of every
  // second row
  const int W = g.b_vec ? 4 : 1, kb = tid / (TH_N / W), nb = (tid % (TH_N / W)) * W, kb_step = TH_COPY / (TH_N / W);
  const bool nb_in = n0 + nb < g.N;
  const float *pb = B + kb * g.b_sk + n0 + nb, *pa = A + (tid / TH_BK) * g.a_sm + (tid % TH_BK) * g.a_sk;
  const int64_t b_step = kb_step * g.b_sk, b_next = TH_BK * g.b_sk, a_next = TH_BK * g.a_sk;
  auto fetch = [&](int s) {
    if (s < steps) {
      float *st = th_smem + (s % TH_STAGES) * TH_STAGE;
      const int left = int(min(g.K - int64_t(s) * TH_BK, int64_t(TH_BK)));
      const float *q = pb;
      float *d = st + kb * TH_N + nb;
      if (W == 4) {
#pragma unroll
        for (int i = 0; i < TH_BK * TH_N / 4 / TH_COPY; ++i, q += b_step, d += kb_step * TH_N) {
          const bool live = nb_in && kb + i * kb_step < left;
          cp_async16(d, live ? q : B, live);
        }
      } else {
#pragma unroll 4
        for (int i = 0; i < TH_BK * TH_N / TH_COPY; ++i, q += b_step, d += kb_step * TH_N) {
          const bool live = nb_in && kb + i * kb_step < left;
          cp_async4(d, live ? q : B, live);
        }
      }
      const float *qa = pa;
      for (int m = tid / TH_BK; m < g.M; m += TH_COPY / TH_BK, qa += (TH_COPY / TH_BK) * g.a_sm) {
        const bool live = tid % TH_BK < left;
        cp_async4(st + TH_BK * TH_N + m * TH_BK + tid % TH_BK, live ? qa : A, live);
      }
      pb += b_next;
      pa += a_next;
    }
    cp_async_commit();
  };
  float acc[2] = {0.0f, 0.0f};
  if (copies)
    for (int s = 0; s < TH_STAGES - 1; ++s) fetch(s);
  for (int s = 0; s < steps; ++s) {
    cp_async_wait<TH_STAGES - 2>();
    __syncthreads(); // slice s has landed for everyone, slice s - 1 has been read by everyone
    if (copies) {
      fetch(s + TH_STAGES - 1);
      continue;
    }
    const float *bs = th_smem + (s % TH_STAGES) * TH_STAGE + lane, *as = th_smem + (s % TH_STAGES) * TH_STAGE + TH_BK * TH_N + warp * TH_BK;
    if (warp < g.M) {
      // 16 values of k at a time, the next 16 on their way while these multiply
      float b[2][16], r0[2][16], r1[2][16];
      auto operands = [&](int to, int k) {
#pragma unroll
        for (int e = 0; e < 16; ++e) b[to][e] = bs[(k + e) * TH_N];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          *reinterpret_cast<float4 *>(&r0[to][4 * e]) = *reinterpret_cast<const float4 *>(as + k + 4 * e);
          if constexpr (!FOUR) *reinterpret_cast<float4 *>(&r1[to][4 * e]) = *reinterpret_cast<const float4 *>(as + 4 * TH_BK + k + 4 * e);
        }
      };
      operands(0, 0);
#pragma unroll
      for (int k = 0; k < TH_BK; k += 16) {
        const int cur = (k >> 4) & 1;
        if (k + 16 < TH_BK) operands(cur ^ 1, k + 16);
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          acc[0] = mad<FUSED>(r0[cur][e], b[cur][e], acc[0]);
          if constexpr (!FOUR) acc[1] = mad<FUSED>(r1[cur][e], b[cur][e], acc[1]); // without a row: what lies in its slot, unused
        }
      }
    }
  }
  if (copies) return;
  const int64_t n = n0 + lane;
  float *C = g.C + int64_t(blockIdx.z) * g.M * g.N;
#pragma unroll
  for (int h = 0; h < (FOUR ? 1 : 2); ++h) {
    const int64_t m = warp + 4 * h;
    if (m < g.M && n < g.N) C[m * g.N + n] = g.bias ? acc[h] + __ldg(g.bias + n * g.bias_stride) : acc[h];
  }
}

// ---------------------------------------------------------------------------------------------
// Large products: 128 x 256 tiles, 256 threads of 8 x 16 outputs.
constexpr int LG_M = 128, LG_N = 256, LG_BK = 8, LG_NT = 256, LG_STAGES = 4;
constexpr int LG_AP = LG_M + 4, LG_BP = LG_N + 4; // pitches of the shared rows [k][m|n], in floats
constexpr int LG_SMEM = LG_STAGES * LG_BK * (LG_AP + LG_BP) * 4;

using f32x2 = unsigned long long;
template <bool FUSED> __device__ __forceinline__ void mad2(f32x2 &c, f32x2 a, f32x2 b) {
  if constexpr (FUSED) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
  } else { // as scalars: results of a packed multiply and a packed add did not have the bits of two roundings
    float x, y, a0, a1, b0, b1;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(c));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a0), "=f"(a1) : "l"(a));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(b0), "=f"(b1) : "l"(b));
    x = __fadd_rn(x, __fmul_rn(a0, b0));
    y = __fadd_rn(y, __fmul_rn(a1, b1));
    asm("mov.b64 %0, {%1, %2};" : "=l"(c) : "f"(x), "f"(y));
  }
}
__device__ __forceinline__ f32x2 twice(float x) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}

// A [R rows][8 k] slice into shared rows [k][row]: 16 bytes at a time along aligned rows, else value by value (along k,
// a lane per k, where that is the unit stride).  What lies outside the operand is zero.
template <int R, bool K_MAJOR>
__device__ __forceinline__ void lg_load(float *st, const float *base, int64_t s_r, int64_t s_k, int64_t rows, bool vec, int64_t k0, int64_t K) {
  constexpr int P = R + 4;
  const int tid = threadIdx.x;
  if (!K_MAJOR && vec) {
#pragma unroll
    for (int i = 0; i < R / 128; ++i) {
      const int v = tid + 256 * i, r = (v * 4) % R, k = (v * 4) / R;
      const bool live = r < rows && k0 + k < K;
      cp_async16(st + k * P + r, live ? base + r + (k0 + k) * s_k : base, live);
    }
  } else {
#pragma unroll
    for (int i = 0; i < R / 32; ++i) {
      const int v = tid + 256 * i;
      const int r = K_MAJOR ? v / LG_BK : v % R, k = K_MAJOR ? v % LG_BK : v / R;
      const bool live = r < rows && k0 + k < K;
      cp_async4(st + k * P + r, live ? base + r * s_r + (k0 + k) * s_k : base, live);
    }
  }
}

// Two warps per scheduler is all that 8 x 16 outputs leave registers for, so latencies are covered inside a warp: the
// operands of step k + 1 are loaded while step k multiplies, and slices arrive by cp.async three steps ahead.
template <bool A_K, bool B_K, bool FUSED> __global__ void __launch_bounds__(LG_NT, 1) sgemm_large(GemmArgs g) {
  extern __shared__ __align__(16) float lg_smem[];
  constexpr int AF = LG_BK * LG_AP, SF = LG_BK * (LG_AP + LG_BP); // floats of A's part and of a stage
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int64_t m0 = int64_t(blockIdx.y) * LG_M, n0 = int64_t(blockIdx.x) * LG_N;
  const float *A = g.A, *B = g.B;
  gemm_batch_base(g, blockIdx.z, A, B);
  A += m0 * g.a_sm;
  B += n0 * g.b_sn;
  const int steps = int((g.K + LG_BK - 1) / LG_BK);
  auto fetch = [&](int s) {
    if (s < steps) {
      float *st = lg_smem + (s % LG_STAGES) * SF;
      lg_load<LG_M, A_K>(st, A, g.a_sm, g.a_sk, g.M - m0, g.a_vec, int64_t(s) * LG_BK, g.K);
      lg_load<LG_N, B_K>(st + AF, B, g.b_sn, g.b_sk, g.N - n0, g.b_vec, int64_t(s) * LG_BK, g.K);
    }
    cp_async_commit();
  };
  // rows {4 ty .. + 3, 64 + 4 ty .. + 3}; columns 64 h + 4 tx .. + 3 for h = 0 .. 3, as pairs
  f32x2 acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
  float4 a[2][2];
  ulonglong2 b[2][4];
  auto operands = [&](int to, int s, int k) {
    const float *st = lg_smem + (s % LG_STAGES) * SF;
#pragma unroll
    for (int h = 0; h < 2; ++h) a[to][h] = *reinterpret_cast<const float4 *>(st + k * LG_AP + 64 * h + 4 * ty);
#pragma unroll
    for (int h = 0; h < 4; ++h) b[to][h] = *reinterpret_cast<const ulonglong2 *>(st + AF + k * LG_BP + 64 * h + 4 * tx);
  };

#pragma unroll
  for (int s = 0; s < LG_STAGES - 1; ++s) fetch(s);
  cp_async_wait<LG_STAGES - 2>();
  __syncthreads();
  operands(0, 0, 0);
  for (int s = 0; s < steps; ++s) {
#pragma unroll
    for (int k = 0; k < LG_BK; ++k) {
      const int cur = k & 1;
      if (k == 0) fetch(s + LG_STAGES - 1); // into the slot that every warp left before the last barrier
      if (k < LG_BK - 1) {
        operands(cur ^ 1, s, k + 1);
      } else { // the first operands of the next slice (of a stale slot after the last one, unused)
        cp_async_wait<LG_STAGES - 2>();
        __syncthreads();
        operands(cur ^ 1, s + 1, 0);
      }
      const f32x2 bb[8] = {b[cur][0].x, b[cur][0].y, b[cur][1].x, b[cur][1].y, b[cur][2].x, b[cur][2].y, b[cur][3].x, b[cur][3].y};
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float aa[4] = {a[cur][h].x, a[cur][h].y, a[cur][h].z, a[cur][h].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const f32x2 pair = twice(aa[i]);
#pragma unroll
          for (int j = 0; j < 8; ++j) mad2<FUSED>(acc[4 * h + i][j], pair, bb[j]);
        }
      }
    }
  }

  float *C = g.C + int64_t(blockIdx.z) * g.M * g.N;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t m = m0 + (i < 4 ? 4 * ty + i : 64 + 4 * ty + i - 4);
    if (m >= g.M) continue;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int64_t n = n0 + 64 * h + 4 * tx;
      float v[4];
      *reinterpret_cast<f32x2 *>(v) = acc[i][2 * h];
      *reinterpret_cast<f32x2 *>(v + 2) = acc[i][2 * h + 1];
      float *dst = C + m * g.N + n;
      if (g.c_vec && !g.bias && n < g.N) {
        *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (n + e < g.N) dst[e] = g.bias ? v[e] + __ldg(g.bias + (n + e) * g.bias_stride) : v[e];
      }
    }
  }
}

} // namespace ntb

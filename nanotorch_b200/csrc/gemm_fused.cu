// 3xTF32 products of small and middle size on the tensor cores, without operand planes.
//
// The plane-fed kernel of gemm_tc.cu is built for products of many 128 x 256 tiles: each operand is split into TF32
// planes by a launch of its own and a tile then streams 48 KB per 16 values of k.  A product of a few tiles leaves most
// SMs idle for the length of the whole contraction (256 x 784 x 256: two CTAs, 34 us, and 4 us for the splits).  Here
//   - producer warps read the fp32 operands in place (any strides), split them in registers and write hi and lo
//     into K-major, 128-byte-swizzled shared tiles: one launch, no planes, and no transpose anywhere else;
//   - the tile is 128 x BN with BN = 32, 64 or 128, so that there are tiles for more SMs;
//   - the contraction is shared out in its 256-deep accumulation chains ("periods"): with fewer tiles than SMs a
//     cluster of up to 8 CTAs takes one period each, the period sums meet in distributed shared memory and are added in
//     period order.
// Per output the sequence of tensor-core instructions and of fp32 additions is that of the plane-fed kernel -- the
// periods, their order, and the k-parts of its split-K -- so the bits of the result do not depend on which of the two
// kernels ran.
//
// What bounds it: the producers.  A 32-deep block of a 128 x BN tile takes 0.72 / 0.87 / 1.5 us for BN = 32 / 64 / 128
// (loads, splits, (128 + BN) * 256 bytes of shared-memory stores); with the tensor-core instructions left out it took
// 3 % less.  256 x 784 x 256: 15 us (34 + 4 for the splits through planes); 784 x 256 x 256: 11.5 (16 + 4); 100 x 2000 x 60:
// 17 (40 + 4).  From one full wave of tiles on, planes pay off again (1024^3: 38 against 35 + 5).
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "gemm_common.cuh"
#include "launch.cuh"
#include "nt_core.cuh"
#include "tf32_split.cuh"
#include "tma.cuh"

namespace ntb {

constexpr int FG_BM = 128, FG_BK = 32;
template <int BN> constexpr int fg_stages = BN == 32 ? 4 : 3;
constexpr int FG_PERIOD_BLOCKS = TC_PERIOD / FG_BK;         // 8 blocks of 32
template <int BN> constexpr int fg_epi_warps = BN == 128 ? 8 : 4;
constexpr int FG_PRODUCERS = 256; // threads, in two groups
template <int BN> constexpr int fg_threads = fg_epi_warps<BN> * 32 + FG_PRODUCERS + 32;
template <int BN> constexpr uint32_t fg_stage_bytes = (FG_BM + BN) * FG_BK * 4 * 2; // hi and lo of both operands
template <int BN> constexpr uint32_t fg_part_bytes = FG_BM * (BN + 4) * 4;          // a period's tile, for the cluster
template <int BN> constexpr uint32_t fg_ring_bytes = fg_stages<BN> * fg_stage_bytes<BN> + 1024 /*align*/ + 256 /*barriers*/;

struct FgOperand {
  const float *p;
  int64_t rows;         // M or N
  int64_t s_r, s_k, s_b; // element strides
  int k_vec;            // unit stride along k, 16-byte loads aligned and whole
  int k_unit;           // unit stride along k
};
struct FgArgs {
  FgOperand a, b;
  float *C;
  const float *bias;
  int64_t bias_stride;
  int64_t M, N, K;
  int periods, part_periods; // chains along k; chains per k-part (the parts' sums are added in order)
  int csize;                 // CTAs of a cluster: they take the periods in turn
  int part_buf;              // the buffer behind the ring exists
  int c_vec;
  int *error_flag;
  long long wait_limit;
};

// K-major operand tile, rows of 128 bytes (32 fp32) in the 128-byte swizzle: 8-row groups of 1024 bytes; layout type 2.
__device__ __forceinline__ uint64_t fg_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= uint64_t((smem_addr & 0x3FFFF) >> 4);
  d |= uint64_t(1) << 16;
  d |= uint64_t(1024 >> 4) << 32;
  d |= uint64_t(1) << 46;
  d |= uint64_t(2) << 61;
  return d;
}

// A producer thread's share of a [R rows][32 k] block: N = 8 R / NP groups of 4 values along k.  Where k is the unit
// stride (K_UNIT) eight lanes read the 128 bytes of a row and a thread's groups lie NP / 8 rows apart; otherwise lanes run
// along the rows, each value is a load of its own and a thread's groups lie along k.  Two groups of producers take the
// blocks in turn, each holding its next block's values in registers while they arrive: a block's loads, splits, stores
// and fence follow one another in a warp, and with every warp in the same phase they added up (1640 clocks per block of
// 160 rows).  All addresses are one pointer and uniform steps: index arithmetic written out per load took 2300.
template <int R, int NP> struct FgShare {
  static constexpr int N = 8 * R / NP;
  const float *p;  // first group: row, k of block 0 of the period
  int64_t step;    // elements between groups
  int64_t s_k;
  int k;           // first group's k inside a block
  unsigned rows;   // bit i: group i's row exists
  uint32_t at;     // byte offset of the first group in a swizzled tile
  int row7;        // its row modulo 8
  bool k_unit, k_vec;

  __device__ __forceinline__ void init(const FgOperand &o, const float *base, int64_t r0, int64_t k0, int t) {
    k_unit = o.k_unit;
    k_vec = o.k_vec;
    s_k = o.s_k;
    const int r = k_unit ? t / 8 : t % R;
    k = (k_unit ? t % 8 : t / R) * 4;
    p = base + (r0 + r) * o.s_r + (k0 + k) * o.s_k;
    step = k_unit ? (NP / 8) * o.s_r : (4 * NP / R) * o.s_k;
    rows = 0;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (r0 + r + (k_unit ? i * (NP / 8) : 0) < o.rows) rows |= 1u << i;
    row7 = r & 7;
    at = uint32_t(r * 128 + (((k >> 2) ^ row7) << 4));
  }
  // loads the block whose first k is 0 of `left` values that remain, and moves on by `blocks` blocks
  __device__ __forceinline__ void fetch(int left, int blocks, float4 (&v)[N]) {
    const float *q = p;
#pragma unroll
    for (int i = 0; i < N; ++i, q += step) {
      v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      const int here = (rows >> i & 1) ? left - (k_unit ? k : k + i * (4 * NP / R)) : 0;
      if (k_vec) { // left is a multiple of 4
        if (here > 0) v[i] = __ldg(reinterpret_cast<const float4 *>(q));
      } else {
        if (here > 0) v[i].x = __ldg(q);
        if (here > 1) v[i].y = __ldg(q + s_k);
        if (here > 2) v[i].z = __ldg(q + 2 * s_k);
        if (here > 3) v[i].w = __ldg(q + 3 * s_k);
      }
    }
    p += int64_t(blocks) * FG_BK * s_k;
  }
  __device__ __forceinline__ uint32_t offset(int i) const {
    return k_unit ? at + uint32_t(i * (NP / 8) * 128) : (at & ~127u) | uint32_t((((k >> 2) + i * (NP / R)) ^ row7) << 4);
  }
};
// hi and lo of tf32_split.cuh in integer arithmetic -- cvt.rna.tf32 runs at a fraction of the rate, and two per value
// would be most of a producer's time.  Values whose rounding could overflow, and what is not finite, take the originals.
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void split4(float4 x, float4 &h, float4 &l) {
  const float top = max_nan(max_nan(fabsf(x.x), fabsf(x.y)), max_nan(fabsf(x.z), fabsf(x.w)));
  if (!(top < __uint_as_float(0x7f7ff000u))) {
    h = make_float4(split_hi(x.x), split_hi(x.y), split_hi(x.z), split_hi(x.w));
    l = make_float4(split_lo(x.x, h.x), split_lo(x.y, h.y), split_lo(x.z, h.z), split_lo(x.w, h.w));
    return;
  }
  auto rna = [](float v) { return __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xffffe000u); };
  h = make_float4(rna(x.x), rna(x.y), rna(x.z), rna(x.w));
  l = make_float4(rna(x.x - h.x), rna(x.y - h.y), rna(x.z - h.z), rna(x.w - h.w));
}
template <int R, int NP>
__device__ __forceinline__ void fg_split(const FgShare<R, NP> &o, const float4 (&v)[FgShare<R, NP>::N], char *hi, char *lo) {
#pragma unroll
  for (int i = 0; i < FgShare<R, NP>::N; ++i) {
    float4 h, l;
    split4(v[i], h, l);
    const uint32_t at = o.offset(i);
    *reinterpret_cast<float4 *>(hi + at) = h;
    *reinterpret_cast<float4 *>(lo + at) = l;
  }
}

// CLUSTER: g.csize > 1.  The [128][BN + 4] buffer behind the ring holds a period's tile for the cluster, or -- one CTA
// per tile, contraction in several k-parts -- the sum of the finished parts; g.part_buf says whether it is there.
template <int BN, bool CLUSTER> __global__ void __launch_bounds__(fg_threads<BN>, 1) gemm_fused_split(FgArgs g) {
  namespace cg = cooperative_groups;
  constexpr int EW = fg_epi_warps<BN>, CW = BN / (EW / 4); // epilogue warps; columns of an epilogue thread
  constexpr int NP = FG_PRODUCERS / 2, STAGES = fg_stages<BN>; // threads of a producer group
  constexpr uint32_t A_PLANE = FG_BM * FG_BK * 4, B_PLANE = BN * FG_BK * 4;
  constexpr uint32_t IDESC = (1u << 4) | (2u << 7) | (2u << 10) | (uint32_t(BN >> 3) << 17) | (uint32_t(FG_BM >> 4) << 24);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  char *ring = reinterpret_cast<char *>(smem_raw + (smem_base - smem_u32(smem_raw)));
  const uint32_t part_off = STAGES * fg_stage_bytes<BN>;
  float *part = reinterpret_cast<float *>(ring + part_off); 
  const uint32_t bar_off = part_off + (g.part_buf ? fg_part_bytes<BN> : 0u);
  const uint32_t bar = smem_base + bar_off;
  // full[s] at +8 s, empty[s] at +32 + 8 s, acc_full[b] at +64 + 8 b, acc_empty[b] at +80 + 8 b, tmem slot at +96
  const uint32_t full0 = bar, empty0 = bar + 32, acc_full0 = bar + 64, acc_empty0 = bar + 80;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(ring + bar_off + 96);
  volatile int *poison_slot = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int rank = CLUSTER ? int(blockIdx.x % unsigned(g.csize)) : 0;
  const int64_t n0 = int64_t(blockIdx.x / unsigned(g.csize)) * BN, m0 = int64_t(blockIdx.y) * FG_BM;
  const int rounds = (g.periods + g.csize - 1) / g.csize;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full0 + 8 * s, NP / 32);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(acc_full0 + 8 * i, 1);
      mbar_init(acc_empty0 + 8 * i, EW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *poison_slot = *reinterpret_cast<volatile int *>(g.error_flag); // an earlier wait ran out: do nothing, see gemm_tc.cu
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * BN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_acc = __shfl_sync(0xffffffffu, *tmem_slot, 0); // uniform, and the compiler knows
  const bool poisoned = *poison_slot != 0;

  // blocks of 32 k in period p
  auto blocks_of = [&](int p) {
    const int64_t k = g.K - int64_t(p) * TC_PERIOD;
    return int(k >= TC_PERIOD ? FG_PERIOD_BLOCKS : (k + FG_BK - 1) / FG_BK);
  };
  bool ok = !poisoned;
  // Every thread passes the cluster's two barriers of a round, whatever became of its role: after the first the round's
  // tiles can be read, after the second they may be written again (and nobody leaves while its tile is being read).
  auto cluster_barrier = [&] {
    if constexpr (CLUSTER) {
      __syncwarp();
      cg::this_cluster().sync();
    }
  };

  if (warp >= EW && warp < EW + FG_PRODUCERS / 32) {
    // ------------------------------------------------------------------ producers
    const int t = (int(threadIdx.x) - EW * 32) % NP, group = (int(threadIdx.x) - EW * 32) / NP;
    const float *A = g.a.p + int64_t(blockIdx.z) * g.a.s_b, *B = g.b.p + int64_t(blockIdx.z) * g.b.s_b;
    int done = 0; // blocks of the rounds before: they take the stages in turn
    for (int round = 0; round < rounds; ++round) {
      const int p = round * g.csize + rank;
      const int nblk = p < g.periods ? blocks_of(p) : 0;
      const int64_t kp = int64_t(p) * TC_PERIOD;
      if (nblk && ok) {
        FgShare<FG_BM, NP> sa;
        FgShare<BN, NP> sb;
        sa.init(g.a, A, m0, kp + group * FG_BK, t);
        sb.init(g.b, B, n0, kp + group * FG_BK, t);
        int left = int(min(g.K - kp, int64_t(TC_PERIOD))) - group * FG_BK;
        float4 va[FgShare<FG_BM, NP>::N], vb[FgShare<BN, NP>::N];
        if (group < nblk) {
          sa.fetch(left, 2, va);
          sb.fetch(left, 2, vb);
        }
        for (int blk = group; blk < nblk; blk += 2) {
          const int s = (done + blk) % STAGES;
          ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, ((done + blk) / STAGES & 1) ^ 1, g.wait_limit));
          if (!ok) {
            atomicExch(g.error_flag, 1);
            break;
          }
          char *st = ring + s * fg_stage_bytes<BN>;
          fg_split(sa, va, st, st + A_PLANE);
          fg_split(sb, vb, st + 2 * A_PLANE, st + 2 * A_PLANE + B_PLANE);
          left -= 2 * FG_BK;
          if (blk + 2 < nblk) {
            sa.fetch(left, 2, va);
            sb.fetch(left, 2, vb);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(full0 + 8 * s);
        }
      }
      done += nblk;
      cluster_barrier();
      cluster_barrier();
    }
  } else if (warp == EW + FG_PRODUCERS / 32) {
    // ------------------------------------------------------------------ MMA issuer
    const uint32_t lead = elect_lane();
    int s = 0;
    uint32_t phase = 0;
    for (int round = 0; round < rounds; ++round) {
      const int p = round * g.csize + rank, buf = round & 1;
      const int nblk = p < g.periods ? blocks_of(p) : 0;
      if (nblk && ok) {
        if (!mbar_wait(acc_empty0 + 8 * buf, ((round >> 1) & 1) ^ 1, g.wait_limit)) {
          if (lead) atomicExch(g.error_flag, 4);
          ok = false;
        }
        tcgen05_fence_after();
        const uint32_t d = tmem_acc + uint32_t(buf * BN);
        bool first = true;
        for (int blk = 0; blk < nblk && ok; ++blk) {
          if (!mbar_wait(full0 + 8 * s, phase, g.wait_limit)) {
            if (lead) atomicExch(g.error_flag, 2);
            ok = false;
            break;
          }
          tcgen05_fence_after();
          const uint32_t st = smem_base + uint32_t(s) * fg_stage_bytes<BN>;
#pragma unroll
          for (int ks = 0; ks < FG_BK / 8; ++ks) {
            const uint32_t pa = st + ks * 32u, pb = st + 2 * A_PLANE + ks * 32u;
            const uint64_t a_hi = fg_desc(pa), a_lo = fg_desc(pa + A_PLANE), b_hi = fg_desc(pb), b_lo = fg_desc(pb + B_PLANE);
            umma_tf32_idesc(d, a_hi, b_lo, IDESC, first ? 0u : 1u, lead); // small terms first, the large one last
            umma_tf32_idesc(d, a_lo, b_hi, IDESC, 1, lead);
            umma_tf32_idesc(d, a_hi, b_hi, IDESC, 1, lead);
            first = false;
          }
          umma_commit(empty0 + 8 * s, lead);
          if (++s == STAGES) {
            s = 0;
            phase ^= 1;
          }
        }
        if (ok) umma_commit(acc_full0 + 8 * buf, lead);
        else if (lead) mbar_arrive(acc_full0 + 8 * buf); // release the epilogue
      }
      cluster_barrier();
      cluster_barrier();
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    // cur: the running part's sums -- of a row's CW columns, or of this CTA's slice of the tile; total, for a slice: the
    // finished parts'
    constexpr int SL = CLUSTER ? FG_BM * BN / 2 / (EW * 32) : CW; // values per thread (a slice's at most)
    const int quad = warp & 3, col0 = (warp >> 2) * CW;
    float cur[SL], total[CLUSTER ? SL : 1];
#pragma unroll
    for (int i = 0; i < SL; ++i) cur[i] = 0.0f;
#pragma unroll
    for (int i = 0; i < (CLUSTER ? SL : 1); ++i) total[i] = 0.0f;
    for (int round = 0; round < rounds; ++round) {
      const int p = round * g.csize + rank, buf = round & 1;
      const int nblk = p < g.periods ? blocks_of(p) : 0;
      if (nblk && ok) {
        ok = __all_sync(0xffffffffu, mbar_wait(acc_full0 + 8 * buf, (round >> 1) & 1, g.wait_limit));
        if (!ok) atomicExch(g.error_flag, 3);
        ok = __all_sync(0xffffffffu, ok && *reinterpret_cast<volatile int *>(g.error_flag) == 0);
      }
      if (nblk && ok) {
        tcgen05_fence_after();
        const uint32_t taddr = tmem_acc + (uint32_t(quad * 32) << 16) + uint32_t(buf * BN + col0);
        float *row = part + (quad * 32 + lane) * (BN + 4) + col0;
#pragma unroll
        for (int c = 0; c < CW / 32; ++c) {
          uint32_t v[32];
          tmem_ld32(taddr + uint32_t(c * 32), v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if constexpr (CLUSTER) {
#pragma unroll
            for (int q = 0; q < 8; ++q)
              *reinterpret_cast<float4 *>(row + c * 32 + 4 * q) = make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]),
                                                                              __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3]));
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) cur[c * 32 + e] = cur[c * 32 + e] + __uint_as_float(v[e]);
          }
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty0 + 8 * buf);
        if constexpr (!CLUSTER) {
          if (g.part_buf && (p + 1 == g.periods || (p + 1) % g.part_periods == 0)) { // a k-part is complete
            if (p >= g.part_periods) {
#pragma unroll
              for (int i = 0; i < CW; ++i) cur[i] = row[i] + cur[i];
            }
            if (p + 1 < g.periods) {
#pragma unroll
              for (int i = 0; i < CW; ++i) {
                row[i] = cur[i];
                cur[i] = 0.0f;
              }
            }
          }
        }
      }
      cluster_barrier();
      if constexpr (CLUSTER) { // this round's periods, added in period order to the slice of the tile that this CTA owns
        const int here = min(g.csize, g.periods - round * g.csize);
        const int rows = FG_BM / g.csize; // csize is a power of two
        for (int q = 0; q < here; ++q) {
          const float *tile = cg::this_cluster().map_shared_rank(part, unsigned(q));
          const int at = round * g.csize + q;
          const bool part_ends = at + 1 == g.periods || (at + 1) % g.part_periods == 0, first_part = at < g.part_periods;
#pragma unroll
          for (int i = 0; i < SL; ++i) {
            const int e = int(threadIdx.x) + i * EW * 32;
            const int r = e / BN, c = e % BN;
            if (r < rows) {
              cur[i] = cur[i] + tile[(rank * rows + r) * (BN + 4) + c];
              if (part_ends) {
                total[i] = first_part ? cur[i] : total[i] + cur[i];
                cur[i] = 0.0f;
              }
            }
          }
        }
      }
      cluster_barrier();
    }

    ok = ok && *reinterpret_cast<volatile int *>(g.error_flag) == 0;
    float *C = g.C + int64_t(blockIdx.z) * g.M * g.N;
    if constexpr (CLUSTER) {
      const int rows = FG_BM / g.csize;
#pragma unroll
      for (int i = 0; i < SL; ++i) {
        const int e = int(threadIdx.x) + i * EW * 32;
        const int64_t m = m0 + rank * rows + e / BN, n = n0 + e % BN;
        if (ok && e / BN < rows && m < g.M && n < g.N) C[m * g.N + n] = g.bias ? total[i] + __ldg(g.bias + n * g.bias_stride) : total[i];
      }
    } else {
      const int64_t m = m0 + quad * 32 + lane;
      if (ok && m < g.M) {
        const int64_t n = n0 + col0;
        float *crow = C + m * g.N;
        if (g.bias) {
#pragma unroll
          for (int i = 0; i < CW; ++i)
            if (n + i < g.N) cur[i] = cur[i] + __ldg(g.bias + (n + i) * g.bias_stride);
        }
#pragma unroll
        for (int q = 0; q < CW / 4; ++q) {
          const int64_t nn = n + 4 * q;
          if (g.c_vec && nn + 3 < g.N) {
            *reinterpret_cast<float4 *>(crow + nn) = make_float4(cur[4 * q], cur[4 * q + 1], cur[4 * q + 2], cur[4 * q + 3]);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (nn + e < g.N) crow[nn + e] = cur[4 * q + e];
          }
        }
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 0) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_acc), "r"(2 * BN) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
struct FgPlan {
  int bn = 0, csize = 1;
  double us = 1e30;
};
// Tile width and cluster size by expected time, from measurements: 0.72 / 0.87 / 1.5 us per 32-deep block for BN = 32 /
// 64 / 128, half as much again once a second wave of tiles competes for the L2; 5.4 us around it; 4 (BN = 32) or 6 us per
// round of a cluster's reduction.  A cluster of 8 does not fit everywhere: clusters of 2, 4, 8 fill 144, 136, 128 SMs.
static FgPlan fg_plan(int64_t batch, int64_t M, int64_t N, int64_t K, bool parts) {
  FgPlan best;
  const int64_t periods = ceil_div(K, TC_PERIOD);
  for (int bn : {32, 64, 128}) {
    if (bn == 128 && parts) continue; // no room for the parts' buffer
    const double block = bn == 32 ? 0.72 : bn == 64 ? 0.87 : 1.5;
    const double tiles = double(ceil_div(M, FG_BM)) * double(ceil_div(N, bn)) * double(batch);
    for (int cs = 1; cs <= 8; cs *= 2) {
      if (cs > 1 && (bn == 128 || cs >= 2 * periods)) continue;
      const double sms = cs == 1 ? sm_count() : cs == 2 ? 144 : cs == 4 ? 136 : 128;
      const double rounds = double(ceil_div(periods, cs)), waves = std::ceil(tiles * cs / sms);
      const double blocks = cs == 1 ? double(ceil_div(K, FG_BK)) : cs >= periods ? std::min<double>(FG_PERIOD_BLOCKS, double(ceil_div(K, FG_BK)))
                                                                                : rounds * FG_PERIOD_BLOCKS;
      const double us = 5.4 + waves * blocks * block * (waves > 1 ? 1.5 : 1.0) + (cs > 1 ? (bn == 32 ? 4.0 : 6.0) * rounds * waves : 0.0);
      if (us < best.us) best = FgPlan{bn, cs, us};
    }
  }
  return best;
}
static thread_local FgPlan t_forced; // nt_matmul_force_fused
bool gemm_fused_forced() { return t_forced.bn != 0; }
void gemm_fused_force(int tile_n, int cluster) { t_forced = tile_n ? FgPlan{tile_n, cluster, 0.0} : FgPlan{}; }
double gemm_fused_expected_us(int64_t batch, int64_t M, int64_t N, int64_t K) {
  return fg_plan(batch, M, N, K, gemm_tc_k_split(batch, M, N, K).splits > 1).us;
}

template <int BN, bool CLUSTER> static void fg_launch(const FgArgs &g, dim3 grid) {
  const uint32_t smem = fg_ring_bytes<BN> + (g.part_buf ? fg_part_bytes<BN> : 0u);
  auto *kernel = gemm_fused_split<BN, CLUSTER>;
  static uint32_t configured = 0;
  if (smem > configured) {
    NT_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    configured = smem;
  }
  launch_with(false, CLUSTER ? unsigned(g.csize) : 1u, kernel, grid, fg_threads<BN>, smem, g);
}

// C = A @ B (+ bias), one collapsed batch stride per operand; false when the shape is outside one launch's limits.
bool gemm_fused(const float *A, const float *B, float *C, int64_t batch, int64_t M, int64_t N, int64_t K, int64_t a_sb, int64_t a_sm,
                int64_t a_sk, int64_t b_sb, int64_t b_sk, int64_t b_sn, const float *bias, int64_t bias_stride) {
  if (batch < 1 || batch > 65535 || M < 1 || N < 1 || K < 1 || ceil_div(M, FG_BM) > 65535 || ceil_div(N, 32) * 8 > 0x7fffffff) return false;
  gemm_tc_prepare();
  // an operand without a unit-stride dim goes through the transposing split there, which never cuts k into parts
  const bool natural = (a_sk == 1 || a_sm == 1 || M == 1 || K == 1) && (b_sk == 1 || b_sn == 1 || N == 1 || K == 1);
  const KSplit ks = natural ? gemm_tc_k_split(batch, M, N, K) : KSplit{};
  const FgPlan plan = gemm_fused_forced() ? t_forced : fg_plan(batch, M, N, K, ks.splits > 1);
  if (plan.bn == 128 && ks.splits > 1) return false; // no room for the parts' buffer
  auto aligned = [](const float *p, int64_t s_r, int64_t s_k, int64_t s_b, int64_t K, int64_t batch) {
    return s_k == 1 && (reinterpret_cast<uintptr_t>(p) & 15) == 0 && s_r % 4 == 0 && K % 4 == 0 && (batch == 1 || s_b % 4 == 0);
  };
  FgArgs g{};
  g.a = FgOperand{A, M, a_sm, a_sk, batch > 1 ? a_sb : 0, aligned(A, a_sm, a_sk, a_sb, K, batch), a_sk == 1 && a_sm != 1};
  g.b = FgOperand{B, N, b_sn, b_sk, batch > 1 ? b_sb : 0, aligned(B, b_sn, b_sk, b_sb, K, batch), b_sk == 1 && b_sn != 1};
  g.a.k_vec = g.a.k_vec && g.a.k_unit;
  g.b.k_vec = g.b.k_vec && g.b.k_unit;
  g.C = C;
  g.bias = bias;
  g.bias_stride = bias_stride;
  g.M = M;
  g.N = N;
  g.K = K;
  g.periods = int(ceil_div(K, TC_PERIOD));
  g.part_periods = ks.splits > 1 ? ks.kb_per_split * 16 / TC_PERIOD : g.periods;
  g.csize = plan.csize;
  g.part_buf = plan.csize > 1 || ks.splits > 1;
  g.c_vec = N % 4 == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
  g.error_flag = pipeline_error_flag();
  g.wait_limit = wait_limit_clocks();
  const dim3 grid{unsigned(ceil_div(N, plan.bn) * plan.csize), unsigned(ceil_div(M, FG_BM)), unsigned(batch)};
  matmul_profile_begin();
  if (plan.bn == 128) fg_launch<128, false>(g, grid);
  else if (plan.bn == 64) plan.csize > 1 ? fg_launch<64, true>(g, grid) : fg_launch<64, false>(g, grid);
  else plan.csize > 1 ? fg_launch<32, true>(g, grid) : fg_launch<32, false>(g, grid);
  matmul_profile_end();
  check_launch("gemm_fused_split");
  return true;
}

} // namespace ntb

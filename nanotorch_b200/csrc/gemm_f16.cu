// fp32 products of fp32 grade from three fp16 products on the tensor cores, over the planes of f16_split.cuh.
//
//   a b  =  hi_a hi_b + 2^-12 (hi_a lo_b + lo_a hi_b)      (per block of 64 x 64, times the two blocks' factors)
//
// The tensor cores multiply fp16 at twice the rate of TF32, and fp16 has TF32's significand: the same three products as the
// kernel of gemm_tc.cu, from half the bytes.  What fp16 lacks is exponent, which the planes make up with a factor per block
// and a lo that is stored 2^12 times too large.  A chain of accumulations is the 64 values of k of one block: first all of its
// cross terms, then the large ones on top, whose first instruction scales what has accumulated by 2^-12 (the scale-input-d of
// tcgen05.mma).  So one accumulator does, exactly, and the chains are short: the tensor core's rounding toward zero reaches
// over 4 large terms, and the epilogue warps add the chains up in fp32 registers, times the factors, rounding to nearest.
//
// A persistent CTA per SM walks over 128 x 256 tiles as in gemm_tc.cu.  Warp 8 loads the hi planes and warp 10 the lo planes,
// in blocks of 32 k (24 KB of each), into two rings of four: the cross terms are through with a lo block half a chain before
// the large ones are with its hi block, and the lo ring runs ahead.  Warp 9 issues the products, warps 0-7 drain the two
// halves of tensor memory in turn.
//
// 4096^3 294 us (536 over TF32 planes): 89 % of the clocks that the instructions take, at 1.55 GHz
// under the power cap.  What is left: 256 clocks of every chain's 1536 in which tensor memory is read, and 100 for the scaled
// instruction.  Error against 64 bits, uniform and normal operands, norm-wise: 1.2e-7 to 1.8e-7 (1.8e-6 over TF32 planes).
#include <cuda.h>

#include "f16_split.cuh"
#include "gemm_common.cuh"
#include "gemm_f16.cuh"
#include "gemm_tile.cuh"
#include "launch.cuh"
#include "nt_core.cuh"
#include "tma.cuh"

namespace ntb {

constexpr int FH_BK = 32;                // values of k per block of a ring
constexpr int FH_CHAIN = 64 / FH_BK;     // blocks per accumulation chain
constexpr int FH_SLOTS = 4;              // blocks in each ring
constexpr uint32_t FH_A_BYTES = TC_BM * FH_BK * 2, FH_B_BYTES = TC_BN * FH_BK * 2;
constexpr uint32_t FH_SLOT_BYTES = FH_A_BYTES + FH_B_BYTES; // 24 KB
constexpr uint32_t FH_SMEM_BYTES = 2 * FH_SLOTS * FH_SLOT_BYTES + 1024 /*align*/ + 256 /*barriers*/ + 8 * TC_CORNER_BYTES;
constexpr int FH_THREADS = 384;
constexpr int FH_LO_SHIFT = 12; // lo is stored 2^12 times too large

// D format F32 (1) in bits [4,6); A and B format F16 (0); majors in bits 15, 16; N >> 3 in [17,23); M >> 4 in [24,29).
constexpr uint32_t FH_IDESC = (1u << 4) | (uint32_t(TC_BN >> 3) << 17) | (uint32_t(TC_BM >> 4) << 24);

__device__ __forceinline__ void umma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, uint32_t lead) {
  asm volatile("{\n\t.reg .pred p, e;\n\t"
               "setp.ne.b32 p, %4, 0;\n\t"
               "setp.ne.b32 e, %5, 0;\n\t"
               "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(lead)
               : "memory");
}
// d = a b + 2^-FH_LO_SHIFT d
__device__ __forceinline__ void umma_f16_scaled(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t lead) {
  asm volatile("{\n\t.reg .pred p, e;\n\t"
               "setp.eq.b32 p, 0, 0;\n\t"
               "setp.ne.b32 e, %5, 0;\n\t"
               "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, %4;\n\t}"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "n"(FH_LO_SHIFT), "r"(lead)
               : "memory");
}

// K-major operand block, rows of 64 bytes (32 values of k) in the 64-byte swizzle: 8-row groups of 512 bytes, layout type 4.
// An instruction consumes 16 values of k, 32 bytes of a row.
// MN-major: rows of 128 bytes hold 64 consecutive values of m (or n) for one k, in the 128-byte swizzle over groups of 8
// rows (1024 bytes), layout type 2; an instruction consumes 16 rows = 2 groups, `stride byte offset` = 1024 apart, and the
// next 64 values of m (or n) lie a block's 32 rows further, the `leading byte offset`.
template <bool MN> __device__ __forceinline__ uint64_t fh_desc(uint32_t smem_addr) {
  constexpr uint32_t lbo = MN ? FH_BK * 128 : 16, sbo = MN ? 1024 : 512;
  uint64_t d = 0;
  d |= uint64_t((smem_addr & 0x3FFFF) >> 4);
  d |= uint64_t(lbo >> 4) << 16;
  d |= uint64_t(sbo >> 4) << 32;
  d |= uint64_t(1) << 46;
  d |= uint64_t(MN ? 2 : 4) << 61;
  return d;
}
template <bool MN> constexpr uint32_t FH_STEP = MN ? 16 * 128 : 32; // bytes to the next 16 values of k

struct F16Args {
  TileArgs t;
  F16Scales a, b; // factors of the blocks along m (or n) and along k
  const int *wide_a, *wide_b;
  F16Fallback f;
};

// Waits until every CTA of the grid, which runs all of them at once, has come here; false when that takes longer than a
// pipeline wait may.
__device__ __forceinline__ bool grid_wait(unsigned int *arrived, int *error_flag, long long limit) {
  __shared__ bool all;
  asm volatile("fence.proxy.async.global;" ::: "memory"); // what this thread wrote is for the copy engines of all SMs
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(arrived, 1u);
    const long long t0 = clock64();
    while ((all = *reinterpret_cast<volatile unsigned int *>(arrived) >= gridDim.x) == false && clock64() - t0 <= limit) {
    }
    if (!all) atomicExch(error_flag, 7);
    else if (atomicAdd(arrived, 1u) == 2 * gridDim.x - 1) *arrived = 0; // the last to leave
    __threadfence();
  }
  __syncthreads();
  asm volatile("fence.proxy.async.global;" ::: "memory");
  return all;
}

// What a CTA does where an operand is wide.  Inside this launch and not behind it: two launches that only looked whether they
// were needed took 6 us of every product (32 x 512^3 with both gradients 170 us, now 157).  Out of line, so that it does not
// take part in the kernel's registers.
template <bool A_MN, bool B_MN> __device__ __noinline__ void fh_fallback(const F16Fallback &f) {
  if (threadIdx.x < 256)
    for (int i = 0; i < 2; ++i) {
      const NatSplitArgs &s = i ? f.b : f.a;
      const int64_t pc = (s.Cp + 255) / 256, pr = (s.R + 15) / 16;
      for (int64_t p = blockIdx.x; p < pc * pr * f.t.batch; p += gridDim.x) split_piece(s, p % pc, p / pc % pr, p / (pc * pr));
    }
  if (grid_wait(f.arrived, f.t.error_flag, f.t.wait_limit)) tf32_tiles<A_MN, B_MN>(f.map_a, f.map_b, f.t);
}

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(FH_THREADS, 1)
gemm_3xf16_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ F16Args args) {
  constexpr uint32_t IDESC = FH_IDESC | (A_MN ? (1u << 15) : 0u) | (B_MN ? (1u << 16) : 0u);
  const TileArgs &g = args.t;
  if (*args.wide_a | *args.wide_b) {
    fh_fallback<A_MN, B_MN>(args.f);
    return;
  }
  static_assert(FH_SMEM_BYTES >= TC_SMEM_BYTES);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t hi_ring = smem_base, lo_ring = smem_base + FH_SLOTS * FH_SLOT_BYTES;
  const uint32_t bar_base = smem_base + 2 * FH_SLOTS * FH_SLOT_BYTES;
  // full and empty of the hi ring at +8 s and +32 + 8 s, of the lo ring at +64 and +96; acc_full at +128, acc_empty at +144;
  // the tensor memory's address at +160
  const uint32_t acc_full0 = bar_base + 128, acc_empty0 = bar_base + 144;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem_raw + (bar_base - smem_u32(smem_raw)) + 160);
  volatile int *poison_slot = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 4 * FH_SLOTS; ++i) mbar_init(bar_base + 8 * i, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(acc_full0 + 8 * i, 1);
      mbar_init(acc_empty0 + 8 * i, 8); // one arrival per epilogue warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    // a wait already ran out in this launch (or an earlier one since the last synchronisation): the whole CTA does nothing
    *poison_slot = *reinterpret_cast<volatile int *>(g.error_flag);
    poison_slot[1] = 0; // split-K: an epilogue warp gave up
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_acc = __shfl_sync(0xffffffffu, *tmem_slot, 0); // uniform, and the compiler knows
  const bool poisoned = *poison_slot != 0;

  // 384 x 168 registers at the launch = 256 x 192 + 128 x 120.  The epilogue's sums and a drained part of a chain take 160;
  // what it spills costs power and so clock, and with fewer registers the issuing warp falls behind: 16384 x 4096 x 4096
  // 1138 us, 1231 without the exchange, 1152 with 208 + 88, 1172 with 224 + 56.
  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 120;");
    if (warp == 8 || warp == 10) {
      // ------------------------------------------------------------------ a plane's producer
      if (lane == 0 && !poisoned) {
        const uint32_t ring = warp == 8 ? hi_ring : lo_ring, full0 = bar_base + (warp == 8 ? 0 : 64), empty0 = full0 + 32;
        const int first = warp == 8 ? 0 : g.batch;
        uint32_t phase = 0;
        int s = 0;
        bool ok = true;
        for (int w = blockIdx.x; w < g.work && ok; w += gridDim.x) {
          const TileItem it = tile_item<FH_CHAIN>(g, w);
          const int m0 = it.tile_m * TC_BM, n0 = it.tile_n * TC_BN, p = first + it.b;
          for (int kb = 0; kb < it.nkb; ++kb) {
            if (!mbar_wait(empty0 + 8 * s, phase ^ 1, g.wait_limit)) {
              atomicExch(g.error_flag, 1);
              ok = false;
              break;
            }
            const uint32_t st = ring + s * FH_SLOT_BYTES, bar = full0 + 8 * s;
            mbar_expect_tx(bar, FH_SLOT_BYTES);
            const int k = (it.kb0 + kb) * FH_BK;
            if constexpr (A_MN) tma_load_4d(st, &map_a, bar, 0, k, m0 >> 6, p);
            else tma_load_3d(st, &map_a, bar, k, m0, p);
            if constexpr (B_MN) tma_load_4d(st + FH_A_BYTES, &map_b, bar, 0, k, n0 >> 6, p);
            else tma_load_3d(st + FH_A_BYTES, &map_b, bar, k, n0, p);
            if (++s == FH_SLOTS) {
              s = 0;
              phase ^= 1;
            }
          }
        }
      }
    } else if (warp == 9) {
      // ------------------------------------------------------------------ MMA issuer
      if (!poisoned) {
        const uint32_t lead = elect_lane();
        const uint32_t hi_full = bar_base, hi_empty = bar_base + 32, lo_full = bar_base + 64, lo_empty = bar_base + 96;
        uint32_t hs = 0, hp = 0, ls = 0, lp = 0, ms = 0; // slot and phase of the next block in either ring; next large terms' slot
        uint32_t done = 0;  // chains of the items before
        bool ok = true;
        for (int w = blockIdx.x; w < g.work && ok; w += gridDim.x) {
          const TileItem it = tile_item<FH_CHAIN>(g, w);
          for (int q = 0; q < it.periods && ok; ++q) {
            const uint32_t p = done + q;
            const int buf = p & 1;
            // the epilogue must have drained this half (two chains ago) before it is overwritten
            if (!mbar_wait(acc_empty0 + 8 * buf, ((p >> 1) & 1) ^ 1, g.wait_limit)) {
              if (lead) atomicExch(g.error_flag, 4);
              ok = false;
              break;
            }
            tcgen05_fence_after();
            const uint32_t d = tmem_acc + uint32_t(buf * TC_BN);
            const int blocks = min(FH_CHAIN, it.nkb - q * FH_CHAIN);
            for (int j = 0; j < blocks && ok; ++j) {
              if (!mbar_wait(hi_full + 8 * hs, hp, g.wait_limit) || !mbar_wait(lo_full + 8 * ls, lp, g.wait_limit)) {
                if (lead) atomicExch(g.error_flag, 2);
                ok = false;
                break;
              }
              tcgen05_fence_after();
              const uint32_t hi = hi_ring + hs * FH_SLOT_BYTES, lo = lo_ring + ls * FH_SLOT_BYTES;
#pragma unroll
              for (int ks = 0; ks < FH_BK / 16; ++ks) {
                const uint32_t ao = ks * FH_STEP<A_MN>, bo = FH_A_BYTES + ks * FH_STEP<B_MN>;
                umma_f16(d, fh_desc<A_MN>(hi + ao), fh_desc<B_MN>(lo + bo), IDESC, (j | ks) != 0, lead);
                umma_f16(d, fh_desc<A_MN>(lo + ao), fh_desc<B_MN>(hi + bo), IDESC, 1, lead);
              }
              umma_commit(lo_empty + 8 * ls, lead);
              if (++hs == FH_SLOTS) hs = 0, hp ^= 1;
              if (++ls == FH_SLOTS) ls = 0, lp ^= 1;
            }
            for (int j = 0; j < blocks && ok; ++j) {
              const uint32_t hi = hi_ring + ms * FH_SLOT_BYTES;
#pragma unroll
              for (int ks = 0; ks < FH_BK / 16; ++ks) {
                const uint64_t a = fh_desc<A_MN>(hi + ks * FH_STEP<A_MN>), b = fh_desc<B_MN>(hi + FH_A_BYTES + ks * FH_STEP<B_MN>);
                if ((j | ks) == 0) umma_f16_scaled(d, a, b, IDESC, lead);
                else umma_f16(d, a, b, IDESC, 1, lead);
              }
              umma_commit(hi_empty + 8 * ms, lead);
              if (++ms == FH_SLOTS) ms = 0;
            }
            if (ok) umma_commit(acc_full0 + 8 * buf, lead);
          }
          done += it.periods;
        }
        if (!ok && lead) { // release the epilogue warps from whatever they wait on
          for (int i = 0; i < 2; ++i) mbar_arrive(acc_full0 + 8 * i);
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 192;");
    // ------------------------------------------------------------------ epilogue
    const int quad = warp & 3;        // 32-lane group of tensor memory this warp may read
    const int half = warp >> 2;       // which 128 of the 256 columns
    char *corner = reinterpret_cast<char *>(smem_raw + (bar_base - smem_u32(smem_raw))) + 256 + warp * TC_CORNER_BYTES;
    bool ok = !poisoned, reached = false;
    uint32_t done = 0; // chains of the items before
    for (int w = blockIdx.x; w < g.work && ok; w += gridDim.x) {
      const TileItem it = tile_item<FH_CHAIN>(g, w);
      float sum[128];
#pragma unroll
      for (int i = 0; i < 128; ++i) sum[i] = 0.0f;
      // the factors of the blocks that meet in this warp's columns, one chain ahead; blocks past the end stand for values that
      // are zero or not stored
      const float *sa = args.a.at(it.b, it.tile_m * 2 + (quad >> 1), it.kb0 / FH_CHAIN);
      const float *sb0 = args.b.at(it.b, it.tile_n * 4 + half * 2, it.kb0 / FH_CHAIN);
      const float *sb1 = args.b.at(it.b, it.tile_n * 4 + half * 2 + 1, it.kb0 / FH_CHAIN);
      float va = __ldg(sa), vb0 = __ldg(sb0), vb1 = __ldg(sb1);
      for (int q = 0; q < it.periods; ++q) {
        const uint32_t p = done + q;
        const int buf = p & 1;
        const float f0 = va * vb0, f1 = va * vb1;
        if (q + 1 < it.periods) {
          va = __ldg(sa += args.a.s_k);
          vb0 = __ldg(sb0 += args.b.s_k);
          vb1 = __ldg(sb1 += args.b.s_k);
        }
        if (!mbar_wait(acc_full0 + 8 * buf, (p >> 1) & 1, g.wait_limit)) {
          atomicExch(g.error_flag, 3);
          ok = false;
          break;
        }
        tcgen05_fence_after();
        const uint32_t taddr = tmem_acc + (uint32_t(quad * 32) << 16) + uint32_t(buf * TC_BN + half * 128);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t v[32];
          tmem_ld32(taddr + uint32_t(c * 32), v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int e = 0; e < 32; ++e) sum[c * 32 + e] = fmaf(__uint_as_float(v[e]), c < 2 ? f0 : f1, sum[c * 32 + e]);
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty0 + 8 * buf);
      }
      done += it.periods;
      // Whether a wait ran out is read once per tile: the 700 clocks of that read are half of a chain, and with one in every
      // chain the tensor cores waited for the epilogue (63 % busy).
      ok = ok && *reinterpret_cast<volatile int *>(g.error_flag) == 0;
      if (!poisoned) finish_tile(g, it, ok, sum, corner, quad, half, lane, int(threadIdx.x), poison_slot);
      reached = reached || it.shared >= 0;
    }
    if (!poisoned && !ok) give_up_tile(g, reached, poison_slot);
  }

  if (!poisoned && *reinterpret_cast<volatile int *>(g.error_flag) != 0) {
    const long long t0 = clock64(); // copies in flight land before this shared memory is another CTA's
    while (clock64() - t0 < 2000000) {
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 9) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_acc), "r"(512) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// Rows of an operand (m or n) across the planes, k along them: 3-D {k, rows, plane}; k along the rows: 4-D {64 m|n, k, (m|n) /
// 64, plane}.  Reads past k or the rows are zero filled.
static CUtensorMap fh_map(const F16Operand &o, int64_t batch, uint32_t box_rows) {
  CUtensorMap m;
  const cuuint64_t row = cuuint64_t(o.p.Cp) * 2, plane = cuuint64_t(o.R) * row;
  const cuuint32_t ones[4] = {1, 1, 1, 1};
  CUresult rc;
  if (o.mn) {
    const cuuint64_t dims[4] = {64, cuuint64_t(o.R), cuuint64_t(o.p.Cp / 64), cuuint64_t(2 * batch)}, strides[3] = {row, 128, plane};
    const cuuint32_t box[4] = {64, FH_BK, box_rows / 64, 1};
    rc = tensor_map_encoder()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, o.p.planes, dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  } else {
    const cuuint64_t dims[3] = {cuuint64_t(o.C), cuuint64_t(o.R), cuuint64_t(2 * batch)}, strides[2] = {row, plane};
    const cuuint32_t box[3] = {FH_BK, box_rows, 1};
    rc = tensor_map_encoder()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, o.p.planes, dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  }
  if (rc != CUDA_SUCCESS) fail_runtime("cuTensorMapEncodeTiled (fp16 planes) failed with code " + std::to_string(int(rc)));
  return m;
}

template <bool A_MN, bool B_MN> static void fh_launch(const CUtensorMap &ma, const CUtensorMap &mb, const F16Args &g, unsigned grid) {
  static bool configured = false;
  if (!configured) {
    NT_CUDA_CHECK(cudaFuncSetAttribute(gemm_3xf16_kernel<A_MN, B_MN>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(FH_SMEM_BYTES)));
    configured = true;
  }
  launch_at_once(gemm_3xf16_kernel<A_MN, B_MN>, grid, FH_THREADS, FH_SMEM_BYTES, ma, mb, g);
}

void gemm_f16_launch(const F16Operand &a, const F16Operand &b, TileArgs t, int64_t K, const F16Fallback &f) {
  F16Args g{};
  t.num_kb = int32_t(ceil_div(K, FH_BK));
  t.kb_per_split = t.kb_per_split * 16 / FH_BK; // whole chains: a multiple of 256 values of k
  g.wide_a = &a.p.header->wide;
  g.wide_b = &b.p.header->wide;
  g.f = f;
  g.t = t;
  g.a = f16_scales(a);
  g.b = f16_scales(b);
  const CUtensorMap ma = fh_map(a, t.batch, TC_BM), mb = fh_map(b, t.batch, TC_BN);
  const unsigned grid = unsigned(std::min(t.work, sm_count()));
  if (a.mn && b.mn) fh_launch<true, true>(ma, mb, g, grid);
  else if (a.mn) fh_launch<true, false>(ma, mb, g, grid);
  else if (b.mn) fh_launch<false, true>(ma, mb, g, grid);
  else fh_launch<false, false>(ma, mb, g, grid);
  check_launch("gemm_3xf16_kernel");
}

} // namespace ntb

// Tensor-core path with zero points, above 16 rows where the GEMV's passes do not run side by side: tcgen05.mma with the WEIGHTS IN TENSOR MEMORY, scales and
// zero points applied outside the product.
//
//   y[m, n] = 2^(8-b) * sum_g s[n, g] * (sum_{k in g} (code - Z) x[m, k]  -  z'[n, g] * sum_{k in g} x[m, k])
//
// (Z = 2^(b-1); z' = (zero - 128) / 2^(8-b).)  One CTA owns 4, 8 or 16 row tiles of the packed
// layout (16 out-features each) and a batch block; a pipeline stage is a block of 128 in-features:
//
//   * sixteen producer warps decode their tiles' blocks to the exact integers (code - Z), two instructions per pair of
//     weights (five for 8-bit codes in bf16), and store them with tcgen05.st as the A operand in tensor memory, so that the weights do not pass through
//     shared memory (written and read there they take 512 of its cycles for every 256 x 64 weights).  The packed layout gives a
//     lane eight neighbouring in-features of a row, the store puts pairs of words side by side, and so it fixes an order of the
//     in-features of its own;
//   * the activations come with TMA, eight blocks ahead, into raw stages; two warps copy them into the 128-byte-swizzled B tile
//     in that same order, eight bytes a lane, free of bank conflicts;
//   * one warp requests activations and issues the MMAs (M = 128 out-features, N = batch rows, K = 16), every group of
//     in-features into an accumulator of its own;
//   * eight warps read a group's accumulator with tcgen05.ld, scale it in fp32 and add it to the sums that they hold in
//     registers, while the next group runs; and they sum the activations of the next group (mma.sync with a matrix of ones
//     over the B tile).
//
// The weights are never rounded: scale and zero point act in fp32, as in the GEMV (gemv.cu).  K is split over the CTAs of a
// thread-block cluster, which add their sums through distributed shared memory in the order of the K ranges.  Every mbarrier
// wait is bounded.  A warp that gives up hands nothing on any more, so that the others give up in turn; the issuing warp stays
// until its copies and MMAs have ended (again with a limit), and tensor memory is freed on every path.
//
// The tiles of gemm_tc.cu hold scale * (code - zero) rounded to 16 bits, 1.4 times the error; the GEMV
// scales in fp32 but takes a pass, with its own decoding, for every 16 rows.  What bounds it (B200, from the launches that the plan
// below is fitted to): a launch takes 4 to 6 us around its main loop, a cluster's reduction included; a block of 128 in-features
// takes 0.8 us for 8 row tiles at 32 batch rows and 1.0 at 64 with groups of 128, 1.3 and 1.8 with groups of 32, 0.5 and 0.6 with
// one scale per row.  The difference is the scaling and the sums of the activations, a chain of waits between the warps: at
// 4096 x 4096, 128 rows, 4 bits, 22.2 us, the tensor pipe is busy 15 % of the time and 0.44 instructions are issued a cycle.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "async.cuh"
#include "decode.cuh"
#include "gemv_common.cuh"
#include "host_util.h"
#include "kernels.h"
#include "tc_common.cuh"

namespace mg {

constexpr int kTsProducers = 16, kTsScalers = 8, kTsStagers = 2;  // warps; one more requests activations and issues MMAs
constexpr int kTsWarps = kTsProducers + kTsScalers + kTsStagers + 1;
constexpr int kTsMaxStages = 6;   // of weights (tensor memory) and activations (shared memory) as the MMAs read them
constexpr int kTsRawStages = 8;   // of activations as they come from global memory; a power of two
constexpr int kTsUnitBytes = 16 * 128;  // 16 rows x 64 in-features
constexpr int kTsMaxCols = 64;  // batch rows of a block

struct TsParams {
  const uint32_t *w;
  const uint16_t *s;
  const uint16_t *z;  // zero points in master units, laid out like the scales
  const uint16_t *x;
  uint16_t *y;
  int N, K, M;
  int kblocks;   // K / 128
  int split;     // CTAs along K
  int tiles;     // row tiles of a CTA: 4, 8 or 16 (16 with at most 32 batch rows)
  int ncols;     // UMMA N: batch rows of a CTA, a multiple of 16
  int stages;
  int accumulators;  // 2 or 4
};

// Shared memory: barriers (8 bytes each) and the address of the tensor memory, the groups' activation sums, the B stages, the
// raw stages.
constexpr int kTsBarFull = 0, kTsBarDone = 8 * kTsMaxStages, kTsBarDEmpty = 16 * kTsMaxStages, kTsBarRawFull = kTsBarDEmpty + 32,
              kTsBarEnd = kTsBarRawFull + 8 * kTsRawStages, kTsTmemSlot = kTsBarEnd + 8;
constexpr int kTsOffSums = 1024, kTsOffStages = 4096;
static_assert(kTsTmemSlot + 4 <= kTsOffSums && kTsOffSums + 3 * 4 * kTsMaxCols * 4 <= kTsOffStages, "shared-memory plan");

// Row tile i of a CTA: tensor-memory lanes [32 (i % 4) + 16 ((i / 4) % 2), + 16) of row block i / 8.  A warp reaches the
// lanes 32 (warp % 4) .. + 31 only, and warps with equal warp % 4 share a scheduler: consecutive tiles go to different ones.
__host__ __device__ inline int ts_row_blocks(int tiles) { return tiles > 8 ? 2 : 1; }
__host__ __device__ inline int ts_dcols(int ncols) { return (ncols + 31) / 32 * 32; }

// 32 in-features (JJ = 0..3) of a block of one tile to tensor memory, 16 columns.  Lane (g, t) holds words (pairs) 4 t .. + 3
// of rows g and g + 8; 16x256b puts its words 0 and 1 into columns 2 t and 2 t + 1, words 2 and 3 into columns 8 + 2 t and
// 9 + 2 t.
template <int B, bool BF16, int JJ> __device__ __forceinline__ void ts_put_quarter(const uint32_t (&w)[2 * B], uint32_t taddr) {
  uint32_t r[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) r[i] = dense_int<B, BF16>(w, 8 * JJ + i);  // pair P: row P & 1, word (P >> 1) & 3, quarter P >> 3
  asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr + 16 * JJ), "r"(r[0]), "r"(r[2]),
               "r"(r[1]), "r"(r[3]), "r"(r[4]), "r"(r[6]), "r"(r[5]), "r"(r[7])
               : "memory");
}

__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      "  .reg .pred p;\n"
      "  setp.ne.b32 p, %4, 0;\n"
      "  tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ uint4 lds_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts_v2(uint32_t addr, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(x), "r"(y) : "memory");
}

// c += ones . B for fp16 or bf16 B fragments: every row of the result holds the column sums
template <bool BF16> __device__ __forceinline__ void mma_ones(float (&c)[4], uint32_t b0, uint32_t b1) {
  if constexpr (BF16) {
    constexpr uint32_t one = 0x3F803F80u;
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%4,%4,%4}, {%5,%6}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(one), "r"(b0), "r"(b1));
  } else {
    const uint32_t ones[4] = {0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u};
    mma16816<false>(c, ones, b0, b1);
  }
}

// Position in a ring of stages
struct TsRing {
  uint32_t idx, parity;
  __device__ __forceinline__ TsRing(uint32_t first, uint32_t first_parity) : idx(first), parity(first_parity) {}
  __device__ __forceinline__ void advance(uint32_t by, uint32_t stages) {  // by <= stages
    idx += by;
    if (idx >= stages) {
      idx -= stages;
      parity ^= 1;
    }
  }
};

template <int B, int GS, bool BF16>
__global__ void __launch_bounds__(kTsWarps * 32, 1) gemm_ts_kernel(const TsParams p, const __grid_constant__ CUtensorMap xmap) {
  extern __shared__ unsigned char ts_smem_raw[];
  const uint32_t raw_u32 = smem_u32(ts_smem_raw);
  const uint32_t base = (raw_u32 + 1023u) & ~1023u;
  unsigned char *base_ptr = ts_smem_raw + (base - raw_u32);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int sk = blockIdx.y;
  const int m0 = blockIdx.z * p.ncols;
  const int mrows = min(p.M - m0, p.ncols);
  const int kb_lo = sk * p.kblocks / p.split, kb_hi = (sk + 1) * p.kblocks / p.split;
  const int nblk = kb_hi - kb_lo;
  const int tile0 = blockIdx.x * p.tiles;            // first row tile of this CTA
  const int tiles = min(p.tiles, p.N / 16 - tile0);  // its row tiles
  const int rbs = ts_row_blocks(tiles);
  const int accs = p.accumulators;
  const uint32_t dcols = ts_dcols(p.ncols);          // tensor-memory columns of an accumulator
  const uint32_t a_col0 = accs * rbs * dcols;         // first column of the A stages, 64 columns a row block each
  const uint32_t stages = p.stages;
  const uint32_t b_half_bytes = p.ncols * 128, b_stage_bytes = 2 * b_half_bytes;
  const int quad = warp & 3;

  constexpr int kFirstScaler = kTsProducers, kFirstStager = kTsProducers + kTsScalers, kMma = kFirstStager + kTsStagers;
  if (warp == kMma) {
    int scalers = 0;  // scaling warps whose lanes hold out-features
    for (int q = 0; q < 4; ++q)
      for (int h = 0; h < 2; ++h) scalers += (q + (rbs == 2 ? 8 * h : 0)) < tiles ? 1 : 0;
    // a lane per index
    if (lane < kTsMaxStages) {
      mbar_init(base + kTsBarFull + 8 * lane, tiles + 2);  // a producer a tile, a stager a half
      mbar_init(base + kTsBarDone + 8 * lane, 1 + kTsScalers);
    }
    if (lane < kTsRawStages) {
      mbar_init(base + kTsBarRawFull + 8 * lane, 1);
    }
    if (lane < 4) {
      mbar_init(base + kTsBarDEmpty + 8 * lane, scalers);
    }
    if (lane == 0) mbar_init(base + kTsBarEnd, 1);
    mbar_init_fence();
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(base + kTsTmemSlot) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }

  // Producers: the four warps of a quadrant share its p.tiles / 4 tiles, 4 / that many warps a tile take its blocks in turn.
  // The first loads go out before anything is waited for.
  constexpr int BW = BlockTraits<B>::WORDS;
  constexpr int kAhead = (B >= 6) ? 2 : (B == 4 ? 3 : 4);
  const int per_quad = p.tiles >> 2;                                       // 1, 2 or 4
  const int j = (warp >> 2) & (per_quad - 1);                              // tile of the quadrant
  const int phase = per_quad == 1 ? warp >> 2 : (per_quad == 2 ? warp >> 3 : 0), step = 4 / per_quad;  // its blocks
  const int my_blocks = (warp < kTsProducers && quad + 4 * j < tiles) ? nblk : 0;
  const uint32_t *wnext = p.w + (static_cast<size_t>(tile0 + quad + 4 * j) * p.kblocks + kb_lo + phase) * BW;
  uint32_t wq[kAhead][2 * B];
#pragma unroll
  for (int a = 0; a < kAhead; ++a)
    if (phase + a * step < my_blocks) {
      load_block<B>(wnext, lane, wq[a]);
      wnext += step * BW;
    }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(base_ptr + kTsTmemSlot);
  // Weights, scales and zero points are never written by a kernel: only the activations and the results have to wait for
  // the kernel before this one.  Every warp waits for it before its first wait on a barrier that hangs on the activations: that
  // kernel may take longer than the limit of such a wait.
  asm volatile("griddepcontrol.launch_dependents;");

  // With K split the B stages, and where these are fewer than the sums need (16 row tiles) the first raw stages behind them,
  // hold [batch row][128 x row blocks out-feature slots] of sums once the last group is complete (and with it everything that
  // writes or reads a stage: every raw stage has been copied by then, and the last sums of activations come before the barrier
  // of their block).
  float *staging = reinterpret_cast<float *>(base_ptr + kTsOffStages);
  const int slots = 128 * rbs;
  bool failed = false;
  if (warp < kTsProducers) {
    // ------------------------------------------------------------------ producers
    TsRing ring(0, 1);
    ring.advance(phase, stages);
    bool ahead = true;  // in the first pass through the stages, which are free from the start
    const uint32_t a_lane = tmem + a_col0 + (static_cast<uint32_t>(quad * 32 + (j & 1) * 16) << 16) + (j >> 1) * 64;
    for (int kb = phase; kb < my_blocks && !failed; kb += step * kAhead) {
#pragma unroll
      for (int a = 0; a < kAhead; ++a) {
        if (kb + a * step < my_blocks && !failed) {
          if (ahead && ring.parity == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            ahead = false;
          }
          if (!mbar_wait_chain(base + kTsBarDone + 8 * ring.idx, ring.parity)) {
            failed = true;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t taddr = a_lane + ring.idx * (rbs * 64);
          ts_put_quarter<B, BF16, 0>(wq[a], taddr);
          ts_put_quarter<B, BF16, 1>(wq[a], taddr);
          ts_put_quarter<B, BF16, 2>(wq[a], taddr);
          ts_put_quarter<B, BF16, 3>(wq[a], taddr);
          if (kb + (a + kAhead) * step < my_blocks) {  // this block's registers are free
            load_block<B>(wnext, lane, wq[a]);
            wnext += step * BW;
          }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(base + kTsBarFull + 8 * ring.idx);
          ring.advance(step, stages);
        }
      }
    }
    if (failed) report_status(kStatusMmaTimeout);
  } else if (warp < kFirstStager) {
    // ------------------------------------------------------------------ scalers
    const int half = (warp >> 2) & 1;  // row block, or half of the chunks of 16 batch rows
    const int rb = rbs == 2 ? half : 0;
    const int chunk0 = rbs == 2 ? 0 : half, chunk_step = rbs == 2 ? 1 : 2;
    const int nchunks = p.ncols / 16;
    const bool scales_any = quad + 8 * rb < tiles;        // this warp's lanes hold out-features
    const int my_tile = quad + 4 * (lane >> 4) + 8 * rb;  // this lane's row tile
    const bool my_valid = my_tile < tiles;
    float yacc[32];  // sums of this lane's out-feature, up to 32 batch rows
#pragma unroll
    for (int i = 0; i < 32; ++i) yacc[i] = 0.f;
    constexpr int NG = (GS == 32) ? 4 : 1;  // groups that end with a block (none but the last for GS == -1)
    const int groups = (GS == -1) ? 1 : p.K / GS;
    const size_t s_off = (static_cast<size_t>(my_valid ? tile0 + my_tile : tile0) * groups + (GS == -1 ? 0 : kb_lo * NG)) * 16 + (lane & 15);
    const uint16_t *sp = p.s + s_off, *zp = p.z + s_off;
    uint16_t s_next[NG], z_next[NG];
    auto load_scales = [&]() {
#pragma unroll
      for (int i = 0; i < NG; ++i) {
        s_next[i] = ldg_u16_tc(sp + i * 16);
        z_next[i] = ldg_u16_tc(zp + i * 16);
      }
      if constexpr (GS != -1) {
        sp += NG * 16;
        zp += NG * 16;
      }
    };
    load_scales();
    asm volatile("griddepcontrol.wait;" ::: "memory");  // for the activations, and before anything is written
    TsRing b_ring(0, 0);
    const int sw = warp - kFirstScaler;
    float csum[NG][4];  // the groups' sums of the activations of batch rows 8 sw .. + 7
#pragma unroll
    for (int q = 0; q < NG; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) csum[q][e] = 0.f;
    // Sums of the activations of the block the ring stands at, into buffer `buf` of three (4 groups x kTsMaxCols batch rows
    // each).  They run a block ahead of the scaling: whoever writes a buffer again has passed the barrier of a block that comes
    // after its last reader's.
    float *sums = reinterpret_cast<float *>(base_ptr + kTsOffSums);
    auto sum_block = [&](int buf, bool group_ends) {
      if (!failed && !mbar_wait_chain(base + kTsBarFull + 8 * b_ring.idx, b_ring.parity)) failed = true;
      if (failed) return;
      if (8 * sw < p.ncols) {
        const int g = lane >> 2, t = lane & 3;
        const uint32_t row = base + kTsOffStages + b_ring.idx * b_stage_bytes + (8 * sw + g) * 128;
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // 32 in-features each
          // the order within a group does not matter: rows of odd g read the other quarter first, free of bank conflicts
          const int chunk = (GS == 32) ? 4 * (q & 1) + t : 4 * ((q ^ g) & 1) + t;
          const uint4 v = lds_v4(row + (q >> 1) * b_half_bytes + ((chunk ^ g) << 4));
          float(&c)[4] = csum[GS == 32 ? q : 0];
          mma_ones<BF16>(c, v.x, v.y);
          mma_ones<BF16>(c, v.z, v.w);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(base + kTsBarDone + 8 * b_ring.idx);
      b_ring.advance(1, stages);
      if (group_ends) {
        if (8 * sw < p.ncols && lane < 4) {
#pragma unroll
          for (int q = 0; q < NG; ++q)
            *reinterpret_cast<float2 *>(sums + (buf * 4 + q) * kTsMaxCols + 8 * sw + 2 * lane) = make_float2(csum[q][0], csum[q][1]);
        }
        if constexpr (GS != -1) {
#pragma unroll
          for (int q = 0; q < NG; ++q)
#pragma unroll
            for (int e = 0; e < 4; ++e) csum[q][e] = 0.f;
        }
      }
    };
    sum_block(0, GS != -1 || nblk == 1);
    int sum_buf = 0;  // of block blk
    TsRing d_ring(0, 0), done(0, 0);
    for (int blk = 0; blk < nblk; ++blk) {
      uint16_t s_cur[NG], z_cur[NG];
#pragma unroll
      for (int i = 0; i < NG; ++i) {
        s_cur[i] = s_next[i];
        z_cur[i] = z_next[i];
      }
      if (GS != -1 && blk + 1 < nblk) load_scales();
      const float *my_sums = sums + (GS == -1 ? 0 : sum_buf * 4 * kTsMaxCols);
      __syncwarp();
      asm volatile("bar.sync 1, %0;" ::"n"(kTsScalers * 32) : "memory");  // the sums of block blk are there
      sum_buf = sum_buf == 2 ? 0 : sum_buf + 1;
      if (blk + 1 < nblk) sum_block(GS == -1 ? 0 : sum_buf, GS != -1 || blk + 2 == nblk);
      if (!scales_any || failed) continue;  // all eight warps pass every named barrier
      if (!mbar_wait_chain(base + kTsBarDone + 8 * done.idx, done.parity)) {
        failed = true;
        continue;
      }
      done.advance(1, stages);
      if (GS == -1 && blk + 1 < nblk) continue;  // waited for all the same: a parity tells neighbouring phases apart only
#pragma unroll
      for (int q = 0; q < NG; ++q) {
        const uint32_t buf = d_ring.idx;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const float sc = scale_to_float<BF16>(s_cur[q]);
        // zero point relative to the integers in the tile: (code - Z) * DensePre = (master - 128) / rest
        constexpr float kPerMaster = static_cast<float>(DensePre<B>::value) / static_cast<float>(1 << (8 - B));
        const float nz = (128.f - scale_to_float<BF16>(z_cur[q])) * kPerMaster;
        const float4 *xs = reinterpret_cast<const float4 *>(my_sums + q * kTsMaxCols);
        const uint32_t d = tmem + (static_cast<uint32_t>(quad * 32) << 16) + (buf * rbs + rb) * dcols;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int ci = chunk0 + c * chunk_step;
          if (ci < nchunks) {
            uint32_t v[16];
            tmem_ld16(d + ci * 16, v);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float4 xv = xs[ci * 4 + i];
              float *ya = yacc + c * 16 + 4 * i;
              ya[0] = fmaf(sc, fmaf(nz, xv.x, __uint_as_float(v[4 * i + 0])), ya[0]);
              ya[1] = fmaf(sc, fmaf(nz, xv.y, __uint_as_float(v[4 * i + 1])), ya[1]);
              ya[2] = fmaf(sc, fmaf(nz, xv.z, __uint_as_float(v[4 * i + 2])), ya[2]);
              ya[3] = fmaf(sc, fmaf(nz, xv.w, __uint_as_float(v[4 * i + 3])), ya[3]);
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(base + kTsBarDEmpty + 8 * buf);
        if constexpr (NG > 1) __syncwarp();  // before the next group's reads
        d_ring.advance(1, accs);
      }
    }
    if (failed) report_status(kStatusMmaTimeout);
    constexpr float kRest = static_cast<float>(1 << (8 - B)) / static_cast<float>(DensePre<B>::value);
    const int n = (tile0 + my_tile) * 16 + (lane & 15);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int ci = chunk0 + c * chunk_step;
      if (ci < nchunks && my_valid && !failed) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float v = yacc[c * 16 + i] * kRest;
          const int m = ci * 16 + i;
          if (p.split > 1)
            staging[m * slots + rb * 128 + quad * 32 + lane] = v;
          else if (m < mrows)
            p.y[static_cast<size_t>(m0 + m) * p.N + n] = to_out16<BF16>(v);
        }
      }
    }
  } else if (warp < kMma) {
    // ------------------------------------------------------------------ activation tiles, from raw to B stages
    // This warp's half (64 in-features) of every block.  Of a row's 16-byte chunk c, words 0 and 1 go to word 2 (c % 2) of the
    // tile's chunk 4 (c / 4) + (c % 4) / 2, words 2 and 3 to the same place two chunks on.  Lanes 8 i .. + 7 take rows 0, 2, 1, 3
    // of four, which keeps the stores of half a warp in different banks.
    const int h = warp - kFirstStager;
    const int sub = ((lane >> 3) & 1) * 2 + (lane >> 4), ci = lane & 7;
    const int nunits = p.ncols / 16;  // 16 rows each
    const uint32_t raw0 = base + kTsOffStages + stages * b_stage_bytes + h * b_half_bytes + sub * 128 + ci * 16;
    const uint32_t tile0_addr = base + kTsOffStages + h * b_half_bytes + sub * 128 + (ci & 1) * 8;
    const uint32_t c_even = ((((ci & 4) | ((ci >> 1) & 1)) ^ sub) << 4), c_odd = c_even ^ 64;  // rows sub and sub + 4 of eight
    TsRing ring(0, 1);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int blk = 0; blk < nblk; ++blk) {
      const int slot = blk & (kTsRawStages - 1);
      if (!mbar_wait_chain(base + kTsBarRawFull + 8 * slot, (blk / kTsRawStages) & 1) ||
          !mbar_wait_chain(base + kTsBarDone + 8 * ring.idx, ring.parity)) {
        failed = true;
        break;
      }
      uint32_t raw = raw0 + slot * b_stage_bytes, dst = tile0_addr + ring.idx * b_stage_bytes;
      for (int u = 0; u < nunits; ++u) {
        uint4 v[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) v[r] = lds_v4(raw + r * 512);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const uint32_t at = dst + r * 512 + ((r & 1) ? c_odd : c_even);
          sts_v2(at, v[r].x, v[r].y);
          sts_v2(at ^ 32, v[r].z, v[r].w);
        }
        raw += kTsUnitBytes;
        dst += kTsUnitBytes;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy accesses before the tensor pipe's and TMA's
      __syncwarp();
      if (lane == 0) mbar_arrive(base + kTsBarFull + 8 * ring.idx);
      ring.advance(1, stages);
    }
    if (failed) report_status(kStatusActivationCopyTimeout);
  } else {
    // ------------------------------------------------------------------ activation requests and MMAs
    // The activations come eight blocks ahead: every CTA reads the same lines at about the same time, and a request takes one
    // to two microseconds.  A block that is ready for its MMAs has left its raw stage.  Rows past the batch arrive as zeros.
    const uint32_t raw0 = base + kTsOffStages + stages * b_stage_bytes;
    auto request = [&](int blk) {  // by one lane
      const int slot = blk & (kTsRawStages - 1);
      const uint32_t bar = base + kTsBarRawFull + 8 * slot;
      mbar_arrive_expect_tx(bar, b_stage_bytes);
      tma_load_2d(raw0 + slot * b_stage_bytes, &xmap, (kb_lo + blk) * 128, m0, bar);
      tma_load_2d(raw0 + slot * b_stage_bytes + b_half_bytes, &xmap, (kb_lo + blk) * 128 + 64, m0, bar);
    };
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the activations may come from the kernel launched just before
    if (elect_one())
      for (int blk = 0; blk < min(nblk, kTsRawStages); ++blk) request(blk);
    __syncwarp();
    const uint32_t idesc = umma_instr_desc(BF16 ? 1 : 0, p.ncols);
    const uint64_t db0 = umma_smem_desc(base + kTsOffStages, 16, 1024, 2);
    const uint32_t b_stage16 = b_stage_bytes >> 4, b_half16 = b_half_bytes >> 4;
    TsRing ring(0, 0), d_ring(0, 1);
    int blk = 0;
    for (; blk < nblk; ++blk) {
      if (!mbar_wait_chain(base + kTsBarFull + 8 * ring.idx, ring.parity)) {
        failed = true;
        break;
      }
      const uint32_t a = tmem + a_col0 + ring.idx * (rbs * 64);
      const uint64_t db = db0 + ring.idx * b_stage16;
      constexpr int NG = GS == 32 ? 4 : 1, KS = 8 / NG;  // groups of a block, K steps of a group
#pragma unroll
      for (int q = 0; q < NG; ++q) {
        const bool first = GS != -1 || blk == 0;  // block of the group
        if (first && !mbar_wait_chain(base + kTsBarDEmpty + 8 * d_ring.idx, d_ring.parity)) {
          failed = true;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d = tmem + d_ring.idx * (rbs * dcols);
        if (elect_one()) {
          for (int r = 0; r < rbs; ++r) {
#pragma unroll
            for (int k = q * KS; k < (q + 1) * KS; ++k)
              umma_f16_ts(d + r * dcols, a + r * 64 + k * 8, db + static_cast<uint64_t>((k >> 2) * b_half16 + (k & 3) * 2), idesc,
                          (k > q * KS || !first) ? 1u : 0u);
          }
          if (q + 1 == NG) {
            // one commit for the stage and the accumulators: commits are what a short block's MMAs wait for
            umma_commit(base + kTsBarDone + 8 * ring.idx);
            if (blk + kTsRawStages < nblk) request(blk + kTsRawStages);
          }
        }
        __syncwarp();
        if (GS != -1) d_ring.advance(1, accs);
      }
      if (failed) break;
      ring.advance(1, stages);
    }
    // Nothing of this CTA may be in flight when it frees its memory.  A scaling warp that gave up has not waited for the MMAs,
    // and where this warp gives up at a block, the activations of that and the following ones may still be on their way.
    if (elect_one()) umma_commit(base + kTsBarEnd);
    __syncwarp();
    if (!mbar_wait_chain(base + kTsBarEnd, 0)) failed = true;
    for (int i = blk; i < min(nblk, blk + kTsRawStages); ++i)
      if (!mbar_wait_chain(base + kTsBarRawFull + 8 * (i & (kTsRawStages - 1)), (i / kTsRawStages) & 1)) break;
    if (failed) report_status(kStatusWeightCopyTimeout);
  }

  // ---------------------------------------------------------------------- sums of a split K
  __syncwarp();
  if (p.split > 1) {
    // The CTAs of one cluster share the tiles along K.  Each adds, in the order of the K ranges, the batch rows it owns.
    cluster_sync_all();
    if (warp < kFirstStager) {
      asm volatile("griddepcontrol.wait;" ::: "memory");  // a producer with few blocks has not waited yet
      const int per = (p.ncols + p.split - 1) / p.split;
      const int c_lo = sk * per, c_hi = min(min(c_lo + per, p.ncols), mrows);
      const int vecs = slots / 4;  // four out-features a step
      for (int idx = threadIdx.x; idx < (c_hi - c_lo) * vecs; idx += kFirstStager * 32) {
        const int c = rbs == 2 ? idx >> 6 : idx >> 5, v4 = idx - c * vecs, slot = v4 * 4;
        const int tile = ((slot >> 5) & 3) + 4 * ((slot >> 4) & 1) + 8 * (slot >> 7);
        if (tile < tiles) {
          const uint32_t local = base + kTsOffStages + ((c_lo + c) * slots + slot) * 4;
          float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int s = 0; s < p.split; s += 2) {
            const float4 a = ld_cluster_f32x4(map_to_cta(local, s));
            float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
            if (s + 1 < p.split) b = ld_cluster_f32x4(map_to_cta(local, s + 1));
            sum.x = (sum.x + a.x) + b.x;
            sum.y = (sum.y + a.y) + b.y;
            sum.z = (sum.z + a.z) + b.z;
            sum.w = (sum.w + a.w) + b.w;
          }
          uint16_t *dst = p.y + static_cast<size_t>(m0 + c_lo + c) * p.N + (tile0 + tile) * 16 + (slot & 15);
          const uint16_t o0 = to_out16<BF16>(sum.x), o1 = to_out16<BF16>(sum.y), o2 = to_out16<BF16>(sum.z), o3 = to_out16<BF16>(sum.w);
          if ((reinterpret_cast<uintptr_t>(dst) & 7u) == 0) {
            *reinterpret_cast<uint2 *>(dst) = make_uint2(o0 | (static_cast<uint32_t>(o1) << 16), o2 | (static_cast<uint32_t>(o3) << 16));
          } else {
            dst[0] = o0;
            dst[1] = o1;
            dst[2] = o2;
            dst[3] = o3;
          }
        }
      }
    }
    __syncwarp();
    cluster_sync_all();  // nobody leaves while its sums are still being read
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kMma) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// ----------------------------------------------------------------------------
// host side
// ----------------------------------------------------------------------------
// What a block of 128 in-features takes, in microseconds: 4, 8 and 16 row tiles a CTA at 32 columns, and for every column above.
// Groups of 32 scale and sum four times a block, one scale per row once in all.
struct TsBlockCost {
  float tiles4, tiles8, tiles16, column;
};
static TsBlockCost ts_block_cost(int group_size) {
  if (group_size == 32) return {1.27f, 1.31f, 1.74f, 0.0165f};
  if (group_size == 128) return {0.73f, 0.78f, 1.04f, 0.0066f};
  return {0.44f, 0.48f, 0.59f, 0.0028f};
}

// Batch blocks of at most 64 rows; 4, 8 or 16 row tiles a CTA (16 with at most 32 rows: a scaling warp holds 32 sums a lane).
// Among these and the K splits up to `max_split` the cheapest by a model of the kernel fitted on B200 to 16419 launches (every
// plan of 1191 products, 2 to 8 bits, all groups, 17 to 512 rows, cold weights): its figures are within 5 % of the measured
// ones (root mean square), the plans it takes within 3 % of the best one for nine products of ten.  4 bits, group 128, model /
// measured in us: 4096 x 4096 at 32 rows 11.6 / 12.7, 64 rows 14.3 / 15.3, 128 rows 22.2 / 22.3; 1024 x 4096 at 128 rows
// 11.9 / 12.3; 14336 x 4096 at 32 rows 22.6 / 23.5 (29.1 with the plan of a model that left out the sums of the activations).
TsPlan gemm_ts_plan(int N, int K, int M, int group_size, int max_split, int sm_count, const int *clusters_at_once) {
  TsPlan best = {};
  best.blocks = (M + kTsMaxCols - 1) / kTsMaxCols;
  const int rows = (M + best.blocks - 1) / best.blocks;
  best.ncols = (rows + 15) / 16 * 16;
  const int tiles16 = N / 16, kblocks = K / 128;
  const TsBlockCost costs = ts_block_cost(group_size);
  const float columns = costs.column * static_cast<float>(best.ncols > 32 ? best.ncols - 32 : 0);
  float best_cost = 1e30f;
  for (int rt = 4; rt <= (best.ncols <= 32 ? 16 : 8); rt *= 2) {
    const long long clusters = static_cast<long long>((tiles16 + rt - 1) / rt) * best.blocks;
    const float block = (rt == 4 ? costs.tiles4 : rt == 8 ? costs.tiles8 : costs.tiles16) + columns;
    const float launch = 2.1f + (best.ncols > 32 ? 1.f : 0.f) + (rt == 16 ? 0.87f : 0.f);
    for (int split = 1; split <= max_split && split <= kblocks; ++split) {
      const int at_once = split == 1 ? sm_count : clusters_at_once ? clusters_at_once[split - 2] : tc_clusters_at_once(split);
      const float waves = static_cast<float>((clusters - 1) / at_once + 1);  // at_once may be INT_MAX
      const long long ctas = clusters * split;
      const float cost = launch + 0.0155f * static_cast<float>(ctas < sm_count ? ctas : sm_count) +
                         (split > 1 ? 1.15f + 0.035f * split : 0.f) +  // the cluster's reduction
                         waves * static_cast<float>((kblocks + split - 1) / split) * block +
                         (waves - 1.f) * (split > 1 ? 4.9f : 3.5f);  // a CTA's own start and end, again in every wave
      if (cost < best_cost) {
        best_cost = cost;
        best.tiles = rt;
        best.split = split;
      }
    }
  }
  const int rb = ts_row_blocks(best.tiles);
  // the accumulators first (four, or two where sixteen tiles leave too little for the weights), the rest for the weights
  best.accumulators = group_size == 32 || rb == 1 ? 4 : 2;
  best.stages = (512 - best.accumulators * rb * ts_dcols(best.ncols)) / (64 * rb);
  if (best.stages > kTsMaxStages) best.stages = kTsMaxStages;
  best.smem = kTsOffStages + 1024 + (best.stages + kTsRawStages) * best.ncols * 256;
  return best;
}

template <int B, int GS, bool BF16>
static int launch_ts(const TsParams &p, const TsPlan &plan, cudaStream_t stream, bool pdl) {
  auto kernel = gemm_ts_kernel<B, GS, BF16>;
  static SharedMemoryOptIn opt_in;  // one per instantiation of this launcher
  {
    const int st = opt_in.ensure(kernel, kTsOffStages + 1024 + (4 + kTsRawStages) * kTsMaxCols * 256);
    if (st != MG_OK) return st;
  }
  CUtensorMap xmap;
  if (tc_make_x_tensor_map(&xmap, p.x, p.M, p.K, p.ncols, false) != MG_OK) return MG_ERR_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((p.N / 16 + plan.tiles - 1) / plan.tiles, plan.split, plan.blocks);
  cfg.blockDim = dim3(kTsWarps * 32, 1, 1);
  cfg.dynamicSmemBytes = plan.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  int na = 0;
  if (pdl) {
    attrs[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  if (plan.split > 1) {
    attrs[na].id = cudaLaunchAttributeClusterDimension;
    attrs[na].val.clusterDim.x = 1;
    attrs[na].val.clusterDim.y = static_cast<unsigned>(plan.split);
    attrs[na].val.clusterDim.z = 1;
    ++na;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = na;
  return cudaLaunchKernelEx(&cfg, kernel, p, xmap) == cudaSuccess ? MG_OK : MG_ERR_CUDA;
}

template <int B>
static int launch_ts_group(const TsParams &p, const TsPlan &plan, int group_size, bool bf16, cudaStream_t stream, bool pdl) {
  switch (group_size) {
    case -1: return bf16 ? launch_ts<B, -1, true>(p, plan, stream, pdl) : launch_ts<B, -1, false>(p, plan, stream, pdl);
    case 32: return bf16 ? launch_ts<B, 32, true>(p, plan, stream, pdl) : launch_ts<B, 32, false>(p, plan, stream, pdl);
    case 128: return bf16 ? launch_ts<B, 128, true>(p, plan, stream, pdl) : launch_ts<B, 128, false>(p, plan, stream, pdl);
    default: return MG_ERR_BAD_ARG;
  }
}

static int launch_ts_bits(const TsParams &p, const TsPlan &plan, int bitwidth, int group_size, bool bf16, cudaStream_t stream, bool pdl) {
  switch (bitwidth) {
    case 2: return launch_ts_group<2>(p, plan, group_size, bf16, stream, pdl);
    case 3: return launch_ts_group<3>(p, plan, group_size, bf16, stream, pdl);
    case 4: return launch_ts_group<4>(p, plan, group_size, bf16, stream, pdl);
    case 6: return launch_ts_group<6>(p, plan, group_size, bf16, stream, pdl);
    case 8: return launch_ts_group<8>(p, plan, group_size, bf16, stream, pdl);
    default: return MG_ERR_BAD_ARG;
  }
}

int gemm_ts_launch(int bitwidth, int group_size, int N, int K, int M, const void *w, const void *s, const void *z, const void *x,
                   void *y, bool bf16, bool pdl, cudaStream_t stream) {
  int sm_count = 0;
  {
    const int st = current_device_sm_count(&sm_count);
    if (st != MG_OK) return st;
  }
  TsParams p;
  p.w = static_cast<const uint32_t *>(w);
  p.s = static_cast<const uint16_t *>(s);
  p.z = static_cast<const uint16_t *>(z);
  p.x = static_cast<const uint16_t *>(x);
  p.y = static_cast<uint16_t *>(y);
  p.N = N;
  p.K = K;
  p.M = M;
  p.kblocks = K / 128;
  const auto launch = [&](int max_split, int *split) {
    const TsPlan plan = gemm_ts_plan(N, K, M, group_size, max_split, sm_count, nullptr);
    *split = p.split = plan.split;
    p.tiles = plan.tiles;
    p.ncols = plan.ncols;
    p.accumulators = plan.accumulators;
    p.stages = plan.stages;
    return launch_ts_bits(p, plan, bitwidth, group_size, bf16, stream, pdl);
  };
  int split = 1;
  int r = launch(8, &split);
  if (r == MG_ERR_CUDA && split > 1) {  // a device that cannot place the cluster (a partitioned GPU, say): nothing was launched
    (void)cudaGetLastError();
    r = launch(1, &split);  // with the tiles and stages of a launch without clusters
  }
  return r;
}

MG_DEFINE_STATUS_ACCESSOR(gemm_ts_device_status)

}  // namespace mg

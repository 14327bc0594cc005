// Fused kernels over wide-window images (bxr_format.h, BXR_MODE_WINDOW4): 4-bit exponent codes inside a 16-binade
// row window, so that a weight outside its window is a rarity (fewer than one in ten thousand on Gaussian rows) and
// the decoded words never have to touch shared memory:
//   * kUmma  : a lane holds the 32 weights of its row and phase in 16 registers and writes them with one tcgen05.st
//              into tensor memory, where tcgen05.mma takes them as its A operand (M = 128 weight rows; the batch is
//              N, read from shared memory).  Shared memory carries only what comes from outside the SM: chunk blobs
//              and activation tiles.  One elected lane issues all MMAs of an item into one accumulator.  (In the 3-bit
//              window kernel the operand tile lives in shared memory, and its stores plus the tensor core's reads of it
//              are more than 40 % of all shared-memory traffic, which sets that kernel's pace; its per-chunk exception patching is what keeps it from using tensor memory: done
//              in registers it costs more instructions than the decode itself.)
//   * kDense : decode twin (parity tests, ResidentWeight.decode).
// Same persistent, warp-specialised pipeline and work partition as the other fused kernels; any batch size, the
// batch of one padded to the narrowest tile.
#pragma once
#include "bxr_kernels.cuh"

namespace grb {

constexpr int kWideWarpLoader = 16;    // bulk copies of chunk blobs
constexpr int kWideWarpMma = 17;       // TMEM owner and MMA issuer
constexpr int kWideWarpXLoader = 18;   // TMA loads of activation tiles
constexpr int kWideWarpSlices = 19;    // partial tiles of the closing reduction
constexpr int kWideWarpEpilogue = 20;  // 4 warps: warp % 4 = the tensor-memory lane quarter a warp may read

// Tensor memory: columns [0, 256) accumulators, FP32, one of NB columns per item.  Up to NB = 128 two items fit, one being
// multiplied while the other is drained.  (Two issuing threads with an accumulator each, chunk about, which the epilogue
// added, left room for one item at NB = 128, whose drain the issuers then waited for; since the issuing lane is an elected
// one it keeps up alone.  34816 x 5120 at 128 rows 61.6 -> 59.7 us, 5120 x 17408 35.7 -> 35.2 us, 5120 x 5120 at 192 rows
// 17.8 -> 17.2 us; one row unchanged.)  An item's sum is one chain of FP32 additions in K order, twice as long as either of
// the two that were added before: y's rms and largest errors against a 64-bit product are the same to five digits, but 0.25 %
// of 34816 x 5120's outputs are not the BF16 nearest to it, where 0.13 % were not (5120 x 17408: 0.28 and 0.15 %).  Columns
// [256, 512): the decoded weights of four chunks, 64 columns each (two 128 x 64
// atoms, two BF16 per column).  (The narrow tiles would leave room for six or seven stages and a deeper activation ring;
// measured at NB = 16 with 7 stages, 8 activation stages and 6 requests in flight, every M = 1 launch got slower, gate|up by
// 4.6 us.)
constexpr int kWideNextBlobs = 8;      // blobs per CTA of the next launch that a finishing CTA asks the L2 for
constexpr uint32_t kWideTmemCols = 512;
// The 192-column tile, for batches above 128 rows: room for one item's accumulator.  Such a batch is bound by
// the number of its passes over the weights: at 128 columns the tensor core is busy for 38 % of a pass, and a pass costs
// little more at 192 (34816 x 5120: 60 -> 72.5 us by single CTAs).
//
// Pairs of CTAs (PAIR, cta_group::2), for batches above 128 rows.  Such a batch is bound by the power cap (a pass of 192 rows
// by single CTAs settles at 1.25 GHz), that is by what a multiply costs in energy besides the multiply: decoding and
// streaming a chunk, and bringing its activations in through L2.  Two CTAs of a cluster walk the same chunks of two row blocks side by
// side; the one of even rank issues MMAs of M = 256 for both, each CTA's tensor memory holding the decoded weights and the
// accumulators of its own row block and each CTA's shared memory half of the activation rows.  With that and two
// accumulator tiles (T = 2) a pass takes 384 rows, so that a chunk is streamed, decoded and written to tensor memory once for
// twice the rows and meets half the activation bytes per row.  At 384 rows, two passes before and one now: 34816 x 5120 147 ->
// 106 us, 5120 x 17408 86 -> 64 us, 7168 x 5120 42 -> 30 us, 5120 x 5120 36 -> 25 us.  (Barriers that a peer arrives on with
// release and acquire at cluster scope cost 1.4 us a chunk; the plain forms order what matters here, the completed tensor
// memory stores and bulk copies.  At 128 rows pairs gain nothing: 34816 x 5120 58.4 against 59.4 us, 7168 x 5120 18.4 against
// 17.0 us.)
template <int NB, int T>
constexpr int kWideAccBufs = T == 1 && NB <= 128 ? 2 : 1;  // items whose accumulators fit tensor memory at once
template <int NB, int T>
constexpr int kWideStages = T * NB <= 256 ? 4 : 2;         // (two are enough at 384 columns: a chunk's multiply takes 1536 tensor-core cycles)
template <int NB, int T>
constexpr uint32_t kWideOperandCol = kWideTmemCols - 64u * kWideStages<NB, T>;

// Shared-memory plan: a ring of chunk blobs and a ring of activation tiles (T x two atoms of 64 columns per chunk, each of the
// rows this CTA brings in).
template <int MODE, int NB, int T, bool PAIR>
struct BxqSmem {
  static constexpr int kOp = (MODE == kUmma) ? kWideStages<NB, T> : 0;
  static constexpr uint32_t kXRows = NB / (PAIR ? 2 : 1);     // activation rows of one tile that this CTA holds
  static constexpr uint32_t kXAtom = kXRows * 128;
  static constexpr uint32_t kXStage = T * 2 * kXAtom;
  static constexpr int kX = (MODE != kUmma) ? 0 : kXStage <= 16384 ? (PAIR ? 5 : 4) : kXStage <= 24576 ? 4 : 3;
  static constexpr bool kXOwn = kX != kOp;                    // activation stages are handed back on barriers of their own
  static constexpr uint32_t kReserve = 1024 /* alignment slack */ + 512 /* barriers, flags */;
  // the epilogue warps turn their accumulator columns around in shared memory (a lane holds one weight row, memory
  // wants consecutive rows together): so many columns x 32 rows x 2 bytes per warp
  static constexpr uint32_t kTurnCols = NB >= 32 && kXStage <= 32768 ? 32 : 16, kTurn = (MODE == kUmma) ? kTurnCols * 64 : 0;
  static constexpr int kInFit = int((232448u - kReserve - kX * kXStage - 4 * kTurn) / BXQ_BLOB_MAX);
  static constexpr int kIn = kInFit > 7 ? 7 : kInFit;   // (more barriers would not fit the one-per-lane set-up)
  static constexpr uint32_t xs = 0;
  static constexpr uint32_t turn = xs + kX * kXStage;
  static constexpr uint32_t in = turn + 4 * kTurn;
  static constexpr uint32_t bars = in + kIn * BXQ_BLOB_MAX;
  // barrier order: in_full, in_empty [kIn each]; op_full, op_empty [kOp each]; x_full [kX]; x_empty [kX, if kXOwn];
  // acc_full, acc_empty [2 each]; final; slice_full, slice_used [kSlices each], swap_used, swap_full (the closing reduction); meet (the epilogue warps)
  // the closing reduction: the CTA's own tile of NB batch rows, and slices of kSliceRows batch rows of the others' on their way
  static constexpr uint32_t kSliceRows = T * NB <= 128 ? NB : 64, kSlice = kSliceRows * BXR_ROWS * 4;
  static constexpr uint32_t kSlicesFit = MODE == kUmma ? (bars - NB * 512u) / kSlice : 0, kSlices = kSlicesFit > 8 ? 8 : kSlicesFit;
  static constexpr uint32_t nbars = 2 * kIn + 2 * kOp + (kXOwn ? 2 : 1) * kX + 4 + 1 + 2 * kSlices + 3;
  static constexpr uint32_t misc = (bars + 8 * nbars + 15) & ~15u;  // tmem base, abort flag, decision
  static constexpr uint32_t total = misc + 48;
  static constexpr uint32_t alloc = total + 1024;
  static_assert(MODE != kUmma || kIn >= 3, "ring too shallow");
  static_assert(MODE != kUmma || T * NB * kWideAccBufs<NB, T> <= int(kWideOperandCol<NB, T>), "accumulators overlap the operand columns");
  static_assert(8 * nbars + 64 <= 512, "barrier area");
  static_assert(MODE != kUmma || (T * NB * 512u <= bars && kSlices >= 2), "kept tiles and slices would overwrite the barriers");
  static_assert(alloc <= 232448, "exceeds the 227 KB of shared memory a CTA may opt into");
};

// A code word holds four column pairs: pair k has the code of its even column in bits [4k, 4k+4) and that of its odd
// column 16 bits higher.  One mask and one multiply-add (whose addend is the row base in both halves) put a pair into
// packed-BF16 exponent position; `hi` is the word shifted right by 8, which brings pairs 2 and 3 to where pairs 0
// and 1 are.  The mask runs on the integer pipe, the multiply-add on the FMA pipe (the multipliers are kernel
// parameters so that the compiler does not turn them back into shifts).
template <int K>
__device__ __forceinline__ uint32_t bxq_exponents(uint32_t lo, uint32_t hi, const BxwPowers& p, uint32_t base2) {
  if constexpr (K == 0) return (lo & BXQ_PAIR_MASK) * p.p7 + base2;
  else if constexpr (K == 1) return (lo & (BXQ_PAIR_MASK << 4)) * p.p3 + base2;
  else if constexpr (K == 2) return (hi & BXQ_PAIR_MASK) * p.p7 + base2;
  else return (hi & (BXQ_PAIR_MASK << 4)) * p.p3 + base2;
}
// raw bytes (sign << 7 | mantissa) of two columns merged with their exponents
__device__ __forceinline__ uint32_t bxq_join(uint32_t raw4, uint32_t selector, uint32_t exponents) {
  return (__byte_perm(raw4, 0, selector) & 0x807F807Fu) | exponents;
}
// The 32 weights of a lane, two per register in column order: four code words and the raw bytes of its two
// 16-column pieces.
__device__ __forceinline__ void bxq_decode32(const uint32_t (&w)[4], const uint4& rf, const uint4& rb, const BxwPowers& p,
                                             uint32_t base2, uint32_t (&out)[16]) {
  const uint32_t raw[8] = {rf.x, rf.y, rf.z, rf.w, rb.x, rb.y, rb.z, rb.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t lo = w[j], hi = w[j] >> 8;
    out[4 * j + 0] = bxq_join(raw[2 * j], 0x1100, bxq_exponents<0>(lo, hi, p, base2));
    out[4 * j + 1] = bxq_join(raw[2 * j], 0x3322, bxq_exponents<1>(lo, hi, p, base2));
    out[4 * j + 2] = bxq_join(raw[2 * j + 1], 0x1100, bxq_exponents<2>(lo, hi, p, base2));
    out[4 * j + 3] = bxq_join(raw[2 * j + 1], 0x3322, bxq_exponents<3>(lo, hi, p, base2));
  }
}
// An exception entry applied to the registers of the lane that owns it: the exponent field of one half of one
// register is replaced.  The register index is data, so the choice is sixteen predicated operations; this runs only
// for the rare warp that has entries at all.
__device__ __forceinline__ void bxq_patch(uint32_t (&out)[16], uint32_t column, uint32_t exponent) {
  const uint32_t reg = column >> 1, sh = (column & 1u) ? 16u : 0u;
#pragma unroll
  for (int i = 0; i < 16; ++i)
    if (reg == uint32_t(i)) out[i] = (out[i] & ~(0x7F80u << sh)) | (exponent & 0xFFu) << (7 + sh);
}

// The work of a CTA is a contiguous range of the (row block, chunk) sequence; an item is the part of it that lies in
// one row block.  Everything but the epilogue needs only the geometry of an item, which follows from the range by
// arithmetic: no load stands between the start of a CTA and its first blob, window base and multiply.  (The item
// list in the image holds the same geometry plus the partial-tile bookkeeping - part, parts, slot - which the
// epilogue reads with plenty of time to spare; bxr_validate checks that the two agree.)
//
// Paired images: workers 2p and 2p + 1 have the same share, share p of the (pair of row blocks, chunk) sequence; worker 2p + r
// takes row block 2g + r of pair g.  `row_block` below counts pairs then.
struct WideSpan {
  uint32_t row_block, chunk_begin, chunk_end;
};
__device__ __forceinline__ WideSpan wide_span(uint32_t unit, uint32_t unit_end, uint32_t chunks) {
  const uint32_t rb = unit / chunks, c0 = unit - rb * chunks;
  return {rb, c0, min(chunks, c0 + (unit_end - unit))};
}

__device__ __forceinline__ uint32_t wide_pack(float lo, float hi) {
  const __nv_bfloat162 pair = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&pair);
}

// The closing reduction of a row block whose parts belong to the CTAs of one thread-block cluster (the partition is
// "aligned": workers = row blocks x P, CTA rank r of cluster b owns part r of row block b, in K order).  Every CTA has
// left its FP32 tile at the start of its shared memory; after the cluster barrier each CTA adds the P tiles of ITS share
// of the batch columns (m = rank, rank + P, ...) in rank order - its own from local shared memory, the others over
// distributed shared memory - and writes y.  No partial tile goes to global memory, no counter, no fence, and the work
// of the reduction is spread over the P SMs.  t = index of the calling thread among the (kDecoderWarps + 4) x 32.  In a cluster
// of pairs (two row blocks side by side) part p of this CTA's row block belongs to rank 2p + (own rank mod 2).
// A peer's shared memory answers after some 1.5 us with all SMs asking, so what a thread needs is loads in flight: U positions
// of up to MAXP parts at once, so that 128 batch rows are one round (5120 x 5120 in clusters of three at 384 rows: 27.2 -> 25.1
// us, 7168 x 5120 in clusters of two 32.6 -> 30.4).
template <bool PAIR, int MAXP, int U>
__device__ __forceinline__ void bxq_reduce_in_cluster(const BxrArgs& args, uint32_t row_block, uint32_t smem, uint32_t t) {
  constexpr uint32_t kThreads = (kDecoderWarps + 4) * 32;
  const uint32_t parts = args.cluster, in_cluster = cluster_rank(), rank = PAIR ? in_cluster >> 1 : in_cluster;
  const uint32_t mine = rank < args.m ? (args.m - rank + parts - 1) / parts : 0;  // batch columns rank, rank + P, ... below m
  const uint32_t row4 = row_block * BXR_ROWS + (t & 31) * 4;    // (kThreads is a multiple of 32: the same for all of a thread's positions)
  if (row4 >= args.rows) return;
  float bias4[4] = {0.f, 0.f, 0.f, 0.f};
  if (args.bias)
    for (int k = 0; k < 4; ++k)
      if (row4 + k < args.rows) bias4[k] = __bfloat162float(args.bias[row4 + k]);
  uint32_t tile[MAXP];
#pragma unroll
  for (uint32_t p = 0; p < MAXP; ++p)
    if (p < parts) tile[p] = cluster_map(smem, PAIR ? 2 * p + (in_cluster & 1u) : p);
  for (uint32_t i0 = t; i0 < mine * 32; i0 += U * kThreads) {
    uint4 u[U][MAXP];
#pragma unroll
    for (uint32_t j = 0; j < U; ++j) {
      const uint32_t i = i0 + j * kThreads, m = rank + (i >> 5) * parts;
#pragma unroll
      for (uint32_t p = 0; p < MAXP; ++p)
        if (i < mine * 32 && p < parts) u[j][p] = p == rank ? lds128(smem + ((m << 5) | (i & 31)) * 16) : lds128_cluster(tile[p] + ((m << 5) | (i & 31)) * 16);
    }
#pragma unroll
    for (uint32_t j = 0; j < U; ++j) {
      const uint32_t i = i0 + j * kThreads, m = rank + (i >> 5) * parts;
      if (i >= mine * 32) break;
      // part 0 is taken as it is: adding it to zero would lose the sign of a -0
      float f[4] = {__uint_as_float(u[j][0].x), __uint_as_float(u[j][0].y), __uint_as_float(u[j][0].z), __uint_as_float(u[j][0].w)};
#pragma unroll
      for (uint32_t p = 1; p < MAXP; ++p)
        if (p < parts) {
          f[0] = __fadd_rn(f[0], __uint_as_float(u[j][p].x));
          f[1] = __fadd_rn(f[1], __uint_as_float(u[j][p].y));
          f[2] = __fadd_rn(f[2], __uint_as_float(u[j][p].z));
          f[3] = __fadd_rn(f[3], __uint_as_float(u[j][p].w));
        }
      if (args.bias)
        for (int k = 0; k < 4; ++k) f[k] = __fadd_rn(f[k], bias4[k]);
      __nv_bfloat16* dst = args.y + size_t(m) * args.ldy + row4;
      if (row4 + 3 < args.rows && (reinterpret_cast<uintptr_t>(dst) & 7u) == 0) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(wide_pack(f[0], f[1]), wide_pack(f[2], f[3]));
      } else {
        for (int k = 0; k < 4; ++k)
          if (row4 + k < args.rows) dst[k] = __float2bfloat16_rn(f[k]);
      }
    }
  }
}
// The closing reduction of a split row block by the 16 decoder warps: y[m, row] = bf16(sum of the row block's FP32 tiles in K
// order (+ bias)), for the batch rows [m_at, m_end) of one accumulator tile.  The others' tiles come from L2, a round trip of
// 1.4 us with all SMs asking and up to 4 x 196 KB of them, so they are brought in by bulk copies slice by slice (BxqSmem), in the
// order they are added, as many ahead as shared memory holds; warp kWideWarpSlices asks for them.  The CTA's own tile (part
// `own`, none if >= parts) lies at the start of shared memory.  A thread owns the same few positions of four weight rows in every
// slice.  Slices are whole tiles up to 128 columns (5120 x 17408 at 128 rows: 34.0 us, 35.6 with 32 rows a slice) and 64 batch
// rows above (at 384 rows: whole 192-row tiles, one at a time, 75 us; 64 rows 64 us; 32 rows 67 us).
// `n` counts slices through the launch (ring position and barrier phase).
template <class L>
__device__ __forceinline__ void bxq_add_tiles(const BxrArgs& args, const RoleCtx& ctx, uint32_t row_block, uint32_t parts, uint32_t own,
                                              uint32_t smem, uint32_t ring, uint32_t bar_full, uint32_t bar_used, uint32_t t, uint32_t m_at, uint32_t m_end,
                                              uint32_t& n) {
  constexpr uint32_t kThreads = kDecoderWarps * 32, kMine = (L::kSliceRows * 32 + kThreads - 1) / kThreads;
  const uint32_t row4 = row_block * BXR_ROWS + (t & 31) * 4;
  float bias4[4] = {0.f, 0.f, 0.f, 0.f};
  if (args.bias)
    for (int i = 0; i < 4; ++i)
      if (row4 + i < args.rows) bias4[i] = __bfloat162float(args.bias[row4 + i]);
  for (uint32_t m0 = m_at; m0 < m_end; m0 += L::kSliceRows) {
    float4 sum[kMine];
    for (uint32_t p = 0; p < parts; ++p) {
      uint32_t src = smem + (m0 - m_at) * BXR_ROWS * 4;
      const uint32_t b = n % L::kSlices;
      if (p != own) {
        if (!ctx.wait_warp(bar_full + 8 * b, (n / L::kSlices) & 1)) return;
        src = ring + b * L::kSlice;
      }
#pragma unroll
      for (uint32_t k = 0; k < kMine; ++k) {
        const uint32_t at = t + k * kThreads;
        if (m0 + (at >> 5) >= m_end || at >= L::kSliceRows * 32) continue;
        const uint4 u = lds128(src + at * 16);
        if (p == 0) {  // taken as it is: adding it to zero would lose the sign of a -0
          sum[k] = make_float4(__uint_as_float(u.x), __uint_as_float(u.y), __uint_as_float(u.z), __uint_as_float(u.w));
        } else {
          sum[k].x = __fadd_rn(sum[k].x, __uint_as_float(u.x));
          sum[k].y = __fadd_rn(sum[k].y, __uint_as_float(u.y));
          sum[k].z = __fadd_rn(sum[k].z, __uint_as_float(u.z));
          sum[k].w = __fadd_rn(sum[k].w, __uint_as_float(u.w));
        }
      }
      if (p != own) {
        __syncwarp();
        if ((t & 31) == 0) mbar_arrive(bar_used + 8 * b);
        ++n;
      }
    }
#pragma unroll
    for (uint32_t k = 0; k < kMine; ++k) {
      const uint32_t at = t + k * kThreads, m = m0 + (at >> 5);
      if (m >= m_end || at >= L::kSliceRows * 32 || m >= args.m || row4 >= args.rows) continue;
      float f[4] = {sum[k].x, sum[k].y, sum[k].z, sum[k].w};
      if (args.bias)
        for (int i = 0; i < 4; ++i) f[i] = __fadd_rn(f[i], bias4[i]);
      __nv_bfloat16* dst = args.y + size_t(m) * args.ldy + row4;
      if (row4 + 3 < args.rows && (reinterpret_cast<uintptr_t>(dst) & 7u) == 0) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(wide_pack(f[0], f[1]), wide_pack(f[2], f[3]));
      } else {
        for (int i = 0; i < 4; ++i)
          if (row4 + i < args.rows) dst[i] = __float2bfloat16_rn(f[i]);
      }
    }
  }
}
// Waits until `tiles` parts of a row block are in memory and clears the block's counter.  All have been declared, by CTAs that
// wait for nobody before they publish.  False if the limit ran out: the counter is then left as it is, since parts may still
// be counted into it, and the host has to clear the workspace before the next launch over it.
__device__ __forceinline__ bool bxq_parts_in_memory(const BxrArgs& args, const RoleCtx& ctx, uint32_t row_block, uint32_t tiles) {
  const unsigned long long t0 = global_ns();
  while ((ld_acquire_gpu(args.counters + row_block) >> 16) < tiles)
    if (global_ns() - t0 > kWaitLimitNs) {
      ctx.abort(kStatusTimeout);
      return false;
    }
  args.counters[row_block] = 0;
  return true;
}
// (batch rows of one accumulator tile that there are, in whole eights)
__device__ __forceinline__ uint32_t wide_tile_cols(uint32_t m, uint32_t tile, uint32_t nb) { return (min(m - min(m, tile * nb), nb) + 7) & ~7u; }

template <int MODE, int NB, int T = 1, bool PAIR = false>
__global__ void __launch_bounds__(MODE == kUmma ? kThreadsUmma : kThreadsSimt, 1)
bxq_kernel(const BxrArgs args, const __grid_constant__ CUtensorMap tmap_x) {
  using L = BxqSmem<MODE, NB, T, PAIR>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // A row block cut into P = args.cluster parts belongs to P workers in a row.  Pairs: a cluster of 2P CTAs has two row blocks,
  // part and row block alternating by rank.
  uint32_t worker = blockIdx.x;
  if (PAIR && args.cluster > 1) {
    const uint32_t n = blockIdx.x / (2 * args.cluster), in_cluster = blockIdx.x - n * 2 * args.cluster;
    worker = (2 * n + (in_cluster & 1u)) * args.cluster + (in_cluster >> 1);
  }
  const uint32_t my_rank = PAIR ? cluster_rank() : 0u;
  const bool leader = (my_rank & 1u) == 0;                 // issues the MMAs of its pair

  RoleCtx ctx;
  ctx.smem = smem;
  ctx.bars = smem + L::bars;
  ctx.abort_addr = smem + L::misc + 4;
  ctx.status = args.status;
  ctx.suspend = false;  // this pipeline is latency-bound: plain probes wake up sooner
  const uint32_t bar_in_full = ctx.bars, bar_in_empty = bar_in_full + 8 * L::kIn;
  const uint32_t bar_op_full = bar_in_empty + 8 * L::kIn, bar_op_empty = bar_op_full + 8 * L::kOp;
  const uint32_t bar_x_full = bar_op_empty + 8 * L::kOp;
  const uint32_t bar_x_empty = L::kXOwn ? bar_x_full + 8 * L::kX : bar_op_empty;   // (rings of one length: stage i of both is free together)
  const uint32_t bar_acc_full = bar_x_full + 8 * L::kX * (L::kXOwn ? 2 : 1), bar_acc_empty = bar_acc_full + 16, bar_final = bar_acc_empty + 16;
  const uint32_t bar_slice_full = bar_final + 8, bar_slice_used = bar_slice_full + 8 * L::kSlices;
  const uint32_t bar_swap_used = bar_slice_used + 8 * L::kSlices, bar_swap_full = bar_swap_used + 8, bar_meet = bar_swap_full + 8;
  constexpr uint32_t kTmemCols = kWideTmemCols;
  constexpr uint32_t kOpN = L::kOp ? L::kOp : 1;
  constexpr uint32_t kXN = L::kX ? L::kX : 1;
  constexpr uint32_t kAccBufs = kWideAccBufs<NB, T>, kOperandCol = kWideOperandCol<NB, T>;
  // accumulator `tile` of the CTA's n-th item: its place in tensor memory (T = 2: one per tile) and which use of the place it is
  auto acc_slot = [](uint32_t n_item, uint32_t tile) { return T == 1 ? n_item % kAccBufs : tile; };
  auto acc_use = [](uint32_t n_item) { return T == 1 ? n_item / kAccBufs : n_item; };

  // The blob loader's own barriers first of all (blobs of one size: it needs nothing else to start its copies): their
  // fences complete while the CTA's share of the work is being computed.
  if (warp == kWideWarpLoader && args.blob_stride16 && lane == 0) {
    for (uint32_t n = 0; n < uint32_t(L::kIn); ++n) mbar_init(bar_in_full + 8 * n, 1);
    mbar_fence_init();
    fence_proxy_async_smem();
  }
  // Work of this CTA, known from the arguments alone; the blob loader asks for its first offsets before anything
  // else so that the first copy can leave as soon as the barriers exist.
  const uint32_t group = args.paired ? 2u : 1u, in_group = args.paired ? worker & 1u : 0u;   // row block = (unit / chunks) * group + in_group
  const uint64_t units = uint64_t(args.row_blocks / group) * args.chunks;
  const uint32_t share = worker / group, shares = args.workers / group;
  const uint32_t unit_begin = uint32_t(units * share / shares);
  const uint32_t unit_count = uint32_t(units * (share + 1) / shares) - unit_begin;
  auto blob_of = [&](uint32_t unit) { const uint32_t g = unit / args.chunks; return (g * group + in_group) * args.chunks + (unit - g * args.chunks); };
  uint32_t first_i0 = 0, first_i1 = 0;
  if (warp == kWideWarpLoader && unit_count && !args.blob_stride16) {
    const uint32_t mine = unit_begin + min(uint32_t(lane), unit_count - 1);
    first_i0 = __ldg(args.blob_index + mine);
    first_i1 = __ldg(args.blob_index + mine + 1);
  }
  const uint32_t unit_end = unit_begin + unit_count;
  // Decoders: the window base of this thread's row in the CTA's first item, asked for before anything else.
  uint32_t first_base = 0;
  if (warp < kDecoderWarps && unit_count) first_base = args.base[((unit_begin / args.chunks) * group + in_group) * BXR_ROWS + (warp & 3) * 32 + lane];
  // Epilogue: where the CTA's items are in the image's list (their partial-tile bookkeeping); needed much later.
  uint32_t item_begin = 0, item_end = 0;
  if (MODE == kUmma && warp >= kWideWarpEpilogue) {
    item_begin = __ldg(args.worker_items + worker);
    item_end = __ldg(args.worker_items + worker + 1);
  }
  // An SM runs the launches of a stream back to back, so whatever a CTA does before its first multiply is not hidden
  // behind the previous launch on the SM that finished last.  The longest wait in it is the first blob's trip from
  // HBM: with blobs of one size the loader needs nothing but its own barriers to start it, and sets those up itself.
  uint32_t early = 0;
  if (warp == kWideWarpLoader && args.blob_stride16) {
    const uint32_t bytes = args.blob_stride16 << 4;
    if (bytes <= BXQ_BLOB_MAX && bytes >= BXQ_LIST_AT) early = min(unit_count, uint32_t(L::kIn));
    if (lane == 0) {
      const uint64_t once = l2_policy_evict_first();
      for (uint32_t u = 0; u < early; ++u) {
        mbar_arrive_expect_tx(bar_in_full + 8 * u, bytes);
        bulk_g2s(smem + L::in + u * BXQ_BLOB_MAX, args.blobs + size_t(blob_of(unit_begin + u)) * bytes, bytes, bar_in_full + 8 * u, once);
      }
    }
    __syncwarp();
  }
  if (warp == 0) {  // one or two barriers per lane
    static_assert(L::nbars <= 64, "two barriers per lane at most");
    const uint32_t i = lane;
#pragma unroll
    for (uint32_t n = i; n < L::nbars; n += 32) {
      if (n < uint32_t(L::kIn) && args.blob_stride16) continue;                    // in_full: the loader's own (above)
      constexpr uint32_t kCtas = PAIR ? 2 : 1;   // CTAs whose warps arrive on a leader's barriers
      uint32_t count = 1;                                                          // in_full, op_empty, x_full, x_empty
      if (n >= uint32_t(L::kIn) && n < 2u * L::kIn) count = kDecoderWarps;          // in_empty
      else if (n >= 2u * L::kIn && n < 2u * L::kIn + L::kOp) count = kDecoderWarps * kCtas;  // op_full
      else if (n >= 2u * L::kIn + 2 * L::kOp + (L::kXOwn ? 2 : 1) * L::kX) {
        const uint32_t j = n - (2u * L::kIn + 2 * L::kOp + (L::kXOwn ? 2 : 1) * L::kX);  // acc_full x2, acc_empty x2, final, slice_full, slice_used, swap_used, swap_full, meet
        count = j < 2 ? 1u : j < 4 ? 4u * kCtas : j < 5 ? 4u : j < 5 + L::kSlices ? 1u : j < 6 + 2 * L::kSlices ? uint32_t(kDecoderWarps) : 4u;
      }
      mbar_init(ctx.bars + 8 * n, count);
    }
    // flags: abort at misc + 4, epilogue decision at misc + 8, final decision at misc + 16 (misc + 0 receives the TMEM
    // base address from the allocating warp and is left alone here)
    if (i == 0) asm volatile("st.shared.v2.u32 [%0], {%1, %1};" ::"r"(smem + L::misc + 8), "r"(0u) : "memory");
    if (i == 1) asm volatile("st.shared.u32 [%0], %1;" ::"r"(smem + L::misc + 4), "r"(0u) : "memory");
    if (i == 2 || i == 3) asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(smem + L::misc + 16 * (i - 1)), "r"(0u) : "memory");
    mbar_fence_init();
  }
  if (MODE == kUmma && warp == kWideWarpMma) {
    tmem_alloc<PAIR>(smem + L::misc, kTmemCols);
    tmem_relinquish<PAIR>();
  }
  tc_fence_before();
  if (PAIR) cluster_sync();   // the peer arrives on this CTA's barriers
  else __syncthreads();
  tc_fence_after();
  // The image is never written by a kernel: everything up to the first access to x, bias, y or the workspace may
  // overlap the tail of the previous kernel in the stream.
  grid_dependents_may_launch();
  if (MODE == kDense) grid_dependency_wait();
  uint32_t tmem_base = 0;
  if (MODE == kUmma) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(smem + L::misc));


  // Epilogue warps: accumulator tile `t` of the CTA's n-th item, as [batch row][128 weight rows] FP32 (as in memory), to `dst`.
  auto drain_to_smem = [&](uint32_t n_item, uint32_t t, uint32_t dst) {
    constexpr int kStep = NB >= 32 ? 32 : 16;
    const uint32_t e = warp - kWideWarpEpilogue;
#pragma unroll 1
    for (uint32_t m0 = 0; m0 < wide_tile_cols(args.m, t, NB); m0 += kStep) {
      uint32_t v[kStep];
      if constexpr (kStep == 32) tmem_ld32(tmem_base + ((e * 32) << 16) + acc_slot(n_item, t) * NB + m0, v);
      else tmem_ld16(tmem_base + ((e * 32) << 16) + acc_slot(n_item, t) * NB + m0, v);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < kStep; ++i) sts32(dst + ((m0 + i) * BXR_ROWS + e * 32 + lane) * 4, v[i]);
    }
  };

  if (warp < kDecoderWarps) {
    // ------------------------------------------------------------------ decoders: 32 weights per lane and chunk
    const uint32_t q = warp >> 2, rg = warp & 3, r = rg * 32 + lane;
    uint32_t s = 0, ph = 0;    // input ring slot of the current chunk and its phase parity
    uint32_t so = 0, pho = 0;  // operand stage (tensor memory) of the current chunk
    const uint32_t raw_at = BXQ_RAW_AT + ((2 * q) * BXR_ROWS + r) * 16;
    const uint32_t code_at = BXQ_CODES_AT + 4 * (q * BXR_ROWS + r);
    // this lane's 16 operand columns: lane = row, columns = its 32 weights inside the chunk's atom
    const uint32_t operand_at = ((rg * 32u) << 16) + kOperandCol + (q >> 1) * 32 + (q & 1) * 16;
    const uint32_t op_full_at = PAIR ? cluster_map(bar_op_full, my_rank & ~1u) : bar_op_full;   // the issuer's
    uint32_t next_base = first_base;
    for (uint32_t u = unit_begin; u < unit_end;) {
      const WideSpan item = wide_span(u, unit_end, args.chunks);
      u += item.chunk_end - item.chunk_begin;
      const uint32_t row = (item.row_block * group + in_group) * BXR_ROWS + r;
      const uint32_t base2 = next_base * 0x00800080u;
      if (u < unit_end) next_base = args.base[row + group * BXR_ROWS];  // the next item's base: on its way while this item is decoded
      for (uint32_t c = item.chunk_begin; c < item.chunk_end; ++c) {
        // (On any content of the slot every read stays inside it, and a stage written too early spoils sums that nobody may use.
        // Votes on these two waits: 34816 x 5120 at one row 42.5 -> 44.9 us.)
        ctx.wait_or_go_on(bar_in_full + 8 * s, ph);
        const uint32_t blob = smem + L::in + s * BXQ_BLOB_MAX;
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = lds32(blob + code_at + 4 * BXR_SEGMENTS * j);
        const uint4 raw_f = lds128(blob + raw_at);
        const uint4 raw_b = lds128(blob + raw_at + BXR_ROWS * 16);
        const uint32_t e_lo = lds_u16(blob + BXQ_WARP_END_AT + 2 * warp);
        const uint32_t e_hi = min(lds_u16(blob + BXQ_WARP_END_AT + 2 * warp + 2), uint32_t(BXQ_ENTRY_MAX));
        uint32_t out[16];
        bxq_decode32(w, raw_f, raw_b, args.kw, base2, out);
        // Exceptions (weights outside their row window): rare.  Every lane reads the same entry; its owner acts.
        // Corrupt bounds are clamped so that every read stays inside the slot.
        for (uint32_t i = e_lo; i < e_hi; ++i) {
          const uint32_t v = lds32(blob + BXQ_LIST_AT + 4 * i);
          if (((v >> 5) & 31u) == uint32_t(lane)) bxq_patch(out, v & 31u, v >> 16);
        }
        __syncwarp();   // every lane has what it needs from the blob: hand the slot back
        if (lane == 0) mbar_arrive(bar_in_empty + 8 * s);
        if (MODE == kUmma) {
          ctx.wait_or_go_on(bar_op_empty + 8 * so, pho ^ 1);
          tc_fence_after();
          tmem_st16(tmem_base + operand_at + so * 64, out);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if (leader) mbar_arrive(bar_op_full + 8 * so);
            else mbar_arrive_cluster(op_full_at + 8 * so);
          }
          if (++so == kOpN) { so = 0; pho ^= 1; }
        } else if (row < args.rows) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t col = c * BXR_COLS + q * 32 + i * 8;
            uint16_t* dst = args.dense + size_t(row) * args.cols + col;
            if (col + 8 <= args.cols && (args.cols & 7) == 0) {
              *reinterpret_cast<uint4*>(dst) = make_uint4(out[4 * i], out[4 * i + 1], out[4 * i + 2], out[4 * i + 3]);
            } else {
              for (int e = 0; e < 8; ++e)
                if (col + e < args.cols) dst[e] = uint16_t(out[4 * i + (e >> 1)] >> (16 * (e & 1)));
            }
          }
        }
        if (++s == L::kIn) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == kWideWarpLoader) {
    // ------------------------------------------------------------------ chunk blobs, one bulk copy each
    uint32_t issued = 0;
    const uint64_t once = l2_policy_evict_first();  // a blob is read once per launch
    for (uint32_t u0 = 0; u0 < unit_count; u0 += 32) {
      uint32_t i0 = first_i0, i1 = first_i1;
      if (args.blob_stride16) {  // blobs of one size: no offsets to look up
        i0 = blob_of(unit_begin + min(u0 + lane, unit_count - 1)) * args.blob_stride16;
        i1 = i0 + args.blob_stride16;
      } else if (u0) {
        const uint32_t mine = unit_begin + min(u0 + lane, unit_count - 1);
        i0 = __ldg(args.blob_index + mine);
        i1 = __ldg(args.blob_index + mine + 1);
      }
      const uint32_t n = min(32u, unit_count - u0);
      bool live = true;
      for (uint32_t i = 0; i < n && live; ++i) {
        const uint32_t u = u0 + i, s = u % L::kIn, ph = (u / L::kIn) & 1;
        const uint32_t b0 = __shfl_sync(0xFFFFFFFFu, i0, i), b1 = __shfl_sync(0xFFFFFFFFu, i1, i);
        if (u < early) {  // requested before the set-up
          issued = u + 1;
          continue;
        }
        const uint32_t bytes = (b1 - b0) << 4;
        if (!ctx.go_warp(bar_in_empty + 8 * s, ph ^ 1)) { live = false; break; }
        if (b1 < b0 || bytes > BXQ_BLOB_MAX || bytes < BXQ_LIST_AT) {
          ctx.abort(kStatusBadArgument);
          live = false;
          break;
        }
        if (lane == 0) {
          mbar_arrive_expect_tx(bar_in_full + 8 * s, bytes);
          bulk_g2s(smem + L::in + s * BXQ_BLOB_MAX, args.blobs + (size_t(b0) << 4), bytes, bar_in_full + 8 * s, once);
        }
        issued = u + 1;
      }
      if (!live) break;
    }
    // Every load of this CTA is on its way: from here on it asks HBM for nothing.  Ask the L2 for what the next launch
    // of the stream will want first - the leading blobs of its CTAs w, w + workers, ... (consecutive in memory) - so
    // that they arrive during this launch's tail and the next launch's set-up.
    if (MODE == kUmma && args.next_blobs && lane == 0 && !ctx.aborted()) {
      for (uint32_t w2 = worker; w2 < args.next_workers; w2 += args.workers) {
        uint32_t first;
        const uint32_t n = bxr_leading_blobs(args.next_row_blocks, args.next_chunks, args.next_workers, args.next_paired, w2, kWideNextBlobs, &first);
        for (uint32_t b = 0; b < n; ++b) bulk_prefetch_l2(args.next_blobs + size_t(first + b) * args.next_blob_bytes, args.next_blob_bytes);
      }
    }
    // after an abort: give copies still in flight a bounded time to land before the CTA exits
    if (ctx.aborted() && lane == 0)
      for (uint32_t u = (issued > uint32_t(L::kIn) ? issued - L::kIn : 0); u < issued; ++u) mbar_wait(bar_in_full + 8 * (u % L::kIn), (u / L::kIn) & 1);
  } else if (MODE == kUmma && warp == kWideWarpXLoader) {
    // ------------------------------------------------------------------ activation tiles by TMA
    // One thread.  Chunk v of this CTA (in the order the items list them) uses activation stage v % kX, which is free once
    // chunk v - kX has been multiplied.  Of a pair, each CTA brings in half of every tile's rows; both halves complete on the
    // issuer's barrier.
    if (lane == 0) {
      grid_dependency_wait();
      const uint64_t stay = l2_policy_evict_last();  // every CTA reads the same activation tiles
      const uint32_t x_full_at = PAIR ? cluster_map(bar_x_full, my_rank & ~1u) : bar_x_full;
      uint32_t c_v = unit_begin % args.chunks;  // the chunk (column block) to request next: wraps at the end of a row block
      uint32_t v = 0;
      for (; v < unit_count; ++v) {
        const uint32_t sx = v % kXN, stage = smem + L::xs + sx * L::kXStage;
        if (ctx.aborted() || !ctx.wait(bar_x_empty + 8 * sx, ((v / kXN) & 1) ^ 1)) break;
        if (leader) mbar_arrive_expect_tx(bar_x_full + 8 * sx, L::kXStage * (PAIR ? 2 : 1));
#pragma unroll
        for (uint32_t t = 0; t < uint32_t(T); ++t)
#pragma unroll
          for (uint32_t a = 0; a < 2; ++a) {
            const uint32_t dst = stage + (2 * t + a) * L::kXAtom;
            const int col = int(c_v * BXR_COLS + 64 * a), row = int(t * NB + (PAIR ? (my_rank & 1u) * L::kXRows : 0u));
            if (PAIR) tma_load_2d_pair(dst, &tmap_x, col, row, x_full_at + 8 * sx, stay);
            else tma_load_2d(dst, &tmap_x, col, row, bar_x_full + 8 * sx, stay);
          }
        if (++c_v == args.chunks) c_v = 0;
      }
      // after an abort: tiles on their way land before the CTA exits (of a pair, the issuer's barriers know of both halves, and
      // its peer waits for it)
      if (ctx.aborted() && leader)
        for (uint32_t u = v > kXN ? v - kXN : 0; u < v; ++u) mbar_wait(bar_x_full + 8 * (u % kXN), (u / kXN) & 1);
    }
  } else if (MODE == kUmma && warp == kWideWarpMma) {
    // ------------------------------------------------------------------ MMA issue: eight per chunk and tile, then the stages go back
    constexpr uint32_t idesc = umma_idesc_bf16(NB, PAIR ? 256 : 128);
    const uint16_t both = uint16_t(3u << (my_rank & ~1u));
    auto commit = [&](uint32_t bar) {
      if (PAIR) umma_commit_pair(bar, both);
      else umma_commit(bar);
    };
    uint32_t n_item = 0, so = 0, pho = 0, sx = 0, phx = 0;
    bool live = leader;
    for (uint32_t u = unit_begin; u < unit_end && live; ++n_item) {
      const WideSpan item = wide_span(u, unit_end, args.chunks);
      u += item.chunk_end - item.chunk_begin;
      const uint32_t drained = (acc_use(n_item) & 1) ^ 1;
      for (uint32_t c = item.chunk_begin; c < item.chunk_end && live; ++c) {
        const bool first = c == item.chunk_begin, last = c + 1 == item.chunk_end;
        if (first && !ctx.go_warp(bar_acc_empty + 8 * acc_slot(n_item, 0), drained)) { live = false; break; }
        if (!ctx.wait_warp(bar_x_full + 8 * sx, phx) || !ctx.wait_warp(bar_op_full + 8 * so, pho)) { live = false; break; }
        const uint32_t a_tmem = tmem_base + kOperandCol + so * 64;
#pragma unroll
        for (uint32_t t = 0; t < uint32_t(T); ++t) {
          const uint32_t slot = acc_slot(n_item, t);
          if (t && first && !ctx.wait_warp(bar_acc_empty + 8 * slot, drained)) { live = false; break; }
          tc_fence_after();
          if (elect_one()) {
            const uint64_t bdesc = umma_desc_sw128(smem + L::xs + sx * L::kXStage + 2 * t * L::kXAtom);
            uint32_t accumulate = first ? 0u : 1u;
#pragma unroll
            for (uint32_t a = 0; a < 2; ++a)
#pragma unroll
              for (uint32_t k = 0; k < 4; ++k) {
                const uint64_t b = bdesc + a * (L::kXAtom >> 4) + 2 * k;
                if (PAIR) umma_bf16_ts_pair(tmem_base + slot * NB, a_tmem + a * 32 + k * 8, b, idesc, accumulate);
                else umma_bf16_ts(tmem_base + slot * NB, a_tmem + a * 32 + k * 8, b, idesc, accumulate);
                accumulate = 1;
              }
            if (t + 1 == uint32_t(T)) {
              commit(bar_op_empty + 8 * so);
              if (L::kXOwn) commit(bar_x_empty + 8 * sx);
            }
            if (last) commit(bar_acc_full + 8 * slot);
          }
          __syncwarp();
        }
        if (++so == kOpN) { so = 0; pho ^= 1; }
        if (++sx == kXN) { sx = 0; phx ^= 1; }
      }
    }
  } else if (MODE == kUmma && warp >= kWideWarpEpilogue) {
    // ------------------------------------------------------------------ TMEM -> y, or -> FP32 partial tile
    const uint32_t e = warp - kWideWarpEpilogue;  // == warp % 4: the TMEM lane quarter this warp may read
    const uint32_t r = e * 32 + lane;
    const uint32_t acc_empty_at = PAIR ? cluster_map(bar_acc_empty, my_rank & ~1u) : bar_acc_empty;   // the issuer's
    uint32_t n_item = 0, met = 0;
    bool live = true;
    // Split row blocks that this CTA is the last to declare, and so adds up: that of its last item (misc + 16) and that of its
    // first (misc + 32), as {1 | (index + 1 of the tile kept in shared memory) << 8, row block, first slot, parts}.
    auto decide = [&](uint32_t at, uint32_t own, const bxr_item& i) {
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(smem + L::misc + at), "r"(1u | own << 8), "r"(i.row_block), "r"(i.slot - i.part), "r"(i.parts) : "memory");
    };
    const uint64_t stay = l2_policy_evict_last();  // partial tiles are read back within the launch
    grid_dependency_wait();  // bias, y, partial tiles and counters may belong to the previous kernel
    bxr_item item = {};
    if (item_begin < item_end) item = args.items[item_begin];
    // A row block's counter: parts declared in the low half, parts in memory in the high half.  A part may be declared by any CTA
    // that runs, since it waits for nobody before the part is in memory, and the last to declare adds.  A first item with another
    // after it is declared right here: declared with its tile, it was now and then the last of its row block, and its CTA added
    // up two row blocks one after the other.  8704 x 5120 at 128 rows 25.7 -> 22.5 us, 5120 x 8704 26.4 -> 23.1, 4096 x
    // 14336 30.3 -> 26.8.
    const bool early = args.cluster <= 1 && item_end - item_begin > 1 && item.parts > 1;
    uint32_t first_declared = 0;
    if (early && e == 0 && lane == 0) first_declared = atomicAdd(args.counters + item.row_block, 1u);
    for (uint32_t it = item_begin; it < item_end && live; ++it, ++n_item) {
      if (it != item_begin) item = args.items[it];
      const uint32_t row = item.row_block * BXR_ROWS + r, row0 = item.row_block * BXR_ROWS + e * 32;
      // The CTA's last item, if it is part of a split row block, keeps its tile in shared memory (all of it is free
      // by now: every blob and every activation tile has been multiplied).  If the other parts of the row block have been
      // declared by then, this CTA adds them up and its own tile never goes to memory.  Only the first and the last item of a
      // CTA can be part of a split row block.
      const bool in_cluster = args.cluster > 1;  // the CTA's one item is a part of its cluster's row block
      const bool keep = item.parts > 1 && (it + 1 == item_end || in_cluster);
      if (!ctx.go_warp(bar_acc_full + 8 * acc_slot(n_item, 0), acc_use(n_item) & 1)) { live = false; break; }
      if (keep) {
        // (the second tile's last multiply may still be reading the activations in whose place the first one goes)
        if (T == 2 && !ctx.wait_warp(bar_acc_full + 8, acc_use(n_item) & 1)) { live = false; break; }
        tc_fence_after();
        uint32_t declared = 0;
        if (!in_cluster && e == 0 && lane == 0) declared = atomicAdd(args.counters + item.row_block, 1u);   // (looked at after the drain)
        if (in_cluster) {
#pragma unroll 1
          for (uint32_t t = 0; t < uint32_t(T); ++t) drain_to_smem(n_item, t, smem + t * NB * BXR_ROWS * 4);
        } else {
          drain_to_smem(n_item, 0, smem);
          if (e == 0 && lane == 0) asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(smem + L::misc + 8), "r"(declared) : "memory");
          fence_proxy_async_smem();  // the tile may leave through a bulk copy
          if (!ctx.meet(bar_meet, met)) { live = false; break; }
          asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(declared) : "r"(smem + L::misc + 8));
          if ((declared & 0xFFFFu) == item.parts - 1) {   // (T = 2: the second tile waits in tensor memory until the first has been added)
            if (e == 0 && lane == 0) decide(16, item.part + 1u, item);
          } else {   // another CTA will be the last: publish the tiles like any other
            if (T == 2) {
              drain_to_smem(n_item, 1, smem + NB * BXR_ROWS * 4);
              fence_proxy_async_smem();
              if (!ctx.meet(bar_meet, met)) { live = false; break; }
            }
            if (e == 0 && lane == 0) {
              bulk_s2g(args.partials + size_t(item.slot) * T * NB * BXR_ROWS, smem, ((args.m + 7) & ~7u) * BXR_ROWS * 4);
              bulk_commit_and_wait();
              fence_proxy_async_all();
              __threadfence();
              atomicAdd(args.counters + item.row_block, 1u << 16);
            }
          }
        }
        continue;   // (the CTA's last item: nobody waits for the accumulator)
      }
      tc_fence_after();
      // A lane holds one weight row and 16 batch columns; y keeps the rows of one batch column together, so its columns are
      // turned around by stmatrix and leave as 16-byte stores.  Partial tiles do so as they are: a store per column is one
      // whole 128-byte line.  A drain is a chain of trips to tensor memory, beside the multiplies of the next item up to 128
      // columns and in front of them above: so many columns a trip as the registers hold.  34816 x 5120, an item of 128
      // columns 3.0-3.6 -> 1.9-2.2 us, of 384 7-9 -> 5 us.
      const uint32_t turn = smem + L::turn + e * L::kTurn;
      const bool y_wide = (reinterpret_cast<uintptr_t>(args.y) & 15u) == 0 && (args.ldy & 7u) == 0 && row0 + 32 <= args.rows;
#pragma unroll 1
      for (uint32_t t = 0; t < uint32_t(T); ++t) {
        if (t) {
          if (!ctx.wait_warp(bar_acc_full + 8 * acc_slot(n_item, t), acc_use(n_item) & 1)) { live = false; break; }
          tc_fence_after();
        }
        const uint32_t taddr = tmem_base + ((e * 32) << 16) + acc_slot(n_item, t) * NB, m_at = t * NB, mcols = wide_tile_cols(args.m, t, NB);
        if (item.parts > 1) {
          constexpr int kStep = NB >= 32 ? 32 : 16;
          float* dst = args.partials + (size_t(item.slot) * T + t) * NB * BXR_ROWS + r;
#pragma unroll 1
          for (uint32_t m0 = 0; m0 < mcols; m0 += kStep, dst += kStep * BXR_ROWS) {
            uint32_t v[kStep];
            if constexpr (kStep == 32) tmem_ld32(taddr + m0, v);
            else tmem_ld16(taddr + m0, v);
            tmem_ld_wait();
#pragma unroll
            for (int h = 0; h < kStep; h += 8)
              if (m0 + h < mcols) {
#pragma unroll
                for (int i = 0; i < 8; ++i) stg32(dst + (h + i) * BXR_ROWS, v[h + i], stay);
              }
          }
        } else if (y_wide) {
          // this lane's weight rows in the accumulator layout, and where its column of a matrix goes: unit j of a batch row's
          // 64 bytes, the units permuted by the batch row (stores and loads free of bank conflicts)
          float b[4];
          if (args.bias)
#pragma unroll
            for (int k = 0; k < 4; ++k) b[k] = __bfloat162float(args.bias[row0 + 8 * k + (lane >> 2)]);
          const uint32_t put_at = turn + (lane & 7) * 64 + (((lane >> 3) ^ ((lane >> 1) & 3)) << 4);
          const uint32_t ml = lane >> 2, get_at = turn + ml * 64 + (((lane & 3) ^ ((ml >> 1) & 3)) << 4);
          __nv_bfloat16* dst = args.y + size_t(m_at + ml) * args.ldy + row0 + (lane & 3) * 8;
          constexpr int kStep = L::kTurnCols, kPieces = kStep / 16;
          uint32_t v[kPieces][16];   // 16 columns: [weight rows 0-15, 16-31][columns 0-7, 8-15][4]
          auto load = [&](uint32_t m0) {
#pragma unroll
            for (int k = 0; k < kPieces; ++k) {
              tmem_ld_16x16(taddr + m0 + 16 * k, v[k]);
              tmem_ld_16x16(taddr + m0 + 16 * k + (16u << 16), v[k] + 8);
            }
          };
          load(0);
#pragma unroll 1
          for (uint32_t m0 = 0; m0 < mcols; m0 += kStep) {
            tmem_ld_wait();
            uint32_t w[kPieces][8];
#pragma unroll
            for (int k = 0; k < kPieces; ++k) {
              if (args.bias)
#pragma unroll
                for (int i = 0; i < 16; ++i) v[k][i] = __float_as_uint(__fadd_rn(__uint_as_float(v[k][i]), b[(i >> 3) * 2 + ((i >> 1) & 1)]));
#pragma unroll
              for (int i = 0; i < 8; ++i) w[k][i] = wide_pack(__uint_as_float(v[k][2 * i]), __uint_as_float(v[k][2 * i + 1]));
            }
            if (m0 + kStep < mcols) load(m0 + kStep);   // the next columns are on their way while these are stored
#pragma unroll
            for (int k = 0; k < kPieces; ++k) {
              stsm_x4_trans(put_at + 1024 * k, w[k][0], w[k][1], w[k][4], w[k][5]);           // columns 0-7: rows 0-7, 8-15, 16-23, 24-31
              stsm_x4_trans(put_at + 1024 * k + 512, w[k][2], w[k][3], w[k][6], w[k][7]);     // columns 8-15
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 2 * kPieces; ++k) {
              const uint4 piece = lds128(get_at + 512 * k);
              if (m_at + m0 + 8 * k + ml < args.m) *reinterpret_cast<uint4*>(dst + 8 * k * args.ldy) = piece;
            }
            dst += kStep * args.ldy;
            __syncwarp();
          }
        } else {
          const float b = (args.bias && row < args.rows) ? __bfloat162float(args.bias[row]) : 0.f;
#pragma unroll 1
          for (uint32_t m0 = 0; m0 < mcols; m0 += 16) {
            uint32_t v[16];
            tmem_ld16(taddr + m0, v);
            tmem_ld_wait();
            if (row < args.rows)
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if (m_at + m0 + i < args.m) {
                  const float f = __uint_as_float(v[i]);
                  args.y[size_t(m_at + m0 + i) * args.ldy + row] = __float2bfloat16_rn(args.bias ? __fadd_rn(f, b) : f);
                }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (leader) mbar_arrive(bar_acc_empty + 8 * acc_slot(n_item, t));
          else mbar_arrive_cluster(acc_empty_at + 8 * acc_slot(n_item, t));
        }
      }
      if (!live) break;
      if (item.parts > 1) {
        fence_proxy_async_all();   // the tile, written by ordinary stores, is read by bulk copies
        __threadfence();
        if (!ctx.meet(bar_meet, met)) { live = false; break; }
        if (e == 0 && lane == 0) {
          atomicAdd(args.counters + item.row_block, 1u << 16);
          if ((first_declared & 0xFFFFu) == item.parts - 1) decide(32, 0, item);
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_final);
  }

  if (MODE == kUmma && args.cluster > 1) {
    // A row block's CTAs in one cluster: every CTA's tile is in its shared memory once its epilogue is through; the cluster
    // barrier makes the tiles visible to the peers, the second one keeps every CTA's shared memory alive until the
    // peers have read it.  Every thread of every CTA gets here on every path (all other waits are bounded).
    const bool worker_thread = warp < kDecoderWarps || warp >= kWideWarpEpilogue;
    const bool drained = worker_thread ? ctx.wait_warp(bar_final, 0) : true;
    __syncwarp();
    cluster_sync();
    if (worker_thread && drained && unit_count) {
      const uint32_t row_block = (unit_begin / args.chunks) * group + in_group, t = (warp < kDecoderWarps ? warp : warp - 4) * 32 + lane;
      // (narrow tiles: a position a thread at most, and a shorter way through code that is read once a launch: 5120 x 5120 at
      // one row reads one position)
      if constexpr (NB <= 32) bxq_reduce_in_cluster<PAIR, 8, 1>(args, row_block, smem, t);
      else if (args.cluster == 2) bxq_reduce_in_cluster<PAIR, 2, 4>(args, row_block, smem, t);
      else if (PAIR || args.cluster == 3) bxq_reduce_in_cluster<PAIR, 3, 3>(args, row_block, smem, t);   // (pairs: clusters of two or three parts)
      else if constexpr (!PAIR) {
        if (args.cluster == 4) bxq_reduce_in_cluster<PAIR, 4, 2>(args, row_block, smem, t);
        else bxq_reduce_in_cluster<PAIR, 8, 1>(args, row_block, smem, t);
      }
    }
    __syncwarp();
    cluster_sync();
  }

  // Row blocks that fell to this CTA are added up: warp kWideWarpSlices brings the others' tiles in, the decoder warps add.
  if (MODE == kUmma && args.cluster <= 1 && (warp < kDecoderWarps || warp >= kWideWarpSlices)) {
    const uint32_t ring = smem + NB * BXR_ROWS * 4;
    bool live = ctx.wait_warp(bar_final, 0);
    uint32_t n = 0;
#pragma unroll 1
    for (uint32_t at = 32; at >= 16; at -= 16) {
      const uint4 decision = lds128(smem + L::misc + at);  // {reduce? | own tile << 8, row block, first slot, parts}
      if (!decision.x) continue;
      const uint32_t own = (decision.x >> 8) - 1u, parts = decision.w;
      // The warp that asks for the tiles is the one that waits for them: with the wait in the epilogue, a fence and the meeting at
      // bar_final stood between a tile's arrival and its copy (5120 x 1280 at one row 6.64 -> 6.44 us).
      if (warp == kWideWarpSlices && lane == 0) {
        live = live && bxq_parts_in_memory(args, ctx, decision.y, parts - (own < parts ? 1u : 0u));
        // Bulk copies read tiles that other CTAs stored, and write over turn-around buffers that this CTA's epilogue stored:
        // ordinary stores of others, which the counter and the barrier order before here, and this before the copies.
        fence_proxy_async_all();
      }
#pragma unroll 1
      for (uint32_t t = 0; t < uint32_t(T); ++t) {
        const uint32_t cols = wide_tile_cols(args.m, t, NB);
        if (T == 2 && t && own < parts) {   // the second tile takes the place of the first once that has been added
          if (warp < kDecoderWarps) {
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_swap_used);
            live = live && ctx.wait_warp(bar_swap_full, 0);
          } else if (warp >= kWideWarpEpilogue) {
            live = live && ctx.wait_warp(bar_swap_used, 0);
            if (live) drain_to_smem(0, t, smem);
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_swap_full);
          }
        }
        if (warp < kDecoderWarps) {
          if (live) bxq_add_tiles<L>(args, ctx, decision.y, parts, own, smem, ring, bar_slice_full, bar_slice_used, warp * 32 + lane, t * NB, t * NB + cols, n);
        } else if (warp == kWideWarpSlices && lane == 0 && live) {
          for (uint32_t m0 = 0; m0 < cols && live; m0 += L::kSliceRows)
            for (uint32_t p = 0; p < parts && live; ++p) {
              if (p == own) continue;
              const uint32_t b = n % L::kSlices, bytes = min(L::kSliceRows, cols - m0) * BXR_ROWS * 4;
              if (!ctx.wait(bar_slice_used + 8 * b, ((n / L::kSlices) & 1) ^ 1)) { live = false; break; }
              mbar_arrive_expect_tx(bar_slice_full + 8 * b, bytes);
              bulk_g2s(ring + b * L::kSlice, args.partials + ((size_t(decision.z + p) * T + t) * NB + m0) * BXR_ROWS, bytes, bar_slice_full + 8 * b, l2_policy_evict_first());
              ++n;
            }
          // copies still in flight must land before the CTA may exit
          if (!live)
            for (uint32_t k = n > L::kSlices ? n - L::kSlices : 0; k < n; ++k) mbar_wait(bar_slice_full + 8 * (k % L::kSlices), (k / L::kSlices) & 1);
        }
      }
    }
  }

  tc_fence_before();
  __syncwarp();
  if (PAIR) cluster_sync();   // what the peer has in flight ends at this CTA's barriers, shared memory and tensor memory
  else __syncthreads();
  if (MODE == kUmma && warp == kWideWarpMma) {
    tc_fence_after();
    tmem_dealloc<PAIR>(tmem_base, kTmemCols);
  }
}

}  // namespace grb

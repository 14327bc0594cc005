// Indexed decode of unchanged BCTX streams with every model in shared memory: the kernel for frames whose packed tables
// (bcx_model.h, PackedShape) fit one SM, which the default 16 x 4 classes do with room to spare, with raw residuals (mode 0)
// or coded ones (mode 128).  bctx_decode_kernel (bctx_decode.cuh) serves every other frame.
//
// What bounds it.  A lane's walk is a serial chain, so nothing slow may stand on it, and a warp executes the rare branches
// of all its lanes.  Global loads stand on the chain even when a lane asks for its stream bytes long before it needs them:
// the lanes of a warp renew their windows at different steps, a warp waits for a register whichever of its lanes has a load
// outstanding on it, and so nearly every step waits for an L2 round trip that another lane has just begun.  Here stream bytes
// come to shared memory by asynchronous copies, which no register waits for, and everything a symbol needs is there: its
// bucket, its 8-byte entry (first slot, frequency, symbol), every second symbol a word of the stream.  The window moves by
// selects, not by a branch; a bucket tells its two symbols apart, so that the forward scan is left to rare symbols (with one
// rank per bucket some lane of a warp scanned at nearly every symbol).  A main symbol and the residual of the one before it
// are looked up together: their chains are independent.  What is left is 100 instructions per warp and word at 63 % of
// the issue slots, with the integer pipe 66 % and the shared-memory data pipe 73 % busy.
// 4096 x 4096 words with coded residuals, 128 per lane: 305 us before (tables in global memory, one CTA of 64 lanes after
// another), 118 us with the tables of all 64 contexts in shared memory (room for 14 warps), 86 us with one row class per CTA
// (28 warps).  128 rows of 5120 words with raw residuals: 160 us before, 25 us.
#pragma once
#include "bctx_decode.cuh"

namespace grb {

struct BctxPackedArgs {
  const uint8_t* tables;
  uint32_t table_bytes, shift, ctx_bytes;    // main context c: buckets at c * ctx_bytes, entries behind them
  uint32_t resid_shift, resid_at;            // residual contexts: from resid_at on, found through the main entries
  const uint8_t* bytes;                      // main stream
  uint32_t size;
  const uint32_t* states;
  const uint32_t* offsets;
  const uint8_t* raw;                        // 6-bit residuals, or the coded residual stream
  uint64_t raw_size;
  const uint32_t* raw_states;                // coded residuals only
  const uint32_t* raw_offsets;
  const uint8_t* row_class;
  const uint8_t* col_class;
  uint64_t n;
  uint32_t rows, cols, nr, nc, stride;
  const long long* ids;        // nullptr: all blocks; else rows: lane i takes the (i % per_row)-th block that row
  uint32_t per_row;            // ids[i / per_row] touches, and writes what of it lies in the row
  uint64_t count;              // lanes' blocks
  uint32_t per_cta;
  const uint32_t* rows_by_class;   // kByClass
  const uint4* part_of;            // kByClass, all blocks: {row class, place of its first row, first block, end block} per CTA
  uint16_t* out;
  uint32_t* status;
  uint32_t* host_flags;        // optional, host memory: [0] = status bits, [1] = an id was out of range
};

constexpr uint32_t kPackedTablesAt = 128;         // barrier first
constexpr uint32_t kPackedColsMax = 24576;        // column classes kept in shared memory
constexpr uint32_t kPackedRing = 64;              // bytes of a stream per lane
constexpr uint32_t kPackedSmemMax = 232448;       // the 227 KB of shared memory a CTA may opt into
struct Yes { static constexpr bool value = true; };
struct No { static constexpr bool value = false; };
enum PackedResidual { kRaw16, kRaw64, kCoded };   // raw: loaded per 16 symbols, or per 64 (strides that are multiples of 64)
// kByClass: rows are whole blocks, and a CTA decodes rows of one row class - a share of them (part_of), or one row of `ids` -
// with the tables of that class alone, so that buckets are fine and 28 warps' rings fit beside them.  Otherwise a block
// may run from one row into the next, and a CTA keeps the tables of all classes: rows that are a multiple of 16 columns (a
// run of 16 symbols stays in its row and its classes are one 16-byte load), or any rows.
enum PackedRows { kByClass, kRows16, kAnyRows };
constexpr uint32_t kPackedThreads = 1024;
template <int RESIDUAL>
constexpr uint32_t kPackedLaneBytes = RESIDUAL == kCoded ? 2 * kPackedRing : kPackedRing;

// Lanes of a warp stand `stride` columns apart, usually 128: 16 bytes of padding per 128 keep their 16-byte class loads on
// different banks.  Slack at the end: a run of 16 columns that starts before the row's end reads into the next row.
__host__ __device__ constexpr uint32_t packed_class_at(uint32_t col) { return col + ((col >> 7) << 4); }
__host__ __device__ constexpr uint32_t packed_class_bytes(uint32_t cols) { return (packed_class_at(cols + 15) + 16) & ~15u; }

__device__ __forceinline__ void packed_report(const BctxPackedArgs& a, uint32_t bad, bool index) {
  atomicOr(a.status, bad);
  if (a.host_flags) *reinterpret_cast<volatile uint32_t*>(a.host_flags + (index ? 1 : 0)) = bad;
}

// One stream of one lane.  Bytes: global -> a ring of four 16-byte pieces in shared memory (asynchronous copies) -> a window
// of three words: w0 w1 hold the eight bytes from word `word` on, most significant first, w2 the four after them; `bit` is
// how far the window has been used up.  Symbols are taken in pairs, at most 32 bits each pair.
struct PackedStream {
  uint32_t ring;           // shared address
  uint32_t x, w0, w1, w2, ahead, bit, word, next_piece, first_take;

  // The next piece; what lies beyond the stream reads as zero.  Pieces count from the stream's address rounded down to 16.
  __device__ __forceinline__ void request(const uint8_t* bytes, uint32_t size) {
    const uint32_t skew = uint32_t(reinterpret_cast<uintptr_t>(bytes) & 15u), end = size + skew, from = next_piece << 4;
    const bool in = from < end;
    cp_async_16(ring + ((next_piece & 3u) << 4), bytes - skew + (in ? from : 0u), in ? min(16u, end - from) : 0u);
    ++next_piece;
  }
  __device__ __forceinline__ uint32_t ring_word(uint32_t i) const { return __byte_perm(lds32(ring + ((i & 15u) << 2)), 0, 0x0123); }
  __device__ __forceinline__ void ask(const uint8_t* bytes, uint32_t size, uint32_t offset) {
    const uint32_t skew = uint32_t(reinterpret_cast<uintptr_t>(bytes) & 15u);
    word = (offset + skew) >> 2;
    bit = ((offset + skew) & 3u) * 8;
    next_piece = word >> 2;
#pragma unroll
    for (int k = 0; k < 4; ++k) request(bytes, size);
  }
  __device__ __forceinline__ void open() {
    w0 = ring_word(word);
    w1 = ring_word(word + 1);
    w2 = ring_word(word + 2);
  }
  // Before every eight symbols (at most 16 bytes; the caller commits and waits for all copies but the newest): a piece is
  // asked for when one has been used up, and the one asked for eight symbols ago has arrived.  64 bytes are then requested
  // from the start of the current piece on and 48 are there, so at least 33 from the read position on, of which the eight
  // symbols and the window touch at most 28.
  __device__ __forceinline__ void refill(const uint8_t* bytes, uint32_t size) {
    if (next_piece - (word >> 2) < 4) request(bytes, size);
  }
  __device__ __forceinline__ void begin_pair() {
    const bool roll = bit >= 32;
    w0 = roll ? w1 : w0;
    w1 = roll ? w2 : w1;
    word += roll ? 1 : 0;
    bit &= 31u;
    w2 = ring_word(word + 2);
    ahead = __funnelshift_l(w1, w0, bit);
  }
  __device__ __forceinline__ void mid_pair() { ahead = __funnelshift_l(__funnelshift_l(w2, w1, bit), ahead, first_take); }
  // The state after a step is at least 2^7: it takes 0, 1 or 2 bytes.
  __device__ __forceinline__ void advance(uint32_t frequency_minus_1, uint32_t above_first, bool second) {
    const uint32_t hi = x >> 16;
    x = frequency_minus_1 * hi + (hi + above_first);
    const uint32_t take = (uint32_t(__clz(int(x))) - 1u) & 24u;   // 0 from 2^23 on, 8 from 2^15 on, else 16 bits
    x = __funnelshift_l(ahead, x, take);
    if (second) bit += first_take + take;
    else first_take = take;
  }
  __device__ __forceinline__ void end_odd() { bit += first_take; }   // a pair of which only the first symbol was taken
  // stream bytes used so far (the window may stand at a word's end)
  __device__ __forceinline__ uint32_t used(const uint8_t* bytes) const {
    return word * 4 + (bit >> 3) - uint32_t(reinterpret_cast<uintptr_t>(bytes) & 15u);
  }
};

template <int ROWS, int RESIDUAL>
__global__ void __launch_bounds__(kPackedThreads, 1) bctx_packed_kernel(const BctxPackedArgs a) {
  constexpr bool CODED = RESIDUAL == kCoded, ALIGNED = ROWS != kAnyRows, BY_CLASS = ROWS == kByClass;
  extern __shared__ __align__(128) uint8_t packed_smem[];
  const uint32_t main_bytes = BY_CLASS ? a.nc * a.ctx_bytes : a.resid_at, resid_bytes = a.table_bytes - a.resid_at;
  const uint32_t bar = smem_u32(packed_smem), tables = bar + kPackedTablesAt, rtables = tables + main_bytes, rings = rtables + resid_bytes;
  const uint32_t classes = rings + blockDim.x * kPackedLaneBytes<RESIDUAL>;
  uint4 part = {0, 0, 0, 0};
  uint64_t lane_begin = uint64_t(blockIdx.x) * a.per_cta, lane_end = min(a.count, lane_begin + a.per_cta);
  if (BY_CLASS) {
    if (a.ids) {
      const long long id = a.ids[blockIdx.x];
      if (id < 0 || id >= (long long)(a.rows)) {
        if (threadIdx.x == 0) packed_report(a, kStatusBadArgument, true);
        return;
      }
      part.x = __ldg(a.row_class + id);
    } else {
      part = __ldg(a.part_of + blockIdx.x);
      lane_begin = part.z;
      lane_end = part.w;
    }
    if (part.x >= a.nr) {
      if (threadIdx.x == 0) packed_report(a, kStatusBadSymbol, false);
      part.x = 0;
    }
  }
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
    fence_proxy_async_smem();
    mbar_arrive_expect_tx(bar, main_bytes + resid_bytes);
    bulk_g2s(tables, a.tables + size_t(part.x) * main_bytes, main_bytes, bar);
    if (resid_bytes) bulk_g2s(rtables, a.tables + a.resid_at, resid_bytes, bar);
  }
  // Labels outside the model are flagged here, once, and read as the last class.
  const bool wide_classes = (a.cols & 15u) == 0 && (reinterpret_cast<uintptr_t>(a.col_class) & 15u) == 0;
  const uint32_t nc4 = a.nc * 0x01010101u;
  for (uint32_t c = threadIdx.x * (wide_classes ? 16 : 1); c < a.cols + 16; c += blockDim.x * (wide_classes ? 16 : 1)) {
    const uint8_t* const src = a.col_class + (c < a.cols ? c : (c - a.cols) % a.cols);
    if (wide_classes) {
      uint4 v = __ldg(reinterpret_cast<const uint4*>(src));
      if (__vcmpgeu4(v.x, nc4) | __vcmpgeu4(v.y, nc4) | __vcmpgeu4(v.z, nc4) | __vcmpgeu4(v.w, nc4)) {
        packed_report(a, kStatusBadSymbol, false);
        const uint32_t last = nc4 - 0x01010101u;
        v = make_uint4(__vminu4(v.x, last), __vminu4(v.y, last), __vminu4(v.z, last), __vminu4(v.w, last));
      }
      sts128(classes + packed_class_at(c), v);
    } else {
      const uint32_t cls = __ldg(src);
      if (cls >= a.nc) packed_report(a, kStatusBadSymbol, false);
      asm volatile("st.shared.u8 [%0], %1;" ::"r"(classes + packed_class_at(c)), "r"(min(cls, a.nc - 1)) : "memory");
    }
  }
  __syncthreads();
  const uint32_t shift = a.shift, bucket_bytes = 131072u >> shift, place = (1u << shift) - 1;
  const uint32_t rshift = a.resid_shift, rbucket_bytes = 131072u >> rshift, rplace = (1u << rshift) - 1;
  const uint64_t blocks_total = (a.n + a.stride - 1) / a.stride;
  for (uint64_t i = lane_begin + threadIdx.x; i < lane_end; i += blockDim.x) {
    uint64_t block = i;
    uint32_t keep_from = 0, keep_to = a.stride;   // words of the block that are wanted (kByClass: all)
    if (BY_CLASS && !a.ids) {
      const uint32_t q = uint32_t(i) / a.per_row;
      block = uint64_t(__ldg(a.rows_by_class + part.y + q)) * a.per_row + (uint32_t(i) - q * a.per_row);
    }
    uint16_t* out = a.out + block * a.stride;     // where the block's word 0 goes
    if (a.ids) {
      const uint64_t q = i / a.per_row;
      const long long id = a.ids[q];
      if (id < 0 || id >= (long long)(a.rows)) {
        packed_report(a, kStatusBadArgument, true);
        continue;
      }
      const uint64_t begin = uint64_t(id) * a.cols;
      block = begin / a.stride + (i - q * a.per_row);
      const uint64_t first = block * a.stride;
      if (first >= begin + a.cols) continue;
      if (!BY_CLASS) keep_from = first < begin ? uint32_t(begin - first) : 0u;
      if (!BY_CLASS) keep_to = uint32_t(min(uint64_t(a.stride), begin + a.cols - first));
      out = a.out + (q * a.cols + (first - begin));
    }
    const bool has_next = block + 1 < blocks_total;
    PackedStream s, t;
    s.ring = rings + threadIdx.x * kPackedRing;                // each kind of ring together: lanes 64 bytes apart share banks
    t.ring = s.ring + blockDim.x * kPackedRing;                // less than lanes 128 bytes apart
    s.x = a.states[block];
    s.ask(a.bytes, a.size, a.offsets[block]);
    if (CODED) {
      t.x = a.raw_states[block];
      t.ask(a.raw, uint32_t(a.raw_size), a.raw_offsets[block]);
    }
    cp_async_commit();
    const uint64_t start = block * a.stride;
    uint32_t row = uint32_t(start / a.cols), col = uint32_t(start - uint64_t(row) * a.cols);
    const uint32_t steps = uint32_t(min(uint64_t(a.stride), a.n - start));
    const bool wide_out = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
    uint32_t bad = 0;
    auto row_tables = [&](uint32_t r) {   // the tables of row r's class, column class 0
      if (BY_CLASS) return tables;
      const uint32_t cls = __ldg(a.row_class + r);
      if (cls >= a.nr) bad |= kStatusBadSymbol;
      return tables + min(cls, a.nr - 1) * a.nc * a.ctx_bytes;
    };
    uint32_t here = row_tables(row);
    cp_async_wait<0>();
    if (!mbar_wait(bar, 0)) {   // the tables, on their way since the start
      packed_report(a, kStatusTimeout, false);
      break;
    }
    s.open();
    if (CODED) t.open();
    auto refill = [&]() {
      s.refill(a.bytes, a.size);
      if (CODED) t.refill(a.raw, uint32_t(a.raw_size));
      cp_async_commit();
      cp_async_wait<1>();
    };
    // Looks a main symbol up in the tables at `ctx` (MAIN) and / or a residual in those the entry `resid_of` names.
    // Returns their second entry words: symbol << 5 | residual tables / 8 << 16, and the residual's bits of the word.
    auto look_up = [&](auto main_too, auto resid_too, bool main_second, bool resid_second, uint32_t ctx, uint32_t resid_of, uint32_t& main_word,
                       uint32_t& resid_word) {
      constexpr bool MAIN = decltype(main_too)::value, RESID = decltype(resid_too)::value;
      uint32_t me = 0, re = 0, md = 0, rd = 0;
      uint2 m = {0, 0}, r = {0, 0};
      if (MAIN) {   // (bucket + place in it) >> 8 = the rank
        const uint32_t v = lds_u16(ctx + ((s.x >> (shift - 1)) & (bucket_bytes - 2)));
        me = ctx + bucket_bytes + (((v + (s.x & place)) >> 5) & ~7u);
      }
      if (RESID) {
        const uint32_t base = rtables + ((resid_of >> 16) << 3), v = lds_u16(base + ((t.x >> (rshift - 1)) & (rbucket_bytes - 2)));
        re = base + rbucket_bytes + (((v + (t.x & rplace)) >> 5) & ~7u);
      }
      if (MAIN) { m = lds64(me); md = (s.x - m.x) & 0xFFFFu; }   // slot - first slot of the symbol
      if (RESID) { r = lds64(re); rd = (t.x - r.x) & 0xFFFFu; }
      while ((MAIN && md > (m.x >> 16)) || (RESID && rd > (r.x >> 16))) {   // rare: a bucket of several symbols
        if (MAIN && md > (m.x >> 16)) { me += 8; m = lds64(me); md = (s.x - m.x) & 0xFFFFu; }
        if (RESID && rd > (r.x >> 16)) { re += 8; r = lds64(re); rd = (t.x - r.x) & 0xFFFFu; }
      }
      if (MAIN) { s.advance(m.x >> 16, md, main_second); main_word = m.y; }
      if (RESID) { t.advance(r.x >> 16, rd, resid_second); resid_word = r.y; }
    };
    const uint32_t* raw = reinterpret_cast<const uint32_t*>(a.raw + (start >> 2) * 3);   // 12 bytes per 16 symbols
    uint32_t r[12];
    const uint32_t runs = steps >> 4;
    for (uint32_t g = 0; g < runs; ++g, col += 16) {
      if (RESIDUAL == kRaw64) {
        if ((g & 3u) == 0) {
          const uint32_t left = (runs - g) * 3;   // a ragged last block may end before its 48 bytes do
#pragma unroll
          for (int k = 0; k < 3; ++k)
            if (left > uint32_t(4 * k + 3)) {
              const uint4 v = __ldg(reinterpret_cast<const uint4*>(raw + 3 * g) + k);
              r[4 * k] = v.x; r[4 * k + 1] = v.y; r[4 * k + 2] = v.z; r[4 * k + 3] = v.w;
            } else {
#pragma unroll
              for (int q = 0; q < 4; ++q) r[4 * k + q] = left > uint32_t(4 * k + q) ? __ldg(raw + 3 * g + 4 * k + q) : 0u;
            }
        } else {
#pragma unroll
          for (int k = 0; k < 9; ++k) r[k] = r[k + 3];
        }
      } else if (RESIDUAL == kRaw16) {
#pragma unroll
        for (int k = 0; k < 3; ++k) r[k] = __ldg(raw + 3 * g + k);
      }
      uint4 cls = {0, 0, 0, 0};
      uint32_t below = here;
      if (ALIGNED) {
        if (!BY_CLASS && col >= a.cols) {
          col -= a.cols;
          here = row_tables(++row);
        }
        cls = lds128(classes + packed_class_at(col));
      } else if (col + 16 >= a.cols) {   // a run of 16 reaches at most one row end (cols >= 16)
        if (row + 1 < a.rows) below = row_tables(row + 1);
      }
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        refill();
        const uint32_t c_lo = half ? cls.z : cls.x, c_hi = half ? cls.w : cls.y;
        // eight raw residuals: six bytes, most significant first
        uint32_t r32 = 0, r16 = 0;
        if (!CODED) {
          r32 = half ? __byte_perm(r[1], r[2], 0x2345) : __byte_perm(r[0], 0, 0x0123);
          r16 = half ? __byte_perm(r[2], 0, 0x4423) : __byte_perm(r[1], 0, 0x4401);
        }
        uint32_t packed[4] = {0, 0, 0, 0}, main_word = 0, before = 0, unused = 0;
        auto keep = [&](int j, uint32_t word) {
          packed[j >> 1] |= (j & 1) ? word << 16 : word;
        };
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          uint32_t ctx;
          if (ALIGNED) {
            ctx = here + __byte_perm(j < 4 ? c_lo : c_hi, 0, 0x4440 + (j & 3)) * a.ctx_bytes;
          } else {
            const uint32_t c = col + half * 8 + j;
            ctx = (c >= a.cols ? below : here) + lds_u8(classes + packed_class_at(c)) * a.ctx_bytes;
          }
          if (j & 1) s.mid_pair();
          else s.begin_pair();
          if (CODED) {
            uint32_t resid_word = 0;
            if (j == 0) {
              look_up(Yes{}, No{}, false, false, ctx, 0, main_word, unused);
            } else {
              if (j & 1) t.begin_pair();    // the residual of symbol j - 1
              else t.mid_pair();
              look_up(Yes{}, Yes{}, j & 1, !(j & 1), ctx, before, main_word, resid_word);
              keep(j - 1, (before & 0xFFFFu) | resid_word);
            }
            before = main_word;
          } else {
            look_up(Yes{}, No{}, j & 1, false, ctx, 0, main_word, unused);
            const uint32_t res = j < 5 ? (r32 >> (26 - 6 * j)) & 63u : j == 5 ? ((r32 & 3u) << 4) | (r16 >> 12) : j == 6 ? (r16 >> 6) & 63u : r16 & 63u;
            keep(j, (main_word & 0xFFFFu) | (res & 31u) | ((res & 32u) << 10));
          }
        }
        if (CODED) {
          uint32_t resid_word = 0;
          t.mid_pair();
          look_up(No{}, Yes{}, false, true, 0, before, unused, resid_word);
          keep(7, (before & 0xFFFFu) | resid_word);
        }
        const uint32_t k = 16 * g + 8 * half;
        if (BY_CLASS || (wide_out && k >= keep_from && k + 8 <= keep_to)) {
          *reinterpret_cast<uint4*>(out + k) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (k + j >= keep_from && k + j < keep_to) out[k + j] = uint16_t(packed[j >> 1] >> (16 * (j & 1)));
        }
      }
      if (!ALIGNED && col + 16 >= a.cols) {   // col wraps below zero; the increment of the loop brings it back
        col -= a.cols;
        here = below;
        ++row;
      }
    }
    if (ROWS == kRows16 && col >= a.cols) {
      col -= a.cols;
      if (++row < a.rows) here = row_tables(row);
    }
    for (uint32_t step = runs << 4; step < steps; ++step) {   // the ragged end of the tensor
      if ((step & 7u) == 0) refill();
      uint32_t main_word = 0, word = 0, unused = 0;
      s.begin_pair();
      look_up(Yes{}, No{}, false, false, here + lds_u8(classes + packed_class_at(col)) * a.ctx_bytes, 0, main_word, unused);
      s.end_odd();
      if (CODED) {
        t.begin_pair();
        look_up(No{}, Yes{}, false, false, 0, main_word, unused, word);
        t.end_odd();
      } else {
        const uint64_t bits = (start + step) * 6, byte = bits >> 3;
        const uint32_t hi = byte < a.raw_size ? __ldg(a.raw + byte) : 0u, lo = byte + 1 < a.raw_size ? __ldg(a.raw + byte + 1) : 0u;
        const uint32_t res = (((hi << 8) | lo) >> (10 - uint32_t(bits & 7))) & 63u;
        word = (res & 31u) | ((res & 32u) << 10);
      }
      if (step >= keep_from && step < keep_to) out[step] = uint16_t((main_word & 0xFFFFu) | word);
      if (++col == a.cols) {
        col = 0;
        if (++row < a.rows) here = row_tables(row);
      }
    }
    // The block must end exactly where the next one starts (or at the canonical end of the stream).
    auto check = [&](const PackedStream& q, const uint8_t* bytes, uint32_t size, const uint32_t* states, const uint32_t* offsets) {
      const uint32_t ip = q.used(bytes);
      if (ip > size) bad |= kStatusOverrun;
      if (q.x != (has_next ? states[block + 1] : (1u << 23)) || ip != (has_next ? offsets[block + 1] : size)) bad |= kStatusCheckpoint;
    };
    check(s, a.bytes, a.size, a.states, a.offsets);
    if (CODED) check(t, a.raw, uint32_t(a.raw_size), a.raw_states, a.raw_offsets);
    if (bad) packed_report(a, bad, false);
    // The piece asked for last may still be under way, and copies keep no order among themselves: without this wait it
    // could land on top of the next block's bytes in the same ring.
    cp_async_wait<0>();
  }
  if (threadIdx.x == 0) mbar_wait(bar, 0);   // no copy may be under way when the CTA ends
}

}  // namespace grb

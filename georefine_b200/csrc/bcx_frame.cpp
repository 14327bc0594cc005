// Whole-frame passes of the BCTX coder on the host: what encode(), decode() and index_frame() do between the container and
// the streams.  Same arithmetic as the bcx_* functions (bcx_host.cpp), which stay the reference for every malformed input:
// a pass that meets one gives up with a nonzero status, and the caller takes the stream through them to learn why.
//
// What bounds it.  A stream is one serial chain of state updates, so the time of a frame is symbols x the latency of one
// update; the rest has to be short or run beside it.  Decoding an update is slot -> entry of its bucket -> multiply-add ->
// renormalisation, about 20 cycles when nothing is mispredicted: the number of bytes a renormalisation takes is computed, not
// branched on, and the tables of the four contexts a row can meet (32 KB) stay in the first-level cache.  The residual
// chain (mode 128), the raw residuals and the joining of the words fit beside the main chain.  Encoding replaces the division
// by a multiplication with a precomputed reciprocal and writes its bytes unconditionally.
// 1024 x 2048 words: encode() 47 -> 13 ms, decode() 38 -> 16 ms (with hashing and compression on other threads).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <new>
#include <thread>
#include <vector>

#include "bcx_model.h"

#if defined(__x86_64__) && defined(__GNUC__) && !defined(__clang__)
#define GRB_CLONES __attribute__((target_clones("default", "arch=haswell")))   // three-operand shifts, mulx
#else
#define GRB_CLONES
#endif
#define GRB_INLINE inline __attribute__((always_inline))

namespace grb {
namespace {

constexpr uint32_t kTotal = 1u << 16;
constexpr uint32_t kLow = 1u << 23;

// fn(0) .. fn(threads - 1), each on a thread of its own where one can be started, else on this one.  What a share throws is
// thrown here, once all of them are over.
template <class Fn>
void on_threads(uint32_t threads, const Fn& fn) {
  std::vector<std::exception_ptr> failed(threads);
  const auto share = [&](uint32_t t) noexcept {
    try {
      fn(t);
    } catch (...) {
      failed[t] = std::current_exception();
    }
  };
  std::vector<std::thread> pool;
  pool.reserve(threads);
  uint32_t t = 1;
  try {
    for (; t < threads; ++t) pool.emplace_back(share, t);
  } catch (...) {   // no thread to be had, or no memory for it
  }
  share(0);
  for (; t < threads; ++t) share(t);
  for (auto& th : pool) th.join();
  for (const auto& e : failed)
    if (e) std::rethrow_exception(e);
}
// Threads worth starting for n words: one per 128 K words, at most 8.
uint32_t threads_for(uint64_t n) {
  const uint32_t hw = std::max(1u, std::thread::hardware_concurrency());
  return uint32_t(std::max<uint64_t>(1, std::min<uint64_t>({uint64_t(hw), 8, n >> 17})));
}

// ---- decoding -------------------------------------------------------------------------------------------------
struct Entry {
  uint16_t first, last;   // first slot, frequency - 1
  uint16_t what;          // the symbol; kDead in the tables of an empty context
  uint16_t rank;          // among the live symbols
};
constexpr uint32_t kDead = 1u << 15;

// Per context: the live symbols in order, and for every bucket of 2^kShift slots a copy of the one that owns its first slot.
// One load then gives an update everything it needs; the symbols behind it in the bucket are found by a scan, which 3 % of
// the updates have to make with 64-slot buckets (half with 1024).
template <uint32_t kShift>
class EntryTables {
 public:
  // False for tables the fast pass does not take (or that are invalid).
  bool load(const uint32_t* freq, uint32_t nctx, uint32_t vocab) {
    stride_ = 1;
    for (uint32_t cx = 0; cx < nctx; ++cx) {
      uint64_t sum = 0;
      uint32_t live = 0;
      for (uint32_t s = 0; s < vocab; ++s) {
        const uint32_t f = freq[size_t(cx) * vocab + s];
        if (f > kTotal) return false;
        sum += f;
        live += f != 0;
      }
      if (sum != 0 && sum != kTotal) return false;
      stride_ = std::max(stride_, live);
    }
    const Entry dead{0, 0xFFFF, uint16_t(kDead), 0};
    buckets_.assign(size_t(nctx) << (16 - kShift), dead);
    entries_.assign(size_t(nctx) * stride_, dead);
    for (uint32_t cx = 0; cx < nctx; ++cx) {
      Entry* bucket = &buckets_[size_t(cx) << (16 - kShift)];
      Entry* entry = &entries_[size_t(cx) * stride_];
      uint32_t run = 0, r = 0;
      constexpr uint32_t kRound = (1u << kShift) - 1;
      for (uint32_t s = 0; s < vocab; ++s) {
        const uint32_t f = freq[size_t(cx) * vocab + s];
        if (!f) continue;
        entry[r] = Entry{uint16_t(run), uint16_t(f - 1), uint16_t(s), uint16_t(r)};
        std::fill(bucket + ((run + kRound) >> kShift), bucket + ((run + f + kRound) >> kShift), entry[r]);
        ++r;
        run += f;
      }
    }
    return true;
  }
  static constexpr uint32_t shift = kShift;
  const Entry* buckets(uint32_t cx) const { return &buckets_[size_t(cx) << (16 - kShift)]; }
  const Entry* entries(uint32_t cx) const { return &entries_[size_t(cx) * stride_]; }

 private:
  uint32_t stride_ = 1;
  std::vector<Entry> buckets_, entries_;
};
using MainTables = EntryTables<6>;    // 8 KB per context: the four a row can meet stay in the first-level cache
using ResidTables = EntryTables<8>;   // 64 symbols of about 1024 slots, up to a hundred contexts

struct Stream {
  const uint8_t* at;
  const uint8_t* end;
  uint32_t x;
  bool open(const uint8_t* bytes, size_t size) {
    if (size < 4) return false;
    std::memcpy(&x, bytes, 4);   // little endian, as everything in a frame
    at = bytes + 4;
    end = bytes + size;
    return x >= kLow;
  }
  bool closed() const { return at == end && x == kLow; }
};

// One update.  The state after the multiply-add is at least 2^7, so it takes at most two bytes.
template <uint32_t kShift>
GRB_INLINE uint32_t take(Stream& s, const Entry* buckets, const Entry* entries, uint32_t& short_of) {
  const uint32_t slot = s.x & (kTotal - 1);
  const Entry* e = buckets + (slot >> kShift);
  uint32_t d = slot - e->first;
  if (__builtin_expect(d > e->last, 0)) {
    e = entries + e->rank;
    do { ++e; d = slot - e->first; } while (d > e->last);
  }
  const uint32_t hi = s.x >> 16, x = e->last * hi + hi + d;
  const uint32_t n = uint32_t(x < kLow) + uint32_t(x < (1u << 15));
  uint32_t next;
  if (__builtin_expect(s.end - s.at >= 4, 1)) {
    std::memcpy(&next, s.at, 4);
    next = __builtin_bswap32(next);
  } else {
    next = 0;
    for (uint32_t i = 0; i < 2; ++i) next |= (s.end - s.at > int64_t(i) ? uint32_t(s.at[i]) : 0u) << (24 - 8 * i);
    short_of |= uint32_t(int64_t(n) > s.end - s.at);
  }
  s.x = uint32_t((uint64_t(x) << 32 | next) >> (32 - 8 * n));
  s.at += n;
  return e->what;
}

struct FrameJob {
  const uint8_t *rc, *cc, *raw;
  size_t raw_bytes;
  uint32_t rows, cols, nc, stride;
  const MainTables* main_tables;
  const ResidTables* resid_tables;
  uint32_t *main_states, *main_offsets, *resid_states, *resid_offsets;
  const uint8_t *main_bytes, *resid_bytes;
  uint16_t* words;
  volatile uint64_t* progress;
};

// The words of all rows in order; false when a stream is malformed.
template <bool CODED>
GRB_INLINE bool frame_words(const FrameJob& j, Stream s, Stream t) {
  uint32_t flags = 0, short_of = 0, until_mark = 0;
  uint64_t mark = 0, bit = 0;
  const Entry* buckets[16];
  const Entry* entries[16];
  uint16_t* w = j.words;
  for (uint32_t row = 0; row < j.rows; ++row) {
    for (uint32_t c = 0; c < j.nc; ++c) {
      buckets[c] = j.main_tables->buckets(uint32_t(j.rc[row]) * j.nc + c);
      entries[c] = j.main_tables->entries(uint32_t(j.rc[row]) * j.nc + c);
    }
    for (uint32_t col = 0; col < j.cols;) {
      uint32_t stop = j.cols;
      if (j.stride) {
        if (!until_mark) {
          j.main_states[mark] = s.x;
          j.main_offsets[mark] = uint32_t(s.at - j.main_bytes);
          if (CODED) {
            j.resid_states[mark] = t.x;
            j.resid_offsets[mark] = uint32_t(t.at - j.resid_bytes);
          }
          ++mark;
          until_mark = j.stride;
        }
        stop = std::min(j.cols - col, until_mark) + col;
        until_mark -= stop - col;
      }
      for (; col < stop; ++col) {
        const uint32_t c = j.cc[col], m = take<MainTables::shift>(s, buckets[c], entries[c], short_of);
        uint32_t r;
        if (CODED) {
          r = take<ResidTables::shift>(t, j.resid_tables->buckets(m & 1023u), j.resid_tables->entries(m & 1023u), short_of);
        } else {
          const size_t b = size_t(bit >> 3);
          const uint32_t two = uint32_t(j.raw[b]) << 8 | (b + 1 < j.raw_bytes ? j.raw[b + 1] : 0u);
          r = (two >> (10 - uint32_t(bit & 7))) & 63u;
          bit += 6;
        }
        flags |= m | r;
        *w++ = join_word(m, r);
      }
    }
    if ((flags & kDead) || short_of) return false;
    if (j.progress) __atomic_store_n(j.progress, uint64_t(row) + 1, __ATOMIC_RELEASE);
  }
  return s.closed() && (!CODED || t.closed());
}
GRB_CLONES bool frame_words_raw(const FrameJob& j, Stream s, Stream t) { return frame_words<false>(j, s, t); }
GRB_CLONES bool frame_words_coded(const FrameJob& j, Stream s, Stream t) { return frame_words<true>(j, s, t); }

// ---- encoding -------------------------------------------------------------------------------------------------
// The division-free form of the update is the one of F. Giesen's public-domain byte-wise rANS coder (ryg_rans: bound, reciprocal,
// bias and complemented frequency per symbol), here with a 64-bit reciprocal, which needs no shift.
// What coding one symbol needs: a renormalisation bound, the reciprocal ceil(2^64 / f) (exact for 32-bit states), and the
// state's new value as q * scale + x + bias with q = floor(x / f).  f == 1 has no such reciprocal: with 2^64 - 1 the quotient
// comes out as x - 1, which its bias makes good.
struct Coding {
  uint64_t reciprocal;
  uint32_t bound, bias, scale, live;
};

GRB_CLONES void emit_rows(const uint16_t* words, uint32_t rows, uint32_t cols, const uint8_t* rc, const uint8_t* cc, uint32_t nc, uint32_t kind,
                          const Coding* table, uint8_t* end, uint8_t** begin, uint32_t* state, uint32_t* dead) {
  uint8_t* p = end;
  uint32_t x = kLow, all_live = 1;
  for (uint32_t row = rows; row-- > 0;) {
    const uint16_t* w = words + size_t(row) * cols;
    const Coding* base = kind ? table : table + size_t(rc[row]) * nc * 1024;
    for (uint32_t col = cols; col-- > 0;) {
      const uint32_t m = main_symbol(w[col]);
      const Coding& c = kind ? base[m * 64 + residual_symbol(w[col])] : base[size_t(cc[col]) * 1024 + m];
      // the bytes go out unconditionally, the position moves by those that count
      const uint64_t bound = c.bound;
      const uint32_t n = uint32_t(x >= bound) + uint32_t(x >= bound << 8);
      const uint16_t low = uint16_t(x), out = uint16_t(low << 8 | low >> 8);
      std::memcpy(p - 2, &out, 2);
      p -= n;
      x >>= 8 * n;
      const uint32_t q = uint32_t((unsigned __int128)(x) * c.reciprocal >> 64);
      x += c.bias + q * c.scale;
      all_live &= c.live;
    }
  }
  *begin = p;
  *state = x;
  *dead = !all_live;
}

}  // namespace

// Codes the whole tensor under `freq`; false when a word's symbol has frequency zero.  `out` receives the stream.
bool encode_stream(const uint16_t* words, uint32_t rows, uint32_t cols, const uint8_t* rc, const uint8_t* cc, uint32_t nr, uint32_t nc, uint32_t kind,
                   const uint32_t* freq, uint8_t** stream, size_t* size) {
  const uint32_t vocab = kind ? 64u : 1024u, nctx = kind ? 1024u : nr * nc;
  std::vector<Coding> table(size_t(nctx) * vocab);
  for (uint32_t cx = 0; cx < nctx; ++cx) {
    uint32_t run = 0;
    for (uint32_t s = 0; s < vocab; ++s) {
      const uint32_t f = freq[size_t(cx) * vocab + s];
      Coding& c = table[size_t(cx) * vocab + s];
      if (f == 0 || f > kTotal) continue;   // value-initialised: live = 0
      c.bound = f << 15;                    // ((2^23 >> 16) << 8) f; 2^31 for f = 2^16, which no state reaches
      c.reciprocal = f == 1 ? ~uint64_t(0) : ~uint64_t(0) / f + 1;
      c.bias = f == 1 ? run + kTotal - 1 : run;
      c.scale = kTotal - f;
      c.live = 1;
      run += f;
    }
  }
  const uint64_t n = uint64_t(rows) * cols;
  // at most two bytes per symbol; touched from the end, so that what is not needed is never paged in
  const size_t room = size_t(n) * 2 + 16;
  auto* buffer = static_cast<uint8_t*>(std::malloc(room));
  if (!buffer) throw std::bad_alloc();
  uint8_t* begin = nullptr;
  uint32_t x = 0, dead = 0;
  emit_rows(words, rows, cols, rc, cc, nc, kind, table.data(), buffer + room, &begin, &x, &dead);
  if (dead) { std::free(buffer); return false; }
  const size_t tail = size_t(buffer + room - begin);
  auto* out = static_cast<uint8_t*>(std::malloc(tail + 4));
  if (!out) { std::free(buffer); throw std::bad_alloc(); }
  std::memcpy(out, &x, 4);
  std::memcpy(out + 4, begin, tail);
  std::free(buffer);
  *stream = out;
  *size = tail + 4;
  return true;
}

}  // namespace grb

extern "C" {

using namespace grb;

// Sums of word & 0x7FFF per row and per column.  0 ok, 1 bad arguments, 3 other failure.
int grb_bctx_magnitudes(const uint16_t* words, uint32_t rows, uint32_t cols, uint64_t* row_sum, uint64_t* col_sum) {
  try {
    if (!words || !rows || !cols || !row_sum || !col_sum) return 1;
    const uint32_t threads = std::min(rows, threads_for(uint64_t(rows) * cols));
    std::vector<std::vector<uint64_t>> parts(threads);
    on_threads(threads, [&](uint32_t t) {
      parts[t].assign(cols, 0);
      std::vector<uint32_t> run(cols, 0);
      const uint32_t r0 = uint32_t(uint64_t(rows) * t / threads), r1 = uint32_t(uint64_t(rows) * (t + 1) / threads);
      uint32_t pending = 0;
      auto flush = [&] {
        for (uint32_t c = 0; c < cols; ++c) { parts[t][c] += run[c]; run[c] = 0; }
        pending = 0;
      };
      for (uint32_t r = r0; r < r1; ++r) {
        const uint16_t* w = words + size_t(r) * cols;
        uint64_t sum = 0;
        for (uint32_t c0 = 0; c0 < cols; c0 += 65536) {   // 65536 x 32767 fits 32 bits
          uint32_t part = 0;
          const uint32_t c1 = std::min(cols, c0 + 65536);
          for (uint32_t c = c0; c < c1; ++c) { const uint32_t v = w[c] & 0x7FFFu; part += v; run[c] += v; }
          sum += part;
        }
        row_sum[r] = sum;
        if (++pending == 65536) flush();
      }
      flush();
    });
    for (uint32_t c = 0; c < cols; ++c) {
      col_sum[c] = 0;
      for (const auto& p : parts) col_sum[c] += p[c];
    }
    return 0;
  } catch (...) {
    return 3;
  }
}

// Frequencies of both streams in one pass over the words: what bcx_frequencies gives for kinds 0 and 1.  resid_floor
// receives a lower bound of the conditional residual stream's bytes: a step multiplies the state by at least
// (65536 / f)(1 - 2^-7) (the state is at least 2^7 f when a symbol of frequency f is coded, and coding loses less than one
// unit of state / f), a byte taken out divides it by at most 256 / (1 - 1 / (2^7 f)), at most two are before a symbol, and
// the state starts at 2^23 and ends below 2^32.  0 ok, 1 bad arguments, 3 other failure.
int grb_bctx_frequencies(const uint16_t* words, uint32_t rows, uint32_t cols, const uint8_t* rc, const uint8_t* cc, uint32_t nr, uint32_t nc,
                         uint32_t* main_freq, uint32_t* resid_freq, uint64_t* resid_floor) {
  try {
    if (!words || !rows || !cols || !rc || !cc || !nr || !nc || !main_freq || !resid_freq || !resid_floor) return 1;
    const size_t main_n = size_t(nr) * nc * 1024, resid_n = 1024 * 64;
    // counts of 32 bits: MAX_WORDS words at most
    const uint32_t threads = std::min(rows, threads_for(uint64_t(rows) * cols));
    std::vector<std::vector<uint32_t>> parts(threads);
    on_threads(threads, [&](uint32_t t) {
      auto& counts = parts[t];
      counts.assign(main_n + resid_n, 0);
      const uint32_t r0 = uint32_t(uint64_t(rows) * t / threads), r1 = uint32_t(uint64_t(rows) * (t + 1) / threads);
      for (uint32_t r = r0; r < r1; ++r) {
        const uint16_t* w = words + size_t(r) * cols;
        uint32_t* base = &counts[size_t(rc[r]) * nc * 1024];
        for (uint32_t c = 0; c < cols; ++c) {
          const uint32_t m = main_symbol(w[c]);
          ++base[size_t(cc[c]) * 1024 + m];
          ++counts[main_n + m * 64 + residual_symbol(w[c])];
        }
      }
    });
    std::vector<uint64_t> counts(main_n + resid_n, 0);
    for (const auto& p : parts)
      for (size_t i = 0; i < counts.size(); ++i) counts[i] += p[i];
    for (uint32_t cx = 0; cx < nr * nc; ++cx) quantise_counts(&counts[size_t(cx) * 1024], 1024, main_freq + size_t(cx) * 1024);
    double bits = -9;
    for (uint32_t cx = 0; cx < 1024; ++cx) {
      const uint64_t* n = &counts[main_n + size_t(cx) * 64];
      uint32_t* f = resid_freq + size_t(cx) * 64;
      quantise_counts(n, 64, f);
      for (uint32_t s = 0; s < 64; ++s)
        if (n[s]) bits += double(n[s]) * (16 - std::log2(double(f[s])) + std::log2(1 - 1.0 / 128) + 2 * std::log2(1 - 1 / (128.0 * f[s])));
    }
    *resid_floor = bits > 8 ? uint64_t(bits * (1 - 1e-9) / 8) : 0;
    return 0;
  } catch (...) {
    return 3;
  }
}

// bcx_encode without the counting: one stream under given frequencies.
int grb_bctx_encode_stream(const uint16_t* words, uint32_t rows, uint32_t cols, const uint8_t* rc, const uint8_t* cc, uint32_t nr, uint32_t nc,
                           uint32_t kind, const uint32_t* freq, uint8_t** stream, size_t* stream_bytes) {
  try {
    if (!words || !rows || !cols || !rc || !cc || !nr || !nc || kind > 1 || !freq || !stream || !stream_bytes) return 1;
    return encode_stream(words, rows, cols, rc, cc, nr, nc, kind, freq, stream, stream_bytes) ? 0 : 3;
  } catch (const std::bad_alloc&) {
    return 2;
  } catch (...) {
    return 3;
  }
}

// The words of a frame in one pass over its streams, and (stride > 0) the restart points before every stride-th word.
// resid_freq == NULL: raw residuals.  progress (optional) receives the number of finished rows as they are finished.
// 0 ok; 1 bad arguments; 2 malformed in some way (outputs must be discarded): bcx_decode / bcx_checkpoint say how.
int grb_bctx_frame_words(const uint8_t* main_stream, size_t main_bytes, const uint8_t* resid, size_t resid_bytes, uint32_t rows, uint32_t cols,
                         const uint8_t* rc, const uint8_t* cc, uint32_t nr, uint32_t nc, const uint32_t* main_freq, const uint32_t* resid_freq,
                         uint32_t stride, uint32_t* main_states, uint32_t* main_offsets, uint32_t* resid_states, uint32_t* resid_offsets,
                         uint16_t* words, uint64_t* progress) {
  try {
    if (!main_stream || !resid || !rows || !cols || !rc || !cc || !nr || !nc || nc > 16 || !main_freq || !words) return 1;
    if (stride && (!main_states || !main_offsets || (resid_freq && (!resid_states || !resid_offsets)))) return 1;
    const uint64_t n = uint64_t(rows) * cols;
    if (main_bytes > 0xFFFFFFFFull || (resid_freq && resid_bytes > 0xFFFFFFFFull)) return 2;
    for (uint32_t r = 0; r < rows; ++r) if (rc[r] >= nr) return 2;
    for (uint32_t c = 0; c < cols; ++c) if (cc[c] >= nc) return 2;
    if (!resid_freq) {
      if (resid_bytes != size_t((n * 6 + 7) / 8)) return 2;
      const uint32_t used = uint32_t(n * 6 % 8);
      if (used && (resid[resid_bytes - 1] & (0xFFu >> used))) return 2;
    }
    MainTables main_tables;
    ResidTables resid_tables;
    if (!main_tables.load(main_freq, nr * nc, 1024) || (resid_freq && !resid_tables.load(resid_freq, 1024, 64))) return 2;
    Stream s{}, t{};
    if (!s.open(main_stream, main_bytes) || (resid_freq && !t.open(resid, resid_bytes))) return 2;
    const FrameJob job{rc, cc, resid, resid_bytes, rows, cols, nc, stride, &main_tables, &resid_tables, main_states, main_offsets, resid_states,
                       resid_offsets, main_stream, resid, words, progress};
    return (resid_freq ? frame_words_coded(job, s, t) : frame_words_raw(job, s, t)) ? 0 : 2;
  } catch (...) {
    return 3;
  }
}

}  // extern "C"

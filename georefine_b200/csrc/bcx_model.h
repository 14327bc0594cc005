// Static probability model of one BCTX stream kind: per context, validated prefix sums of the 16-bit
// frequencies and an inverse index from slot to symbol.  Shared by the host walker and (through its
// exported tables) by the CUDA decoder of unchanged streams.
//
// Word split (reference: context-runtime/georefine_context_runtime/bitexact_context_ans.cpp:9-12):
//   main     = exponent(8) << 2 | mantissa[6:5]      10 bits, vocabulary 1024
//   residual = sign << 5 | mantissa[4:0]              6 bits, vocabulary 64
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <vector>

namespace grb {

inline uint32_t main_symbol(uint16_t w) { return (uint32_t(w) >> 5) & 0x3FFu; }
inline uint32_t residual_symbol(uint16_t w) { return ((uint32_t(w) >> 10) & 32u) | (w & 31u); }
inline uint16_t join_word(uint32_t main, uint32_t residual) {
  return uint16_t((main << 5) | (residual & 31u) | ((residual & 32u) << 10));
}

// bcx_host.cpp, bcx_frame.cpp
void quantise_counts(const uint64_t* counts, uint32_t vocab, uint32_t* freq);
bool encode_stream(const uint16_t* words, uint32_t rows, uint32_t cols, const uint8_t* rc, const uint8_t* cc, uint32_t nr, uint32_t nc, uint32_t kind,
                   const uint32_t* freq, uint8_t** stream, size_t* size);

constexpr uint32_t kBucketShift = 4;                   // 16 slots per bucket
constexpr uint32_t kBuckets = 65536u >> kBucketShift;  // 4096 buckets per context

class Model {
 public:
  // False when a frequency exceeds 2^16, or a context's sum is neither 0 nor 2^16.
  bool load(const uint32_t* freq, uint32_t nctx, uint32_t vocab) {
    nctx_ = nctx;
    vocab_ = vocab;
    cum_.assign(size_t(nctx) * (vocab + 1), 0);
    bucket_.assign(size_t(nctx) * kBuckets, 0);
    live_.assign(nctx, 0);
    for (uint32_t cx = 0; cx < nctx; ++cx) {
      uint32_t* c = &cum_[size_t(cx) * (vocab + 1)];
      uint64_t run = 0;
      for (uint32_t s = 0; s < vocab; ++s) {
        const uint32_t f = freq[size_t(cx) * vocab + s];
        c[s] = uint32_t(run);
        if (f > 65536u || run + f > 65536u) return false;
        run += f;
      }
      c[vocab] = uint32_t(run);
      if (run != 0 && run != 65536u) return false;
      live_[cx] = run == 65536u;
      if (!live_[cx]) continue;
      uint16_t* b = &bucket_[size_t(cx) * kBuckets];
      uint32_t s = 0;
      for (uint32_t k = 0; k < kBuckets; ++k) {
        const uint32_t slot = k << kBucketShift;
        while (c[s + 1] <= slot) ++s;
        b[k] = uint16_t(s);
      }
    }
    return true;
  }
  bool live(uint32_t cx) const { return live_[cx] != 0; }
  uint32_t start(uint32_t cx, uint32_t s) const { return cum_[size_t(cx) * (vocab_ + 1) + s]; }
  // The symbol whose slot range contains `slot` (context must be live).
  uint32_t find(uint32_t cx, uint32_t slot) const {
    const uint32_t* c = &cum_[size_t(cx) * (vocab_ + 1)];
    uint32_t s = bucket_[size_t(cx) * kBuckets + (slot >> kBucketShift)];
    while (c[s + 1] <= slot) ++s;
    return s;
  }
  void export_tables(uint32_t* cum, uint16_t* bucket) const {
    std::copy(cum_.begin(), cum_.end(), cum);
    std::copy(bucket_.begin(), bucket_.end(), bucket);
  }

 private:
  uint32_t nctx_ = 0, vocab_ = 0;
  std::vector<uint32_t> cum_;
  std::vector<uint16_t> bucket_;
  std::vector<uint8_t> live_;
};

// The models of a frame packed for shared memory (csrc/bctx_packed.cuh).  A context has few live symbols (60 to 80 of 1024
// on Gaussian weights), so its model is: u16 bucket[65536 >> shift] = rank << 8 | 255 - last, where rank is the rank among the
// live symbols of the one that owns the bucket's first slot and `last` (0..255) the last place in the bucket that symbol owns
// (255 when it owns all of it), so that (bucket + place) >> 8 is the rank at any place up to the bucket's second boundary;
// and entries of 8 bytes in rank order, {first slot u16 | frequency - 1 u16, what the symbol means u32}.  Buckets with more
// boundaries, where rare symbols lie, end in a forward scan of the entries, which always ends: the last live entry reaches up
// to slot 65535, and entries past it match any slot.
// Layout: the main contexts at multiples of ctx_bytes (those of one row class, one per column class, side by side: a kernel
// may keep one row class only, `resident` contexts); from resid_at on the residual contexts (coded residuals only) of the
// main symbols that occur anywhere, each as long as its live symbols need.  The meaning of a main entry is
// symbol << 5 | (offset of its residual context from resid_at) / 8 << 16, that of a residual entry its bits of the word.
struct PackedShape {
  uint32_t shift, ctx_bytes, resid_shift, resid_at, bytes;
};

constexpr uint64_t kPackedImageMax = 4u << 20;   // what the prefix sums of a 64 x 16 frame take, too

class PackedTables {
 public:
  // resid_freq == nullptr: raw residuals.  False when the frequencies are invalid.
  bool load(const uint32_t* main_freq, uint32_t nctx, const uint32_t* resid_freq) {
    main_ = main_freq;
    resid_ = resid_freq;
    nctx_ = nctx;
    ranks_ = 1;
    occurs_.assign(1024, 0);
    for (uint32_t cx = 0; cx < nctx; ++cx) {
      uint32_t live = 0;
      if (!count(main_freq + size_t(cx) * 1024, 1024, live)) return false;
      for (uint32_t s = 0; s < 1024; ++s) occurs_[s] |= main_freq[size_t(cx) * 1024 + s] != 0;
      ranks_ = std::max(ranks_, live);
    }
    resid_live_.assign(1024, 0);
    resid_entries_ = resid_contexts_ = 0;
    unpaired_ = false;
    for (uint32_t s = 0; resid_ && s < 1024; ++s) {
      if (!count(resid_ + size_t(s) * 64, 64, resid_live_[s])) return false;
      if (!occurs_[s]) continue;
      unpaired_ |= !resid_live_[s];
      ++resid_contexts_;
      resid_entries_ += resid_live_[s];
    }
    return true;
  }
  // The bucket widths with the fewest scan steps (rare symbols, which share buckets, are mostly main symbols) whose tables,
  // `resident` main contexts of them, fit `limit` bytes; false when none do, or the packed form cannot hold the models.
  bool shape(uint32_t resident, uint32_t limit, PackedShape& out) const {
    // (a main symbol that has a frequency but no residual model: valid as long as the streams never code it, and left
    // to the kernel whose scan is bounded by the vocabulary)
    if (ranks_ > 255 || unpaired_) return false;
    uint64_t best = ~uint64_t(0);
    for (uint32_t ms = 3; ms <= 8; ++ms)
      for (uint32_t rs = resid_ ? 4 : 8; rs <= 8; ++rs) {
        const uint64_t ctx = ((131072u >> ms) + ranks_ * 8 + 15) & ~15u, resid_at = ctx * nctx_;
        const uint64_t resid = resid_ ? uint64_t(resid_contexts_) * (131072u >> rs) + uint64_t(resid_entries_) * 8 : 0;
        const uint64_t bytes = (resid_at + resid + 15) & ~uint64_t(15), kept = bytes - resid_at + ctx * resident, cost = (uint64_t(ranks_) << ms) + (resid_ ? uint64_t(16) << rs : 0);
        if (kept > limit || bytes > kPackedImageMax || resid > 65535u * 8 || cost >= best) continue;
        best = cost;
        out = PackedShape{ms, uint32_t(ctx), rs, uint32_t(resid_at), uint32_t(bytes)};
      }
    return best != ~uint64_t(0);
  }
  void write(const PackedShape& p, uint8_t* image) const {
    std::memset(image, 0, p.bytes);
    std::vector<uint32_t> resid_of(1024, 0);
    uint32_t at = 0;
    for (uint32_t s = 0; resid_ && s < 1024; ++s) {
      if (!occurs_[s]) continue;
      resid_of[s] = at;
      context(resid_ + size_t(s) * 64, 64, p.resid_shift, resid_live_[s], image + p.resid_at + at,
              [](uint32_t r) { return (r & 31u) | (r & 32u) << 10; });
      at += (131072u >> p.resid_shift) + resid_live_[s] * 8;
    }
    for (uint32_t cx = 0; cx < nctx_; ++cx)
      context(main_ + size_t(cx) * 1024, 1024, p.shift, ranks_, image + size_t(cx) * p.ctx_bytes,
              [&](uint32_t s) { return s << 5 | (resid_of[s] >> 3) << 16; });
  }

 private:
  static bool count(const uint32_t* freq, uint32_t vocab, uint32_t& live) {
    uint64_t sum = 0;
    live = 0;
    for (uint32_t s = 0; s < vocab; ++s) { sum += freq[s]; live += freq[s] != 0; }
    return sum == 0 || sum == 65536u;
  }
  template <class Meaning>
  static void context(const uint32_t* freq, uint32_t vocab, uint32_t shift, uint32_t ranks, uint8_t* at, Meaning meaning) {
    uint8_t* entry = at + (131072u >> shift);
    uint32_t r = 0, run = 0;
    auto put = [&](uint32_t lo, uint32_t last, uint32_t what) {
      const uint32_t words[2] = {lo | last << 16, what};
      std::memcpy(entry + size_t(r++) * 8, words, 8);
    };
    const uint32_t round = (1u << shift) - 1;
    for (uint32_t s = 0; s < vocab; ++s) {
      const uint32_t f = freq[s];
      if (!f) continue;
      const uint32_t first = (run + round) >> shift, end = (run + f + round) >> shift;   // buckets whose first slot is the symbol's
      for (uint32_t b = first; b < end; ++b) {
        const uint32_t last = std::min(run + f - 1 - (b << shift), 255u);
        const uint16_t v = uint16_t(r << 8 | (255u - last));
        std::memcpy(at + 2 * size_t(b), &v, 2);
      }
      put(run, f - 1, meaning(s));
      run += f;
    }
    while (r < ranks) put(0, 65535, 0);
  }

  const uint32_t *main_ = nullptr, *resid_ = nullptr;
  uint32_t nctx_ = 0, ranks_ = 0, resid_entries_ = 0, resid_contexts_ = 0;
  bool unpaired_ = false;
  std::vector<uint8_t> occurs_;
  std::vector<uint32_t> resid_live_;
};

}  // namespace grb

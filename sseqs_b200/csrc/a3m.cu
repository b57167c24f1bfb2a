// Host-side a3m row assembly (sseqs/to_a3m.py:16-72): the rows of the a3m
// file built from traceback results, in a given order, with the reference's
// placement, case and filtering rules.  Plain C++ (no device code); the
// Python layer computes the order (np.argsort of the scores, descending) and
// passes pointers into the traceback's host byte matrices.
//
// Rows are written where they go in the output, in runs rather than byte by byte,
// and repeats are found by a hash of the bytes written (2048 rows of a 413-residue
// query: 2.3 -> 0.7 ms on one host core against a string per row, a formatted
// header and a set of strings).
#include <cstdint>
#include <cstring>
#include <vector>

#include "sseqs_b200.h"

namespace {
inline uint8_t lower_ascii(uint8_t c) { return (uint8_t)((c >= 'A' && c <= 'Z') ? c + 32 : c); }

// First occurrence of needle in hay (both without a preparation that would
// cost more than the search: a fragment usually matches at its first candidate).
inline int64_t find_first(const char* hay, int64_t n, const char* needle, int64_t m) {
  for (const char* p = hay; m <= n - (p - hay);) {
    p = static_cast<const char*>(std::memchr(p, needle[0], (size_t)(n - (p - hay) - m + 1)));
    if (!p) return -1;
    if (std::memcmp(p, needle, (size_t)m) == 0) return p - hay;
    ++p;
  }
  return -1;
}

// 64-bit hash of n bytes, 8 at a time (multiply and xor-shift; the multiplier is
// that of MurmurHash3's 64-bit finaliser, public domain).
inline uint64_t hash_bytes(const char* p, size_t n) {
  uint64_t h = 0x9e3779b97f4a7c15ull ^ (uint64_t)n;
  auto mix = [&](uint64_t w) {
    h = (h ^ w) * 0xff51afd7ed558ccdull;
    h ^= h >> 32;
  };
  for (; n >= 8; p += 8, n -= 8) {
    uint64_t w;
    std::memcpy(&w, p, 8);
    mix(w);
  }
  uint64_t w = 0;
  std::memcpy(&w, p, n);
  mix(w);
  return h;
}

// Rows already in the output, by content (open addressing).
class RowSet {
 public:
  RowSet(const char* base, int64_t rows) : base_(base) {
    size_t cap = 16;
    while (cap < (size_t)rows * 2) cap <<= 1;
    slots_.assign(cap, Slot{0, -1, 0});
  }
  bool insert(int64_t at, size_t n) {           // false: an equal row is there
    const uint64_t h = hash_bytes(base_ + at, n);
    Slot& s = find(base_ + at, n, h);
    if (s.at >= 0) return false;
    s = Slot{h, at, n};
    return true;
  }
  bool contains(const char* row, size_t n) { return find(row, n, hash_bytes(row, n)).at >= 0; }

 private:
  struct Slot {
    uint64_t hash;
    int64_t at;
    size_t n;
  };
  Slot& find(const char* row, size_t n, uint64_t h) {   // an equal row's slot, or a free one
    for (size_t k = h & (slots_.size() - 1);; k = (k + 1) & (slots_.size() - 1)) {
      Slot& s = slots_[k];
      if (s.at < 0 || (s.hash == h && s.n == n && std::memcmp(base_ + s.at, row, n) == 0)) return s;
    }
  }
  const char* base_;
  std::vector<Slot> slots_;
};

inline char* put(char* p, const char* text) {
  const size_t n = std::strlen(text);
  std::memcpy(p, text, n);
  return p + n;
}
inline char* put(char* p, int64_t v) {
  char buf[24];
  int k = 24;
  uint64_t u = v < 0 ? 0 - (uint64_t)v : (uint64_t)v;
  do {
    buf[--k] = (char)('0' + u % 10);
    u /= 10;
  } while (u);
  if (v < 0) buf[--k] = '-';
  std::memcpy(p, buf + k, (size_t)(24 - k));
  return p + (24 - k);
}
}  // namespace

extern "C" int sseqs_a3m_rows(const char* query, int64_t query_len, int64_t n_rows,
                              const int64_t* order, const uint8_t* const* q_rows,
                              const uint8_t* const* t_rows, const int32_t* lens,
                              const int64_t* scores, char* out, int64_t out_cap,
                              int64_t* out_len) {
  if (!query || query_len < 0 || n_rows < 0 || !out || !out_len || out_cap < 0 ||
      (n_rows > 0 && (!order || !q_rows || !t_rows || !lens || !scores)))
    return SSEQS_ERR_ARG;
  *out_len = 0;
  try {
    RowSet seen(out, n_rows);
    std::vector<char> compact, spill;
    std::vector<int32_t> gaps;
    int64_t pos = 0;
    for (int64_t i = 0; i < n_rows; ++i) {
      const int64_t k = order[i];
      if (k < 0 || k >= n_rows) return SSEQS_ERR_ARG;
      const int32_t n = lens[k];
      if (scores[k] == 0 || n <= 0) continue;          // score 0 or no alignment
      const uint8_t* qa = q_rows[k];
      const uint8_t* ta = t_rows[k];
      // the query's residues without gaps, run by run; `gaps`: columns that are one
      if (compact.size() < (size_t)n) compact.resize((size_t)n);
      gaps.clear();
      int64_t m = 0;
      for (int32_t j = 0; j < n;) {
        const void* g = std::memchr(qa + j, '-', (size_t)(n - j));
        const int32_t e = g ? (int32_t)(static_cast<const uint8_t*>(g) - qa) : n;
        std::memcpy(compact.data() + m, qa + j, (size_t)(e - j));
        m += e - j;
        if (g) gaps.push_back(e);
        j = e + 1;
      }
      // first occurrence, as str.find
      const int64_t q0 = m > 0 ? find_first(query, query_len, compact.data(), m) : 0;
      if (q0 < 0) return SSEQS_ERR_UNSUPPORTED;
      const int64_t row_len = query_len - m + n;
      char head[64];                                   // ">target_<i> score=<s>.0"
      const char* head_end = put(put(put(put(put(head, ">target_"), i), " score="), scores[k]), ".0\n");
      const int64_t head_len = head_end - head;
      // a row that does not fit is an error only if it is kept
      const bool fits = pos + head_len + row_len + 1 <= out_cap;
      if (!fits) spill.resize((size_t)row_len);
      char* row = fits ? out + pos + head_len : spill.data();
      char* p = row;
      std::memset(p, '-', (size_t)q0);
      p += q0;
      // upper case over the row, then lower case where the query has a gap
      for (int32_t j = 0; j < n; ++j) {
        const uint8_t tc = ta[j];
        p[j] = (char)(tc - ((uint8_t)(tc - 'a') < 26 ? 32 : 0));
      }
      for (const int32_t j : gaps) p[j] = (char)lower_ascii(ta[j]);
      const bool at_sign = std::memchr(p, '@', (size_t)n) != nullptr;
      p += n;
      std::memset(p, '-', (size_t)(query_len - q0 - m));
      p += query_len - q0 - m;
      if (at_sign) continue;                           // written over
      if (!fits) {
        if (seen.contains(row, (size_t)row_len)) continue;
        return SSEQS_ERR_CAPACITY;
      }
      if (!seen.insert(row - out, (size_t)row_len)) continue;
      std::memcpy(out + pos, head, (size_t)head_len);
      *p++ = '\n';
      pos = p - out;
    }
    *out_len = pos;
  } catch (...) {          // out of memory
    return SSEQS_ERR_CAPACITY;
  }
  return SSEQS_OK;
}

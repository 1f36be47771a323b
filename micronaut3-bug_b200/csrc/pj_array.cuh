/*
 * pj_array.cuh — structural index of array framing (`[rec, rec, ...]`), word-parallel: what its kernels share.
 *
 * A 64-byte word of the input is turned into 64-bit masks (one bit per byte) of backslashes, quotes and brackets.
 * From those follows, exactly as the framing rules of petjson.h say:
 *   escaped bytes      a byte is escaped iff an odd run of backslashes precedes it
 *   in-string mask     prefix-XOR of the unescaped quotes
 *   nesting depth      openers minus closers among the bytes outside strings
 * The three quantities carry from word to word (escape carry c, in-string s, depth d), and every carry is
 * a prefix sum, so words are first summarised as a FUNCTION of their incoming (c, s) — four cases — and the
 * summaries are composed by scans (warp shuffle, block, then tiles); with the incoming state known the separators
 * are `[` at depth 0, `,` and `]` at depth 1 (pj_array_index.cuh).
 */
#ifndef PJ_ARRAY_CUH
#define PJ_ARRAY_CUH

#include "pj_core.cuh"

namespace pj {

PJ_HD uint32_t popc64(uint64_t x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)__popcll(x);
#else
  return (uint32_t)__builtin_popcountll(x);
#endif
}
PJ_HD uint32_t ctz64a(uint64_t x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)(__ffsll((long long)x) - 1);
#else
  return (uint32_t)__builtin_ctzll(x);
#endif
}

/* state carried between words */
struct ArrState {
  uint32_t c, s; /* first byte of the next word is escaped; the next word starts inside a string */
  int32_t d;     /* nesting depth */
};
/* bytes escaped by an odd run of backslashes, and the carry into the next word */
PJ_HD uint64_t escaped_mask(uint64_t backslash, uint32_t carry_in, uint32_t* carry_out) {
  const uint64_t even = 0x5555555555555555ull;
  backslash &= ~(uint64_t)carry_in; /* an escaped backslash does not escape */
  const uint64_t follows = (backslash << 1) | carry_in;
  const uint64_t odd_starts = backslash & ~even & ~follows;
  const uint64_t sum = odd_starts + backslash;
  *carry_out = sum < odd_starts ? 1u : 0u; /* a run of backslashes reaching past the word, of odd length */
  const uint64_t invert = sum << 1;
  return (even ^ invert) & follows;
}
PJ_HD uint64_t prefix_xor(uint64_t x) {
  x ^= x << 1; x ^= x << 2; x ^= x << 4; x ^= x << 8; x ^= x << 16; x ^= x << 32;
  return x;
}
/* A word (or any run of words) as a function of its incoming (c, s): index x = c | s << 1. */
struct ArrFn {
  uint32_t st;  /* four 2-bit outgoing states, entry x in bits 2x..2x+1 */
  int32_t d[4]; /* depth change for each incoming state */
};
PJ_HD ArrFn fn_identity() { ArrFn f; f.st = 0xE4u; f.d[0] = f.d[1] = f.d[2] = f.d[3] = 0; return f; }
PJ_HD int32_t fn_pick(const int32_t* d, uint32_t x) { return x == 0 ? d[0] : (x == 1 ? d[1] : (x == 2 ? d[2] : d[3])); }
/* first f, then g */
PJ_HD ArrFn fn_compose(const ArrFn& f, const ArrFn& g) {
  ArrFn h;
  h.st = 0;
  for (uint32_t x = 0; x < 4; ++x) {
    const uint32_t mid = (f.st >> (2 * x)) & 3u;
    h.st |= ((g.st >> (2 * mid)) & 3u) << (2 * x);
    h.d[x] = f.d[x] + fn_pick(g.d, mid);
  }
  return h;
}
PJ_HD ArrState fn_apply(const ArrFn& f, ArrState in) {
  const uint32_t x = in.c | (in.s << 1);
  const uint32_t o = (f.st >> (2 * x)) & 3u;
  ArrState out;
  out.c = o & 1; out.s = o >> 1; out.d = in.d + fn_pick(f.d, x);
  return out;
}

/* The extent that starts after the separator at byte p (a `[` or `,`; a `]` starts none).
 * sep: separator bitmap, one bit per input byte; first_opener: offset of the first `[` at depth 0. */
struct ExtentOut {
  uint32_t is_record, blank, second_opener;
  uint64_t start, end;
};
PJ_HD ExtentOut arr_extent(const uint8_t* in, uint64_t len, const uint64_t* sep, uint64_t p, uint64_t first_opener) {
  ExtentOut r;
  r.is_record = 0; r.blank = 0; r.second_opener = 0; r.start = p + 1; r.end = len;
  const uint32_t x = ld_byte(in + p);
  if (x == ']') return r;
  const bool left_opener = x == '[';
  r.second_opener = left_opener && p > first_opener;
  /* next separator after p */
  const uint64_t nwords = (len + 63) >> 6;
  uint64_t wi = p >> 6;
  const uint32_t b = (uint32_t)(p & 63);
  uint64_t m = b == 63 ? 0 : (sep[wi] & (~0ull << (b + 1)));
  bool has_right = false;
  for (;;) {
    if (m) { r.end = (wi << 6) + ctz64a(m); has_right = true; break; }
    if (++wi >= nwords) break;
    m = sep[wi];
  }
  uint64_t t = p + 1;
  while (t < r.end) {
    const uint32_t y = ld_byte(in + t);
    if (y == ' ' || y == '\t' || y == '\r' || y == '\n') ++t; else break;
  }
  r.blank = t >= r.end;
  const bool right_closer = has_right && ld_byte(in + r.end) == ']';
  r.is_record = !(r.blank && ((left_opener && right_closer) || !has_right));
  return r;
}

}  // namespace pj
#endif

/*
 * pj_array_ref.h — TEST INFRASTRUCTURE. The separators of array framing word after word, by masks and in order: what k_arr_index
 * (pj_array_index.cuh) is compared with, and what stands in for it where another kernel runs on the host.
 */
#ifndef PJ_ARRAY_REF_H
#define PJ_ARRAY_REF_H

#include "pj_array.cuh"

namespace pj {

struct WordMasks {
  uint64_t B, Q, O, C, M, W, LB, RB, valid; /* backslash, quote, { [, } ], comma, blank, [, ], bytes inside the input */
};

/* bit k of the result: byte k of the 8-byte word w equals c (exact for every byte) */
PJ_HD uint32_t eq_bits8(uint64_t w, uint32_t c) {
  const uint64_t x = w ^ (0x0101010101010101ull * c);
  const uint64_t y = ((x & 0x7F7F7F7F7F7F7F7Full) + 0x7F7F7F7F7F7F7F7Full) | x; /* bit 7 of a byte clear iff the byte is 0 */
  const uint64_t m = (~y & 0x8080808080808080ull) >> 7;
  return (uint32_t)((m * 0x0102040810204080ull) >> 56);
}
/* masks of the 64 bytes at p, of which the first `n` (1..64) are input; the rest read as 0 */
PJ_HD WordMasks word_masks(const uint8_t* p, uint32_t n) {
  WordMasks m;
  m.B = m.Q = m.O = m.C = m.M = m.W = m.LB = m.RB = 0;
  for (uint32_t k = 0; k < 8; ++k) {
    uint64_t w = 0;
    if (8 * k < n) {
      const uint32_t take = n - 8 * k >= 8 ? 8 : n - 8 * k;
      for (uint32_t b = 0; b < take; ++b) w |= (uint64_t)p[8 * k + b] << (8 * b);
    }
    const uint64_t lb = eq_bits8(w, '['), rb = eq_bits8(w, ']'), lc = eq_bits8(w, '{'), rc = eq_bits8(w, '}');
    const uint64_t ws = eq_bits8(w, ' ') | eq_bits8(w, '\t') | eq_bits8(w, '\r') | eq_bits8(w, '\n');
    m.B |= (uint64_t)eq_bits8(w, '\\') << (8 * k);
    m.Q |= (uint64_t)eq_bits8(w, '"') << (8 * k);
    m.M |= (uint64_t)eq_bits8(w, ',') << (8 * k);
    m.LB |= lb << (8 * k); m.RB |= rb << (8 * k);
    m.O |= (lb | lc) << (8 * k); m.C |= (rb | rc) << (8 * k);
    m.W |= ws << (8 * k);
  }
  m.valid = n >= 64 ? ~0ull : ((1ull << n) - 1);
  /* bytes past the input are neither blanks nor anything else */
  m.W &= m.valid;
  return m;
}

struct WordEval {
  uint64_t quotes;   /* unescaped quotes */
  uint64_t interior; /* bytes strictly inside strings */
  uint64_t outside;  /* bytes outside strings that are not quotes */
  ArrState out;
};
PJ_HD WordEval eval_word(const WordMasks& m, ArrState in) {
  WordEval e;
  uint32_t c_out;
  const uint64_t esc = escaped_mask(m.B, in.c, &c_out);
  e.quotes = m.Q & ~esc;
  const uint64_t instr = prefix_xor(e.quotes) ^ (in.s ? ~0ull : 0ull); /* from an opening quote up to, not including, the closing one */
  e.interior = instr & ~e.quotes & m.valid;
  e.outside = ~instr & ~e.quotes & m.valid;
  e.out.c = c_out;
  e.out.s = (uint32_t)(instr >> 63) & 1u;
  e.out.d = in.d + (int32_t)popc64(m.O & e.outside) - (int32_t)popc64(m.C & e.outside);
  return e;
}

PJ_HD ArrFn fn_of_word(const WordMasks& m) {
  ArrFn f;
  f.st = 0;
  for (uint32_t x = 0; x < 4; ++x) {
    ArrState in;
    in.c = x & 1; in.s = x >> 1; in.d = 0;
    const WordEval e = eval_word(m, in);
    f.st |= (e.out.c | (e.out.s << 1)) << (2 * x);
    f.d[x] = e.out.d;
  }
  return f;
}
/* Second pass over a word whose incoming state is known: separators, the lowest byte that breaks
 * `ws [ ... ] ws` (doc_bit, 64 = none) and the lowest opener (opener_bit, 64 = none). */
struct WordMarks {
  uint64_t sep;
  uint32_t doc_bit, opener_bit;
};
PJ_HD WordMarks mark_word(const WordMasks& m, const WordEval& e, int32_t depth_in) {
  WordMarks r;
  uint64_t sep = 0, openers = 0, low = 0; /* low: bytes whose depth is <= 0 */
  int32_t d = depth_in;
  uint32_t seg = 0;
  uint64_t bits = (m.O | m.C) & e.outside;
  while (bits) {
    const uint32_t b = ctz64a(bits);
    const uint64_t bit = 1ull << b;
    bits &= bits - 1;
    /* bytes seg..b see depth d */
    if (d <= 0) low |= (b == 63 ? ~0ull : ((bit << 1) - 1)) & ~((1ull << seg) - 1);
    if (m.O & bit) { if ((m.LB & bit) && d == 0) { sep |= bit; openers |= bit; } d++; }
    else { if ((m.RB & bit) && d == 1) sep |= bit; d--; }
    seg = b + 1;
  }
  if (seg < 64 && d <= 0) low |= ~((1ull << seg) - 1);
  /* commas at depth 1: the bytes at depth exactly 1 are those between the bracket events; redo the walk on commas */
  {
    int32_t dd = depth_in;
    uint64_t ev = (m.O | m.C | m.M) & e.outside;
    while (ev) {
      const uint32_t b = ctz64a(ev);
      const uint64_t bit = 1ull << b;
      ev &= ev - 1;
      if (m.O & bit) dd++;
      else if (m.C & bit) dd--;
      else if (dd == 1) sep |= bit;
    }
  }
  const uint64_t bad = low & ~m.W & ~e.interior & m.valid & ~openers;
  r.sep = sep;
  r.doc_bit = bad ? ctz64a(bad) : 64u;
  r.opener_bit = openers ? ctz64a(openers) : 64u;
  return r;
}

}  // namespace pj
#endif

/*
 * pj_array_index.cuh — k_arr_index<W>: the separators of array framing (see pj_array.cuh for the method) in one pass over the input.
 *
 * One thread = W consecutive 64-byte words, one block = a tile of 16 KB (W = 1) or 64 KB (W = 4). A thread turns its words into masks of
 * quotes, backslashes, openers and closers, 16 bytes per load, and summarises them as a function of the incoming (escape carry, in-string)
 * state; the functions are composed by ordered scans over the warp and the block; the tile's own state comes from one decoupled look-back over the
 * functions of the earlier tiles (two 64-bit words each, and one for a state that is known). With the state known each word's separators are
 * the brackets at depth 0 and 1 and the commas between them; a word that stays deeper has none and is done.
 *
 * Bound by the instructions of the masks, about 9 per byte, and the look-back. 300 k Pets with escapes (91 MB): 480 us in three launches and two passes
 * before, 123 now; 1 M (295 MB): 1600 -> 337, of which 100 are the look-back's. Four blocks per SM (64 registers): with three, five, six
 * of them 355, 370, 375 us; read through shared memory 421 against 415 before that.
 * The bitmap's bits are input bytes; the words are those of the 16-byte aligned addresses, so that any alignment is read alike. Where the two differ the
 * bitmap is zeroed before and words are or-ed into it.
 */
#ifndef PJ_ARRAY_INDEX_CUH
#define PJ_ARRAY_INDEX_CUH

#include "pj_array.cuh"
#include "pj_dev.cuh"
#include "pj_result.h"

namespace pj {

static constexpr uint32_t AI_THREADS = 256, AI_WARPS = AI_THREADS / 32;

struct ArrIndexArgs {
  const uint8_t* in;
  uint64_t len;
  uint64_t* sep; /* one bit per input byte, (len + 63) / 64 words; zeroed when `in` is not 16-byte aligned */
  uint32_t ntiles;
  uint32_t* ticket;
  unsigned long long *fn0, *fn1, *inc; /* [ntiles] each: a tile's function in two words, the state behind it */
  unsigned long long spin_limit_ns;
  DevResult* res;
};

PJ_HD uint32_t arr_tiles(uint32_t mis, uint64_t len, uint32_t words) { /* 64-byte words per thread */
  const uint64_t per = 64ull * words * AI_THREADS;
  return len ? (uint32_t)((mis + len + per - 1) / per) : 1u;
}

__device__ __forceinline__ ArrFn fn_shfl_up(const ArrFn& f, int d) {
  ArrFn g;
  g.st = __shfl_up_sync(0xFFFFFFFFu, f.st, d);
#pragma unroll
  for (int k = 0; k < 4; ++k) g.d[k] = __shfl_up_sync(0xFFFFFFFFu, f.d[k], d);
  return g;
}
__device__ __forceinline__ ArrFn fn_shfl(const ArrFn& f, int lane) {
  ArrFn g;
  g.st = __shfl_sync(0xFFFFFFFFu, f.st, lane);
#pragma unroll
  for (int k = 0; k < 4; ++k) g.d[k] = __shfl_sync(0xFFFFFFFFu, f.d[k], lane);
  return g;
}
/* inclusive ordered scan of the warp's functions (lane 0 first) */
__device__ __forceinline__ ArrFn fn_warp_scan(ArrFn f) {
  const unsigned lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const ArrFn g = fn_shfl_up(f, d);
    if (lane >= (unsigned)d) f = fn_compose(g, f);
  }
  return f;
}
/* a function in two words: states and the first two depths, the other two; a tile's depth changes by 2^16 at most */
__device__ __forceinline__ unsigned long long fn_pack(int32_t a, int32_t b) { return TS_VALID | (unsigned long long)((uint32_t)(a + (1 << 19)) & 0xFFFFFu) | ((unsigned long long)((uint32_t)(b + (1 << 19)) & 0xFFFFFu) << 20); }
__device__ __forceinline__ int32_t fn_depth(unsigned long long w, int k) { return (int32_t)((w >> (20 * k)) & 0xFFFFFu) - (1 << 19); }
__device__ __forceinline__ unsigned long long state_pack(const ArrState& s) { return TS_VALID | (unsigned long long)(uint32_t)s.d | ((unsigned long long)s.s << 32) | ((unsigned long long)s.c << 33); }
__device__ __forceinline__ ArrState state_unpack(unsigned long long w) {
  ArrState s;
  s.d = (int32_t)(uint32_t)w; s.s = (uint32_t)(w >> 32) & 1u; s.c = (uint32_t)(w >> 33) & 1u;
  return s;
}

/* The state before `tile`. Warp 0, all lanes; false when the bounded wait ran out. */
__device__ __forceinline__ bool arr_lookback(const ArrIndexArgs& a, uint32_t tile, uint32_t lane, ArrState* out) {
  ArrFn acc = fn_identity();
  int64_t j = (int64_t)tile - 1;
  const unsigned long long t0 = global_ns();
  for (;;) {
    const int64_t mine = j - (31 - (int64_t)lane); /* the oldest in lane 0 */
    unsigned long long w0, w1, wi;
    uint32_t known;
    for (;;) {
      w0 = w1 = TS_VALID; wi = TS_VALID; /* before the first tile: depth 0, outside strings */
      if (mine >= 0) { wi = ld_relaxed_u64(&a.inc[mine]); w0 = ld_relaxed_u64(&a.fn0[mine]); w1 = ld_relaxed_u64(&a.fn1[mine]); }
      known = __ballot_sync(0xFFFFFFFFu, (wi & TS_VALID) != 0);
      const uint32_t ready = __ballot_sync(0xFFFFFFFFu, (w0 & w1 & TS_VALID) != 0 && mine >= 0) | known;
      const uint32_t need = known ? 0xFFFFFFFFu << (31 - __clz((int)known)) : 0xFFFFFFFFu; /* from the newest known state on */
      if ((ready & need) == need) break;
      uint32_t give_up = 0;
      if (lane == 0) give_up = (global_ns() - t0 > a.spin_limit_ns) || *(volatile uint32_t*)&a.res->timeout;
      give_up = __shfl_sync(0xFFFFFFFFu, give_up, 0);
      if (give_up) { if (lane == 0) atomicExch(&a.res->timeout, 1u); return false; }
      __nanosleep(40);
    }
    const uint32_t from = known ? 31u - (uint32_t)__clz((int)known) : 0u;
    ArrFn f = fn_identity();
    if (known ? lane > from : true) {
      f.st = (uint32_t)(w0 >> 40) & 0xFFu;
      f.d[0] = fn_depth(w0, 0); f.d[1] = fn_depth(w0, 1); f.d[2] = fn_depth(w1, 0); f.d[3] = fn_depth(w1, 1);
    }
    acc = fn_compose(fn_shfl(fn_warp_scan(f), 31), acc);
    if (known) { *out = fn_apply(acc, state_unpack(__shfl_sync(0xFFFFFFFFu, wi, (int)from))); return true; }
    j -= 32;
  }
}

/* 0x80 in every byte of w that equals c (c repeated), exactly */
__device__ __forceinline__ uint32_t arr_eq4(uint32_t w, uint32_t c) { return ~((((w ^ c) & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | (w ^ c)) & 0x80808080u; }
/* 0x80 per byte of four words as 16 bits */
__device__ __forceinline__ uint32_t arr_gather16(uint32_t f0, uint32_t f1, uint32_t f2, uint32_t f3) {
  return (__dp4a(f1, 0x80402010u, __dp4a(f0, 0x08040201u, 0u)) + (__dp4a(f3, 0x80402010u, __dp4a(f2, 0x08040201u, 0u)) << 8)) >> 7;
}
struct ArrWord { uint64_t Q, B, O, C; }; /* quotes, backslashes, openers, closers */

/* 64-byte word at the aligned address p; bytes [lo, hi) of it belong to the input */
__device__ __forceinline__ ArrWord arr_load_word(const uint8_t* p, int32_t lo, int32_t hi) {
  ArrWord m;
  m.Q = m.B = m.O = m.C = 0;
  const uint4* q = reinterpret_cast<const uint4*>(p);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (16 * k >= hi) break; /* never touch a 16-byte block that holds no input byte */
    const uint4 v = q[k];
    const uint32_t x[4] = {v.x, v.y, v.z, v.w};
    uint32_t fq[4], fb[4], fo[4], fc[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t y = x[i] | 0x20202020u; /* [ and { differ in this bit only, ] and } too */
      fq[i] = arr_eq4(x[i], 0x22222222u); fb[i] = arr_eq4(x[i], 0x5C5C5C5Cu); fo[i] = arr_eq4(y, 0x7B7B7B7Bu); fc[i] = arr_eq4(y, 0x7D7D7D7Du);
    }
    m.Q |= (uint64_t)arr_gather16(fq[0], fq[1], fq[2], fq[3]) << (16 * k);
    m.B |= (uint64_t)arr_gather16(fb[0], fb[1], fb[2], fb[3]) << (16 * k);
    m.O |= (uint64_t)arr_gather16(fo[0], fo[1], fo[2], fo[3]) << (16 * k);
    m.C |= (uint64_t)arr_gather16(fc[0], fc[1], fc[2], fc[3]) << (16 * k);
  }
  if (lo > 0 || hi < 64) {
    const uint64_t valid = hi <= 0 ? 0ull : ((hi >= 64 ? ~0ull : (1ull << hi) - 1u) & (lo > 0 ? ~0ull << lo : ~0ull));
    m.Q &= valid; m.B &= valid; m.O &= valid; m.C &= valid;
  }
  return m;
}
/* W words with escape carry c: their unescaped quotes, and what they do to the state: carry out, parity, depth from outside / inside a string */
template <int W>
__device__ __forceinline__ void arr_eval(const ArrWord* m, uint32_t c, uint64_t* q, uint32_t* c_out, uint32_t* par_out, int32_t* d0, int32_t* d1) {
  uint32_t par = 0;
  int32_t a = 0, b = 0;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    q[k] = m[k].Q & ~escaped_mask(m[k].B, c, &c);
    const uint64_t in = prefix_xor(q[k]) ^ (par ? ~0ull : 0ull);
    a += (int32_t)popc64(m[k].O & ~in) - (int32_t)popc64(m[k].C & ~in);
    b += (int32_t)popc64(m[k].O & in) - (int32_t)popc64(m[k].C & in);
    par = (uint32_t)(in >> 63);
  }
  *c_out = c; *par_out = par; *d0 = a; *d1 = b;
}
__device__ __forceinline__ bool arr_blank(uint32_t x) { return x == ' ' || x == '\t' || x == '\r' || x == '\n'; }

/* Separators of one word that starts at depth d outside (in: inside strings) ...; bytes [lo, hi) are input. bad, opener: lowest byte that breaks
 * `ws [ ... ] ws`, lowest `[` at depth 0 (64: none). */
__device__ __forceinline__ uint64_t arr_mark(const uint8_t* p, const ArrWord& m, uint64_t quotes, uint64_t in, int32_t d, int32_t lo, int32_t hi, uint32_t* bad, uint32_t* opener) {
  const uint64_t valid = (hi >= 64 ? ~0ull : (1ull << hi) - 1u) & (lo > 0 ? ~0ull << lo : ~0ull);
  const uint64_t outside = ~in & ~quotes & valid, strange = (~in | quotes) & valid; /* not inside a string: quotes count there */
  uint64_t sep = 0, ev = (m.O | m.C) & outside;
  uint32_t seg = 0;
  for (;;) {
    const uint32_t b = ev ? ctz64a(ev) : 64u;
    /* bytes seg .. b - 1 lie at depth d */
    const uint64_t here = (b >= 64u ? ~0ull : (1ull << b) - 1u) & (seg >= 64u ? 0ull : ~0ull << seg);
    if (d == 1) { for (uint64_t t = here & outside; t; t &= t - 1u) if (p[ctz64a(t)] == ',') sep |= t & (0ull - t); }
    else if (d <= 0 && *bad == 64u) {
      for (uint64_t t = here & strange; t; t &= t - 1u) if (!arr_blank(p[ctz64a(t)])) { *bad = ctz64a(t); break; }
    }
    if (b >= 64u) break;
    const uint64_t bit = 1ull << b;
    ev &= ev - 1u;
    if (m.O & bit) {
      if (d == 0 && p[b] == '[') { sep |= bit; if (*opener == 64u) *opener = b; }
      else if (d <= 0 && *bad == 64u) *bad = b;
      ++d;
    } else {
      if (d == 1) { if (p[b] == ']') sep |= bit; }
      else if (d <= 0 && *bad == 64u) *bad = b;
      --d;
    }
    seg = b + 1u;
  }
  return sep;
}

/* The same for a word that starts at depth 2 or more, as far as it does not come below depth 1 (false: arr_mark() has to look): only the closers
 * that come down to depth 1 matter, and the bytes up to the opener behind them. (1 M Pets: 446 us event by event, 415 so.) */
__device__ __forceinline__ bool arr_mark_deep(const uint8_t* p, const ArrWord& m, uint64_t quotes, uint64_t in, int32_t d, int32_t hi, uint64_t* sep_out) {
  const uint64_t outside = ~in & ~quotes & (hi >= 64 ? ~0ull : (1ull << hi) - 1u);
  const uint64_t O = m.O & outside, C = m.C & outside;
  uint64_t sep = 0;
  for (uint64_t c = C; c; c &= c - 1u) {
    const uint64_t upto = c ^ (c - 1u); /* the closer and the bytes before it */
    if (d + (int32_t)popc64(O & upto) - (int32_t)popc64(C & upto) > 1) continue;
    const uint64_t next = (O | C) & ~upto, first = next & (0ull - next);
    if (first & C) return false; /* down to depth 0 */
    for (uint64_t t = outside & ~upto & (first - 1u); t; t &= t - 1u) if (p[ctz64a(t)] == ',') sep |= t & (0ull - t);
    if (!first) break; /* depth 1 up to the word's end (first - 1 above: all ones) */
  }
  *sep_out = sep;
  return true;
}

template <int W>
__global__ void __launch_bounds__(AI_THREADS, 4) k_arr_index(const __grid_constant__ ArrIndexArgs a) {
  __shared__ ArrFn sh_fn[AI_WARPS];
  __shared__ ArrState sh_in[AI_WARPS];
  __shared__ uint32_t sh_tile, sh_ok;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (tid == 0) sh_tile = atomicAdd(a.ticket, 1u);
  __syncthreads();
  const uint32_t tile = sh_tile;
  if (tile >= a.ntiles) return;
  const uint32_t mis = (uint32_t)(reinterpret_cast<uintptr_t>(a.in) & 15u);
  const uint8_t* base = a.in - mis;
  const uint64_t w0 = ((uint64_t)tile * AI_THREADS + tid) * W, end = a.len ? a.len + mis : 0; /* the thread's first word; bytes from base on */
  ArrWord m[W];
  uint64_t q[W];
#pragma unroll
  for (int k = 0; k < W; ++k) {
    const uint64_t v = (w0 + k) * 64u;
    const int64_t rest = (int64_t)end - (int64_t)v;
    m[k] = arr_load_word(base + v, v ? 0 : (int32_t)mis, rest >= 64 ? 64 : (rest < 0 ? 0 : (int32_t)rest));
  }
  ArrFn f;
  {
    uint32_t c, p;
    arr_eval<W>(m, 0u, q, &c, &p, &f.d[0], &f.d[2]);
    uint32_t c1 = c, p1 = p;
    f.d[1] = f.d[0]; f.d[3] = f.d[2];
    if ((m[0].Q | m[0].B) & 1u) { uint64_t unused[W]; arr_eval<W>(m, 1u, unused, &c1, &p1, &f.d[1], &f.d[3]); } /* (an escape makes a difference) */
    f.st = (c | (p << 1)) | ((c1 | (p1 << 1)) << 2) | ((c | ((p ^ 1u) << 1)) << 4) | ((c1 | ((p1 ^ 1u) << 1)) << 6);
  }
  const ArrFn inc = fn_warp_scan(f);
  if (lane == 31) sh_fn[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    ArrFn g = fn_identity();
    if (lane < AI_WARPS) g = sh_fn[lane];
    g = fn_warp_scan(g);
    const ArrFn all = fn_shfl(g, 31);
    if (lane == 0 && tile) {
      st_relaxed_u64(&a.fn0[tile], fn_pack(all.d[0], all.d[1]) | ((unsigned long long)all.st << 40));
      st_relaxed_u64(&a.fn1[tile], fn_pack(all.d[2], all.d[3]));
    }
    ArrState before;
    before.c = before.s = 0; before.d = 0;
    bool ok = true;
    if (tile) ok = arr_lookback(a, tile, lane, &before);
    const ArrState after = fn_apply(all, before);
    if (lane == 0) {
      if (ok) st_relaxed_u64(&a.inc[tile], state_pack(after));
      if (tile == a.ntiles - 1u) { a.res->arr_final_s = after.s; a.res->arr_final_d = after.d; }
      sh_ok = ok;
    }
    ArrFn prev = fn_shfl_up(g, 1);
    if (lane == 0) prev = fn_identity();
    if (lane < AI_WARPS) sh_in[lane] = fn_apply(prev, before);
  }
  ArrFn prev = fn_shfl_up(inc, 1);
  if (lane == 0) prev = fn_identity();
  __syncthreads();
  const bool ok = sh_ok != 0;
  ArrState st = fn_apply(prev, sh_in[warp]);
  if (st.c) { uint32_t c, p; int32_t x, y; arr_eval<W>(m, 1u, q, &c, &p, &x, &y); }
  uint64_t sep[W];
  uint32_t s = st.s;
  int32_t d = st.d;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    const uint64_t v = (w0 + k) * 64u;
    const uint64_t in = prefix_xor(q[k]) ^ (s ? ~0ull : 0ull);
    const uint32_t up = popc64(m[k].O & ~in & ~q[k]), down = popc64(m[k].C & ~in & ~q[k]);
    sep[k] = 0;
    if (v < end && d - (int32_t)down <= 1) { /* (deeper all through: no separator) */
      uint32_t bad = 64u, opener = 64u;
      const int32_t hi = end - v >= 64u ? 64 : (int32_t)(end - v);
      if (d < 2 || !arr_mark_deep(base + v, m[k], q[k], in, d, hi, &sep[k])) sep[k] = arr_mark(base + v, m[k], q[k], in, d, v ? 0 : (int32_t)mis, hi, &bad, &opener);
      if (ok && bad < 64u) atomicMin(&a.res->doc_err_off, (unsigned long long)(v + bad - mis));
      if (ok && opener < 64u) atomicMin(&a.res->first_opener, (unsigned long long)(v + opener - mis));
    }
    d += (int32_t)up - (int32_t)down;
    s = (uint32_t)(in >> 63);
  }
  const uint64_t nwords = (a.len + 63u) >> 6;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    const uint64_t w = w0 + k, x = ok ? sep[k] : 0ull;
    if (mis == 0) { if (w < nwords) a.sep[w] = x; }
    else if (x) { /* bit b of the word is input byte 64 w + b - mis */
      if (x >> mis) atomicOr((unsigned long long*)&a.sep[w], (unsigned long long)(x >> mis));
      if (w && (x << (64u - mis))) atomicOr((unsigned long long*)&a.sep[w - 1u], (unsigned long long)(x << (64u - mis)));
    }
  }
}

}  // namespace pj
#endif

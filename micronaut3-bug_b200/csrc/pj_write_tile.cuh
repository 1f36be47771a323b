/*
 * pj_write_tile.cuh — k_write_tile<SCHEMA>: columns -> JSON text (rules W1-W5) in one pass over HBM.
 *
 * One thread block = one tile of consecutive records. The steps:
 *
 *  1. The rows of a tile are consecutive in every model's table, so what it reads is ONE piece of every column and arena: bulk copies
 *     (cp.async.bulk) bring them to shared memory, and nothing is read from global memory after that. All threads look the strings over
 *     for bytes that have to be escaped, 16 bytes at a time; the few blocks that hold one are looked at again, a byte per lane, and their
 *     escapes counted for the strings they lie in. Where more than WT_HITS blocks hold one, all strings are looked over instead, one per
 *     lane (200 k Pets with two quotes a name, kernel, us: every block by a warp 138, strings by lanes 84, and the short ones written by the lanes that
 *     meet them 74; 100 k Users with four paths 107 / 66 / 48).
 *  2. Sizes: first the elements of the lists, an element per lane, with running sums; then the records, a record per lane, 32 of one
 *     model at a time.
 *  3. One decoupled look-back over the earlier tiles gives the tile's place in the output.
 *  4. Text: the first half of a record's properties, the second half, the strings of its list and the objects of its list are units
 *     of their own, each a lane's, so that the lanes of a warp do the same and long lists are spread over lanes. A lane puts its text
 *     together in a register and stores whole words into a window in shared memory; words that two units share are or-ed.
 *     Strings with a byte to escape (but short ones where most are) and strings of 512 bytes and more are left out and written afterwards, a warp per string or per 2 KB of it (by the
 *     lane that meets them, 300 MB of Users: strings of 300 bytes 780 us with it, 940 without; of 1000 bytes 666 and 440).
 *  5. The window leaves with one bulk copy. Text longer than the window goes in several rounds of 4 and 5.
 *
 * Tables whose rows a tile does not find in order (a record map of the caller's own making, offsets of written strings that fall, or of any
 * where there is a byte to escape), or whose strings do not fit shared memory, take the general road: a record per thread (pj_write_fast.cuh), its
 * long strings and lists by whole warps. So does a record whose text outgrows the window.
 *
 * What bounds it: instruction issue and waiting for one another. 300 k Pets: 180 instructions of a warp per record, a third of the issue slots
 * used; the warps of a block wait for the first one's offsets and look-back, and two or three blocks per SM (shared memory) cover half of that.
 * Integers and strings are written by functions that are called, not expanded: the instruction cache does not hold the text of three
 * models otherwise (400 k mixed records 449 -> 336 us, Pets the same).
 *
 * Measured (kernel, against a record per thread with byte stores and a pass over the arenas before it; us): 600 k Pets 268 -> 221, Users
 * 205 -> 135, Orders 123 -> 87, Pets with escapes 735 -> 340, mixed records with escapes 925 -> 367, 100 k Pets with long lists 1 670 -> 450.
 */
#ifndef PJ_WRITE_TILE_CUH
#define PJ_WRITE_TILE_CUH

#include "pj_dev.cuh"
#include "pj_result.h"
#include "pj_write_core.cuh"
#include "pj_write_fast.cuh"

namespace pj {

#ifndef PJ_CX
#if defined(__CUDACC__)
#define PJ_CX constexpr __host__ __device__
#else
#define PJ_CX constexpr
#endif
#endif
static constexpr uint32_t WT_MAX_RECS = 256; /* records per tile */
/* Threads of a block, and blocks per SM. 600 k records, us of the kernel: mixed 256 threads / three blocks 520, 512 / two 373 (three models' records
 * fill twice as many groups of 32); Pets, of which 256 share a block that writes them in two windows, 240 and 224; Users 133 and 152, Orders 86
 * and 117: their tiles are short, and more blocks wait in turn. */
template <int SCHEMA> struct WtT {
  static constexpr uint32_t threads = SCHEMA == PJ_SCHEMA_PET || SCHEMA == PJ_SCHEMA_MIXED ? 512u : 256u, blocks = threads == 512u ? 2u : 3u;
  static constexpr uint32_t warps = threads / 32u;
};
static_assert(WT_MAX_RECS <= 256, "a record per thread");
static constexpr uint32_t WT_SHORT_THREADS = 256, WT_SHORT_BLOCKS = 4; /* tables of short Pets, see wt_short() */
inline uint32_t wt_threads(uint32_t schema) { return schema == PJ_SCHEMA_PET ? WtT<1>::threads : (schema == PJ_SCHEMA_ORDER ? WtT<2>::threads : (schema == PJ_SCHEMA_USER ? WtT<3>::threads : WtT<4>::threads)); }
static constexpr uint32_t WT_MOST_WARPS = 16;
static constexpr uint32_t WT_MAX_SMEM = 128 * 1024;
static constexpr uint32_t WT_MIN_WINDOW = 2048;
static constexpr uint32_t WT_ESC = 160;             /* strings with escapes, and long ones, a round keeps for later */
static constexpr uint32_t WT_LONG = 512;            /* bytes of a string that a warp copies */
static constexpr uint32_t WT_LONG_LIST = 8;         /* elements of a list that a warp writes on the general road */
static constexpr uint32_t WT_SHORT = 48;            /* bytes up to which a lane escapes a string where the tile has many of them */
static constexpr uint32_t WT_PART = 2048;           /* bytes of a long string a warp takes at a time */
static constexpr uint32_t WT_HITS = 192;            /* 16-byte blocks with a byte to escape that are kept in a list */
static constexpr uint32_t WT_BACK = 4;              /* tiles a lane looks back at per round */
static constexpr uint32_t WT_COLS = 48;             /* columns of a schema */
static constexpr uint32_t WT_NONE = 0xFFFFFFFFu;

struct WriteArgs {
  uint64_t n;             /* records (mixed) or rows */
  uint32_t schema, array; /* array: wrap as [r,r,...] */
  int inclusion;
  uint32_t hexa;          /* 'A' or 'a': hex letters of \u00xx escapes */
  uint8_t* out;
  uint64_t cap;
  DevResult* res;
  DevCols cols;
};
/* One column (or arena) of the schema, as the tiles stage it. */
struct WtCol {
  const uint8_t* p;
  const uint32_t* off;  /* arenas: the offsets of its strings, else null */
  uint8_t col, shift;   /* number; log2 of an element's bytes */
  uint8_t model, level; /* 0: an element per row, 1: per element of the list of strings, 2: ... of objects */
  uint8_t plus, pad[3]; /* offsets: one element more than rows */
};
struct WTileArgs {
  WriteArgs w;
  WtCol col[WT_COLS]; /* those with an element per row first */
  uint32_t ncol, nrow; /* how many; how many of them have an element per row */
  const uint32_t* list[2]; /* offsets of the list of strings, of the list of objects */
  unsigned long long* agg; /* [ntiles] text bytes of the tile | TS_VALID */
  unsigned long long* inc; /* [ntiles] text bytes of all tiles up to and including it | TS_VALID */
  uint32_t* ticket;
  uint32_t ntiles;
  uint32_t recs;  /* records per tile */
  uint32_t smem;  /* bytes of dynamic shared memory */
  unsigned long long spin_limit_ns;
};

/* Exclusive prefix of `tile` over all earlier tiles. Warp 0 only, all lanes; false when the bounded wait ran out. */
__device__ __forceinline__ bool lookback_u64(const unsigned long long* agg, const unsigned long long* inc, uint32_t* timeout_flag, unsigned long long limit_ns,
                                             uint32_t tile, uint32_t lane, unsigned long long* excl_out) {
  unsigned long long excl = 0;
  int64_t j = (int64_t)tile - 1;
  const unsigned long long t0 = global_ns();
  while (j >= 0) {
    unsigned long long part = 0;
    bool found = false;
    for (;;) { /* WT_BACK times 32 tiles: the nearest with an inclusive total, and the totals of those in between */
      unsigned long long wa[WT_BACK], wi[WT_BACK];
#pragma unroll
      for (uint32_t k = 0; k < WT_BACK; ++k) {
        const int64_t mine = j - (int64_t)(lane + 32u * k);
        wa[k] = TS_VALID; wi[k] = TS_VALID; /* tiles before the first: inclusive total 0 */
        if (mine >= 0) { wi[k] = ld_relaxed_u64(&inc[mine]); wa[k] = ld_relaxed_u64(&agg[mine]); }
      }
      bool ready = true;
      part = 0; found = false;
#pragma unroll
      for (uint32_t k = 0; k < WT_BACK; ++k) {
        const bool has_inc = wi[k] & TS_VALID, has_agg = wa[k] & TS_VALID;
        const uint32_t inc_mask = __ballot_sync(0xFFFFFFFFu, has_inc);
        const uint32_t ready_mask = __ballot_sync(0xFFFFFFFFu, has_inc || has_agg);
        if (found || !ready) continue;
        const uint32_t first_inc = inc_mask ? (uint32_t)(__ffs((int)inc_mask) - 1) : 32u;
        const uint32_t need = first_inc >= 31 ? 0xFFFFFFFFu : ((2u << first_inc) - 1u);
        if ((ready_mask & need) != need) { ready = false; continue; }
        part += lane < first_inc ? (wa[k] & ~TS_VALID) : (lane == first_inc ? (wi[k] & ~TS_VALID) : 0ull);
        found = first_inc < 32;
      }
      if (ready) break;
      uint32_t give_up = 0;
      if (lane == 0) give_up = (global_ns() - t0 > limit_ns) || *(volatile uint32_t*)timeout_flag;
      give_up = __shfl_sync(0xFFFFFFFFu, give_up, 0);
      if (give_up) { if (lane == 0) atomicExch(timeout_flag, 1u); return false; }
      __nanosleep(40);
    }
#pragma unroll
    for (int d = 16; d; d >>= 1) part += __shfl_xor_sync(0xFFFFFFFFu, part, d);
    excl += part;
    if (found) break;
    j -= 32 * WT_BACK;
  }
  *excl_out = excl;
  return true;
}

/* ---- the schema's lists ------------------------------------------------------------------------------------------------ */
/* the property of OBJ that is a list of `kind`, or -1 */
template <int OBJ>
PJ_CX int wt_list_field(uint32_t kind) {
  for (int i = 0; i < CObj<OBJ>::N; ++i) if (CObj<OBJ>::f[i].kind == kind) return i;
  return -1;
}
static constexpr int WT_LIST_STR = wt_list_field<OBJ_PET>(K_LIST_STR), WT_LIST_OBJ = wt_list_field<OBJ_PET>(K_LIST_OBJ);
static_assert(wt_list_field<OBJ_ORDER>(K_LIST_STR) < 0 && wt_list_field<OBJ_ORDER>(K_LIST_OBJ) < 0 && wt_list_field<OBJ_USER>(K_LIST_STR) < 0 &&
              wt_list_field<OBJ_USER>(K_LIST_OBJ) < 0, "only one model has lists");
/* first property of a root's second half */
template <int OBJ> struct WtMid { static constexpr int v = CObj<OBJ>::N / 2; };
static_assert(WT_LIST_STR >= WtMid<OBJ_PET>::v && WT_LIST_OBJ >= WtMid<OBJ_PET>::v, "the lists' places come from one unit");

struct WtEsc { uint32_t at, n, dst; }; /* n: bytes | to be escaped << 31 */
/* General road: a long string or list of a record, measured and written by whole warps. */
struct WtLater {
  uint8_t* dst;    /* where its text goes */
  unsigned long long size; /* bytes of it */
  uint32_t a, b;   /* bytes of the arena, or elements */
  uint16_t rec, link; /* the record of the tile; the record's next one */
  uint8_t kind, col;  /* of the data */
};
static constexpr uint32_t WT_LATERS = 192; /* a tile's */
static constexpr uint16_t WT_LAST = 0xFFFF;
struct WtShared {
  unsigned long long mbar[3], base;                /* copies of: columns with an element per row; those of list elements; arenas */
  unsigned long long row0[3];                      /* per model: the tile's first row */
  uint32_t cnt[3], pre[3];                         /* ... how many, and how many of the models before */
  uint32_t at[PJ_MAX_COLS];                        /* per column: element 0 of it would lie there (modulo 2^32) */
  uint32_t lo[PJ_MAX_COLS], span[PJ_MAX_COLS];     /* arenas: the first staged byte's number, and how many */
  uint32_t str0[PJ_MAX_COLS];                      /* arenas: number of the first string of the tile's */
  uint32_t item0[2], itemn[2];                     /* per list: the tile's first element, and how many */
  uint32_t text, stage, sums, extra, win;          /* where the arenas begin and end; elements' sums, strings' escapes, window */
  uint32_t nstr, flight;                           /* strings; which of the copies are under way */
  uint32_t nhit;                                   /* 16-byte blocks with a byte to escape */
  uint16_t hit[WT_HITS];
  uint32_t odd, ok, tile, nesc;                    /* odd: the tile takes the general road */
  uint32_t longs, nlater;                          /* some string of the tile is long; how many WtLater */
  uint16_t ar0[32], ar1[32];                       /* arenas: their first 16-byte block, and one more than the last */
  uint8_t arcol[32], arlevel[32], armodel[32];
  union { uint32_t wsum[WT_MOST_WARPS]; unsigned long long wsum8[WT_MOST_WARPS]; };
  uint32_t cls[3][WT_MOST_WARPS];
  uint32_t pos[WT_MAX_RECS + 1];                   /* a record's bytes, then where it starts in the tile's text */
  uint32_t mid[WT_MAX_RECS];                       /* where its second half starts | no property before it << 31 */
  union {
    uint32_t list[2][WT_MAX_RECS];                 /* where its lists' elements start, from its first byte; WT_NONE: none are written */
    unsigned long long bytes[WT_MAX_RECS];         /* general road: a record's bytes, then where it starts */
  };
  uint8_t perm[WT_MAX_RECS];                       /* mixed: the tile's records by model */
  WtEsc esc[WT_ESC];
};

/* element `row` of column COL, staged */
template <class T>
__device__ __forceinline__ const T* wt_at(const WtShared& sh, const uint8_t* w8, uint32_t col, uint32_t row) { return reinterpret_cast<const T*>(w8 + (uint32_t)(sh.at[col] + row * (uint32_t)sizeof(T))); }
/* bytes the escapes of a string add: string x of the tile */
__device__ __forceinline__ uint32_t* wt_extras(const WtShared& sh, uint8_t* w8) { return reinterpret_cast<uint32_t*>(w8 + sh.extra); }
__device__ __forceinline__ uint32_t wt_extra(const WtShared& sh, const uint8_t* w8, uint32_t data_col, uint32_t index) {
  return reinterpret_cast<const uint32_t*>(w8 + sh.extra)[sh.str0[data_col] + index];
}

/* ---- sizes ----------------------------------------------------------------------------------------------------------- */
/* Pets whose tiles leave four blocks room on an SM, and more tiles than two blocks of it take at once: a short tile is three trips of its staging and a
 * look-back, and four of them wait in turn. 1 M Pets, 512 threads / 256, us of the kernel: {} 143 / 95, an id and a name of two bytes 167 / 113, 64 bytes of
 * text 197 / 146; 200 k 42 / 30, 46 / 34, 50 / 42. 60 k are one wave either way (22 / 23; with a name of 64 bytes and escapes 40 k 33 / 41). */
inline bool wt_short(uint32_t smem, uint64_t ntiles, uint32_t sms) {
  return smem <= 228u * 1024u / WT_SHORT_BLOCKS - 1024u - (uint32_t)sizeof(WtShared) && ntiles > 2u * (uint64_t)sms;
}
struct WtRead { /* what the units of a tile read */
  int incl;
  bool dirty; /* some string of the tile has to be escaped */
  bool many;  /* most of them: short ones are the lanes' that meet them */
  bool later; /* ... or is long: not all are written where they are met */
  uint32_t hexa;
};
/* length of string [x, y) of arena COL, quotes and escapes included; index: its number among the tile's strings of the arena. Sets bad when it
 * does not lie in what is staged. */
__device__ __forceinline__ uint32_t wt_str_size(const WtRead& r, WtShared& sh, const uint8_t* w8, uint32_t col, uint32_t index, uint32_t x, uint32_t y, bool& bad) {
  const uint32_t lo = sh.lo[col];
  const uint32_t u = x - lo, v = y - lo;
  if (u > v || v > sh.span[col]) { bad = true; return 2; }
  uint32_t n = y - x + 2u;
  if (n >= WT_LONG + 2u) sh.longs = 1u;
  if (r.dirty) n += wt_extra(sh, w8, col, index);
  return n;
}
/* the row-indexed values of properties [LO, HI), loaded together so that their latencies overlap */
template <int OBJ, int LO, int HI>
__device__ __forceinline__ void wt_snap(const WtShared& sh, const uint8_t* w8, uint32_t row, RowSnap& r) {
  if constexpr (LO < HI) {
    constexpr uint32_t kind = FK<OBJ, LO>::kind, col = FK<OBJ, LO>::col;
    if constexpr (kind == K_I64) r.v[LO] = *wt_at<int64_t>(sh, w8, col, row);
    else if constexpr (kind == K_I32) r.v[LO] = *wt_at<int32_t>(sh, w8, col, row);
    else if constexpr (kind == K_BOOL || kind == K_ENUM) r.v[LO] = *wt_at<uint8_t>(sh, w8, col, row);
    else if constexpr (kind == K_DATETIME) {
      r.v[LO] = *wt_at<int64_t>(sh, w8, col, row);
      r.a[LO] = (uint32_t)*wt_at<int32_t>(sh, w8, col + 1, row); r.b[LO] = (uint32_t)*wt_at<int32_t>(sh, w8, col + 2, row);
    } else if constexpr (kind == K_STR || kind == K_LIST_STR || kind == K_LIST_OBJ) {
      r.a[LO] = *wt_at<uint32_t>(sh, w8, col, row); r.b[LO] = *wt_at<uint32_t>(sh, w8, col, row + 1u);
    }
    wt_snap<OBJ, LO + 1, HI>(sh, w8, row, r);
  }
}
template <int OBJ, int LO, int HI>
PJ_CX int wt_child() { /* the flat object among properties [LO, HI), or -1 */
  for (int i = LO; i < HI; ++i) if (CObj<OBJ>::f[i].kind == K_OBJ) return CObj<OBJ>::f[i].child;
  return -1;
}
/* ... with the presence bits, and the flat object's */
template <int OBJ, int LO, int HI>
__device__ __forceinline__ void wt_load(const WtShared& sh, const uint8_t* w8, uint32_t row, RowSnap& r, RowSnap& rc) {
  r.present = *wt_at<uint8_t>(sh, w8, CObj<OBJ>::present_col, row);
  wt_snap<OBJ, LO, HI>(sh, w8, row, r);
  constexpr int E = wt_child<OBJ, LO, HI>();
  if constexpr (E >= 0) { rc.present = *wt_at<uint8_t>(sh, w8, CObj<E>::present_col, row); wt_snap<E, 0, CObj<E>::N>(sh, w8, row, rc); }
}
/* does a string of properties [I, N), present or not, end before it begins? wt_count_block() finds a byte's string by offsets that never fall. */
template <int OBJ, int I = 0>
__device__ __forceinline__ bool wt_falls(const RowSnap& r, const RowSnap& rc) {
  if constexpr (I >= CObj<OBJ>::N) return false;
  else {
    bool f = false;
    if constexpr (FK<OBJ, I>::kind == K_STR) f = r.a[I] > r.b[I];
    else if constexpr (FK<OBJ, I>::kind == K_OBJ) f = wt_falls<FK<OBJ, I>::child>(rc, rc);
    return f || wt_falls<OBJ, I + 1>(r, rc);
  }
}
PJ_HD uint32_t wt_frac_digits(uint32_t u) { /* of 1..999999999, without the zeros at the end */
  uint32_t nd = 9;
  while (u % 10u == 0) { u /= 10u; nd--; }
  return nd;
}
struct WtList { uint32_t a, b, bytes; }; /* elements [a, b) of a list, and their text with a comma or bracket behind each */
/* bytes of properties [I, HI) of an object: a separator and the name before every value. bad: not for this road. */
template <int SCHEMA, int OBJ, int I, int HI>
__device__ __forceinline__ uint32_t wt_size(const WtRead& x, WtShared& sh, const uint8_t* w8, uint32_t index, const RowSnap& r, const RowSnap& rc, const WtList* lists, uint32_t* list_at, uint32_t at, bool& first, bool& bad) {
  if constexpr (I >= HI) return 0;
  else {
    constexpr uint32_t kind = FK<OBJ, I>::kind, col = FK<OBJ, I>::col;
    const bool pr = (r.present >> I) & 1;
    bool empty = false;
    if constexpr (kind == K_STR || kind == K_LIST_STR || kind == K_LIST_OBJ) empty = r.a[I] == r.b[I];
    uint32_t n = 0;
    if (included(x.incl, pr, empty)) {
      first = false;
      n = 1u + FK<OBJ, I>::pat_len;
      if (!pr) n += 4;
      else if constexpr (kind == K_I64 || kind == K_I32) n += (r.v[I] < 0) + ndigits_u64(r.v[I] < 0 ? 0 - (uint64_t)r.v[I] : (uint64_t)r.v[I]);
      else if constexpr (kind == K_BOOL) n += r.v[I] ? 4 : 5;
      else if constexpr (kind == K_ENUM) {
        constexpr int E = FK<OBJ, I>::child;
        static_assert(CEnum<E>::N == 3, "three literals");
        const uint32_t e = (uint32_t)r.v[I] % 3u;
        n += 2u + (e == 0 ? EK<E, 0>::len : (e == 1 ? EK<E, 1>::len : EK<E, 2>::len));
      } else if constexpr (kind == K_DATETIME) {
        if (r.a[I] > 999999999u) bad = true;
        else n += 21u + (r.a[I] ? 1u + wt_frac_digits(r.a[I]) : 0u) + (r.b[I] ? 6u : 1u);
      } else if constexpr (kind == K_STR) n += wt_str_size(x, sh, w8, col + 1, index, r.a[I], r.b[I], bad);
      else if constexpr (kind == K_OBJ) {
        constexpr int E = FK<OBJ, I>::child;
        bool f = true;
        n += wt_size<SCHEMA, E, 0, CObj<E>::N>(x, sh, w8, index, rc, rc, nullptr, nullptr, 0, f, bad) + 1u + f;
      } else if constexpr (kind == K_LIST_STR || kind == K_LIST_OBJ) {
        if (!empty) list_at[kind == K_LIST_OBJ] = at + n + 1u;
        n += empty ? 2u : 1u + lists[kind == K_LIST_OBJ].bytes;
      }
    }
    return n + wt_size<SCHEMA, OBJ, I + 1, HI>(x, sh, w8, index, r, rc, lists, list_at, at + n, first, bad);
  }
}

/* ---- text ------------------------------------------------------------------------------------------------------------- */
/* A lane's text on its way into the window: the bytes that do not fill a word yet are in acc. Window words are zero to begin with. */
struct WtOut {
  uint8_t* w8;
  uint32_t at, acc, fill; /* byte offset of the word; its bytes so far; how many bits */
};
__device__ __forceinline__ void wt_or(uint8_t* w8, uint32_t at, uint32_t v) {
#if defined(__CUDA_ARCH__)
  asm volatile("red.shared.or.b32 [%0], %1;" ::"r"(smem_addr(w8) + at), "r"(v) : "memory");
#else
  atomicOr(reinterpret_cast<uint32_t*>(w8 + at), v);
#endif
}
/* a word of shared memory */
__device__ __forceinline__ uint32_t wt_ld(const uint8_t* w8, uint32_t at) {
#if defined(__CUDA_ARCH__)
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(smem_addr(w8) + at) : "memory");
  return v;
#else
  return *reinterpret_cast<const uint32_t*>(w8 + at);
#endif
}
__device__ __forceinline__ void wt_st(uint8_t* w8, uint32_t at, uint32_t v) {
#if defined(__CUDA_ARCH__)
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(smem_addr(w8) + at), "r"(v) : "memory");
#else
  *reinterpret_cast<uint32_t*>(w8 + at) = v;
#endif
}
__device__ __forceinline__ void wt_begin(WtOut& e, uint32_t pos) { e.at = pos & ~3u; e.fill = (pos & 3u) * 8u; e.acc = 0; }
__device__ __forceinline__ uint32_t wt_pos(const WtOut& e) { return e.at + (e.fill >> 3); }
__device__ __forceinline__ void wt_end(const WtOut& e) { if (e.fill) wt_or(e.w8, e.at, e.acc); }
/* the low `bits` (0 .. 32, whole bytes) of v; the rest of v is zero */
__device__ __forceinline__ void wt_put(WtOut& e, uint32_t v, uint32_t bits) {
  const uint32_t nf = e.fill + bits, a = e.acc | (v << e.fill);
  const bool full = nf >= 32u;
#if defined(__CUDA_ARCH__)
  /* (no branch: the lanes of a warp seldom agree) */
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.u32 p, %0, 32;\n\t@p red.shared.or.b32 [%1], %2;\n\t}" ::"r"(nf), "r"(smem_addr(e.w8) + e.at), "r"(a) : "memory");
#else
  if (full) wt_or(e.w8, e.at, a);
#endif
  e.acc = full ? __funnelshift_l(v, 0u, e.fill) : a;
  e.at += full ? 4u : 0u;
  e.fill = nf & 31u;
}
__device__ __forceinline__ void wt_put4(WtOut& e, uint32_t v) {
  wt_or(e.w8, e.at, e.acc | (v << e.fill));
  e.acc = __funnelshift_l(v, 0u, e.fill);
  e.at += 4u;
}
/* separator c, then property I's name, its colon and, for values that are strings, the opening quote */
template <int OBJ, int I, int QUOTE>
struct WtKey {
  static constexpr uint32_t len = 1u + FK<OBJ, I>::pat_len + QUOTE;
  static PJ_CX uint32_t word(uint32_t k) {
    uint32_t v = 0;
    for (uint32_t b = 0; b < 4; ++b) {
      const uint32_t i = 4 * k + b;
      uint32_t c = 0;
      if (i >= 1 && i - 1 < FK<OBJ, I>::pat_len) c = (uint32_t)(((i - 1) < 8 ? FK<OBJ, I>::pat0 >> (8 * (i - 1)) : FK<OBJ, I>::pat1 >> (8 * (i - 9))) & 0xFF);
      else if (i + 1 == len && QUOTE) c = '"';
      v |= c << (8 * b);
    }
    return v;
  }
};
template <int OBJ, int I, int QUOTE, int K = 0>
__device__ __forceinline__ void wt_put_key(WtOut& e, uint32_t c) {
  using P = WtKey<OBJ, I, QUOTE>;
  if constexpr (4 * K < P::len) {
    constexpr uint32_t w = P::word(K);
    const uint32_t v = K == 0 ? w | c : w;
    if constexpr (4 * K + 4 <= P::len) wt_put4(e, v); else wt_put(e, v, 8u * (P::len - 4 * K));
    wt_put_key<OBJ, I, QUOTE, K + 1>(e, c);
  }
}
/* four decimal digits of v < 10000 as bytes 0..9, the first one lowest */
__device__ __forceinline__ uint32_t wt_digits4(uint32_t v) {
  const uint32_t hi = v / 100u, t = hi | ((v - hi * 100u) << 16);
  const uint32_t tens = ((t * 103u) >> 10) & 0x000F000Fu; /* x / 10 for x < 100 in both halves: 99 * 103 stays below 2^16 */
  return tens | ((t - tens * 10u) << 8);
}
static __device__ __noinline__ WtOut wt_put_i64(WtOut e, int64_t v) {
  if (v < 0) wt_put(e, '-', 8);
  const uint64_t u = v < 0 ? 0 - (uint64_t)v : (uint64_t)v;
  uint32_t lead = (uint32_t)u, mid = 0, low = 0, groups = 0; /* full groups of 8 digits behind the leading one */
  if (u >= 100000000ull) {
    const uint64_t q = u / 100000000ull; /* < 1.85e11 */
    low = (uint32_t)(u - q * 100000000ull);
    if (q >= 100000000ull) { lead = (uint32_t)(q >> 8) / 390625u; mid = (uint32_t)q - lead * 100000000u; groups = 2; }
    else { lead = (uint32_t)q; groups = 1; }
  }
  {
    const uint32_t h = lead / 10000u, w0 = wt_digits4(h), w1 = wt_digits4(lead - h * 10000u);
    /* zeros before the first digit go; of 0 itself one stays */
    const uint32_t z = w0 ? ((uint32_t)__ffs((int)w0) - 1u) >> 3 : 4u + (((uint32_t)__ffs((int)(w1 | 0x01000000u)) - 1u) >> 3);
    const uint32_t a0 = w0 | 0x30303030u, a1 = w1 | 0x30303030u;
    if (z < 4u) wt_put4(e, __funnelshift_r(a0, a1, 8u * z));
    wt_put(e, a1 >> (8u * (z & 3u)), 32u - 8u * (z & 3u));
  }
  if (groups >= 2u) { const uint32_t h = mid / 10000u; wt_put4(e, wt_digits4(h) | 0x30303030u); wt_put4(e, wt_digits4(mid - h * 10000u) | 0x30303030u); }
  if (groups) { const uint32_t h = low / 10000u; wt_put4(e, wt_digits4(h) | 0x30303030u); wt_put4(e, wt_digits4(low - h * 10000u) | 0x30303030u); }
  return e;
}

/* two digits of v < 100 (of any v: the two bytes the general writer gives) */
__device__ __forceinline__ uint32_t wt_2d(uint32_t v) { const uint32_t q = v / 10u; return ((q + '0') & 0xFFu) | (((v - q * 10u + '0') & 0xFFu) << 8); }
/* W5; nanos below 10^9 */
__device__ __forceinline__ void wt_put_datetime(WtOut& e, int64_t epoch, uint32_t nanos, int32_t off) {
  const int64_t local = epoch + off;
  const int64_t days = (local >= 0 ? local : local - 86399) / 86400;
  const uint32_t sod = (uint32_t)(local - days * 86400);
  uint32_t y, m, d;
  if (days >= -719468 && days < 400000000) { /* from the year 0 on, in 32 bits: the same steps as civil_from_days() */
    const uint32_t z = (uint32_t)((int32_t)days + 719468), era = z / 146097u, doe = z - era * 146097u;
    const uint32_t yoe = (doe - doe / 1460u + doe / 36524u - doe / 146096u) / 365u, doy = doe - (365u * yoe + yoe / 4u - yoe / 100u);
    const uint32_t mp = (5u * doy + 2u) / 153u;
    d = doy - (153u * mp + 2u) / 5u + 1u;
    m = mp < 10u ? mp + 3u : mp - 9u;
    y = yoe + era * 400u + (m <= 2u);
    const uint32_t c = y / 100u;
    y = wt_2d(c) | (wt_2d(y - c * 100u) << 16);
  } else {
    int64_t yy;
    civil_from_days(days, &yy, &m, &d);
    y = wt_2d((uint32_t)(yy / 100)) | (wt_2d((uint32_t)(yy % 100)) << 16);
  }
  const uint32_t hh = sod / 3600u, mm = (sod - hh * 3600u) / 60u, ss = sod % 60u;
  wt_put4(e, '"' | (y << 8));
  wt_put4(e, (y >> 24) | ('-' << 8) | (wt_2d(m) << 16));
  wt_put4(e, '-' | (wt_2d(d) << 8) | ('T' << 24));
  wt_put4(e, wt_2d(hh) | (':' << 16) | ((wt_2d(mm) & 0xFFu) << 24));
  wt_put4(e, (wt_2d(mm) >> 8) | (':' << 8) | (wt_2d(ss) << 16));
  if (nanos) {
    uint32_t u = nanos, nd = 9;
    while (u % 10u == 0) { u /= 10u; nd--; }
    u = nanos; /* all nine digits, of which the first nd are written */
    const uint32_t top = u / 100000000u, r8 = u - top * 100000000u, h = r8 / 10000u;
    wt_put(e, '.' | ((top + '0') << 8), 16);
    const uint32_t a0 = wt_digits4(h) | 0x30303030u, a1 = wt_digits4(r8 - h * 10000u) | 0x30303030u;
    const uint32_t n0 = nd - 1u < 4u ? nd - 1u : 4u, n1 = nd > 5u ? nd - 5u : 0u;
    wt_put(e, n0 == 4u ? a0 : a0 & ((1u << (8u * n0)) - 1u), 8u * n0);
    wt_put(e, n1 == 4u ? a1 : a1 & ((1u << (8u * n1)) - 1u), 8u * n1);
  }
  if (off == 0) wt_put(e, 'Z' | ('"' << 8), 16);
  else {
    const uint32_t a = (uint32_t)(off < 0 ? -off : off), h = wt_2d(a / 3600u), q = wt_2d(a % 3600u / 60u);
    wt_put4(e, (off < 0 ? '-' : '+') | (h << 8) | (':' << 24));
    wt_put(e, q | ('"' << 16), 24);
  }
}
template <int E>
__device__ __forceinline__ void wt_put_enum(WtOut& e, uint32_t k) { /* behind its opening quote; with the closing one */
  static_assert(CEnum<E>::N == 3 && EK<E, 0>::len >= 4 && EK<E, 1>::len >= 4 && EK<E, 2>::len >= 4 && EK<E, 0>::len <= 11 && EK<E, 1>::len <= 11 && EK<E, 2>::len <= 11, "three words");
  const uint64_t lo = k == 0 ? EK<E, 0>::lo : (k == 1 ? EK<E, 1>::lo : EK<E, 2>::lo);
  uint64_t hi = k == 0 ? EK<E, 0>::hi : (k == 1 ? EK<E, 1>::hi : EK<E, 2>::hi);
  const uint32_t len = k == 0 ? EK<E, 0>::len : (k == 1 ? EK<E, 1>::len : EK<E, 2>::len);
  uint32_t w1 = (uint32_t)(lo >> 32), w2 = (uint32_t)hi;
  const uint32_t n = len + 1u; /* and the quote */
  if (len < 8u) w1 |= (uint32_t)'"' << (8u * (len - 4u)); else w2 |= (uint32_t)'"' << (8u * (len - 8u));
  wt_put4(e, (uint32_t)lo);
  wt_put(e, w1, n >= 8u ? 32u : 8u * (n - 4u));
  wt_put(e, w2, n > 8u ? 8u * (n - 8u) : 0u);
}
__device__ __forceinline__ uint32_t wt_peek4(const uint8_t* w8, uint32_t s) {
  return __funnelshift_r(wt_ld(w8, s & ~3u), wt_ld(w8, (s & ~3u) + 4u), (s & 3u) * 8u);
}
__device__ __forceinline__ uint32_t wt_low(uint32_t v, uint32_t n) { return n >= 4u ? v : v & ((1u << (8u * n)) - 1u); }
/* byte c as W3 writes it: bytes from the lowest on, and how many */
__device__ __forceinline__ uint64_t wt_escaped(uint32_t c, uint32_t hexa, uint32_t* len) {
  const uint32_t extra = escape_extra_byte(c);
  *len = 1u + extra;
  if (extra == 0u) return c;
  if (extra == 1u) return '\\' | ((c == 8 ? 'b' : (c == 9 ? 't' : (c == 10 ? 'n' : (c == 12 ? 'f' : (c == 13 ? 'r' : c))))) << 8);
  return 0x3030755Cull | (uint64_t)(('0' + (c >> 4)) | (((c & 15) < 10 ? '0' + (c & 15) : hexa + (c & 15) - 10) << 8)) << 32;
}
/* bytes that the escapes of the `have` lowest bytes of x add */
__device__ __forceinline__ uint32_t wt_word_extra(uint32_t x, uint32_t have) {
  if (have < 4u) x |= 0x61616161u << (8u * have); /* (letters) */
  return word_needs_escape(x) ? word_escape_extra(x) : 0u;
}
/* n bytes at byte s, escaped */
static __device__ __noinline__ WtOut wt_put_escaped(WtOut e, uint32_t s, uint32_t n, uint32_t hexa) {
  for (uint32_t i = 0, left = 0; i < n; ++i) {
    if (left == 0) { /* four bytes that stay as they are, or these four one by one */
      const uint32_t have = n - i < 4u ? n - i : 4u, x = wt_low(wt_peek4(e.w8, s + i), have);
      if (!wt_word_extra(x, have)) {
        if (have == 4u) wt_put4(e, x); else wt_put(e, x, 8u * have);
        i += have - 1u;
        continue;
      }
      left = have;
    }
    --left;
    uint32_t len;
    const uint64_t v = wt_escaped(e.w8[s + i], hexa, &len);
    if (len <= 2u) { wt_put(e, (uint32_t)v, 8u * len); continue; }
    wt_put4(e, (uint32_t)v);
    wt_put(e, (uint32_t)(v >> 32), 16);
  }
  return e;
}
/* the len (1 .. 6) bytes of v to byte p of the window */
__device__ __forceinline__ void wt_or_bytes(uint8_t* w8, uint32_t p, uint64_t v, uint32_t len) {
  const uint32_t sh = (p & 3u) * 8u, at = p & ~3u;
  wt_or(w8, at, (uint32_t)(v << sh));
  if ((p & 3u) + len > 4u) wt_or(w8, at + 4u, (uint32_t)((v << sh) >> 32));
  if ((p & 3u) + len > 8u) wt_or(w8, at + 8u, (uint32_t)(v >> (64u - sh)));
}
/* n staged bytes at byte s, escaped, by a warp: a byte per lane, four of a string of more than 256 bytes (Pets whose name has 43 KB 22.9 -> 14.2 ms;
 * short strings take longer so); dst: where it goes */
__device__ __forceinline__ void wt_escape(uint8_t* w8, uint32_t s, uint32_t n, uint32_t dst, uint32_t hexa, uint32_t lane) {
  if (n <= 256u) {
    for (uint32_t i0 = 0; i0 < n; i0 += 32u) {
      uint32_t len = 0;
      const uint64_t v = i0 + lane < n ? wt_escaped(w8[s + i0 + lane], hexa, &len) : 0ull;
      const uint32_t end = warp_incl_scan(len);
      if (len) wt_or_bytes(w8, dst + end - len, v, len);
      dst += __shfl_sync(0xFFFFFFFFu, end, 31);
    }
    return;
  }
  for (uint32_t i0 = 0; i0 < n; i0 += 128u) {
    const uint32_t i = i0 + 4u * lane, have = i >= n ? 0u : (n - i < 4u ? n - i : 4u);
    const uint32_t x = have ? wt_low(wt_peek4(w8, s + i), have) : 0u;
    const uint32_t extra = wt_word_extra(x, have), end = warp_incl_scan(have + extra);
    uint32_t p = dst + end - have - extra;
    if (extra == 0u) { if (have) wt_or_bytes(w8, p, x, have); }
    else
      for (uint32_t k = 0; k < have; ++k) {
        uint32_t len;
        const uint64_t v = wt_escaped((x >> (8u * k)) & 0xFFu, hexa, &len);
        wt_or_bytes(w8, p, v, len);
        p += len;
      }
    dst += __shfl_sync(0xFFFFFFFFu, end, 31);
  }
}
/* n staged bytes at byte s that stay as they are, by a warp, a word of the window per lane */
__device__ __forceinline__ void wt_copy(uint8_t* w8, uint32_t s, uint32_t n, uint32_t dst, uint32_t lane) {
  const uint32_t lead = dst & 3u, end = lead + n; /* (bytes from the word that holds the first on) */
  s -= lead; dst -= lead;
  for (uint32_t k = 4u * lane; k < end; k += 128u) {
    uint32_t v = wt_peek4(w8, s + k);
    if (k >= lead && k + 4u <= end) { wt_st(w8, dst + k, v); continue; }
    if (k < lead) v &= 0xFFFFFFFFu << (8u * (lead - k));
    if (k + 4u > end) v &= 0xFFFFFFFFu >> (8u * (k + 4u - end));
    wt_or(w8, dst + k, v); /* shared with the text beside it */
  }
}
/* n bytes at byte s and a closing quote: up to the next word of the window, then whole words, then the rest */
static __device__ __noinline__ WtOut wt_put_plain(WtOut e, uint32_t s, uint32_t n) {
  const uint32_t room = 4u - (e.fill >> 3), h = n < room ? n : room;
  wt_put(e, wt_low(wt_peek4(e.w8, s), h), 8u * h);
  s += h; n -= h;
  uint32_t q = s & ~3u, x = wt_ld(e.w8, q);
  const uint32_t shift = (s & 3u) * 8u;
  for (; n >= 16u; n -= 16u) {
    const uint32_t y0 = wt_ld(e.w8, q + 4u), y1 = wt_ld(e.w8, q + 8u), y2 = wt_ld(e.w8, q + 12u), y3 = wt_ld(e.w8, q + 16u);
    wt_st(e.w8, e.at, __funnelshift_r(x, y0, shift)); wt_st(e.w8, e.at + 4u, __funnelshift_r(y0, y1, shift));
    wt_st(e.w8, e.at + 8u, __funnelshift_r(y1, y2, shift)); wt_st(e.w8, e.at + 12u, __funnelshift_r(y2, y3, shift));
    x = y3; q += 16u; e.at += 16u;
  }
  for (; n >= 4u; n -= 4u) {
    q += 4u;
    const uint32_t y = wt_ld(e.w8, q);
    wt_st(e.w8, e.at, __funnelshift_r(x, y, shift));
    e.at += 4u;
    x = y;
  }
  const uint32_t y = wt_ld(e.w8, q + 4u);
  wt_put(e, (n ? wt_low(__funnelshift_r(x, y, shift), n) : 0u) | ((uint32_t)'"' << (8u * n)), 8u * n + 8u);
  return e;
}
/* the n staged bytes at byte s, string `index` of the tile's in arena col, and the closing quote, behind the opening one */
__device__ __forceinline__ void wt_put_str(const WtRead& r, WtShared& sh, WtOut& e, uint32_t col, uint32_t index, uint32_t s, uint32_t n) {
  if (r.later) {
    const uint32_t extra = r.dirty ? wt_extra(sh, e.w8, col, index) : 0u;
    if (extra || n >= WT_LONG) {
      const uint32_t k = r.many && n < WT_SHORT ? WT_ESC : atomicAdd(&sh.nesc, 1u);
      if (k < WT_ESC) { /* later, by a warp */
        const uint32_t pos = wt_pos(e);
        sh.esc[k].at = s; sh.esc[k].n = n | (extra ? 0x80000000u : 0u); sh.esc[k].dst = pos;
        wt_end(e);
        wt_begin(e, pos + n + extra);
        wt_put(e, '"', 8);
        return;
      }
      if (extra) { e = wt_put_escaped(e, s, n, r.hexa); wt_put(e, '"', 8); return; }
    }
  }
  e = wt_put_plain(e, s, n);
}
/* properties [I, HI) of an object whose values are in r (its flat object's in rc); sep: what stands before the next property;
 * lists: how many bytes to leave for the elements of its lists */
template <int SCHEMA, int OBJ, int I, int HI>
__device__ __forceinline__ void wt_fields(const WtRead& x, WtShared& sh, uint32_t index, const RowSnap& r, const RowSnap& rc, const WtList* lists, uint32_t& sep, WtOut& e) {
  if constexpr (I < HI) {
    constexpr uint32_t kind = FK<OBJ, I>::kind, col = FK<OBJ, I>::col;
    const bool pr = (r.present >> I) & 1;
    bool empty = false;
    if constexpr (kind == K_STR || kind == K_LIST_STR || kind == K_LIST_OBJ) empty = r.a[I] == r.b[I];
    if (included(x.incl, pr, empty)) {
      constexpr int quote = kind == K_STR || kind == K_ENUM; /* (written with the name) */
      if (!pr) { wt_put_key<OBJ, I, 0>(e, sep); wt_put4(e, 0x6C6C756Eu); }
      else {
        wt_put_key<OBJ, I, quote>(e, sep);
        if constexpr (kind == K_I64 || kind == K_I32) e = wt_put_i64(e, r.v[I]);
        else if constexpr (kind == K_BOOL) { wt_put4(e, r.v[I] ? 0x65757274u : 0x736C6166u); wt_put(e, r.v[I] ? 0u : (uint32_t)'e', r.v[I] ? 0u : 8u); }
        else if constexpr (kind == K_ENUM) wt_put_enum<FK<OBJ, I>::child>(e, (uint32_t)r.v[I] % 3u);
        else if constexpr (kind == K_DATETIME) wt_put_datetime(e, r.v[I], r.a[I], (int32_t)r.b[I]);
        else if constexpr (kind == K_STR) wt_put_str(x, sh, e, col + 1, index, sh.at[col + 1] + r.a[I], r.b[I] - r.a[I]);
        else if constexpr (kind == K_OBJ) {
          constexpr int E = FK<OBJ, I>::child;
          uint32_t s = '{';
          wt_fields<SCHEMA, E, 0, CObj<E>::N>(x, sh, index, rc, rc, nullptr, s, e);
          wt_put(e, s == '{' ? '{' | ('}' << 8) : (uint32_t)'}', s == '{' ? 16u : 8u);
        } else if constexpr (kind == K_LIST_STR || kind == K_LIST_OBJ) {
          constexpr int l = kind == K_LIST_OBJ;
          if (empty) wt_put(e, '[' | (']' << 8), 16);
          else {
            wt_put(e, '[', 8);
            const uint32_t pos = wt_pos(e);
            wt_end(e); /* (the elements are another unit's) */
            wt_begin(e, pos + lists[l].bytes);
          }
        }
      }
      sep = ',';
    }
    wt_fields<SCHEMA, OBJ, I + 1, HI>(x, sh, index, r, rc, lists, sep, e);
  }
}

/* ---- units: 32 rows of one model ----------------------------------------------------------------------------------- */
/* group g of the tile: its model, its first row and which record of the tile a lane's row is (WT_NONE: the lane has none) */
struct WtGroup { uint32_t model, first, n; };
template <int SCHEMA>
__device__ __forceinline__ WtGroup wt_group(const WtShared& sh, uint32_t g) {
  WtGroup o;
  if constexpr (SCHEMA != PJ_SCHEMA_MIXED) { o.model = SCHEMA - 1; o.first = 32u * g; }
  else {
    o.model = 0;
    for (; o.model < 2u; ++o.model) { const uint32_t k = (sh.cnt[o.model] + 31u) / 32u; if (g < k) break; g -= k; }
    o.first = 32u * g;
  }
  const uint32_t rest = sh.cnt[o.model] - o.first;
  o.n = rest < 32u ? rest : 32u;
  return o;
}
template <int SCHEMA>
__device__ __forceinline__ uint32_t wt_record(const WtShared& sh, const WtGroup& g, uint32_t lane) {
  if (lane >= g.n) return WT_NONE;
  const uint32_t k = g.first + lane;
  return SCHEMA == PJ_SCHEMA_MIXED ? (uint32_t)sh.perm[sh.pre[g.model] + k] : k;
}
/* the elements a row's list has, and their bytes by the running sums */
template <int L>
__device__ __forceinline__ WtList wt_list(const WtShared& sh, const uint8_t* w8, uint32_t a, uint32_t b, uint32_t group_first, bool& bad) {
  WtList l;
  const uint32_t u = a - sh.item0[L], v = b - sh.item0[L];
  if (u > v || v > sh.itemn[L]) { bad = true; l.a = l.b = group_first; l.bytes = 0; return l; }
  const uint32_t* sums = reinterpret_cast<const uint32_t*>(w8 + sh.sums) + (L ? sh.itemn[0] : 0u);
  l.a = a; l.b = b;
  l.bytes = v > u ? sums[v - 1u] - (a > group_first ? sums[u - 1u] : 0u) : 0u;
  return l;
}
/* running sums of the elements of list L of the group's rows: text and the comma or bracket behind it */
template <int SCHEMA, int L>
__device__ __forceinline__ void wt_sum_items(const WtRead& x, WtShared& sh, uint8_t* w8, const WtGroup& g, uint32_t lane, bool& bad) {
  constexpr int F = L ? WT_LIST_OBJ : WT_LIST_STR;
  constexpr uint32_t col = FK<OBJ_PET, F>::col;
  const uint32_t row = (uint32_t)sh.row0[0] + g.first;
  uint32_t i0 = *wt_at<uint32_t>(sh, w8, col, row), i1 = *wt_at<uint32_t>(sh, w8, col, row + g.n);
  const uint32_t base = sh.item0[L];
  if (i0 - base > i1 - base || i1 - base > sh.itemn[L]) { bad = true; i1 = i0; }
  uint32_t* sums = reinterpret_cast<uint32_t*>(w8 + sh.sums) + (L ? sh.itemn[0] : 0u);
  uint32_t carry = 0;
  for (uint32_t k0 = i0; k0 < i1; k0 += 32u) {
    const uint32_t k = k0 + lane;
    uint32_t n = 0;
    if (k < i1) {
      if constexpr (L == 0) {
        const uint32_t* so = wt_at<uint32_t>(sh, w8, col + 1, k);
        n = wt_str_size(x, sh, w8, col + 2, k - base, so[0], so[1], bad) + 1u;
      } else {
        constexpr int E = FK<OBJ_PET, F>::child;
        RowSnap r;
        r.present = *wt_at<uint8_t>(sh, w8, CObj<E>::present_col, k);
        wt_snap<E, 0, CObj<E>::N>(sh, w8, k, r);
        if (x.dirty && wt_falls<E>(r, r)) bad = true;
        bool first = true;
        n = wt_size<SCHEMA, E, 0, CObj<E>::N>(x, sh, w8, k - base, r, r, nullptr, nullptr, 0, first, bad) + 2u + first;
      }
    }
    n = warp_incl_scan(n) + carry;
    if (k < i1) sums[k - base] = n;
    carry = __shfl_sync(0xFFFFFFFFu, n, 31);
  }
}
/* bytes of the group's records, and where their second halves start */
template <int SCHEMA, int OBJ>
__device__ __forceinline__ void wt_size_records(const WtRead& x, WtShared& sh, const uint8_t* w8, const WtGroup& g, uint32_t lane, bool& bad) {
  const uint32_t rec = wt_record<SCHEMA>(sh, g, lane);
  if (rec == WT_NONE) return;
  const uint32_t index = g.first + lane, row = (uint32_t)sh.row0[g.model] + index;
  RowSnap r, rc;
  wt_load<OBJ, 0, CObj<OBJ>::N>(sh, w8, row, r, rc);
  WtList lists[2];
  if constexpr (OBJ == OBJ_PET) {
    lists[0] = wt_list<0>(sh, w8, r.a[WT_LIST_STR], r.b[WT_LIST_STR], *wt_at<uint32_t>(sh, w8, FK<OBJ, WT_LIST_STR>::col, row - lane), bad);
    lists[1] = wt_list<1>(sh, w8, r.a[WT_LIST_OBJ], r.b[WT_LIST_OBJ], *wt_at<uint32_t>(sh, w8, FK<OBJ, WT_LIST_OBJ>::col, row - lane), bad);
  }
  if (x.dirty && wt_falls<OBJ>(r, rc)) bad = true;
  bool first = true;
  uint32_t list_at[2] = {WT_NONE, WT_NONE};
  const uint32_t n0 = wt_size<SCHEMA, OBJ, 0, WtMid<OBJ>::v>(x, sh, w8, index, r, rc, lists, list_at, 0, first, bad);
  sh.mid[rec] = n0 | (first ? 0x80000000u : 0u);
  const uint32_t n1 = wt_size<SCHEMA, OBJ, WtMid<OBJ>::v, CObj<OBJ>::N>(x, sh, w8, index, r, rc, lists, list_at, n0, first, bad);
  if constexpr (OBJ == OBJ_PET) { sh.list[0][rec] = list_at[0]; sh.list[1][rec] = list_at[1]; }
  if (n0 >= 0x80000000u) bad = true;
  sh.pos[rec] = n0 + n1 + 2u + first; /* } and what follows the record */
}
/* text of half H of the group's records, those of [ra, rb) of the tile. at0: where the tile's text begins in the window. */
template <int SCHEMA, int OBJ, int H>
__device__ __forceinline__ void wt_half(const WtRead& x, WtShared& sh, uint8_t* w8, const WtGroup& g, uint32_t lane, uint32_t ra, uint32_t rb, uint32_t at0, uint32_t after) {
  constexpr int LO = H ? WtMid<OBJ>::v : 0, HI = H ? CObj<OBJ>::N : WtMid<OBJ>::v;
  const uint32_t rec = wt_record<SCHEMA>(sh, g, lane);
  if (rec == WT_NONE || rec < ra || rec >= rb) return;
  const uint32_t index = g.first + lane, row = (uint32_t)sh.row0[g.model] + index;
  RowSnap r, rc;
  wt_load<OBJ, LO, HI>(sh, w8, row, r, rc);
  WtList lists[2];
  if constexpr (H == 1 && OBJ == OBJ_PET) {
    bool bad = false;
    lists[0] = wt_list<0>(sh, w8, r.a[WT_LIST_STR], r.b[WT_LIST_STR], *wt_at<uint32_t>(sh, w8, FK<OBJ, WT_LIST_STR>::col, row - lane), bad);
    lists[1] = wt_list<1>(sh, w8, r.a[WT_LIST_OBJ], r.b[WT_LIST_OBJ], *wt_at<uint32_t>(sh, w8, FK<OBJ, WT_LIST_OBJ>::col, row - lane), bad);
  }
  WtOut e;
  e.w8 = w8;
  const uint32_t mid = sh.mid[rec];
  wt_begin(e, at0 + sh.pos[rec] + (H ? mid & 0x7FFFFFFFu : 0u));
  uint32_t sep = H == 0 || mid >> 31 ? '{' : ',';
  wt_fields<SCHEMA, OBJ, LO, HI>(x, sh, index, r, rc, lists, sep, e);
  if (H) {
    if (sep == '{') wt_put(e, '{', 8);
    wt_put(e, '}' | (after << 8), 16);
  }
  wt_end(e);
}
/* the elements of list L of the group's records, one per lane, whosever they are */
template <int SCHEMA, int L>
__device__ __forceinline__ void wt_items(const WtRead& x, WtShared& sh, uint8_t* w8, const WtGroup& g, uint32_t lane, uint32_t ra, uint32_t rb, uint32_t at0, uint32_t part, uint32_t parts) {
  constexpr int F = L ? WT_LIST_OBJ : WT_LIST_STR;
  constexpr uint32_t col = FK<OBJ_PET, F>::col;
  const uint32_t rec = wt_record<SCHEMA>(sh, g, lane);
  const bool live = rec != WT_NONE && rec >= ra && rec < rb;
  const uint32_t* c = wt_at<uint32_t>(sh, w8, col, (uint32_t)sh.row0[0] + g.first);
  const uint32_t a = c[lane < g.n ? lane : g.n], b = c[lane < g.n ? lane + 1u : g.n]; /* lanes without a row: no elements, at the group's end */
  const uint32_t base = sh.item0[L], i0 = __shfl_sync(0xFFFFFFFFu, a, 0), i1 = __shfl_sync(0xFFFFFFFFu, b, 31);
  const uint32_t* sums = reinterpret_cast<const uint32_t*>(w8 + sh.sums) + (L ? sh.itemn[0] : 0u);
  uint32_t list_at = live && b > a ? sh.list[L][rec] : WT_NONE;
  const bool any = list_at != WT_NONE;
  if (any) list_at += at0 + sh.pos[rec] - (a > i0 ? sums[a - base - 1u] : 0u); /* (of element k: and the sums before it) */
  const uint32_t mine = __ballot_sync(0xFFFFFFFFu, any);
  if (!mine) return;
  /* from the first record's first element to the last one's last */
  const uint32_t k_lo = __shfl_sync(0xFFFFFFFFu, a, __ffs((int)mine) - 1), k_hi = __shfl_sync(0xFFFFFFFFu, b, 31 - __clz((int)mine));
  for (uint32_t k0 = k_lo + 32u * part; k0 < k_hi; k0 += 32u * parts) {
    const uint32_t k = k0 + lane;
    uint32_t own = 0; /* the last lane whose elements begin at or before k */
#pragma unroll
    for (uint32_t d = 16; d; d >>= 1) { const uint32_t v = __shfl_sync(0xFFFFFFFFu, a, (int)(own + d)); if (v <= k) own += d; }
    const uint32_t at = __shfl_sync(0xFFFFFFFFu, list_at, (int)own), end = __shfl_sync(0xFFFFFFFFu, b, (int)own);
    if (k >= k_hi || !((mine >> own) & 1u)) continue;
    WtOut e;
    e.w8 = w8;
    wt_begin(e, at + (k > i0 ? sums[k - base - 1u] : 0u));
    const uint32_t close = k + 1u < end ? (uint32_t)',' : (uint32_t)']';
    if constexpr (L == 0) {
      const uint32_t* so = wt_at<uint32_t>(sh, w8, col + 1, k);
      const uint32_t s0 = so[0], s1 = so[1];
      wt_put(e, '"', 8);
      wt_put_str(x, sh, e, col + 2, k - base, sh.at[col + 2] + s0, s1 - s0);
      wt_put(e, close, 8);
    } else {
      constexpr int E = FK<OBJ_PET, F>::child;
      RowSnap r;
      r.present = *wt_at<uint8_t>(sh, w8, CObj<E>::present_col, k);
      wt_snap<E, 0, CObj<E>::N>(sh, w8, k, r);
      uint32_t sep = '{';
      wt_fields<SCHEMA, E, 0, CObj<E>::N>(x, sh, k - base, r, r, nullptr, sep, e);
      if (sep == '{') wt_put(e, '{', 8);
      wt_put(e, '}' | (close << 8), 16);
    }
    wt_end(e);
  }
}
/* text of unit k of a group: the halves of its records, (part of) the elements of its lists */
template <int SCHEMA, int OBJ>
__device__ __forceinline__ void wt_unit(const WtRead& x, WtShared& sh, uint8_t* w8, const WtGroup& g, uint32_t k, uint32_t part, uint32_t parts, uint32_t lane, uint32_t ra, uint32_t rb, uint32_t at0, uint32_t after) {
  if (k == 0) wt_half<SCHEMA, OBJ, 0>(x, sh, w8, g, lane, ra, rb, at0, after);
  else if (k == 1) wt_half<SCHEMA, OBJ, 1>(x, sh, w8, g, lane, ra, rb, at0, after);
  else if constexpr (OBJ == OBJ_PET) {
    if (k == 2) wt_items<SCHEMA, 0>(x, sh, w8, g, lane, ra, rb, at0, part, parts); else wt_items<SCHEMA, 1>(x, sh, w8, g, lane, ra, rb, at0, part, parts);
  }
}

/* ---- the tile ------------------------------------------------------------------------------------------------------- */
/* A piece of a column on its way to shared memory at byte `at`: elements [x, y). Returns where the next one goes. All lanes of warp 0. */
__device__ __forceinline__ uint32_t wt_place(WtShared& sh, uint8_t* w8, uint32_t at, const WtCol& c, bool have, uint64_t x, uint64_t y, uint32_t room, uint32_t bar, uint32_t lane, bool& bad) {
  uint32_t n = 0, lead = 0;
  uintptr_t src = 0;
  if (have && y > x) {
    const uintptr_t p = (uintptr_t)c.p + (x << c.shift), q = (uintptr_t)c.p + (y << c.shift);
    src = p & ~(uintptr_t)15;
    lead = (uint32_t)(p - src);
    const uint64_t bytes = ((q + 15u) & ~(uintptr_t)15) - src; /* whole 16-byte blocks that hold a byte of the tile's */
    if (bytes > room) bad = true; else n = (uint32_t)bytes;
  }
  const uint32_t end = warp_incl_scan(n), total = __shfl_sync(0xFFFFFFFFu, end, 31); /* (32 times the room at most) */
  bad = __any_sync(0xFFFFFFFFu, bad || at + total > room);
  if (bad) return at;
  if (have) sh.at[c.col] = at + end - n + lead - ((uint32_t)x << c.shift);
  if (lane == 0 && total) { sh.flight |= 1u << bar; mbar_expect_tx(&sh.mbar[bar], total); }
  __syncwarp();
  if (n) bulk_g2s(w8 + at + end - n, (const void*)src, n, &sh.mbar[bar]);
  return at + total;
}
/* What the tile reads, on its way to shared memory. Warp 0. Sets sh.odd when it does not fit. */
template <int SCHEMA>
__device__ __forceinline__ void wt_stage(const WTileArgs& a, WtShared& sh, uint8_t* w8, uint32_t lane) {
  constexpr bool LISTS = SCHEMA == PJ_SCHEMA_PET || SCHEMA == PJ_SCHEMA_MIXED;
  bool bad = sh.odd != 0;
  bad = __any_sync(0xFFFFFFFFu, bad);
  uint32_t at = 0;
  /* columns with an element per row */
  if (!bad) {
    const bool have = lane < a.nrow;
    const WtCol c = a.col[have ? lane : 0u];
    const uint64_t r0 = sh.row0[c.model];
    const uint32_t n = sh.cnt[c.model];
    at = wt_place(sh, w8, at, c, have && n, r0, r0 + n + c.plus, a.smem, 0u, lane, bad);
  }
  /* the tile's elements of the lists */
  uint32_t i0 = 0, items = 0;
  if (LISTS && !bad && lane < 2u) {
    if (sh.cnt[0]) {
      const uint32_t* o = a.list[lane];
      i0 = o[sh.row0[0]];
      const uint32_t i1 = o[sh.row0[0] + sh.cnt[0]];
      if (i1 < i0 || i1 - i0 > a.smem / 4u) bad = true; else items = i1 - i0;
    }
    sh.item0[lane] = i0; sh.itemn[lane] = items;
  }
  bad = __any_sync(0xFFFFFFFFu, bad);
  const uint32_t n0 = __shfl_sync(0xFFFFFFFFu, items, 0), n1 = __shfl_sync(0xFFFFFFFFu, items, 1), f0 = __shfl_sync(0xFFFFFFFFu, i0, 0), f1 = __shfl_sync(0xFFFFFFFFu, i0, 1);
  /* their columns and the arenas */
  uint32_t strs = 0;
  if (!bad && a.nrow < a.ncol) {
    const bool have = lane < a.ncol - a.nrow;
    const WtCol c = a.col[have ? a.nrow + lane : 0u];
    const uint32_t n = c.level == 0 ? sh.cnt[c.model] : (c.level == 1 ? n0 : n1);
    uint64_t x = c.level == 0 ? sh.row0[c.model] : (c.level == 1 ? f0 : f1), y = x + n + c.plus;
    uint32_t mine = 0;
    if (have && c.off) {
      if (n) { mine = n; const uint32_t lo = c.off[x], hi = c.off[y]; x = lo; y = hi; if (hi < lo) bad = true; }
      else x = y = 0;
      sh.lo[c.col] = (uint32_t)x; sh.span[c.col] = (uint32_t)(y - x);
    }
    const uint32_t upto = warp_incl_scan(mine);
    if (have && c.off) sh.str0[c.col] = upto - mine;
    strs = __shfl_sync(0xFFFFFFFFu, upto, 31);
    /* first what is no text */
    at = wt_place(sh, w8, at, c, have && !c.off && n, x, y, a.smem, 1u, lane, bad);
    if (lane == 0) sh.text = at;
    if (!bad) at = wt_place(sh, w8, at, c, have && c.off, x, y, a.smem, 2u, lane, bad);
    /* whose text a block is: a column starts in a block of its own */
    const bool text = !bad && have && c.off && y > x;
    const uint32_t first = text ? sh.at[c.col] + (uint32_t)x : 0u;
    sh.ar0[lane] = (uint16_t)(first >> 4); sh.ar1[lane] = (uint16_t)(text ? (first + (uint32_t)(y - x) + 15u) >> 4 : 0u);
    sh.arcol[lane] = c.col; sh.arlevel[lane] = c.level; sh.armodel[lane] = c.model;
  }
  else if (lane == 0) sh.text = at;
  const uint32_t sums = at + 16u, extra = (sums + 4u * (n0 + n1) + 15u) & ~15u;
  if (extra + 4u * strs + 16u + WT_MIN_WINDOW > a.smem) bad = true;
  if (lane == 0) { sh.stage = at; sh.sums = sums; sh.extra = sh.win = extra; sh.nstr = strs; if (bad) sh.odd = 1; }
}
/* bytes the escapes of the n bytes at s add, all lanes of a warp: 16-byte blocks, looked at again where there is one */
__device__ __forceinline__ uint32_t wt_warp_extra(const uint8_t* s, uint32_t n, uint32_t lane) {
  const uintptr_t from = reinterpret_cast<uintptr_t>(s), to = from + n;
  uint32_t extra = 0;
  for (uintptr_t p = (from & ~(uintptr_t)15) + 16u * lane; p < to; p += 512u) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    const uint32_t x[4] = {v.x, v.y, v.z, v.w};
    if (word_needs_escape(x[0]) | word_needs_escape(x[1]) | word_needs_escape(x[2]) | word_needs_escape(x[3]))
      for (uint32_t k = 0; k < 16u; ++k) if (p + k >= from && p + k < to) extra += escape_extra_byte((x[k >> 2] >> (8u * (k & 3u))) & 0xFFu);
  }
  return __reduce_add_sync(0xFFFFFFFFu, extra);
}
/* a 16-byte block with a byte to escape: counted for the strings it lies in, by a warp */
__device__ __forceinline__ void wt_count_block(WtShared& sh, uint8_t* w8, uint32_t block, uint32_t lane) {
  const uint32_t who = __ballot_sync(0xFFFFFFFFu, block - sh.ar0[lane] < (uint32_t)sh.ar1[lane] - sh.ar0[lane]);
  if (!who) return;
  const uint32_t c = (uint32_t)__ffs((int)who) - 1u, col = sh.arcol[c], level = sh.arlevel[c], model = sh.armodel[c], p = 16u * block + lane, x = p - sh.at[col];
  const uint32_t extra = lane < 16u && x - sh.lo[col] < sh.span[col] ? escape_extra_byte(w8[p]) : 0u;
  if (!extra) return;
  const uint32_t first = level == 0 ? (uint32_t)sh.row0[model] : sh.item0[level - 1u];
  const uint32_t* o = wt_at<uint32_t>(sh, w8, col - 1u, first); /* (an arena's column follows its offsets') */
  uint32_t lo = 0, hi = level == 0 ? sh.cnt[model] : sh.itemn[level - 1u]; /* the last string that begins at or before it */
  while (lo + 1u < hi) { const uint32_t mid = (lo + hi) >> 1; if (o[mid] <= x) lo = mid; else hi = mid; }
  atomicAdd(wt_extras(sh, w8) + sh.str0[col] + lo, extra);
}
/* All strings of the tile that are staged, one per lane: their escapes. For text with many bytes to escape; bad: one lies outside its arena. */
__device__ __forceinline__ bool wt_count_strings(WtShared& sh, uint8_t* w8, uint32_t warp, uint32_t warps, uint32_t lane) {
  uint32_t todo = __ballot_sync(0xFFFFFFFFu, sh.ar1[lane] > sh.ar0[lane]), turn = 0; /* the first group of 32 goes to this warp */
  bool bad = false;
  for (; todo; todo &= todo - 1u) {
    const uint32_t c = (uint32_t)__ffs((int)todo) - 1u, col = sh.arcol[c], level = sh.arlevel[c], model = sh.armodel[c];
    const uint32_t first = level == 0 ? (uint32_t)sh.row0[model] : sh.item0[level - 1u], n = level == 0 ? sh.cnt[model] : sh.itemn[level - 1u], groups = (n + 31u) / 32u;
    const uint32_t* o = wt_at<uint32_t>(sh, w8, col - 1u, first); /* (an arena's column follows its offsets') */
    for (uint32_t g = (warp + warps - turn) % warps; g < groups; g += warps) {
      const uint32_t k = 32u * g + lane;
      uint32_t a = 0, len = 0;
      if (k < n) {
        const uint32_t b = o[k + 1u];
        a = o[k];
        if (a > b || a < sh.lo[col] || b - sh.lo[col] > sh.span[col]) bad = true;
        else len = b - a;
      }
      const uint8_t* s = w8 + (sh.at[col] + a);
      if (len && len < WT_LONG) wt_extras(sh, w8)[sh.str0[col] + k] = str_escape_extra(s, len);
      for (uint32_t longs = __ballot_sync(0xFFFFFFFFu, len >= WT_LONG); longs; longs &= longs - 1u) { /* those are a warp's, one after the other */
        const int who = __ffs((int)longs) - 1;
        const uint32_t m = __shfl_sync(0xFFFFFFFFu, len, who), from = sh.at[col] + __shfl_sync(0xFFFFFFFFu, a, who), extra = wt_warp_extra(w8 + from, m, lane);
        if (lane == 0) wt_extras(sh, w8)[sh.str0[col] + 32u * g + (uint32_t)who] = extra;
      }
    }
    turn = (turn + groups) % warps;
  }
  return bad;
}
/* Mixed streams: the tile's records by model, in order; odd when the rows of a model do not follow each other. */
__device__ __forceinline__ void wt_sort(const WTileArgs& a, WtShared& sh, uint64_t rec0, uint32_t nrec, uint32_t tid) {
  const uint32_t lane = tid & 31u, warp = tid >> 5;
  uint32_t m = 3, rank = 0;
  uint64_t row = 0;
  if (tid < nrec) {
    uint32_t type;
    if (write_locate(PJ_SCHEMA_MIXED, &a.w.cols, rec0 + tid, &type, &row)) m = type == PJ_TYPE_PET ? 0u : (type == PJ_TYPE_ORDER ? 1u : 2u);
    sh.pos[tid] = 0;
  }
#pragma unroll
  for (uint32_t k = 0; k < 3; ++k) {
    const uint32_t b = __ballot_sync(0xFFFFFFFFu, m == k);
    if (lane == 0) sh.cls[k][warp] = (uint32_t)__popc(b);
    if (m == k) rank = (uint32_t)__popc(b & ((1u << lane) - 1u));
  }
  __syncthreads();
  uint32_t cnt[3] = {0, 0, 0};
#pragma unroll
  for (uint32_t k = 0; k < 3; ++k)
#pragma unroll
    for (uint32_t w = 0; w < WtT<PJ_SCHEMA_MIXED>::warps; ++w) { const uint32_t v = sh.cls[k][w]; if (m == k && w < warp) rank += v; cnt[k] += v; }
  if (m < 3u) {
    sh.perm[(m == 0 ? 0u : (m == 1 ? cnt[0] : cnt[0] + cnt[1])) + rank] = (uint8_t)tid;
    if (rank == 0) sh.row0[m] = row;
  }
  if (tid < 3u) { sh.cnt[tid] = tid == 0 ? cnt[0] : (tid == 1 ? cnt[1] : cnt[2]); sh.pre[tid] = tid == 0 ? 0u : (tid == 1 ? cnt[0] : cnt[0] + cnt[1]); }
  __syncthreads();
  if (m < 3u && row != sh.row0[m] + rank) sh.odd = 1;
}
template <int SCHEMA>
__device__ __forceinline__ uint32_t wt_groups(const WtShared& sh) {
  if constexpr (SCHEMA != PJ_SCHEMA_MIXED) return (sh.cnt[SCHEMA - 1] + 31u) / 32u;
  else return (sh.cnt[0] + 31u) / 32u + (sh.cnt[1] + 31u) / 32u + (sh.cnt[2] + 31u) / 32u;
}
/* ---- the general road: a record per thread, its long strings and lists by whole warps ------------------------------------ */
/* What a record's thread leaves (see WriteAll of pj_write_fast.cuh): noted while it is measured, found again in the same order while it is written. */
struct WtLeave {
  static constexpr bool on = true;
  WtShared* sh;
  WtLater* e;
  uint32_t cap, rec, last;
  template <bool WR>
  __device__ __forceinline__ bool put(uint32_t kind, uint32_t col, uint32_t a, uint32_t b, WOut& w) {
    if (kind == K_STR ? b - a < WT_LONG : b - a < WT_LONG_LIST || b < a) return false;
    if (WR) {
      const uint32_t k = last == WT_NONE ? sh->mid[rec] : (uint32_t)e[last].link;
      if (k == WT_LAST || e[k].kind != kind || e[k].col != col || e[k].a != a || e[k].b != b) return false;
      e[k].dst = w.dst + w.n;
      w.n += e[k].size;
      last = k;
      return true;
    }
    const uint32_t k = atomicAdd(&sh->nlater, 1u);
    if (k >= cap) return false;
    e[k].dst = nullptr; e[k].size = 0; e[k].a = a; e[k].b = b; e[k].rec = (uint16_t)rec; e[k].link = WT_LAST; e[k].kind = (uint8_t)kind; e[k].col = (uint8_t)col;
    if (last == WT_NONE) sh->mid[rec] = k; else e[last].link = (uint16_t)k;
    last = k;
    return true;
  }
};
template <int SCHEMA>
__device__ __forceinline__ uint64_t wt_row(const DevCols& c, uint64_t i) { return SCHEMA == PJ_SCHEMA_MIXED ? (uint64_t)colp<uint32_t>(&c, PJ_COL_REC_ROW)[i] : i; }
/* Record `rec` of the tile, row `row` of model OBJ: bytes of its text and of what follows it, without what is left to the warps (top bit: a byte has
 * to be escaped), or the text itself. PLAIN: no byte has to. */
template <int OBJ, bool WR, bool PLAIN>
__device__ __noinline__ unsigned long long wt_general(const DevCols* c, uint64_t row, int incl, uint32_t hexa, uint8_t* dst, uint32_t after, WtShared* sh, WtLater* e, uint32_t cap, uint32_t rec) {
  WOut w;
  w.dst = dst; w.n = 0; w.hexa = hexa;
  WtLeave l;
  l.sh = sh; l.e = e; l.cap = cap; l.rec = rec; l.last = WT_NONE;
  if (!WR) sh->mid[rec] = WT_LAST;
  fwrite_object<WR, PLAIN, OBJ, 0>(c, row, incl, l, w);
  if (WR) dst[w.n] = (uint8_t)after;
  return (w.n + 1u) | (!WR && w.escapes ? TS_VALID : 0ull);
}
template <int SCHEMA, bool WR>
__device__ __forceinline__ unsigned long long wt_general_any(const DevCols* c, uint32_t model, uint64_t row, int incl, uint32_t hexa, uint8_t* dst, uint32_t after, WtShared* sh, WtLater* e, uint32_t cap, uint32_t rec, bool plain) {
  if constexpr (SCHEMA == PJ_SCHEMA_PET || SCHEMA == PJ_SCHEMA_MIXED)
    if (model == 0) return WR && plain ? wt_general<OBJ_PET, WR, WR>(c, row, incl, hexa, dst, after, sh, e, cap, rec) : wt_general<OBJ_PET, WR, false>(c, row, incl, hexa, dst, after, sh, e, cap, rec);
  if constexpr (SCHEMA == PJ_SCHEMA_ORDER || SCHEMA == PJ_SCHEMA_MIXED)
    if (model == 1) return wt_general<OBJ_ORDER, WR, false>(c, row, incl, hexa, dst, after, sh, e, cap, rec);
  if constexpr (SCHEMA == PJ_SCHEMA_USER || SCHEMA == PJ_SCHEMA_MIXED)
    if (model == 2) return WR && plain ? wt_general<OBJ_USER, WR, WR>(c, row, incl, hexa, dst, after, sh, e, cap, rec) : wt_general<OBJ_USER, WR, false>(c, row, incl, hexa, dst, after, sh, e, cap, rec);
  return 0;
}
/* the n bytes at s to d, as they are, all lanes of a warp: 16-byte blocks of d */
__device__ __forceinline__ void wt_warp_copy(uint8_t* d, const uint8_t* s, uint32_t n, uint32_t lane) {
  const uint32_t head = (0u - (uint32_t)reinterpret_cast<uintptr_t>(d)) & 15u, lead = head < n ? head : n;
  if (lane < lead) d[lane] = s[lane];
  d += lead; s += lead; n -= lead;
  const uint32_t shift = ((uint32_t)reinterpret_cast<uintptr_t>(s) & 3u) * 8u, whole = n & ~15u;
  for (uint32_t k = 16u * lane; k < whole; k += 512u) {
    const uint32_t* p = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(s + k) & ~(uintptr_t)3);
    const uint32_t x0 = p[0], x1 = p[1], x2 = p[2], x3 = p[3], x4 = shift ? p[4] : 0u; /* (never a word that holds none of the n bytes) */
    uint4 v;
    v.x = __funnelshift_r(x0, x1, shift); v.y = __funnelshift_r(x1, x2, shift); v.z = __funnelshift_r(x2, x3, shift); v.w = __funnelshift_r(x3, x4, shift);
    *reinterpret_cast<uint4*>(d + k) = v;
  }
  if (lane < n - whole) d[whole + lane] = s[whole + lane];
}
/* ... escaped, four bytes per lane */
__device__ __forceinline__ void wt_warp_escape(uint8_t* d, const uint8_t* s, uint32_t n, uint32_t hexa, uint32_t lane) {
  const uint32_t shift = ((uint32_t)reinterpret_cast<uintptr_t>(s) & 3u) * 8u;
  for (uint32_t i0 = 0; i0 < n; i0 += 128u) {
    const uint32_t i = i0 + 4u * lane, have = i >= n ? 0u : (n - i < 4u ? n - i : 4u);
    uint32_t x = 0;
    if (have) { /* (never a word that holds none of the n bytes) */
      const uint32_t* p = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(s + i) & ~(uintptr_t)3);
      x = wt_low(__funnelshift_r(p[0], shift + 8u * have > 32u ? p[1] : 0u, shift), have);
    }
    const uint32_t extra = wt_word_extra(x, have), end = warp_incl_scan(have + extra);
    uint8_t* p = d + (end - have - extra);
    for (uint32_t k = 0; k < have; ++k) {
      uint32_t len = 1;
      uint64_t v = (x >> (8u * k)) & 0xFFu;
      if (extra) v = wt_escaped((uint32_t)v, hexa, &len);
      for (uint32_t b = 0; b < len; ++b) p[b] = (uint8_t)(v >> (8u * b));
      p += len;
    }
    d += __shfl_sync(0xFFFFFFFFu, end, 31);
  }
}
/* Element k of a list: its text, measured or written, by one lane. PLAIN: it has no byte to escape. */
template <bool WR, bool PLAIN>
__device__ __forceinline__ void wt_element(const DevCols* c, const WtLater& e, uint32_t k, int incl, WOut& w) {
  if (e.kind == K_LIST_STR) {
    const uint32_t* so = colp<uint32_t>(c, FK<OBJ_PET, WT_LIST_STR>::col + 1);
    fput_str<WR, PLAIN>(w, colp<uint8_t>(c, FK<OBJ_PET, WT_LIST_STR>::col + 2) + so[k], so[k + 1] - so[k]);
  } else {
    WriteAll all;
    fwrite_object<WR, PLAIN, FK<OBJ_PET, WT_LIST_OBJ>::child, 1>(c, k, incl, all, w);
  }
}
/* Measures what the records' threads have left, n of them: a string in parts of WT_PART bytes that go round the warps, a list by one warp, an element
 * per lane. bytes: whether the records' totals are wanted. */
static __device__ __noinline__ void wt_measure_later(const DevCols* c, WtShared& sh, WtLater* e, uint32_t n, int incl, bool bytes, uint32_t warp, uint32_t warps, uint32_t lane) {
  for (uint32_t j = 0; j < n; ++j) {
    WtLater& l = e[j];
    const uint32_t first = (warp + warps - j % warps) % warps; /* the first part that is the warp's */
    unsigned long long size = 0;
    if (l.kind == K_STR) {
      const uint8_t* s = colp<uint8_t>(c, l.col) + l.a;
      const uint32_t len = l.b - l.a;
      for (uint32_t from = first * WT_PART; from < len; from += WT_PART * warps) {
        size += wt_warp_extra(s + from, len - from < WT_PART ? len - from : WT_PART, lane);
        if (len - from <= WT_PART * warps) break; /* (a sum could pass 2^32) */
      }
      if (first == 0) size += 2ull + len;
    } else if (first == 0) {
      unsigned long long sum = 0;
      for (uint32_t k = l.a + lane; k < l.b; k += 32u) {
        WOut w;
        w.dst = nullptr; w.n = 0;
        wt_element<false, false>(c, l, k, incl, w);
        sum += w.n + 1u;
        if (l.b - k <= 32u) break;
      }
      for (int d = 16; d; d >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, d);
      size = sum + 1u;
    }
    if (size && lane == 0) { atomicAdd(&l.size, size); if (bytes) atomicAdd(&sh.bytes[l.rec], size); }
    __syncwarp();
  }
}
/* ... and writes them. */
static __device__ __noinline__ void wt_write_later(const DevCols* c, WtLater* e, uint32_t n, int incl, uint32_t hexa, uint32_t warp, uint32_t warps, uint32_t lane) {
  for (uint32_t j = 0; j < n; ++j) {
    const WtLater& l = e[j];
    const uint32_t first = (warp + warps - j % warps) % warps;
    if (l.kind == K_STR) {
      const uint8_t* s = colp<uint8_t>(c, l.col) + l.a;
      const uint32_t len = l.b - l.a;
      if (first == 0 && lane == 0) { l.dst[0] = '"'; l.dst[l.size - 1u] = '"'; }
      if (l.size != 2ull + len) { if (first == 0) wt_warp_escape(l.dst + 1, s, len, hexa, lane); continue; }
      for (uint32_t from = first * WT_PART; from < len; from += WT_PART * warps) {
        wt_warp_copy(l.dst + 1 + from, s + from, len - from < WT_PART ? len - from : WT_PART, lane);
        if (len - from <= WT_PART * warps) break;
      }
    } else if (first == 0) {
      uint8_t* d = l.dst;
      if (lane == 0) *d = '[';
      ++d;
      for (uint32_t k0 = l.a; k0 < l.b; k0 += 32u) {
        const uint32_t k = k0 + lane;
        const bool have = k0 <= k && k < l.b;
        WOut w;
        w.dst = nullptr; w.n = 0; w.hexa = hexa;
        if (have) { wt_element<false, false>(c, l, k, incl, w); w.n++; }
        const unsigned long long end = warp_incl_scan((unsigned long long)w.n);
        if (have) {
          const bool plain = w.escapes == 0;
          w.dst = d + (end - w.n); w.n = 0;
          if (plain) wt_element<true, true>(c, l, k, incl, w); else wt_element<true, false>(c, l, k, incl, w);
          wput<true>(w, k + 1u < l.b ? ',' : ']');
        }
        d += __shfl_sync(0xFFFFFFFFu, end, 31);
        if (l.b - k0 <= 32u) break;
      }
    }
  }
}
__device__ __forceinline__ void wt_zero(uint8_t* w8, uint32_t from, uint32_t to, uint32_t t, uint32_t nt) {
  for (uint32_t k = from + 16u * t; k < to; k += 16u * nt) *reinterpret_cast<uint4*>(w8 + k) = uint4{0, 0, 0, 0};
}
/* the window's n bytes from `pad` on to gbase[pad..]: the 16-byte multiples in the middle leave with one bulk copy, the odd bytes at both
 * ends with plain stores. All threads, behind a barrier; thread 0 waits until the window has been read. */
template <uint32_t THREADS>
__device__ __forceinline__ void wt_copy_out(uint8_t* gbase, const uint8_t* win, uint32_t pad, uint32_t n, uint32_t tid) {
  const uint32_t end = pad + n, lo16 = (pad + 15u) & ~15u, hi16 = end & ~15u;
  if (hi16 > lo16) {
    if (tid == 0) { bulk_s2g(gbase + lo16, win + lo16, hi16 - lo16); bulk_s2g_wait_read(); }
    if (tid >= 32 && tid < 32 + (lo16 - pad)) gbase[pad + tid - 32] = win[pad + tid - 32];
    if (tid >= 64 && tid < 64 + (end - hi16)) gbase[hi16 + tid - 64] = win[hi16 + tid - 64];
  } else {
    for (uint32_t b = pad + tid; b < end; b += THREADS) gbase[b] = win[b];
  }
}

/* The tile's text has `total` bytes: where it goes (sh.base), and whether it fits (sh.ok). Warp 0. */
__device__ __forceinline__ void wt_find_place(const WTileArgs& a, WtShared& sh, uint32_t tile, unsigned long long total, uint32_t lane) {
  if (lane == 0) {
    st_relaxed_u64(&a.agg[tile], TS_VALID | total);
    if (tile == 0) st_relaxed_u64(&a.inc[tile], TS_VALID | total);
  }
  unsigned long long excl = 0;
  const bool ok = lookback_u64(a.agg, a.inc, &a.w.res->timeout, a.spin_limit_ns, tile, lane, &excl);
  if (lane == 0) {
    if (tile != 0 && ok) st_relaxed_u64(&a.inc[tile], TS_VALID | (excl + total));
    const bool fits = (a.w.array ? 1u : 0u) + excl + total <= a.w.cap; /* (the opening bracket) */
    if (ok && !fits) a.w.res->ok = 0;
    if (tile == a.ntiles - 1) a.w.res->out_bytes = excl + total; /* text bytes of all records */
    sh.base = excl;
    sh.ok = ok && fits;
  }
}
/* cycles per phase: sizes, look-back, text into the window, copy-out */
__device__ __forceinline__ void wt_note_cycles(DevResult* res, long long c0, long long c1, long long c2, long long c3) {
  const long long c4 = clock64();
  atomicAdd(&res->phase_cycles[0], (unsigned long long)(c1 - c0));
  atomicAdd(&res->phase_cycles[1], (unsigned long long)(c2 - c1));
  atomicAdd(&res->phase_cycles[2], (unsigned long long)(c3 - c2));
  atomicAdd(&res->phase_cycles[3], (unsigned long long)(c4 - c3));
}
/* A tile on the general road: a record per thread, those of one model side by side; the warps measure and write what the threads leave. The text goes
 * through a window behind the list of that, if it fits, else straight to global memory. Out of line, like the next one: few tiles come here.
 * 300 MB against a record per thread with all of its strings (kernel, us): Users of 72 KB 30 200 -> 430, of 1.2 MB 67 600 -> 425, Pets of 3000 short
 * strings 31 700 -> 1 230; 100 k Users of which one in a thousand has 96 KB 6 270 -> 117; 300 k records of three models in the caller's own order 490 -> 260, with escapes 590 -> 355 (and 240 and 435 in tiles of 128
 * records of 128 threads, five to an SM, whose strings were looked over for escapes by a kernel of their own, 40 us more). */
template <int SCHEMA, uint32_t THREADS>
__device__ __noinline__ void wt_general_tile(const WTileArgs& a, WtShared& sh, uint8_t* smem, uint64_t rec0, uint32_t nrec, uint32_t tile, long long c0) {
  constexpr uint32_t WARPS = THREADS / 32u;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, ngroups = wt_groups<SCHEMA>(sh);
  WtLater* const e = reinterpret_cast<WtLater*>(smem);
  if (tid < nrec) sh.bytes[tid] = 0;
  __syncthreads();
  bool esc = false; /* a byte has to be escaped, but for what is left to the warps */
  for (uint32_t u = warp; u < ngroups; u += WARPS) {
    const WtGroup g = wt_group<SCHEMA>(sh, u);
    const uint32_t rec = wt_record<SCHEMA>(sh, g, lane);
    if (rec == WT_NONE) continue;
    const unsigned long long n = wt_general_any<SCHEMA, false>(&a.w.cols, g.model, wt_row<SCHEMA>(a.w.cols, rec0 + rec), a.w.inclusion, a.w.hexa, nullptr, 0, &sh, e, WT_LATERS, rec, false);
    sh.bytes[rec] = n & ~TS_VALID;
    esc = esc || n >> 63;
  }
  const bool plain = !__syncthreads_or((int)esc);
  const uint32_t nlater = sh.nlater < WT_LATERS ? sh.nlater : WT_LATERS;
  wt_measure_later(&a.w.cols, sh, e, nlater, a.w.inclusion, true, warp, WARPS, lane);
  __syncthreads();
  const unsigned long long len = tid < nrec ? sh.bytes[tid] : 0ull;
  unsigned long long at = warp_incl_scan(len), total = 0;
  if (lane == 31) sh.wsum8[warp] = at;
  at -= len;
  __syncthreads();
  const long long c1 = clock64();
  for (uint32_t q = 0; q < WARPS; ++q) { const unsigned long long v = sh.wsum8[q]; if (q < warp) at += v; total += v; }
  if (tid < nrec) sh.bytes[tid] = at; /* where it starts */
  if (warp == 0) wt_find_place(a, sh, tile, total, lane);
  __syncthreads();
  const long long c2 = clock64();
  if (!sh.ok) return;
  uint8_t* const out0 = a.w.out + (a.w.array ? 1 : 0) + sh.base;
  constexpr uint32_t win = WT_LATERS * (uint32_t)sizeof(WtLater);
  static_assert(win % 16u == 0 && win + WT_MIN_WINDOW <= 8192u, "the smallest tile has a window");
  const bool inside = total + 48u <= a.smem - win;
  const uint32_t pad = (uint32_t)(reinterpret_cast<uintptr_t>(out0) & 15u);
  for (uint32_t u = warp; u < ngroups; u += WARPS) {
    const WtGroup g = wt_group<SCHEMA>(sh, u);
    const uint32_t rec = wt_record<SCHEMA>(sh, g, lane);
    if (rec != WT_NONE) (void)wt_general_any<SCHEMA, true>(&a.w.cols, g.model, wt_row<SCHEMA>(a.w.cols, rec0 + rec), a.w.inclusion, a.w.hexa, (inside ? smem + win + pad : out0) + sh.bytes[rec], a.w.array ? ',' : '\n', &sh, e, WT_LATERS, rec, plain);
  }
  __syncthreads();
  wt_write_later(&a.w.cols, e, nlater, a.w.inclusion, a.w.hexa, warp, WARPS, lane);
  fence_async_smem();
  __syncthreads();
  const long long c3 = clock64();
  if (inside) wt_copy_out<THREADS>(out0 - pad, smem + win, pad, (uint32_t)total, tid);
  __syncthreads();
  if (tid == 0) wt_note_cycles(a.w.res, c0, c1, c2, c3);
}
/* One record of a staged tile whose text has no window: the same steps, straight to dst. w8: `bytes` of shared memory that are free. */
template <int SCHEMA, uint32_t WARPS>
__device__ __noinline__ void wt_general_one(const WTileArgs& a, WtShared& sh, uint8_t* w8, uint32_t bytes, uint64_t i, uint32_t rec, uint8_t* dst) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, most = bytes / (uint32_t)sizeof(WtLater), cap = most < WT_LATERS ? most : WT_LATERS;
  WtLater* const e = reinterpret_cast<WtLater*>(w8);
  uint32_t model = SCHEMA - 1u; /* thread 0's */
  bool plain = true;
  if (tid == 0) {
    if constexpr (SCHEMA == PJ_SCHEMA_MIXED) { const uint32_t type = colp<uint8_t>(&a.w.cols, PJ_COL_REC_TYPE)[i]; model = type == PJ_TYPE_PET ? 0u : (type == PJ_TYPE_ORDER ? 1u : 2u); }
    sh.nlater = 0;
    plain = !(wt_general_any<SCHEMA, false>(&a.w.cols, model, wt_row<SCHEMA>(a.w.cols, i), a.w.inclusion, a.w.hexa, nullptr, 0, &sh, e, cap, rec, false) >> 63);
  }
  __syncthreads();
  const uint32_t nlater = sh.nlater < cap ? sh.nlater : cap;
  wt_measure_later(&a.w.cols, sh, e, nlater, a.w.inclusion, false, warp, WARPS, lane);
  __syncthreads();
  if (tid == 0) (void)wt_general_any<SCHEMA, true>(&a.w.cols, model, wt_row<SCHEMA>(a.w.cols, i), a.w.inclusion, a.w.hexa, dst, a.w.array ? ',' : '\n', &sh, e, cap, rec, plain);
  __syncthreads();
  wt_write_later(&a.w.cols, e, nlater, a.w.inclusion, a.w.hexa, warp, WARPS, lane);
  __syncthreads();
}

template <int SCHEMA, uint32_t THREADS = WtT<SCHEMA>::threads>
__global__ void __launch_bounds__(THREADS, THREADS == WtT<SCHEMA>::threads ? WtT<SCHEMA>::blocks : WT_SHORT_BLOCKS) k_write_tile(const __grid_constant__ WTileArgs a) {
  constexpr uint32_t WARPS = THREADS / 32u;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ __align__(16) WtShared sh;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (tid == 0) { sh.tile = atomicAdd(a.ticket, 1u); for (uint32_t k = 0; k < 3u; ++k) mbar_init(&sh.mbar[k], 1u); sh.odd = 0; sh.nesc = 0; sh.ok = 0; sh.nhit = 0; sh.flight = 0; sh.longs = 0; sh.nlater = 0; }
  __syncthreads();
  const uint32_t tile = sh.tile;
  if (tile >= a.ntiles) return;
  const long long c0 = clock64();
  const uint64_t rec0 = (uint64_t)tile * a.recs;
  const uint32_t nrec = rec0 >= a.w.n ? 0u : (a.w.n - rec0 < a.recs ? (uint32_t)(a.w.n - rec0) : a.recs);
  if constexpr (SCHEMA == PJ_SCHEMA_MIXED) wt_sort(a, sh, rec0, nrec, tid);
  else if (tid == 0) { sh.row0[SCHEMA - 1] = rec0; sh.cnt[SCHEMA - 1] = nrec; }
  __syncthreads();
  if (warp == 0) wt_stage<SCHEMA>(a, sh, smem, lane);
  __syncthreads();
  WtRead x;
  x.incl = a.w.inclusion; x.hexa = a.w.hexa; x.dirty = x.later = x.many = false;
  bool odd = sh.odd != 0;
  const uint32_t ngroups = wt_groups<SCHEMA>(sh);
  if (sh.flight) {
    bool landed = true;
    if (warp == 0)
      for (uint32_t k = 0; k < 3u; ++k) if ((sh.flight >> k) & 1u) landed = mbar_wait_bounded(&sh.mbar[k], 0, a.spin_limit_ns) && landed;
    if (__syncthreads_or(!landed)) {
      if (tid == 0) { /* (the copies still write here) */
        atomicExch(&a.w.res->timeout, 1u);
        for (uint32_t k = 0; k < 3u; ++k) if ((sh.flight >> k) & 1u) (void)mbar_wait_bounded(&sh.mbar[k], 0, a.spin_limit_ns);
      }
      return;
    }
  }
  if (!odd) {
    const uint32_t b0 = sh.text >> 4, b1 = sh.stage >> 4;
    bool bad = false;
    uint32_t any = 0;
    for (uint32_t b = b0 + tid; b < b1; b += THREADS) {
      const uint4 v = *reinterpret_cast<const uint4*>(smem + 16u * b);
      if (word_needs_escape(v.x) | word_needs_escape(v.y) | word_needs_escape(v.z) | word_needs_escape(v.w)) {
        const uint32_t k = atomicAdd(&sh.nhit, 1u);
        if (k < WT_HITS) sh.hit[k] = (uint16_t)b;
        any = 1;
      }
    }
    if (__syncthreads_or((int)any)) {
      x.dirty = true;
      uint32_t* ex = wt_extras(sh, smem); /* (the window begins behind them) */
      if (tid == 0) sh.win = (sh.extra + 4u * sh.nstr + 15u) & ~15u;
      for (uint32_t k = tid; k < sh.nstr; k += THREADS) ex[k] = 0;
      __syncthreads();
      x.many = sh.nhit > WT_HITS;
      if (x.many) bad = wt_count_strings(sh, smem, warp, WARPS, lane);
      else for (uint32_t k = warp; k < sh.nhit; k += WARPS) wt_count_block(sh, smem, sh.hit[k], lane);
      __syncthreads();
    }
    if constexpr (SCHEMA == PJ_SCHEMA_PET || SCHEMA == PJ_SCHEMA_MIXED) {
      const uint32_t npet = (sh.cnt[0] + 31u) / 32u;
      for (uint32_t u = warp; u < 2u * npet; u += WARPS) {
        const WtGroup g = wt_group<SCHEMA>(sh, u >> 1);
        if (u & 1u) wt_sum_items<SCHEMA, 1>(x, sh, smem, g, lane, bad); else wt_sum_items<SCHEMA, 0>(x, sh, smem, g, lane, bad);
      }
      __syncthreads();
    }
    for (uint32_t u = warp; u < ngroups; u += WARPS) {
      const WtGroup g = wt_group<SCHEMA>(sh, u);
      if constexpr (SCHEMA == PJ_SCHEMA_PET || SCHEMA == PJ_SCHEMA_MIXED) if (g.model == 0) wt_size_records<SCHEMA, OBJ_PET>(x, sh, smem, g, lane, bad);
      if constexpr (SCHEMA == PJ_SCHEMA_ORDER || SCHEMA == PJ_SCHEMA_MIXED) if (g.model == 1) wt_size_records<SCHEMA, OBJ_ORDER>(x, sh, smem, g, lane, bad);
      if constexpr (SCHEMA == PJ_SCHEMA_USER || SCHEMA == PJ_SCHEMA_MIXED) if (g.model == 2) wt_size_records<SCHEMA, OBJ_USER>(x, sh, smem, g, lane, bad);
    }
    odd = __syncthreads_or((int)bad) != 0;
    x.later = x.dirty || sh.longs;
  }
  if (odd) { wt_general_tile<SCHEMA, THREADS>(a, sh, smem, rec0, nrec, tile, c0); return; }
  /* where the records start */
  const uint32_t len = tid < nrec ? sh.pos[tid] : 0u;
  uint32_t at = warp_incl_scan(len);
  if (lane == 31) sh.wsum[warp] = at;
  at -= len;
  __syncthreads();
  const long long c1 = clock64();
  uint32_t total = 0;
#pragma unroll
  for (uint32_t q = 0; q < WARPS; ++q) { const uint32_t v = sh.wsum[q]; if (q < warp) at += v; total += v; }
  if (tid < nrec) sh.pos[tid] = at;
  if (tid == 0) sh.pos[nrec] = total;
  const uint32_t win = sh.win, room = a.smem - win - 48u; /* (the last word and the output's alignment) */
  if (warp == 0) wt_find_place(a, sh, tile, total, lane);
  else wt_zero(smem, win, win + 32u + (total < room ? total : room), tid - 32u, THREADS - 32u);
  __syncthreads();
  const long long c2 = clock64();
  if (!sh.ok) return;
  uint8_t* const out0 = a.w.out + (a.w.array ? 1 : 0) + sh.base; /* where the tile's text starts */
  const uint32_t after = a.w.array ? (uint32_t)',' : (uint32_t)'\n';
  long long c3 = c2;
  uint32_t ra = 0;
  while (ra < nrec) { /* a window of records at a time; mostly all of them */
    const uint32_t start = sh.pos[ra];
    uint32_t rb = nrec;
    if (total - start > room) { /* the records whose text ends inside the window */
      uint32_t lo = ra, hi = nrec;
      while (lo + 1u < hi) { const uint32_t mid = (lo + hi) >> 1; if (sh.pos[mid] - start <= room) lo = mid; else hi = mid; }
      rb = lo - ra > 32u ? lo - (lo - ra) % 32u : lo; /* whole groups */
    }
    uint8_t* const dst0 = out0 + start;
    if (rb == ra) { wt_general_one<SCHEMA, WARPS>(a, sh, smem + win, room + 48u, rec0 + ra, ra, dst0); ++ra; continue; } /* no window for this one */
    const uint32_t pad = (uint32_t)(reinterpret_cast<uintptr_t>(dst0) & 15u), bytes = sh.pos[rb] - start;
    /* the window mirrors the output's alignment: window byte k goes to (dst0 - pad)[k] */
    if (ra) { wt_zero(smem, win, win + 32u + bytes, tid, THREADS); if (tid == 0) sh.nesc = 0; __syncthreads(); }
    const uint32_t at0 = win + pad - start;
    /* the units of all groups, the long ones first: a unit's number turns with its group, so that a warp's are not all of one kind */
    constexpr uint32_t KINDS = SCHEMA == PJ_SCHEMA_PET || SCHEMA == PJ_SCHEMA_MIXED ? 4u : 2u;
    const bool single = KINDS == 4u && ngroups == 1u; /* a tile of long lists: their elements are spread over the warps */
    constexpr uint32_t PARTS = (WARPS - 2u) / 2u;
    for (uint32_t u = warp; u < (single ? 2u + 2u * PARTS : KINDS * ngroups); u += WARPS) {
      const WtGroup g = wt_group<SCHEMA>(sh, single ? 0u : u / KINDS);
      const uint32_t k = single ? (u < 2u ? u : 2u + (u & 1u)) : (u + u / KINDS) % KINDS, part = single && u >= 2u ? (u - 2u) / 2u : 0u, parts = single ? PARTS : 1u;
      if constexpr (SCHEMA == PJ_SCHEMA_PET || SCHEMA == PJ_SCHEMA_MIXED) if (g.model == 0) wt_unit<SCHEMA, OBJ_PET>(x, sh, smem, g, k, part, parts, lane, ra, rb, at0, after);
      if constexpr (SCHEMA == PJ_SCHEMA_ORDER || SCHEMA == PJ_SCHEMA_MIXED) if (g.model == 1) wt_unit<SCHEMA, OBJ_ORDER>(x, sh, smem, g, k, part, parts, lane, ra, rb, at0, after);
      if constexpr (SCHEMA == PJ_SCHEMA_USER || SCHEMA == PJ_SCHEMA_MIXED) if (g.model == 2) wt_unit<SCHEMA, OBJ_USER>(x, sh, smem, g, k, part, parts, lane, ra, rb, at0, after);
    }
    if (x.later) {
      __syncthreads();
      const uint32_t n = sh.nesc < WT_ESC ? sh.nesc : WT_ESC;
      for (uint32_t k = warp; k < n; k += WARPS) if (sh.esc[k].n >> 31) wt_escape(smem, sh.esc[k].at, sh.esc[k].n & 0x7FFFFFFFu, sh.esc[k].dst, x.hexa, lane);
      if (sh.longs)
        for (uint32_t k = 0; k < n; ++k) {
          const WtEsc l = sh.esc[k];
          if (l.n >> 31 || (l.n <= WT_PART && k % WARPS != warp)) continue;
          for (uint32_t from = (warp + WARPS - k % WARPS) % WARPS * WT_PART; from < l.n; from += WT_PART * WARPS) wt_copy(smem, l.at + from, l.n - from < WT_PART ? l.n - from : WT_PART, l.dst + from, lane);
        }
    }
    fence_async_smem();
    __syncthreads();
    c3 = clock64();
    wt_copy_out<THREADS>(dst0 - pad, smem + win, pad, bytes, tid);
    ra = rb;
    if (ra < nrec) __syncthreads();
  }
  __syncthreads();
  if (tid == 0) wt_note_cycles(a.w.res, c0, c1, c2, c3);
}

/* ---- host: the schema's columns as the tiles stage them ---------------------------------------------------------------- */
/* How many wt_add_columns() makes of OBJ's properties from I on: with an element per row of the root's (ROWS), or the others. */
template <int OBJ, int LEVEL, bool ROWS, int I = -1>
PJ_CX uint32_t wt_count_columns() {
  constexpr uint32_t own = (LEVEL == 0) == ROWS; /* a column that has an element wherever OBJ has one */
  if constexpr (I < 0) return own + wt_count_columns<OBJ, LEVEL, ROWS, 0>(); /* presence */
  else if constexpr (I >= CObj<OBJ>::N) return 0;
  else {
    constexpr uint32_t kind = CObj<OBJ>::f[I].kind;
    uint32_t n = 0;
    if constexpr (kind == K_DATETIME) n = 3u * own;
    else if constexpr (kind == K_STR) n = own + !ROWS;
    else if constexpr (kind == K_OBJ) n = wt_count_columns<CObj<OBJ>::f[I].child, LEVEL, ROWS>();
    else if constexpr (kind == K_LIST_STR) n = own + 2u * !ROWS;
    else if constexpr (kind == K_LIST_OBJ) n = own + wt_count_columns<CObj<OBJ>::f[I].child, 2, ROWS>();
    else n = own;
    return n + wt_count_columns<OBJ, LEVEL, ROWS, I + 1>();
  }
}
static constexpr uint32_t WT_ROW_COLS = wt_count_columns<OBJ_PET, 0, true>() + wt_count_columns<OBJ_ORDER, 0, true>() + wt_count_columns<OBJ_USER, 0, true>();
static constexpr uint32_t WT_OTHER_COLS = wt_count_columns<OBJ_PET, 0, false>() + wt_count_columns<OBJ_ORDER, 0, false>() + wt_count_columns<OBJ_USER, 0, false>();
static_assert(WT_ROW_COLS <= 32u && WT_OTHER_COLS <= 32u, "wt_stage() takes a column per lane");
static_assert(WT_ROW_COLS + WT_OTHER_COLS <= WT_COLS, "room for the columns");
inline void wt_add_columns(const Schema& S, const ObjDesc& O, const DevCols& cols, uint32_t model, uint32_t level, bool rows, WTileArgs* a) {
  auto add = [&](uint32_t col, uint32_t shift, uint32_t lev, uint32_t plus, int off) {
    if ((lev == 0 && off < 0) != rows) return;
    WtCol& c = a->col[a->ncol++];
    c.p = (const uint8_t*)cols.ptr[col]; c.off = off >= 0 ? (const uint32_t*)cols.ptr[off] : nullptr;
    c.col = (uint8_t)col; c.shift = (uint8_t)shift; c.model = (uint8_t)model; c.level = (uint8_t)lev; c.plus = (uint8_t)plus;
  };
  add(O.present_col, 0, level, 0, -1);
  for (int i = 0; i < (int)O.nfields; ++i) {
    const FieldDesc& F = O.f[i];
    switch (F.kind) {
      case K_I64: add(F.col, 3, level, 0, -1); break;
      case K_I32: add(F.col, 2, level, 0, -1); break;
      case K_BOOL: case K_ENUM: add(F.col, 0, level, 0, -1); break;
      case K_DATETIME: add(F.col, 3, level, 0, -1); add(F.col + 1u, 2, level, 0, -1); add(F.col + 2u, 2, level, 0, -1); break;
      case K_STR: add(F.col, 2, level, 1, -1); add(F.col + 1u, 0, level, 0, F.col); break;
      case K_OBJ: wt_add_columns(S, S.obj[F.child], cols, model, level, rows, a); break;
      case K_LIST_STR: add(F.col, 2, level, 1, -1); add(F.col + 1u, 2, 1, 1, -1); add(F.col + 2u, 0, 1, 0, F.col + 1); a->list[0] = (const uint32_t*)cols.ptr[F.col]; break;
      case K_LIST_OBJ: add(F.col, 2, level, 1, -1); a->list[1] = (const uint32_t*)cols.ptr[F.col]; wt_add_columns(S, S.obj[F.child], cols, model, 2, rows, a); break;
      default: break;
    }
  }
}
inline void wt_columns(const Schema& S, uint32_t schema, const DevCols& cols, WTileArgs* a) {
  const uint32_t roots[3] = {OBJ_PET, OBJ_ORDER, OBJ_USER};
  a->ncol = 0;
  a->list[0] = a->list[1] = nullptr;
  for (int rows = 1; rows >= 0; --rows) {
    for (uint32_t m = 0; m < 3; ++m) if (schema == PJ_SCHEMA_MIXED || schema == m + 1) wt_add_columns(S, S.obj[roots[m]], cols, m, 0, rows != 0, a);
    if (rows) a->nrow = a->ncol;
  }
}

}  // namespace pj
#endif

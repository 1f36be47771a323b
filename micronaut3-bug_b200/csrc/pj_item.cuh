/*
 * pj_item.cuh — k_parse_items<SCHEMA>: JSON records to typed columns in one kernel and one pass over HBM, with the work
 * spread over bytes, strings and fields instead of records.
 *
 * One thread block = one tile of the input, staged in shared memory by one bulk copy. A tile owns the lines (in array
 * framing: the extents) whose preceding separator lies in it and follows its last one to its end. The steps:
 *
 *  1. item_index: 144 bytes per thread. Byte-parallel masks of quotes and control characters give the positions of all
 *     quotes of the tile in order: string k = (open, close); and the lines: first byte and first string. Backslashes, bytes
 *     beyond ASCII and control characters take extra work only where they are; strings with escapes are decoded in place.
 *  2. item_walk: one line per thread. A record as a serialiser writes it is walked property by property; every string's end
 *     is known, so nothing is scanned, and nothing is decoded either: REFERENCES to the values' text go to the line's row.
 *  3. item_pack: the lines the walk did not recognise (blanks, another order of keys, null, errors), 32 strings at a time,
 *     a string and the gap behind it per lane. The punctuation of a gap alone tells where in the record it stands (`}],`
 *     closes an element, its list and is followed by a key of the root; `,` and `:` leave the place as it is), so the object a
 *     string lies in is what the nearest telling gap before it left: one ballot and one shuffle instead of a walk. Keys are
 *     looked up in a hash table.
 *  4. item_value: groups of 32 lines and one field: the references are decoded by lanes that all do the same.
 *  5. Counts per record are added up, ONE decoupled look-back over the earlier tiles gives the tile's place in every
 *     column and arena, and the columns are written, again by groups of 32 lines.
 *
 * The steps detect every deviation from a valid record of the model; the common failures (wrong JSON type, unknown
 * literal, bad date-time, missing property, record ending inside a string) are reported with the exact parser's kind
 * and offset, because the smallest offset of a record's deviations is its first failure. Any other deviation sends the
 * record to the exact parser (pj_core.cuh); a record that one accepts (unknown keys with nested values, repeated keys, ...) stands apart:
 * its counts take part in the sums, and it is parsed once more to write its columns (item_emit_apart). Does the tile not fit
 * the shared memory laid out for it (many more lines or strings than its bytes suggest), every thread of the block walks lines
 * where they lie (item_slow_tile); a record that runs out of the window is read where it lies as well.
 */
#ifndef PJ_ITEM_CUH
#define PJ_ITEM_CUH

#include "pj_dev.cuh"
#include "pj_fast.cuh"
#include "pj_index.cuh"
#include "pj_array.cuh"
#include "pj_item_tables.h"
#include "pj_result.h"
#include "pj_schema_const.cuh"
#include "pj_stream.cuh"

namespace pj {

#ifndef PJ_IT_BLOCKS
#define PJ_IT_BLOCKS 3 /* resident blocks per SM the kernel is compiled for */
#endif
static constexpr uint32_t IT_BLOCKS = PJ_IT_BLOCKS;
#ifndef PJ_IT_THREADS
#define PJ_IT_THREADS 256
#endif
static constexpr uint32_t IT_THREADS = PJ_IT_THREADS;
static constexpr uint32_t IT_WARPS = IT_THREADS / 32;
static constexpr uint32_t IT_BLK = 9;                /* 16-byte blocks a thread indexes per step: odd, so that a warp's 128-bit loads are free of bank conflicts */
static constexpr uint32_t IT_SPAN = IT_BLK * 16;
static constexpr uint32_t IT_SPANW = (IT_SPAN + 31) / 32;
static constexpr uint32_t IT_STEP = IT_THREADS * IT_SPAN; /* bytes the block indexes per step */
static constexpr uint32_t IT_FRONT = 32;             /* bytes before the window that may be read (and mean nothing) */
static constexpr uint32_t IT_PAD = IT_SPAN + 16;               /* ... and behind it */
static constexpr uint32_t IT_MAX_LINES = IT_THREADS; /* lines per tile */
static constexpr uint32_t IT_MAX_STRS = 4096;        /* strings per tile */
static constexpr uint32_t IT_MAX_SPECIAL = 512;     /* strings per tile that need a closer look and are kept in a list */
static constexpr uint32_t IT_MAX_WIN = 65536 - 64;   /* window offsets are 16-bit */
static constexpr uint32_t IT_STAGE = 256;            /* words of a warp to put strings together in */
static constexpr uint32_t IT_MAX_DYN_SMEM = 200 * 1024; /* dynamic shared memory of a block */
static constexpr uint32_t IT_NONE = 0xFFFFFFFFu;

static constexpr uint32_t IT_NLB = 16;    /* look-back counters: the NSLOT counters and the record count */
static constexpr uint32_t IT_REC = NSLOT; /* number of the record counter */
static_assert(NSLOT + 1 == IT_NLB, "one more than counters");
static constexpr uint32_t IT_AGG_BITS = 20; /* a tile's own totals are published three to a word */
struct ItemTile {
  unsigned long long inc[IT_NLB];
  unsigned long long agg[6];
  unsigned long long pad[2];
};
static_assert(sizeof(ItemTile) == 192, "whole sectors");

struct ItemArgs {
  const uint8_t* in;
  uint64_t len, limit, goff;
  uint32_t is_first, is_last;
  uint32_t tile_bytes, ntiles;
  uint32_t win_bytes;  /* bytes staged per tile: the tile and what its last record may need behind it */
  uint32_t str_words;  /* 32-bit words for strings */
  uint32_t row_cap;    /* rows of lines */
  uint32_t opts;       /* PJ_OPT_* bits that change a rule */
  unsigned long long spin_limit_ns;
  const uint64_t* sep; /* array framing: one bit per input byte, set for `[`, the commas and `]` that delimit records; else null */
  ItemTile* tiles;
  uint32_t* ticket;
  DevResult* res;
  const DevResult* prev;    /* totals of the pieces of the same call parsed by earlier launches (null: none) */
  const uint32_t* looks;    /* several models: [ND_LOOKS] line feeds in pieces of the input (null: whatever it is) */
  uint64_t slot_cap[NSLOT]; /* largest total per slot the caller's buffers can take */
  uint64_t rec_cap;         /* records the per-record and row-indexed buffers can take */
  FinalizePlan plan;
  DevCols cols;
};

/* counter slots a schema uses */
template <int SCHEMA>
struct ItemSlots {
  static constexpr uint32_t lo = SCHEMA == PJ_SCHEMA_PET ? (uint32_t)SLOT_PET_CAT_NAME : (SCHEMA == PJ_SCHEMA_USER ? (uint32_t)SLOT_USR_STR0 : 0u);
  static constexpr uint32_t hi = SCHEMA == PJ_SCHEMA_PET ? (uint32_t)SLOT_USR_STR0 : (SCHEMA == PJ_SCHEMA_ORDER ? 0u : (uint32_t)NSLOT);
  static constexpr uint32_t mask = ((hi > lo ? ((1u << hi) - (1u << lo)) : 0u)) | (1u << IT_REC);
  static constexpr uint32_t count = (hi > lo ? hi - lo : 0u) + 1u;
  static constexpr uint32_t nagg = (count + 2u) / 3u;
  static constexpr bool lists = SCHEMA == PJ_SCHEMA_PET || SCHEMA == PJ_SCHEMA_MIXED;
};
static_assert((ItemSlots<PJ_SCHEMA_MIXED>::nagg) <= 6, "packed totals fit");

/* shared memory of a tile: what the dynamic part holds, from a 16-byte aligned base */
struct ItemLayout { uint32_t win, strs, rows, total; };
PJ_HD ItemLayout item_layout(uint32_t win_bytes, uint32_t str_words, uint32_t row_cap, uint32_t stride) {
  ItemLayout l;
  l.win = IT_FRONT;
  l.strs = (l.win + win_bytes + IT_PAD + 15u) & ~15u;
  l.rows = (l.strs + str_words * 4u + 15u) & ~15u;
  l.total = l.rows + row_cap * stride * 4u;
  return l;
}

struct ItemShared {
  union { /* what reads the input, and what writes the columns */
    struct {
      __align__(16) uint32_t key[IT_SLOTS][8];
      __align__(16) ItGapEntry gap[IG_SLOTS];
      uint32_t field[3][IT_SLOTS];
      uint32_t broken[IT_MAX_STRS / 32]; /* strings that are not valid */
      uint16_t special_list[IT_MAX_SPECIAL];
    };
    uint32_t stage[IT_WARPS][IT_STAGE];
  };
  uint32_t special[IT_MAX_STRS / 32 + 1u]; /* per string: it holds a backslash, a control character or a byte beyond ASCII; later: it was decoded in place */
  uint32_t line[IT_MAX_LINES + 1];         /* window offset of a line's first byte | strings before it << 16 */
  uint32_t oddline[IT_MAX_LINES / 32];     /* lines the walk leaves alone from the start */
  uint32_t movedline[IT_MAX_LINES / 32];   /* lines with a string that was decoded in place or is not valid */
  uint32_t oddmask[IT_WARPS];              /* lines the walk did not recognise */
  uint8_t owner[IT_WARPS][32];
  uint8_t perm[IT_THREADS], cls[4][IT_WARPS]; /* mixed streams: lines by model */
  uint32_t csum[IT_NLB][IT_WARPS];         /* counters: sums per 32 lines, then exclusive prefixes */
  uint32_t tot[IT_NLB], base[IT_NLB];
  uint32_t recs[IT_WARPS];                 /* lines that are records */
  uint32_t wsum[IT_WARPS], wmin[3][IT_WARPS];
  uint32_t nspecial, odd;                  /* odd: some record ends inside a string */
  uint32_t open_end;                       /* the last line runs out of the window */
  uint32_t nstr, nline, stop;              /* strings, lines, last separator */
  uint32_t free_word;                      /* first free word behind the strings */
  uint32_t ndense;                         /* lines the dense walk took */
  uint32_t ok, slow, tile, next, apart;    /* apart: a record of the tile stands apart */
  uint32_t aside;                          /* the input is left to k_parse_stream */
  unsigned long long mbar;
};

/* ---- look-back --------------------------------------------------------------------------------------------------
 * Tiles take their number from an atomic ticket, so every predecessor of a running tile is running or done. A tile
 * publishes its own totals (three to a 64-bit word, when they fit 20 bits) as soon as its records are sized, and its inclusive
 * totals once it has the sum of all before it. One round looks at 32 predecessors: each lane reads one tile's own totals and
 * the first of its inclusive words; the nearest tile with inclusive totals then gives the rest in one coalesced read.
 * Every word carries its own valid bit; every wait is bounded. */
template <int SCHEMA>
__device__ __forceinline__ bool item_lookback(const ItemArgs& a, uint32_t tile, uint32_t lane, uint32_t* excl) {
  using SL = ItemSlots<SCHEMA>;
#pragma unroll
  for (uint32_t k = 0; k < SL::count; ++k) excl[k] = 0;
  int64_t j = (int64_t)tile - 1;
  const unsigned long long t0 = global_ns();
  unsigned polls = 0, rounds = 0;
  auto give_up = [&]() -> bool {
    uint32_t g = 0;
    if (lane == 0) g = (global_ns() - t0 > a.spin_limit_ns) || *(volatile uint32_t*)&a.res->timeout;
    g = __shfl_sync(0xFFFFFFFFu, g, 0);
    if (g && lane == 0) atomicExch(&a.res->timeout, 1u);
    return g != 0;
  };
  while (j >= 0) {
    const int64_t mine = j - lane;
    unsigned long long w[SL::nagg];
    uint32_t first_inc;
    for (;;) {
      bool has_inc = mine < 0, has_agg = true; /* tiles before the first count as "inclusive, zero" */
#pragma unroll
      for (uint32_t k = 0; k < SL::nagg; ++k) w[k] = TS_VALID;
      if (mine >= 0) {
        has_inc = (ld_relaxed_u64(&a.tiles[mine].inc[0]) & TS_VALID) != 0;
#pragma unroll
        for (uint32_t k = 0; k < SL::nagg; ++k) { w[k] = ld_relaxed_u64(&a.tiles[mine].agg[k]); has_agg = has_agg && (w[k] & TS_VALID); }
      }
      const uint32_t inc_mask = __ballot_sync(0xFFFFFFFFu, has_inc);
      const uint32_t ready_mask = __ballot_sync(0xFFFFFFFFu, has_inc || has_agg);
      first_inc = inc_mask ? (uint32_t)(__ffs((int)inc_mask) - 1) : 32u;
      const uint32_t need = first_inc >= 31 ? 0xFFFFFFFFu : ((2u << first_inc) - 1u);
      if ((ready_mask & need) == need) break;
      ++polls;
      if (give_up()) return false;
      __nanosleep(40);
    }
    ++rounds;
#pragma unroll
    for (uint32_t k = 0; k < SL::count; ++k) {
      const uint32_t v = (uint32_t)(w[k / 3] >> (IT_AGG_BITS * (k % 3))) & ((1u << IT_AGG_BITS) - 1u);
      excl[k] += __reduce_add_sync(0xFFFFFFFFu, lane < first_inc ? v : 0u);
    }
    if (first_inc < 32) {
      const int64_t src = j - first_inc;
      if (src >= 0) {
        unsigned long long v = TS_VALID;
        for (;;) { /* the words of a tile are stored together: this ends at once */
          if (lane < SL::count) v = ld_relaxed_u64(&a.tiles[src].inc[lane]);
          if (__all_sync(0xFFFFFFFFu, (v & TS_VALID) != 0)) break;
          if (give_up()) return false;
        }
#pragma unroll
        for (uint32_t k = 0; k < SL::count; ++k) excl[k] += __shfl_sync(0xFFFFFFFFu, (uint32_t)v, (int)k);
      }
      break;
    }
    j -= 32;
  }
  if (lane == 0 && polls) atomicAdd(&a.res->lookback_polls, (unsigned long long)polls);
  if (lane == 0 && rounds) atomicAdd(&a.res->lookback_rounds, (unsigned long long)rounds);
  return true;
}

/* Warp 0 of a tile whose totals stand in sh.tot[]: publishes them, looks back, publishes the inclusive totals, checks the
 * caller's capacities and leaves in sh.base[] where the tile starts over the whole call and in sh.ok whether to emit. The
 * last tile also leaves the call's totals. */
template <int SCHEMA>
__device__ __forceinline__ void item_resolve(const ItemArgs& a, ItemShared& sh, uint32_t tile, uint32_t lane) {
  using SL = ItemSlots<SCHEMA>;
  ItemTile* me = &a.tiles[tile];
  /* lane k < count holds used counter k */
  const uint32_t slot = lane + 1 == SL::count ? IT_REC : SL::lo + lane;
  const bool have = lane < SL::count;
  const uint32_t mine = have ? sh.tot[slot] : 0u;
  if (tile == 0) { if (have) st_relaxed_u64(&me->inc[lane], TS_VALID | mine); }
  else {
    const bool small = __all_sync(0xFFFFFFFFu, mine < (1u << IT_AGG_BITS));
    const uint32_t m1 = __shfl_down_sync(0xFFFFFFFFu, mine, 1), m2 = __shfl_down_sync(0xFFFFFFFFu, mine, 2);
    if (small && have && lane % 3 == 0)
      st_relaxed_u64(&me->agg[lane / 3], TS_VALID | mine | ((unsigned long long)m1 << IT_AGG_BITS) | ((unsigned long long)m2 << (2 * IT_AGG_BITS)));
  }
  uint32_t excl_all[SL::count];
  const bool ok = item_lookback<SCHEMA>(a, tile, lane, excl_all);
  uint32_t excl = 0;
#pragma unroll
  for (uint32_t k = 0; k < SL::count; ++k) if (lane == k) excl = excl_all[k];
  if (tile != 0 && ok && have) st_relaxed_u64(&me->inc[lane], TS_VALID | (unsigned long long)(excl + mine));
  uint64_t prior = 0; /* what earlier launches of the call produced comes first */
  if (a.prev && have) prior = slot == IT_REC ? a.prev->n_records : a.prev->total[slot];
  const uint64_t before = prior + excl;
  if (have) sh.base[slot] = (uint32_t)before;
  const uint64_t cap = slot == IT_REC ? a.rec_cap : a.slot_cap[have ? slot : 0];
  const uint32_t any_over = __ballot_sync(0xFFFFFFFFu, have && before + mine > cap);
  if (lane == 0) {
    sh.ok = ok && !any_over;
    if (any_over) a.res->over = 1u;
  }
  if (tile == a.ntiles - 1 && have) {
    if (slot == IT_REC) a.res->n_records = before + mine;
    else a.res->total[slot] = before + mine;
  }
}

/* Closing entries of the offset columns, by the last tile of a launch. */
__device__ __forceinline__ void item_close_offsets(const ItemArgs& a, const ItemShared& sh, uint32_t tid) {
  if (tid < a.plan.n) {
    const FinalizeItem it = a.plan.item[tid];
    if (it.sentinel_slot != 0xFF) {
      const uint32_t rs = it.rows_slot == 0xFF ? IT_REC : it.rows_slot;
      colp<uint32_t>(&a.cols, it.col)[(uint64_t)sh.base[rs] + sh.tot[rs]] = sh.base[it.sentinel_slot] + sh.tot[it.sentinel_slot];
    }
  }
}

/* ---- 1. index ------------------------------------------------------------------------------------------------ */
__device__ __forceinline__ uint32_t item_low(int32_t n) { return n <= 0 ? 0u : (n >= 32 ? 0xFFFFFFFFu : ((1u << n) - 1u)); }
/* 0x80 in every byte of w that equals c (c repeated), exactly */
__device__ __forceinline__ uint32_t item_eq4(uint32_t w, uint32_t c) { return ~((((w ^ c) & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | (w ^ c)) & 0x80808080u; }
/* 0x80 per byte of four words as 16 bits */
__device__ __forceinline__ uint32_t item_gather16(uint32_t f0, uint32_t f1, uint32_t f2, uint32_t f3) {
  return (__dp4a(f1, 0x80402010u, __dp4a(f0, 0x08040201u, 0u)) + (__dp4a(f3, 0x80402010u, __dp4a(f2, 0x08040201u, 0u)) << 8)) >> 7;
}
__device__ __forceinline__ uint32_t item_prefix_xor(uint32_t x) {
  x ^= x << 1; x ^= x << 2; x ^= x << 4; x ^= x << 8; x ^= x << 16;
  return x;
}
/* for the shape of the next call's tiles */
__device__ __forceinline__ void item_note_strings(const ItemArgs& a, uint32_t n, uint32_t bytes) { if (bytes > 1024u) atomicMax(&a.res->strs_per_kb, n * 1024u / bytes); }
/* The strings and lines the tile owns. False (for every thread): the tile does not fit, the block has to take the other road. The last line may
 * run out of the window. A record may end
 * inside a string: its separator then counts as the string's closing quote. */
template <bool ARR>
__device__ __forceinline__ bool item_index(const ItemArgs& a, const StreamGeom& g, ItemShared& sh, uint8_t* win, uint32_t* strs, uint32_t tid, uint32_t tile) {
  const uint32_t lane = tid & 31, warp = tid >> 5;
  bool started = !ARR && tile == 0 && a.is_first && a.limit > 0, done = false, fine = true, open_end = false;
  uint32_t start = g.mis, stop = 0, nq = 0, nline = 0;
  const int32_t end_valid = (int32_t)g.hi_valid + (g.to_limit ? 1 : 0), lo_valid = (int32_t)g.lo_valid; /* the end of the input counts as a separator */
  uint16_t* q16 = reinterpret_cast<uint16_t*>(strs);
  if (tid == 0 && started) sh.line[0] = start;
  for (uint32_t o = 0; !done; o += IT_STEP) {
    if ((int32_t)o >= end_valid) { open_end = started; break; } /* the last record runs out of the window */
    if (!started && o >= g.own_end) break;
    const int32_t p0 = (int32_t)(o + IT_SPAN * tid);
    /* quotes, separators, control characters (later: all that takes a closer look), a bit per byte of the thread's */
    uint32_t q[IT_SPANW], t[IT_SPANW], c[IT_SPANW];
    uint32_t bs = 0, hb = 0;
#pragma unroll
    for (uint32_t i = 0; i < IT_SPANW; ++i) q[i] = t[i] = c[i] = 0;
    const uint4* src = reinterpret_cast<const uint4*>(win + p0);
    if (p0 < end_valid) {
#pragma unroll
      for (uint32_t b = 0; b < IT_BLK; ++b) {
        const uint4 v = src[b];
        const uint32_t x[4] = {v.x, v.y, v.z, v.w};
        /* Bytes below 0x23 are few: of them, bit 5 tells the printable ones from the control characters, and of the printable
           ones ( space ! " ) bit 1 tells the quotes. Or-ed up over the words: backslashes, bytes beyond ASCII. */
        uint32_t fq[4], fc[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t low = ~(((x[k] & 0x7F7F7F7Fu) + 0x5D5D5D5Du) | x[k]) & 0x80808080u;
          fq[k] = low & (x[k] << 2) & (x[k] << 6);
          fc[k] = low & ~(x[k] << 2);
          bs |= ~(((x[k] ^ 0x5C5C5C5Cu) & 0x7F7F7F7Fu) + 0x7F7F7F7Fu);
          hb |= x[k];
        }
        q[b >> 1] |= item_gather16(fq[0], fq[1], fq[2], fq[3]) << (16u * (b & 1u));
        c[b >> 1] |= item_gather16(fc[0], fc[1], fc[2], fc[3]) << (16u * (b & 1u));
      }
      if (p0 < lo_valid || p0 + (int32_t)IT_SPAN > end_valid) {
#pragma unroll
        for (uint32_t i = 0; i < IT_SPANW; ++i) {
          const int32_t p = p0 + (int32_t)(32u * i);
          const uint32_t vm = item_low(end_valid - p) & ~item_low(lo_valid - p);
          q[i] &= vm; c[i] &= vm;
        }
      }
      if (ARR) {
        const int64_t bit = (int64_t)g.v0 + p0 - (int64_t)g.mis; /* input offset of the thread's first byte */
        const int64_t nwords32 = (int64_t)((a.len + 31) >> 5);
        const uint32_t* sw = reinterpret_cast<const uint32_t*>(a.sep);
        const int64_t i0 = bit >> 5; /* floor: the first tile may begin a few bytes before the input */
        uint32_t b0 = i0 >= 0 && i0 < nwords32 ? sw[i0] : 0u;
#pragma unroll
        for (uint32_t i = 0; i < IT_SPANW; ++i) {
          const int64_t n = i0 + 1 + (int64_t)i;
          const uint32_t b1 = n >= 0 && n < nwords32 ? sw[n] : 0u;
          const int32_t p = p0 + (int32_t)(32u * i);
          const int32_t room = p0 + (int32_t)IT_SPAN < end_valid ? p0 + (int32_t)IT_SPAN : end_valid;
          t[i] = __funnelshift_r(b0, b1, (uint32_t)(bit & 31)) & item_low(room - p) & ~item_low(lo_valid - p);
          if (g.to_limit && (int32_t)g.hi_valid >= p && (int32_t)g.hi_valid < p + 32 && (int32_t)g.hi_valid < room) t[i] |= 1u << (g.hi_valid - (uint32_t)p);
          c[i] &= ~t[i];
          b0 = b1;
        }
      } else {
#pragma unroll
        for (uint32_t i = 0; i < IT_SPANW; ++i) {
          for (uint32_t m = c[i]; m; m &= m - 1u) {
            const uint32_t b = (uint32_t)__ffs((int)m) - 1u;
            if (win[p0 + (int32_t)(32u * i + b)] == '\n') t[i] |= 1u << b;
          }
          c[i] &= ~t[i];
        }
      }
    }
    /* Escaped quotes, and the bytes that make a string one to decode. A quote is escaped when an odd run of backslashes ends
       before it. */
    const bool my_sp = p0 < end_valid && (((bs | hb) & 0x80808080u) != 0 || (p0 > lo_valid && win[p0 - 1] == '\\'));
    if (__any_sync(0xFFFFFFFFu, my_sp)) {
      if (my_sp) {
#pragma unroll
        for (uint32_t b = 0; b < IT_BLK; ++b) {
          const uint4 v = src[b];
          const uint32_t B = item_gather16(item_eq4(v.x, 0x5C5C5C5Cu), item_eq4(v.y, 0x5C5C5C5Cu), item_eq4(v.z, 0x5C5C5C5Cu), item_eq4(v.w, 0x5C5C5C5Cu));
          const uint32_t H = item_gather16(v.x & 0x80808080u, v.y & 0x80808080u, v.z & 0x80808080u, v.w & 0x80808080u);
          const int32_t p = p0 + (int32_t)(16u * b);
          const uint32_t before = p > lo_valid && win[p - 1] == '\\' ? 1u : 0u;
          for (uint32_t m = (q[b >> 1] >> (16u * (b & 1u))) & ((B << 1) | before) & 0xFFFFu; m; m &= m - 1u) {
            const int32_t at = p + __ffs((int)m) - 1;
            int32_t r = at - 1;
            while (r >= lo_valid && win[r] == '\\' && at - r < 4096) --r;
            if (at - r >= 4096) sh.slow = 1;
            if ((at - 1 - r) & 1) q[b >> 1] &= ~((m & (0u - m)) << (16u * (b & 1u)));
          }
          c[b >> 1] |= (B | H) << (16u * (b & 1u)); /* (only those inside a string will count) */
        }
      }
    }
    /* where the first own line begins and the last one ends */
    {
      uint32_t m0 = IT_NONE, m1 = IT_NONE;
#pragma unroll
      for (int i = (int)IT_SPANW - 1; i >= 0; --i) {
        const int32_t p = p0 + 32 * i;
        const uint32_t own = item_low((int32_t)g.own_end - p), t0 = t[i] & own, t1 = t[i] & ~own;
        if (t0) m0 = (uint32_t)(p + __ffs((int)t0)); /* behind the separator */
        if (t1) m1 = (uint32_t)(p + __ffs((int)t1) - 1);
      }
      m0 = __reduce_min_sync(0xFFFFFFFFu, m0); m1 = __reduce_min_sync(0xFFFFFFFFu, m1);
      if (lane == 0) { sh.wmin[0][warp] = m0; sh.wmin[1][warp] = m1; }
      __syncthreads();
      uint32_t x0 = IT_NONE, x1 = IT_NONE;
#pragma unroll
      for (uint32_t k = 0; k < IT_WARPS; ++k) { const uint32_t y0 = sh.wmin[0][k], y1 = sh.wmin[1][k]; x0 = y0 < x0 ? y0 : x0; x1 = y1 < x1 ? y1 : x1; }
      if (!started && x0 != IT_NONE) { started = true; start = x0; if (tid == 0) sh.line[0] = start; }
      if (!started) { __syncthreads(); continue; }
      int32_t last = 0x7FFFFFFF;
      if (x1 != IT_NONE) { stop = x1; done = true; last = (int32_t)x1 + 1; }
      if (p0 < (int32_t)start || p0 + (int32_t)IT_SPAN > last) {
#pragma unroll
        for (uint32_t i = 0; i < IT_SPANW; ++i) {
          const int32_t p = p0 + (int32_t)(32u * i);
          const uint32_t act = item_low(last - p) & ~item_low((int32_t)start - p);
          q[i] &= act; t[i] &= act; c[i] &= act;
        }
      }
    }
    /* order of the quotes (low half) and separators (high half); twice when some record ends inside a string */
    uint32_t at, total, any = 0;
#pragma unroll
    for (uint32_t i = 0; i < IT_SPANW; ++i) any |= t[i];
    for (uint32_t round = 0;; ++round) {
      uint32_t n = 0;
#pragma unroll
      for (uint32_t i = 0; i < IT_SPANW; ++i) n += (uint32_t)__popc(q[i]) + ((uint32_t)__popc(t[i]) << 16);
      const uint32_t inc = warp_incl_scan(n);
      if (lane == 31) sh.wsum[warp] = inc;
      __syncthreads();
      at = inc - n; total = 0;
#pragma unroll
      for (uint32_t k = 0; k < IT_WARPS; ++k) { const uint32_t x = sh.wsum[k]; if (k < warp) at += x; total += x; }
      if (round) break;
      /* A record that ends inside a string has an odd number of quotes: it changes the parity from separator to separator. */
      const uint32_t n0 = nq + (at & 0xFFFFu);
      uint32_t last = 0, odd = 0; /* parity at the thread's last separator; at any of them */
      if (any) {
        uint32_t m0 = n0;
#pragma unroll
        for (uint32_t i = 0; i < IT_SPANW; ++i) {
          for (uint32_t m = t[i]; m; m &= m - 1u) { last = (m0 + (uint32_t)__popc(q[i] & ((m & (0u - m)) - 1u))) & 1u; odd |= last; }
          m0 += (uint32_t)__popc(q[i]);
        }
      }
      if (!__syncthreads_or((int)odd)) break;
      if (tid == 0) sh.odd = 1;
      const uint32_t has = __ballot_sync(0xFFFFFFFFu, any != 0), par = __ballot_sync(0xFFFFFFFFu, last != 0);
      if (lane == 0) sh.wmin[2][warp] = has ? 2u | ((par >> (31 - __clz((int)has))) & 1u) : 0u;
      __syncthreads();
      uint32_t prev = 0; /* at the separator before the thread's first: even before the step's first one */
#pragma unroll
      for (uint32_t k = 0; k < IT_WARPS; ++k) { const uint32_t x = sh.wmin[2][k]; if (k < warp && x) prev = x & 1u; }
      const uint32_t below = has & ((1u << lane) - 1u);
      if (below) prev = (par >> (31 - __clz((int)below))) & 1u;
      if (any) {
        uint32_t m0 = n0;
#pragma unroll
        for (uint32_t i = 0; i < IT_SPANW; ++i) {
          const uint32_t raw = q[i];
          for (uint32_t m = t[i]; m; m &= m - 1u) {
            const uint32_t bit = m & (0u - m), here = (m0 + (uint32_t)__popc(raw & (bit - 1u))) & 1u;
            if (here != prev) q[i] |= bit; /* closed there */
            prev = here;
          }
          m0 += (uint32_t)__popc(raw);
        }
      }
    }
    {
      const uint32_t n = nq + (total & 0xFFFFu), nl = nline + (total >> 16);
      if (n / 2u + 2u > a.str_words || n / 2u >= IT_MAX_STRS || nl > IT_MAX_LINES || nl > a.row_cap) {
        if (tid == 0) item_note_strings(a, n / 2u, (int32_t)(o + IT_STEP) < end_valid ? o + IT_STEP - start : (uint32_t)end_valid - start);
        fine = false;
        break;
      }
      uint32_t k = nq + (at & 0xFFFFu), ln = nline + (at >> 16) + 1u;
#pragma unroll
      for (uint32_t i = 0; i < IT_SPANW; ++i) {
        const uint32_t p = (uint32_t)(p0 + 32 * (int32_t)i);
        for (uint32_t m = c[i] & (item_prefix_xor(q[i]) ^ (0u - (k & 1u))); m; m &= m - 1u) { /* strings that need a closer look */
          const uint32_t z = (k + (uint32_t)__popc(q[i] & ((m & (0u - m)) - 1u))) >> 1;
          if (z < IT_MAX_STRS) {
            const uint32_t bit = 1u << (z & 31u);
            if (!(atomicOr(&sh.special[z >> 5], bit) & bit)) {
              const uint32_t e = atomicAdd(&sh.nspecial, 1u);
              if (e < IT_MAX_SPECIAL) sh.special_list[e] = (uint16_t)z;
            }
          }
          /* on behind this string's end */
          const uint32_t rest = q[i] & ~((m & (0u - m)) - 1u);
          if (!rest) break;
          m &= ~((rest & (0u - rest)) - 1u) | (m & (0u - m));
        }
        for (uint32_t m = t[i]; m; m &= m - 1u, ++ln) { /* the line behind every separator */
          const uint32_t bit = m & (0u - m);
          sh.line[ln] = (p + (uint32_t)__ffs((int)m)) | (((k + (uint32_t)__popc(q[i] & (bit | (bit - 1u)))) >> 1) << 16);
        }
        for (uint32_t m = q[i]; m; m &= m - 1u) q16[k++] = (uint16_t)(p + (uint32_t)__ffs((int)m) - 1u);
      }
      nq = n; nline = nl;
    }
  }
  if (open_end && (nline >= IT_MAX_LINES || nline >= a.row_cap)) fine = false;
  if (open_end) __syncthreads(); /* (the line's entry) */
  if (tid == 0) {
    const bool any = fine && started && (done || open_end);
    /* a line that runs out of the window keeps none of its strings: it is a whole line up to the window's end for those who size lines, and
       the exact parser's (item_walk_line) */
    if (open_end) { nq = 2u * (sh.line[nline] >> 16); stop = g.hi_valid; if (any) sh.line[nline + 1u] = (stop + 1u) | ((nq >> 1) << 16); ++nline; }
    sh.nstr = any ? nq >> 1 : 0u; sh.nline = any ? nline : 0u; sh.stop = stop; sh.open_end = open_end;
    sh.free_word = (any ? nq >> 1 : 0u) + 1u;
    if (any) strs[nq >> 1] = (stop + 1u) | ((stop + 1u) << 16);
  }
  return fine;
}

/* 8 bytes at p, which may lie up to IT_FRONT bytes before the window */
__device__ __forceinline__ uint64_t item_back8(const uint8_t* win, int32_t p) {
  const uint32_t* a = reinterpret_cast<const uint32_t*>(win) + (p >> 2);
  const uint32_t sh = ((uint32_t)p & 3u) * 8u, x0 = a[0], x1 = a[1], x2 = a[2];
  return (uint64_t)__funnelshift_r(x0, x1, sh) | ((uint64_t)__funnelshift_r(x1, x2, sh) << 32);
}
__device__ __forceinline__ bool item_blank(uint32_t x) { return x <= ' ' && ((0x100002600ull >> x) & 1u); } /* (a line feed is none in a line, and then no line holds one) */
__device__ __forceinline__ uint32_t item_peek4(const uint8_t* win, uint32_t p) {
  Win w;
  w.s = win; w.w0 = 0;
  return wpeek4(w, p);
}
/* 0x80 in every byte of x that is a blank */
__device__ __forceinline__ uint32_t item_blank4(uint32_t x) { return item_eq4(x, 0x20202020u) | item_eq4(x, 0x09090909u) | item_eq4(x, 0x0A0A0A0Au) | item_eq4(x, 0x0D0D0D0Du); }
/* from p over blanks, up to end; four bytes a step, because the lanes of a warp wait for the one with the most blanks, and a byte's load takes as
 * long as a word's */
__device__ __forceinline__ uint32_t item_skip(const uint8_t* win, uint32_t p, uint32_t end) {
  if (p >= end) return p;
  for (;;) {
    const uint32_t no = ~item_blank4(item_peek4(win, p)) & 0x80808080u;
    if (no) { p += ((uint32_t)__ffs((int)no) - 1u) >> 3; break; }
    p += 4u;
    if (p >= end) break;
  }
  return p < end ? p : end;
}
/* from p back over blanks, down to `from`: the first position behind them, where p - 1 is none */
__device__ __forceinline__ uint32_t item_skip_back(const uint8_t* win, uint32_t from, uint32_t p) {
  if (p <= from) return p;
  for (;;) {
    const uint32_t no = ~item_blank4((uint32_t)(item_back8(win, (int32_t)p - 8) >> 32)) & 0x80808080u;
    if (no) { p -= (uint32_t)__clz((int)no) >> 3; break; }
    p = p < from + 4u ? from : p - 4u;
    if (p <= from) break;
  }
  return p > from ? p : from;
}
__device__ __forceinline__ bool item_only_blanks(const uint8_t* win, uint32_t p, uint32_t end) { return item_skip(win, p, end) == end; }
/* bytes that string k, which ends at close, lost when it was decoded; moved: bit per string, null when there is none */
__device__ __forceinline__ uint32_t item_freed(const uint8_t* win, const uint32_t* moved, uint32_t k, uint32_t close) {
  if (!moved || !((moved[k >> 5] >> (k & 31u)) & 1u)) return 0;
  const uint32_t n = win[close - 1u];
  return n < 255u ? n : (uint32_t)win[close - 3u] | ((uint32_t)win[close - 2u] << 8);
}
/* One string that holds a backslash, a control character or a byte beyond ASCII: decoded in place (the decoded text is
 * never longer); what is left over up to the old closing quote becomes blanks. False: not a valid string. */
static __device__ __noinline__ bool item_decode_string(uint8_t* win, uint32_t open, uint32_t close, uint32_t opts, uint32_t* moved) {
  uint32_t p = open + 1u, d = p;
  *moved = 0;
  if (win[close] != '"') return false; /* the record ends inside it */
  while (p < close) {
    if (p + 4u <= close) { /* four characters that stay as they are */
      const uint32_t x4 = item_peek4(win, p), b4 = x4 ^ 0x5C5C5C5Cu;
      if (!((x4 | ((x4 - 0x20202020u) & ~x4) | ((b4 - 0x01010101u) & ~b4)) & 0x80808080u)) {
        if (d != p) { win[d] = (uint8_t)x4; win[d + 1u] = (uint8_t)(x4 >> 8); win[d + 2u] = (uint8_t)(x4 >> 16); win[d + 3u] = (uint8_t)(x4 >> 24); }
        d += 4u; p += 4u;
        continue;
      }
    }
    const uint32_t x = win[p];
    if (x < 0x20) return false;
    if (x == '\\') {
      const uint32_t y = p + 1 < close ? win[p + 1] : 0u;
      uint32_t cp;
      switch (y) {
        case '"': case '\\': case '/': cp = y; break;
        case 'b': cp = 8; break;
        case 'f': cp = 12; break;
        case 'n': cp = 10; break;
        case 'r': cp = 13; break;
        case 't': cp = 9; break;
        case 'u': {
          Win w;
          w.s = win; w.w0 = 0;
          if (p + 6 > close || !fast_hex4(w, p + 2, &cp)) return false;
          if (cp - 0xD800u < 0x400u && p + 12 <= close && win[p + 6] == '\\' && win[p + 7] == 'u') {
            uint32_t lo;
            if (!fast_hex4(w, p + 8, &lo)) return false;
            if (lo - 0xDC00u < 0x400u) { cp = 0x10000u + ((cp - 0xD800u) << 10) + (lo - 0xDC00u); p += 6; }
          }
          if (cp - 0xD800u < 0x800u) {
            if (!(opts & PJ_OPT_LONE_SURROGATE_REPLACE)) return false;
            cp = 0xFFFDu;
          }
          p += 4;
          break;
        }
        default: return false;
      }
      p += 2;
      *moved = 1;
      if (cp < 0x80) win[d++] = (uint8_t)cp;
      else if (cp < 0x800) { win[d++] = (uint8_t)(0xC0 | (cp >> 6)); win[d++] = (uint8_t)(0x80 | (cp & 63)); }
      else if (cp < 0x10000) { win[d++] = (uint8_t)(0xE0 | (cp >> 12)); win[d++] = (uint8_t)(0x80 | ((cp >> 6) & 63)); win[d++] = (uint8_t)(0x80 | (cp & 63)); }
      else { win[d++] = (uint8_t)(0xF0 | (cp >> 18)); win[d++] = (uint8_t)(0x80 | ((cp >> 12) & 63)); win[d++] = (uint8_t)(0x80 | ((cp >> 6) & 63)); win[d++] = (uint8_t)(0x80 | (cp & 63)); }
      continue;
    }
    uint32_t n = 1; /* RFC 3629, the table of lex_string() */
    if (x >= 0x80) {
      uint32_t lo = 0x80, hi = 0xBF;
      if (x - 0xC2u <= 0x1Du) n = 2;
      else if (x == 0xE0) { n = 3; lo = 0xA0; }
      else if (x == 0xED) { n = 3; hi = 0x9F; }
      else if (x - 0xE1u <= 0x0Eu) n = 3;
      else if (x == 0xF0) { n = 4; lo = 0x90; }
      else if (x - 0xF1u <= 2u) n = 4;
      else if (x == 0xF4) { n = 4; hi = 0x8F; }
      else return false;
      if (p + n > close) return false;
      const uint32_t y1 = win[p + 1];
      if (y1 < lo || y1 > hi) return false;
      if (n >= 3 && win[p + 2] - 0x80u > 0x3Fu) return false;
      if (n >= 4 && win[p + 3] - 0x80u > 0x3Fu) return false;
    }
    for (uint32_t k = 0; k < n; ++k) win[d++] = win[p++];
  }
  /* The text ends earlier now. The closing quote stays where it is, so that the gap behind it does too; the bytes between
     hold how many were freed. */
  if (d != close) {
    const uint32_t freed = close - d;
    win[close - 1u] = (uint8_t)(freed < 255u ? freed : 255u);
    if (freed >= 255u) { win[close - 3u] = (uint8_t)freed; win[close - 2u] = (uint8_t)(freed >> 8); }
  }
  return true;
}
/* One string item_index() marked. */
__device__ __forceinline__ void item_special(const ItemArgs& a, ItemShared& sh, uint8_t* win, const uint32_t* pairs, uint32_t k) {
  const uint32_t pr = pairs[k], open = pr & 0xFFFFu, close = pr >> 16;
  uint32_t moved;
  const bool ok = item_decode_string(win, open, close, a.opts, &moved);
  if (!ok || !moved) atomicAnd(&sh.special[k >> 5], ~(1u << (k & 31u)));
  if (ok && !moved) return; /* plain after all */
  if (!ok) atomicOr(&sh.broken[k >> 5], 1u << (k & 31u));
  uint32_t lo = 0, hi = sh.nline; /* its line: the last one that begins at or before it and has a string */
  while (lo + 1u < hi) { const uint32_t mid = (lo + hi) >> 1; if (sh.line[mid] >> 16 <= k) lo = mid; else hi = mid; }
  atomicOr(&sh.movedline[lo >> 5], 1u << (lo & 31u));
  /* a line with a broken string, or with a key in another spelling, is not for the walk */
  const uint32_t sep = (sh.line[lo + 1u] & 0xFFFFu) - 1u;
  uint32_t p = close + 1u;
  while (p < sep && item_blank(win[p])) ++p;
  if (!ok || win[p] == ':') atomicOr(&sh.oddline[lo >> 5], 1u << (lo & 31u));
}
/* All of them: off the list, one per thread, while it holds them, and as many for every warp: its lanes part in them (31 strings of a tile of Pets
 * in the lanes of one warp took 55 000 cycles, four for each warp take 30 000, a warp per string with a byte per lane 27 000). Text where more of
 * the strings are of this kind (another script, \/ for every slash) fills the lanes without one: a warp then takes 32 strings that follow each other. */
__device__ __forceinline__ void item_specials(const ItemArgs& a, ItemShared& sh, uint8_t* win, const uint32_t* pairs, uint32_t tid) {
  if (sh.nspecial <= IT_MAX_SPECIAL) {
    for (uint32_t i = (tid & 31u) * IT_WARPS + (tid >> 5); i < sh.nspecial; i += IT_THREADS) {
      const uint32_t k = sh.special_list[i];
      if (k < sh.nstr) item_special(a, sh, win, pairs, k); /* (a line that runs out of the window has none) */
    }
    return;
  }
  for (uint32_t k = tid; k < sh.nstr; k += IT_THREADS) if ((sh.special[k >> 5] >> (k & 31u)) & 1u) item_special(a, sh, win, pairs, k);
}

/* first byte of a value that is no number: a literal, an object, a list (as the walk takes whatever is between colon and comma) */
__device__ __forceinline__ bool item_other_type(uint32_t x) { return x == 't' || x == 'f' || x == '[' || x == '{'; }
__device__ __forceinline__ bool item_number_start(uint32_t x) { return x - (uint32_t)'0' <= 9u || x == '-'; }
/* -?(0|[1-9][0-9]*) in the n bytes at pos, within int64 / int32. Read from its end, eight digits at a time. */
__device__ __forceinline__ bool item_int(const uint8_t* win, uint32_t pos, uint32_t n, bool is64, int64_t* out) {
  const bool neg = n && win[pos] == '-';
  pos += neg; n -= neg;
  if (n == 0 || n > 19) return false;
  if (win[pos] == '0' && n > 1) return false;
  const uint32_t e = pos + n;
  uint64_t mag, bad;
  {
    uint64_t x = item_back8(win, (int32_t)e - 8);
    const uint32_t k = n < 8 ? n : 8u;
    if (k < 8) x = (x & (~0ull << (64 - 8 * k))) | (0x3030303030303030ull >> (8 * k));
    bad = swar_nondigit(x);
    mag = swar_parse8(x);
  }
  if (n > 8) {
    uint64_t x = item_back8(win, (int32_t)e - 16);
    const uint32_t k = n - 8 < 8 ? n - 8 : 8u;
    if (k < 8) x = (x & (~0ull << (64 - 8 * k))) | (0x3030303030303030ull >> (8 * k));
    bad |= swar_nondigit(x);
    mag += (uint64_t)swar_parse8(x) * 100000000ull;
  }
  if (n > 16) {
    const uint32_t k = n - 16; /* 1..3 */
    uint32_t x = (uint32_t)item_back8(win, (int32_t)e - 20);
    x = (x & (~0u << (32 - 8 * k))) | (0x30303030u >> (8 * k));
    const uint32_t d0 = (x & 0xFFu) - 48u, d1 = ((x >> 8) & 0xFFu) - 48u, d2 = ((x >> 16) & 0xFFu) - 48u, d3 = (x >> 24) - 48u;
    bad |= (d1 > 9u) | (d2 > 9u) | (d3 > 9u) | (d0 > 9u);
    mag += (uint64_t)(d1 * 100u + d2 * 10u + d3) * 10000000000000000ull;
  }
  const uint64_t lim = is64 ? 0x7FFFFFFFFFFFFFFFull + neg : 0x7FFFFFFFull + neg;
  *out = neg ? (int64_t)(0 - mag) : (int64_t)mag;
  return !bad && mag <= lim;
}
__device__ __forceinline__ bool item_true(const uint8_t* win, uint32_t pos, uint32_t n) { return n == 4 && item_peek4(win, pos) == 0x65757274u; }
__device__ __forceinline__ bool item_false(const uint8_t* win, uint32_t pos, uint32_t n) { return n == 5 && win[pos] == 'f' && item_peek4(win, pos + 1) == 0x65736C61u; }

__device__ __forceinline__ void item_error(uint32_t* row, uint32_t pos, uint32_t kind) {
  atomicMin(&row[IW_ERR], (pos << 8) | kind);
}
/* A scalar token that belongs to no property: only what is cheap to see as valid (integers, literals) passes. */
static __device__ __noinline__ bool item_plain_scalar(const uint8_t* win, uint32_t s, uint32_t n) {
  if (n == 4 && (item_peek4(win, s) == 0x65757274u || item_peek4(win, s) == 0x6C6C756Eu)) return true;
  if (n == 5 && win[s] == 'f' && item_peek4(win, s + 1) == 0x65736C61u) return true;
  uint32_t i = win[s] == '-' ? 1u : 0u;
  if (i >= n || (win[s + i] == '0' && i + 1 < n)) return false;
  for (; i < n; ++i) if (win[s + i] - (uint32_t)'0' > 9u) return false;
  return true;
}

template <int E>
PJ_CX int it_string_field() { /* the one string property of a flat object */
  int at = -1;
  for (int i = 0; i < CObj<E>::N; ++i) if (CObj<E>::f[i].kind == K_STR) at = i;
  return at;
}
/* ---- 2. the walk ------------------------------------------------------------------------------------------------
 * Records as serialisers write them: properties in model order, any of them missing or null, blanks between the tokens or
 * none. One line per thread, every string's end known from the index, so only the gaps are looked at; references to the
 * values' text go to the row. The first deviation ends a line's walk, and item_pack() looks at it.
 * Bound by instructions and, in lines with blanks, by the chain of byte loads; 200k Users with blanks took 292 us when
 * item_pack() took all of them and take 115 us with the walk. */
struct ItemWalk {
  const uint8_t* win;
  const uint32_t* pairs;
  const uint32_t* moved;
  uint32_t p;            /* at the brace or comma before the next member, or at the closing brace */
  uint32_t k, kend, sep; /* next string, end of the line's strings, its separator */
  bool ok, open;         /* open: p is no closing brace */
};
/* is `"name"` of property I at p? */
template <int OBJ, int I>
__device__ __forceinline__ bool item_at_key(const uint8_t* win, uint32_t p) {
  constexpr uint32_t n = FK<OBJ, I>::pat_len - 1u; /* without the colon */
  constexpr uint64_t t0 = FK<OBJ, I>::pat0, t1 = FK<OBJ, I>::pat1;
  const uint32_t* a = reinterpret_cast<const uint32_t*>(win) + (p >> 2);
  const uint32_t s = (p & 3u) * 8u;
  const uint32_t y0 = a[0], y1 = a[1];
  uint32_t d = __funnelshift_r(y0, y1, s) ^ (uint32_t)t0;
  static_assert(n >= 4, "a name of two letters");
  if constexpr (n > 4) {
    const uint32_t y2 = a[2];
    const uint32_t x = __funnelshift_r(y1, y2, s) ^ (uint32_t)(t0 >> 32);
    d |= n >= 8 ? x : x & ((1u << (8 * (n & 3u))) - 1u);
    if constexpr (n > 8) {
      const uint32_t y3 = a[3];
      const uint32_t z = __funnelshift_r(y2, y3, s) ^ (uint32_t)t1;
      d |= n >= 12 ? z : z & ((1u << (8 * (n & 3u))) - 1u);
      if constexpr (n > 12) {
        const uint32_t v = __funnelshift_r(y3, a[4], s) ^ (uint32_t)(t1 >> 32);
        d |= n >= 16 ? v : v & ((1u << (8 * (n & 3u))) - 1u);
      }
    }
  }
  return d == 0;
}
/* from p over blanks to c and over the blanks behind it; the position there */
__device__ __forceinline__ uint32_t item_over(ItemWalk& f, uint32_t p, uint32_t c) {
  if (f.win[p] != c) {
    p = item_skip(f.win, p, f.sep);
    f.ok = f.ok && f.win[p] == c;
  }
  return item_skip(f.win, p + 1u, f.sep);
}
/* back from q over blanks to a comma (or closing brace: last) and over the blanks before it; where the comma is, and in *end
 * the end of what is before it */
__device__ __forceinline__ uint32_t item_back(ItemWalk& f, uint32_t from, uint32_t q, bool last, uint32_t* end) {
  const uint32_t c = last ? '}' : ',';
  uint32_t r = q - 1u;
  if (f.win[r] != c) {
    r = item_skip_back(f.win, from + 1u, q) - 1u;
    f.ok = f.ok && f.win[r] == c;
  }
  *end = item_skip_back(f.win, from, r);
  return r;
}
/* the flat object E whose brace is behind the blanks from at on, all of its properties there: bytes of its string in *bytes,
 * the position behind its brace returned */
template <int E, int I = 0>
__device__ __forceinline__ uint32_t item_walk_flat(ItemWalk& f, uint32_t at, uint32_t* bytes) {
  constexpr uint32_t kind = CObj<E>::f[I].kind;
  constexpr bool last = I + 1 == CObj<E>::N;
  static_assert(kind == K_STR ? last : (!last && (kind == K_I64 || kind == K_I32)), "integers, then a string");
  const uint32_t key = f.pairs[f.k < f.kend ? f.k : f.kend], nx = f.pairs[f.k + 1u < f.kend ? f.k + 1u : f.kend];
  const uint32_t ko = item_over(f, at, I == 0 ? '{' : ',');
  f.ok = f.ok && f.k + 1u < f.kend && ko == (key & 0xFFFFu) && item_at_key<E, I>(f.win, ko);
  if (!f.ok) return at;
  const uint32_t v = item_over(f, (key >> 16) + 1u, ':');
  if constexpr (!last) {
    uint32_t end;
    const uint32_t comma = item_back(f, v, nx & 0xFFFFu, false, &end);
    f.ok = f.ok && end > v && end - v < 32u;
    f.k++;
    return item_walk_flat<E, I + 1>(f, comma, bytes);
  } else {
    const uint32_t open = nx & 0xFFFFu, close = nx >> 16;
    f.ok = f.ok && open == v && close - open < 0x1000u; /* a length that fits its row */
    *bytes = close - open - 1u - item_freed(f.win, f.moved, f.k + 1u, close);
    f.k += 2u;
    const uint32_t p = item_skip(f.win, close + 1u, f.sep);
    f.ok = f.ok && f.win[p] == '}';
    return p + 1u;
  }
}
template <int N> struct ItInteger { static constexpr int value = N; };
struct ItemLists { uint32_t k_str, n_str, k_obj, n_obj, bytes; };
/* the list whose bracket is at v; the position behind it */
template <int OBJ, int I>
__device__ __forceinline__ uint32_t item_walk_list(ItemWalk& f, uint32_t v, ItemLists& l) {
  constexpr uint32_t kind = CObj<OBJ>::f[I].kind;
  f.ok = f.ok && f.win[v] == '[';
  uint32_t n = 0, p = v + 1u;
  const uint32_t k0 = f.k;
  p = item_skip(f.win, p, f.sep);
  bool go = f.ok && f.win[p] != ']';
  p += go ? 0u : 1u;
  while (go) {
    if constexpr (kind == K_LIST_STR) {
      const uint32_t pr = f.pairs[f.k < f.kend ? f.k : f.kend], open = pr & 0xFFFFu, close = pr >> 16;
      f.ok = f.k < f.kend && open == p && close - open < 0x8000u;
      l.bytes += close - open - 1u - (f.ok ? item_freed(f.win, f.moved, f.k, close) : 0u);
      f.k++;
      p = close + 1u;
    } else {
      uint32_t bytes = 0;
      p = item_walk_flat<CObj<OBJ>::f[I].child>(f, p, &bytes);
      l.bytes += bytes << 16;
    }
    ++n;
    p = item_skip(f.win, f.ok ? p : v, f.sep);
    const uint32_t x = f.win[p];
    go = f.ok && x == ',';
    f.ok = f.ok && (x == ',' || x == ']');
    ++p;
    if (go) p = item_skip(f.win, p, f.sep);
  }
  if constexpr (kind == K_LIST_STR) { l.k_str = k0; l.n_str = n; } else { l.k_obj = k0; l.n_obj = n; }
  return p;
}
/* The members of OBJ from property I on, each tried once, in model order. f.p: at the brace or comma before the first; left at
 * the closing brace. A root's values go to its row's words, an embedded object's to the words behind WORD0. */
template <int OBJ, int I, bool ROOT = true, uint32_t WORD0 = 0, uint32_t BIT0 = 0>
__device__ __forceinline__ void item_walk_members(ItemWalk& f, uint32_t* row, uint32_t& flags, ItemLists& l) {
  if constexpr (I < CObj<OBJ>::N) {
    constexpr uint32_t kind = CObj<OBJ>::f[I].kind, word = ROOT ? it_root_word<OBJ>(I) : WORD0 + it_flat_word<OBJ>(I);
    if (f.ok && f.open && f.k < f.kend) {
      const uint32_t key = f.pairs[f.k], ko = key & 0xFFFFu;
      if (item_at_key<OBJ, I>(f.win, ko)) {
        f.ok = ko == f.p + 1u || item_only_blanks(f.win, f.p + 1u, ko);
        f.k++;
        const bool more = f.k < f.kend; /* strings follow: the next key, or the value */
        const uint32_t nx = f.pairs[f.k]; /* (or the entry behind the last one) */
        const uint32_t v = item_over(f, (key >> 16) + 1u, ':'), x0 = f.win[v];
        uint32_t end = v; /* at the delimiter behind the value */
        uint32_t bit = 1u << (IF_PRESENT + BIT0 + I);
        bool to_delimiter = true; /* end is still behind the value, blanks may follow */
        if (x0 == 'n') {
          f.ok = f.ok && item_peek4(f.win, v) == 0x6C6C756Eu;
          end = v + 4u;
          bit = 0;
        } else if constexpr (kind == K_I64 || kind == K_I32 || kind == K_BOOL) {
          uint32_t e;
          if (ROOT || more) {
            end = item_back(f, v, more ? nx & 0xFFFFu : f.sep, !more, &e);
            if (!ROOT && f.win[e - 1u] == '}') { /* the embedded object ends here, and the comma is its root's */
              end = --e;
              e = item_skip_back(f.win, v, e);
            }
          } else {
            e = v;
            while (e < f.sep && ((uint32_t)f.win[e] - '0' <= 9u || f.win[e] == '-')) ++e;
            end = e;
          }
          f.ok = f.ok && e > v && e - v < 32u;
          row[word] = v | ((e - v) << 16);
          to_delimiter = !ROOT; /* (an embedded object's own brace may come first) */
        } else if constexpr (kind == K_STR || kind == K_ENUM || kind == K_DATETIME) {
          const uint32_t close = nx >> 16;
          f.ok = f.ok && more && (nx & 0xFFFFu) == v && close - v < 0x7FF0u;
          row[word] = (v + 1u) | ((close - v - 1u - (f.ok ? item_freed(f.win, f.moved, f.k, close) : 0u)) << 16);
          end = close + 1u;
          f.k++;
        } else if constexpr (kind == K_OBJ) {
          f.ok = f.ok && x0 == '{';
          f.p = v;
          item_walk_members<CObj<OBJ>::f[I].child, 0, false, ItModel<OBJ>::child_word, IB_CHILD>(f, row, flags, l);
          if (f.ok && f.open) { /* no member at all: `{}` */
            const uint32_t q = item_over(f, v, '{');
            f.ok = f.p == v && f.win[q] == '}';
            f.p = q;
          }
          f.open = true;
          end = f.p + 1u;
        } else end = item_walk_list<OBJ, I>(f, v, l);
        end = f.ok ? end : f.p;
        if (to_delimiter) end = item_skip(f.win, end, f.sep);
        const uint32_t x = f.win[end];
        f.open = x == ',';
        f.ok = f.ok && (x == ',' || x == '}');
        flags |= bit;
        f.p = end;
      }
    }
    item_walk_members<OBJ, I + 1, ROOT, WORD0, BIT0>(f, row, flags, l);
  }
}
/* The same for records without a blank and without null, and with embedded objects whole: no byte is looked at twice. (Strings that were
 * decoded are shorter than their quotes tell.) It is tried first, because most producers write this way (1M Pets: 617 us against 790 us with the walk above alone). */
/* is `"name":` of property I at p? */
template <int OBJ, int I>
__device__ __forceinline__ bool item_at_key_colon(const uint8_t* win, uint32_t p) {
  constexpr uint32_t n = FK<OBJ, I>::pat_len;
  constexpr uint64_t t0 = FK<OBJ, I>::pat0, t1 = FK<OBJ, I>::pat1;
  const uint32_t* a = reinterpret_cast<const uint32_t*>(win) + (p >> 2);
  const uint32_t s = (p & 3u) * 8u;
  const uint32_t y0 = a[0], y1 = a[1];
  uint32_t d = __funnelshift_r(y0, y1, s) ^ (uint32_t)t0;
  if constexpr (n < 4) d &= (1u << (8 * (n & 3u))) - 1u;
  if constexpr (n > 4) {
    const uint32_t y2 = a[2];
    const uint32_t x = __funnelshift_r(y1, y2, s) ^ (uint32_t)(t0 >> 32);
    d |= n >= 8 ? x : x & ((1u << (8 * (n & 3u))) - 1u);
    if constexpr (n > 8) {
      const uint32_t y3 = a[3];
      const uint32_t z = __funnelshift_r(y2, y3, s) ^ (uint32_t)t1;
      d |= n >= 12 ? z : z & ((1u << (8 * (n & 3u))) - 1u);
      if constexpr (n > 12) {
        const uint32_t v = __funnelshift_r(y3, a[4], s) ^ (uint32_t)(t1 >> 32);
        d |= n >= 16 ? v : v & ((1u << (8 * (n & 3u))) - 1u);
      }
    }
  }
  return d == 0;
}
/* the flat object E at position at: `{"a":1,"b":"c"}`, all of its properties; references to its values in ref[]; returns the
 * position behind its brace */
template <int E, int I = 0>
__device__ __forceinline__ uint32_t item_dense_flat(ItemWalk& f, uint32_t at, uint32_t* ref) {
  if constexpr (I == 0) f.ok = f.ok && f.win[at] == '{';
  if constexpr (I < CObj<E>::N) {
    constexpr uint32_t kind = CObj<E>::f[I].kind;
    static_assert(kind == K_I64 || kind == K_I32 || kind == K_STR, "flat objects: integers and strings");
    f.ok = f.ok && item_at_key_colon<E, I>(f.win, at + 1u);
    const uint32_t v = at + 1u + FK<E, I>::pat_len;
    f.k++;
    const uint32_t nx = f.pairs[f.k < f.kend ? f.k : f.kend];
    uint32_t end;
    if constexpr (kind == K_STR) {
      f.ok = f.ok && f.k < f.kend && (nx & 0xFFFFu) == v;
      end = (nx >> 16) + 1u;
      f.ok = f.ok && end - v < 0x1000u; /* a length that fits its row */
      ref[I] = (v + 1u) | ((end - v - 2u - (f.ok ? item_freed(f.win, f.moved, f.k, nx >> 16) : 0u)) << 16);
      f.k++;
    } else {
      static_assert(I + 1 < CObj<E>::N, "an integer is followed by another property");
      end = (nx & 0xFFFFu) - 1u; /* the comma before the next key */
      f.ok = f.ok && f.k < f.kend && end > v && end - v < 32u && item_number_start(f.win[v]) && f.win[end - 1u] > ' ';
      ref[I] = v | ((end - v) << 16);
    }
    f.ok = f.ok && f.win[f.ok ? end : at] == (I + 1 < CObj<E>::N ? ',' : '}');
    return item_dense_flat<E, I + 1>(f, end, ref);
  } else return at + 1u;
}
template <int OBJ, int CH, int J = 0>
__device__ __forceinline__ void item_dense_child(uint32_t* row, const uint32_t* ref) {
  if constexpr (J < CObj<CH>::N) {
    row[ItModel<OBJ>::child_word + it_flat_word<CH>(J)] = ref[J];
    item_dense_child<OBJ, CH, J + 1>(row, ref);
  }
}
/* the members of root OBJ from property I on, each tried once, in model order */
template <int OBJ, int I>
__device__ __forceinline__ void item_dense_members(ItemWalk& f, uint32_t* row, uint32_t& flags, ItemLists& l) {
  if constexpr (I < CObj<OBJ>::N) {
    constexpr uint32_t kind = CObj<OBJ>::f[I].kind, word = it_root_word<OBJ>(I);
    if (f.ok && f.k < f.kend && item_at_key_colon<OBJ, I>(f.win, f.p + 1u)) {
      const uint32_t v = f.p + 1u + FK<OBJ, I>::pat_len;
      f.k++;
      const bool more = f.k < f.kend; /* strings follow: the next key, or the value */
      const uint32_t nx = f.pairs[more ? f.k : f.kend];
      uint32_t end = v; /* behind the value */
      if constexpr (kind == K_I64 || kind == K_I32 || kind == K_BOOL) {
        end = more ? (nx & 0xFFFFu) - 1u : f.sep - 1u;
        const uint32_t x0 = f.win[v];
        f.ok = end > v && end - v < 32u && (kind == K_BOOL ? x0 == 't' || x0 == 'f' : item_number_start(x0)) && f.win[end - 1u] > ' ';
        row[word] = v | ((end - v) << 16);
      } else if constexpr (kind == K_STR || kind == K_ENUM || kind == K_DATETIME) {
        end = (nx >> 16) + 1u;
        f.ok = more && (nx & 0xFFFFu) == v && end - v <= 0x8000u;
        row[word] = (v + 1u) | ((end - v - 2u - (f.ok ? item_freed(f.win, f.moved, f.k, nx >> 16) : 0u)) << 16);
        f.k++;
      } else if constexpr (kind == K_OBJ) {
        constexpr int CH = CObj<OBJ>::f[I].child;
        uint32_t ref[8];
        end = item_dense_flat<CH>(f, v, ref);
        item_dense_child<OBJ, CH>(row, ref);
        flags |= ((1u << CObj<CH>::N) - 1u) << (IF_PRESENT + IB_CHILD);
      } else { /* a list */
        f.ok = f.win[v] == '[';
        uint32_t n = 0;
        const uint32_t k0 = f.k;
        bool go = f.ok && f.win[v + 1u] != ']';
        end = v + (go ? 1u : 2u);
        while (go) {
          uint32_t behind;
          if constexpr (kind == K_LIST_STR) {
            const uint32_t pr = f.pairs[f.k < f.kend ? f.k : f.kend];
            behind = (pr >> 16) + 1u;
            f.ok = f.k < f.kend && (pr & 0xFFFFu) == end && behind - end < 0x8000u;
            l.bytes += behind - end - 2u - (f.ok ? item_freed(f.win, f.moved, f.k, pr >> 16) : 0u);
            f.k++;
          } else {
            uint32_t ref[8];
            behind = item_dense_flat<CObj<OBJ>::f[I].child>(f, end, ref);
            l.bytes += ref[it_string_field<CObj<OBJ>::f[I].child>()] & 0xFFFF0000u;
          }
          ++n;
          const uint32_t x = f.win[f.ok ? behind : end];
          end = behind + 1u;
          go = f.ok && x == ',';
          f.ok = f.ok && (x == ',' || x == ']');
        }
        if constexpr (kind == K_LIST_STR) { l.k_str = k0; l.n_str = n; } else { l.k_obj = k0; l.n_obj = n; }
      }
      flags |= 1u << (IF_PRESENT + I);
      const uint32_t x = f.win[f.ok ? end : f.p];
      f.ok = f.ok && (x == ',' || (x == '}' && end + 1u == f.sep));
      f.p = f.ok ? end : f.p;
    }
    item_dense_members<OBJ, I + 1>(f, row, flags, l);
  }
}
__device__ __forceinline__ ItemWalk item_walk_open(const ItemShared& sh, const uint8_t* win, const uint32_t* pairs, uint32_t i) {
  const uint32_t me = sh.line[i], next = sh.line[i + 1u];
  ItemWalk f;
  f.win = win; f.pairs = pairs; f.moved = sh.nspecial ? sh.special : nullptr;
  f.p = me & 0xFFFFu; f.k = me >> 16; f.kend = next >> 16; f.sep = (next & 0xFFFFu) - 1u;
  f.ok = true; f.open = true;
  return f;
}
/* a record of its schema's or, in a stream of several models, of type's model */
template <int SCHEMA, bool DENSE>
__device__ __forceinline__ void item_walk_model(ItemWalk& f, uint32_t* row, uint32_t& flags, ItemLists& l, uint32_t type) {
  auto members = [&](auto obj) {
    constexpr int OBJ = decltype(obj)::value;
    if constexpr (DENSE) item_dense_members<OBJ, 0>(f, row, flags, l);
    else item_walk_members<OBJ, 0>(f, row, flags, l);
  };
  if constexpr (SCHEMA != PJ_SCHEMA_MIXED) members(ItInteger<RootOf<SCHEMA>::obj>());
  else {
    if (type == PJ_TYPE_PET) { members(ItInteger<OBJ_PET>()); flags |= 6u << IF_NOTMODEL; }
    else if (type == PJ_TYPE_ORDER) { members(ItInteger<OBJ_ORDER>()); flags |= 5u << IF_NOTMODEL; }
    else if (type == PJ_TYPE_USER) { members(ItInteger<OBJ_USER>()); flags |= 3u << IF_NOTMODEL; }
    else f.ok = false;
  }
  if constexpr (DENSE) f.ok = f.ok && f.k == f.kend && f.win[f.p] == '}' && f.p + 1u == f.sep;
  else f.ok = f.ok && f.k == f.kend && !f.open && item_only_blanks(f.win, f.p + 1u, f.sep);
}
/* is the line at input offset s0, which runs out of the window, a record? */
static __device__ __noinline__ bool item_long_is_record(const ItemArgs& a, uint64_t s0) {
  return a.sep ? arr_extent(a.in, a.len, a.sep, s0 - 1u, a.res->first_opener).is_record != 0 : nd_is_record(a.in, s0, a.limit, (int)a.is_last);
}
/* One line: its row, or IF_ODD there. */
template <int SCHEMA, bool ARR, bool DENSE>
__device__ __forceinline__ void item_walk_line(const ItemArgs& a, const StreamGeom& g, ItemShared& sh, const uint8_t* win, const uint32_t* pairs, uint32_t* rows, uint32_t i, uint32_t type) {
  constexpr uint32_t STRIDE = ItStride<SCHEMA>::n;
  ItemWalk f = item_walk_open(sh, win, pairs, i);
  uint32_t* row = rows + i * STRIDE;
  const uint32_t start = f.p;
  uint32_t flags = 0, err = IE_NONE;
  ItemLists l;
  l.k_str = l.n_str = l.k_obj = l.n_obj = l.bytes = 0;
  const bool cut = f.sep >= g.hi_valid && !a.is_last; /* the readable bytes end here, the stream does not */
  /* array framing: what the separator before the line is. Nothing follows `]`; documents of several arrays are in error at the second one. */
  const uint32_t before = ARR ? win[start - 1u] : 0u;
  if (ARR && before == '[') {
    const uint64_t at = g.v0 + start - 1u - g.mis;
    if (at > a.res->first_opener) atomicMin(&a.res->doc_err_off, (unsigned long long)at);
  }
  const bool long_line = sh.open_end && i + 1u == sh.nline;
  if (ARR && before == ']') f.p = start;
  else if (long_line) {
    if (item_long_is_record(a, g.v0 + start - g.mis)) { flags = IF_RECORD; err = (start << 8) | IE_REFUSED; }
  } else if (f.k == f.kend) { /* no string */
    uint32_t p = start;
    while (p < f.sep && item_blank(win[p])) ++p;
    if (p < f.sep || cut) { flags = IF_RECORD; err = (start << 8) | IE_REFUSED; } /* for the exact parser */
    else if (ARR && f.sep < g.hi_valid && !(before == '[' && win[f.sep] == ']')) { flags = IF_RECORD; err = (f.sep << 8) | (uint32_t)PJ_E_SYNTAX; } /* an extent without a value */
    f.p = start;
  } else {
    const uint32_t n = f.kend - f.k, bit = 1u << (i & 31u);
    const bool plain = !(sh.movedline[i >> 5] & bit), fit = !cut && !(sh.oddline[i >> 5] & bit);
    /* A warp waits for its longest line, which takes some 300 cycles a string (1000 with blanks), while the warps together take 10 (25) in
       item_pack() for every string of the tile, whoever's it is: lines much longer than the others are its. (50 k Pets with long lists 610 -> 575 us,
       with blanks 1620 -> 1270, the line for both at a quarter and a twelfth of the tile's strings before.) */
    if constexpr (DENSE) f.ok = fit && win[start] == '{' && (n <= 32u || n * 30u <= sh.nstr);
    else {
      f.p = item_skip(win, f.p, f.sep);
      f.ok = fit && win[f.p] == '{' && (n <= 16u || n * 40u <= sh.nstr);
    }
    item_walk_model<SCHEMA, DENSE>(f, row, flags, l, type);
    if (!plain) flags |= IF_MOVED;
    flags = IF_RECORD | (f.ok ? flags : IF_ODD);
  }
  row[IW_FLAGS] = flags; row[IW_ERR] = err; row[IW_POS] = start | (f.p << 16);
  if constexpr (ItemSlots<SCHEMA>::lists) {
    row[IW_LIST] = l.k_str | (l.n_str << 16);
    if (SCHEMA == PJ_SCHEMA_PET || type == PJ_TYPE_PET) { row[ItWords<OBJ_PET>::n] = l.k_obj | (l.n_obj << 16); row[ItWords<OBJ_PET>::n + 1u] = l.bytes; }
  }
}
static_assert(ItStride<PJ_SCHEMA_PET>::n >= ItWords<OBJ_PET>::n + 2u && ItStride<PJ_SCHEMA_MIXED>::n >= ItWords<OBJ_PET>::n + 2u, "two words behind a Pet's for its lists");
static_assert(CObj<OBJ_TAG>::N == 2 && CObj<OBJ_TAG>::f[0].kind == K_I64 && CObj<OBJ_TAG>::f[1].kind == K_STR, "list elements: an integer and a string");

/* perm[]: the lines by class (0 to 3; 4: none), in order within a class; a line per thread. Ends of the classes in ends[]. */
__device__ __forceinline__ void item_sort(ItemShared& sh, uint32_t tid, uint32_t cls, uint32_t* ends) {
  const uint32_t lane = tid & 31, warp = tid >> 5;
  uint32_t rank = 0;
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) {
    const uint32_t bal = __ballot_sync(0xFFFFFFFFu, cls == k);
    if (lane == 0) sh.cls[k][warp] = (uint8_t)__popc(bal);
    if (cls == k) rank = (uint32_t)__popc(bal & ((1u << lane) - 1u));
  }
  __syncthreads();
  uint32_t at = 0;
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) {
#pragma unroll
    for (uint32_t q = 0; q < IT_WARPS; ++q) {
      if (cls == k && q == warp) rank += at;
      at += sh.cls[k][q];
    }
    ends[k] = at;
  }
  if (cls < 4) sh.perm[rank] = (uint8_t)tid;
  __syncthreads();
}
/* All lines: one per thread, in order, or, in a stream of several models, sorted by the model the key behind `id` decides,
 * so that a warp walks one model. */
template <int SCHEMA, bool ARR>
__device__ __forceinline__ uint32_t item_walk(const ItemArgs& a, const StreamGeom& g, ItemShared& sh, const uint8_t* win, const uint32_t* pairs, uint32_t* rows, uint32_t tid) {
  const uint32_t lane = tid & 31, warp = tid >> 5, nline = sh.nline;
  uint32_t i = tid, type = 0;
  if constexpr (SCHEMA == PJ_SCHEMA_MIXED) {
    uint32_t cls = 4; /* threads without a line go last */
    if (tid < nline) {
      const ItemWalk f = item_walk_open(sh, win, pairs, tid);
      cls = 3; /* no idea */
      if (f.k < f.kend) {
        uint32_t pr = f.pairs[f.k], x = item_peek4(win, (pr & 0xFFFFu) + 1u);
        if ((x & 0xFFFFFFu) == 0x226469u && f.k + 1u < f.kend) x = item_peek4(win, (f.pairs[f.k + 1u] & 0xFFFFu) + 1u); /* `id` is everyone's */
        const uint32_t c0 = x & 0xFFu, c1 = (x >> 8) & 0xFFu, c3 = x >> 24;
        if (c0 == 'n' || c0 == 't' || (c0 == 'c' && c1 == 'a') || (c0 == 'p' && c3 == 't')) cls = 0;
        else if (c0 == 'q' || (c0 == 'c' && c1 == 'o') || (c0 == 'p' && c1 == 'e') || (c0 == 's' && c1 == 'h')) cls = 1;
        else if (c0 == 'u' || c0 == 'f' || c0 == 'l' || c0 == 'e' || c0 == 'p') cls = 2;
      }
    }
    uint32_t ends[4];
    item_sort(sh, tid, cls, ends);
    type = tid < ends[0] ? (uint32_t)PJ_TYPE_PET : (tid < ends[1] ? (uint32_t)PJ_TYPE_ORDER : (tid < ends[2] ? (uint32_t)PJ_TYPE_USER : (uint32_t)PJ_TYPE_NONE));
    if (tid < nline) i = sh.perm[tid];
  }
  if (tid < nline) item_walk_line<SCHEMA, ARR, true>(a, g, sh, win, pairs, rows, i, type);
  return i | (type << 16);
}
/* The second look at the lines the dense walk left: by the same threads. Out of line, so that the tiles that need none keep
 * their instructions close together; every thread of the block calls it. */
template <int SCHEMA, bool ARR>
__device__ __noinline__ void item_walk_again(const ItemArgs& a, const StreamGeom& g, ItemShared& sh, const uint8_t* win, const uint32_t* pairs, uint32_t* rows, uint32_t tid, uint32_t mine) {
  const uint32_t i = mine & 0xFFFFu, type = mine >> 16;
  if (tid < sh.nline && ((sh.oddmask[i >> 5] >> (i & 31u)) & 1u)) item_walk_line<SCHEMA, ARR, false>(a, g, sh, win, pairs, rows, i, type);
  __syncthreads();
  const bool odd = tid < sh.nline && (rows[tid * ItStride<SCHEMA>::n + IW_FLAGS] & IF_ODD);
  const uint32_t m = __ballot_sync(0xFFFFFFFFu, odd);
  if ((tid & 31u) == 0) sh.oddmask[tid >> 5] = m;
  __syncthreads();
}

/* ---- 3. strings and gaps ------------------------------------------------------------------------------------------ */
/* A gap as the tables know it, and the places in it that matter. */
struct ItemView {
  uint32_t desc;       /* ItGap, 0: not one of the texts */
  uint32_t vpos, vend; /* first byte of the value behind the colon, end of a number or literal */
  uint32_t clpos;      /* the record's closing brace */
};
__device__ __forceinline__ uint32_t item_gap_find(const ItemShared& sh, uint32_t lo, uint32_t hi, uint32_t len) {
  const ItGapEntry e = sh.gap[it_gap_hash(lo, hi)];
  return e.lo == lo && e.hi == hi && e.len == len ? e.desc : 0u;
}
/* [from, b) with blanks: its text is put together byte by byte, numbers and literals are skipped. */
template <bool ARR>
__device__ __forceinline__ void item_gap_spaced(const ItemShared& sh, const uint8_t* win, uint32_t from, uint32_t b, ItemView& v) {
  Win w;
  w.s = win; w.w0 = 0;
  uint32_t lo = 0, hi = 0, n = 0, p = from;
  v.vpos = b; v.vend = 0; v.clpos = b;
  while (p < b && n <= 8u) {
    uint32_t c = win[p];
    if (item_blank(c)) { p = item_skip(win, p + 1u, b); continue; }
    if (n == 1u) v.vpos = p;
    if (c - (uint32_t)'0' <= 9u || c == '-' || (c | 0x20u) - (uint32_t)'a' <= 25u) {
      ++p;
      for (;;) {
        const uint64_t m = swar_nondigit(wpeek8(w, p));
        if (!m) { p += 8; if (p > b) break; continue; }
        p += ctz64(m) >> 3;
        const uint32_t x = win[p];
        if ((x | 0x20u) - (uint32_t)'a' <= 25u || x == '.' || x == '+' || x == '-') { ++p; continue; }
        break;
      }
      v.vend = p;
      c = '0';
    } else {
      if (c == '}') v.clpos = p;
      ++p;
    }
    if (n < 4u) lo |= c << (8u * n); else if (n < 8u) hi |= c << (8u * (n - 4u));
    ++n;
  }
  v.desc = n <= 8u && p == b ? item_gap_find(sh, lo, hi, n) : 0u;
}

/* the property (ItField) that the n bytes at `at` name in a root, its embedded object or an element; 0: none */
__device__ __forceinline__ uint32_t item_key(const ItemShared& sh, const uint8_t* win, uint32_t at, uint32_t len, uint32_t s) {
  const uint32_t* kw = reinterpret_cast<const uint32_t*>(win) + (at >> 2);
  const uint32_t ksh = (at & 3u) * 8u;
  const uint32_t y0 = kw[0], y1 = kw[1], y2 = kw[2], y3 = kw[3], y4 = kw[4];
  const uint32_t x0 = __funnelshift_r(y0, y1, ksh), x1 = __funnelshift_r(y1, y2, ksh), x2 = __funnelshift_r(y2, y3, ksh), x3 = __funnelshift_r(y3, y4, ksh);
  const uint32_t slot = it_hash(x0 & 0xFFFFu, len, IT_MUL);
  const uint4 kt = *reinterpret_cast<const uint4*>(&sh.key[slot][0]), km = *reinterpret_cast<const uint4*>(&sh.key[slot][4]);
  const uint32_t f = sh.field[s == IS_ROOT ? 0 : (s == IS_CHILD ? 1 : 2)][slot];
  return (((x0 ^ kt.x) & km.x) | ((x1 ^ kt.y) & km.y) | ((x2 ^ kt.z) & km.z) | ((x3 ^ kt.w) & km.w)) != 0 || len != ItField::len(f) ? 0u : f;
}
/* Lines [i0, i0 + n), each with a string, by a warp: together at most 32 strings, or one line with more. What does not fit its words (a
 * string of 32 KB, more list elements than there is room for) leaves them to the exact parser. */
template <int SCHEMA, bool ARR>
__device__ __noinline__ void item_pack(const ItemArgs& a, const StreamGeom& g, ItemShared& sh, const uint8_t* win, uint32_t* pairs, uint32_t* rows, uint32_t i0, uint32_t n) {
  constexpr uint32_t STRIDE = ItStride<SCHEMA>::n;
  constexpr uint32_t LW = ItWords<OBJ_PET>::n; /* the word of the list of objects, then that of the bytes */
  constexpr int E = OBJ_TAG, ES = it_string_field<E>();
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t lt = (1u << lane) - 1u, le = (2u << lane) - 1u; /* lane 31: 2 << 31 wraps to 0, so all ones */
  const uint32_t nstr = sh.nstr;
  const bool special = sh.nspecial != 0, truncs = sh.odd != 0;
  const uint32_t* moved = special ? sh.special : nullptr;
  const uint32_t k_lo = sh.line[i0] >> 16, k_hi = sh.line[i0 + n] >> 16;
  const bool single = k_hi - k_lo > 32u;
  /* rows start empty */
  uint32_t first_bit = 0;
  if (lane < n) {
    const uint32_t me = sh.line[i0 + lane];
    uint32_t* row = rows + (i0 + lane) * STRIDE;
    row[IW_FLAGS] = IF_RECORD | IF_ROWS; row[IW_ERR] = IE_NONE; row[IW_POS] = me & 0xFFFFu;
    if constexpr (ItemSlots<SCHEMA>::lists) { row[IW_LIST] = 0; row[LW] = 0; row[LW + 1u] = 0; }
    first_bit = 1u << (((me >> 16) - k_lo) & 31u);
  }
  const uint32_t FS = single ? 1u : __reduce_or_sync(0xFFFFFFFFu, first_bit); /* lanes with the first string of a line */
  __syncwarp();
  bool slow = false;
  uint32_t st = IS_ROOT, pk = 0, rows_at = 0, rows_end = 0, nT = 0, nP = 0;
  for (uint32_t k0 = k_lo; k0 < k_hi; k0 += 32) {
    const uint32_t k = k0 + lane;
    const bool live = k < k_hi;
    const bool first_group = k0 == k_lo;
    const uint32_t pr = pairs[live ? k : nstr], nx = pairs[live ? k + 1u : nstr];
    const uint32_t open = pr & 0xFFFFu, close = pr >> 16;
    const uint32_t ln = single ? i0 : i0 + (uint32_t)__popc(FS & le) - 1u; /* this lane's line */
    const bool first = single ? k == k_lo : live && ((FS >> lane) & 1u);
    const uint32_t line_end = live ? sh.line[ln + 1u] : 0u;
    const uint32_t sep = (line_end & 0xFFFFu) - 1u;
    const bool last = live && k + 1u == line_end >> 16;
    const uint32_t b = last ? sep : nx & 0xFFFFu; /* end of the gap: the next string, or the line's separator */
    uint32_t* row = rows + (live ? ln : i0) * STRIDE;
    const bool trunc = truncs && live && close == sep;
    const uint32_t from = trunc ? sep : close + 1u;
    const uint32_t freed = live ? item_freed(win, moved, k, close) : 0u;

    /* ---- the gap behind the string ---- */
    ItemView v;
    v.vpos = b; v.vend = 0; v.clpos = b - 1u;
    {
      /* without blanks: the bytes themselves, or `:0` and what follows the number (found from the gap's end) */
      const uint32_t len0 = b - from;
      const uint32_t* hp = reinterpret_cast<const uint32_t*>(win) + (from >> 2);
      const uint32_t hs = (from & 3u) * 8u, h0 = hp[0], h1 = hp[1], h2 = hp[2];
      uint32_t lo = __funnelshift_r(h0, h1, hs), hi = __funnelshift_r(h1, h2, hs), len = len0;
      const uint32_t c0 = lo & 0xFFu, c1 = (lo >> 8) & 0xFFu;
      bool fits = len0 <= 8u;
      hi = len0 <= 4u ? 0u : (len0 < 8u ? hi & ((1u << (8u * (len0 & 3u))) - 1u) : hi);
      lo = len0 < 4u ? lo & ((1u << (8u * len0)) - 1u) : lo;
      if (c0 == ':' && len0 > 1u) v.vpos = from + 1u;
      if (c0 == ':' && len0 > 2u && (c1 - (uint32_t)'0' <= 9u || c1 == '-' || c1 - (uint32_t)'a' <= 25u)) {
        const uint32_t* tp = reinterpret_cast<const uint32_t*>(win) + ((b - 4u) >> 2);
        const uint32_t ts = (b & 3u) * 8u;
        const uint32_t th = __funnelshift_r(tp[0], tp[1], ts); /* the last four bytes */
        /* bytes 0x30-0x3F and 0x60-0x6F: digits, and the letters a literal ends with */
        const uint32_t x3 = (th ^ 0x30303030u) & 0xF0F0F0F0u, x6 = (th ^ 0x60606060u) & 0xF0F0F0F0u;
        const uint32_t z = ~((((x3 & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x3) & (((x6 & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x6)) & 0x80808080u;
        const uint32_t tail = (uint32_t)__clz((int)z) >> 3; /* bytes behind the last of them; 4: none of the four is one */
        v.vend = b - tail;
        fits = tail <= 3u && (tail >= 1u);
        len = tail + 2u;
        const uint32_t t = fits ? th >> (32u - 8u * tail) : 0u;
        lo = (t << 16) | (uint32_t)':' | ((uint32_t)'0' << 8); hi = t >> 16;
      }
      v.desc = fits ? item_gap_find(sh, lo, hi, len) : 0u;
    }
    if (live && v.desc == 0 && !trunc) item_gap_spaced<ARR>(sh, win, from, b, v);
    if (live && v.desc != 0 && last != ((v.desc & ItGap::ENDS) != 0)) v.desc = 0;
    const bool ok = live && v.desc != 0;
    const uint32_t d = ok ? v.desc : ItGap::make(IV_NONE, 15, IS_ROOT, false, false, false, false), vk = ItGap::vk(d);
    const bool telling = live && ((d & ItGap::TELLS) || last), newelem = live && (d & ItGap::ELEM);
    bool iskey = live && (d & ItGap::KEY);

    /* ---- the object the string lies in: what the nearest telling gap before it left ---- */
    const uint32_t NI = __ballot_sync(0xFFFFFFFFu, telling);
    const uint32_t pm = NI & lt;
    const uint32_t out = last ? (uint32_t)IS_ROOT : ItGap::out(d);
    const uint32_t from_lane = __shfl_sync(0xFFFFFFFFu, out, pm ? 31 - __clz((int)pm) : 0);
    const uint32_t s = pm ? from_lane : st;
    const uint32_t PK = __ballot_sync(0xFFFFFFFFu, iskey && vk == IV_STR);
    const bool isval = !first && (lane ? (PK >> (lane - 1)) & 1u : pk != 0);
    const bool iselem = live && !isval && s == IS_LIST && !iskey;
    const uint32_t need = ItGap::need(d);
    const bool role_ok = isval ? !iskey : (s == IS_LIST ? !iskey : (iskey || trunc));
    if (live) {
      if (first) { /* blanks, a brace, blanks */
        const uint32_t at = sh.line[ln] & 0xFFFFu;
        bool good = win[at] == '{' && open == at + 1u;
        if (!good) {
          uint32_t p = at;
          while (p < open && item_blank(win[p])) ++p;
          if (p < open && win[p] == '{') { ++p; while (p < open && item_blank(win[p])) ++p; good = p == open; }
        }
        if (!good || (sep >= g.hi_valid && !a.is_last)) item_error(row, at, IE_REFUSED);
      }
      if (trunc) { item_error(row, close, (uint32_t)PJ_E_EOF); if (!role_ok) item_error(row, open, IE_REFUSED); }
      else if (!ok || !role_ok || !(need == 15u || need == s)) {
        uint32_t at = close, kind = IE_REFUSED;
        if (!ok && !isval && s != IS_LIST) { /* does a bracket or brace follow the colon that the property's type rules out? */
          uint32_t p = close + 1u;
          while (p < sep && item_blank(win[p])) ++p;
          if (p < sep && win[p] == ':') {
            ++p;
            while (p < sep && item_blank(win[p])) ++p;
            const uint32_t x = p < sep ? win[p] : 0u;
            const uint32_t f = item_key(sh, win, open + 1u, close - freed - open - 1u, s), fk = ItField::kind(f);
            const bool everyones = SCHEMA != PJ_SCHEMA_MIXED || s != IS_ROOT || ItField::models(f) == 7u; /* (another model's property has no type) */
            if (f && everyones && ((x == '[' && fk != K_LIST_STR && fk != K_LIST_OBJ) || (x == '{' && fk != K_OBJ))) { at = p; kind = (uint32_t)PJ_E_TYPE; }
          }
        }
        item_error(row, at, kind);
        iskey = false;
      }
      if (last) reinterpret_cast<uint16_t*>(&row[IW_POS])[1] = (uint16_t)v.clpos;
      if (special) {
        if (((sh.special[k >> 5] | sh.broken[k >> 5]) >> (k & 31u)) & 1u) {
          atomicOr(&row[IW_FLAGS], IF_MOVED);
          if ((sh.broken[k >> 5] >> (k & 31u)) & 1u) item_error(row, open - 1u, IE_REFUSED); /* before anything its text is judged by */
        }
      }
    }
    uint32_t NE = 0, erow = 0;
    if constexpr (ItemSlots<SCHEMA>::lists) {
      const uint32_t EL = __ballot_sync(0xFFFFFFFFu, iselem);
      NE = __ballot_sync(0xFFFFFFFFu, newelem);
      if (EL | NE) {
        /* lanes of this lane's line */
        const uint32_t lo = single ? 0u : 31u - (uint32_t)__clz((int)(FS & le)), up = single ? 0u : FS & ~le;
        const uint32_t mine = (up ? (up & (0u - up)) - 1u : 0xFFFFFFFFu) & ~((1u << lo) - 1u);
        if (iselem) {
          if (close - open > 0x8000u) slow = true;
          atomicAdd(&row[LW + 1u], close - open - 1u - freed);
          if (!single) { if (!(EL & mine & lt)) row[IW_LIST] = k | ((uint32_t)__popc(EL & mine) << 16); }
          else if (nP == 0 && !(EL & lt)) row[IW_LIST] = k;
        }
        if (NE) {
          /* rows of the elements: of a pack, all at once; of a long line, room for as many as its strings can make */
          const uint32_t want = single ? 3u * ((k_hi - k0 + 1u) / 2u + 1u) : 3u * (uint32_t)__popc(NE);
          if (!single || rows_end == 0) {
            if (lane == 0) rows_at = atomicAdd(&sh.free_word, want);
            rows_at = __shfl_sync(0xFFFFFFFFu, rows_at, 0);
            rows_end = rows_at + want;
            if (rows_end > a.str_words) slow = true;
          }
          if (newelem) {
            const uint32_t r = rows_at + 3u * (nT + (uint32_t)__popc(NE & lt));
            if (r + 3u > rows_end) slow = true;
            if (!slow) { pairs[r] = 0; pairs[r + 1u] = 0; pairs[r + 2u] = 0; }
            if (!single) { if (!(NE & mine & lt)) row[LW] = r | ((uint32_t)__popc(NE & mine) << 16); }
            else if (nT == 0 && !(NE & lt)) row[LW] = r;
          }
          slow = __any_sync(0xFFFFFFFFu, slow); /* (and every row is empty before a key writes to it) */
        }
      }
      erow = rows_at + 3u * (nT + (uint32_t)__popc(NE & lt) - 1u);
      nP += (uint32_t)__popc(EL);
    }
    /* ---- keys ---- */
    if (iskey && !slow) {
      const uint32_t len = close - open - 1u - freed;
      const uint32_t f = item_key(sh, win, open + 1u, len, s);
      const uint32_t vlen = v.vend - v.vpos;
      if (!f) {
        if (!(vk == IV_STR || (vk == IV_SCALAR && item_plain_scalar(win, v.vpos, vlen)))) item_error(row, close, IE_REFUSED);
      } else {
        const uint32_t kind = ItField::kind(f), vclose = nx >> 16;
        const bool null = vk == IV_SCALAR && vlen == 4u && item_peek4(win, v.vpos) == 0x6C6C756Eu;
        bool good = ((ItField::allowed(f) >> vk) & 1u) != 0;
        const uint32_t n_val = vk == IV_STR ? vclose - b - 1u - item_freed(win, moved, k + 1u, vclose) : vlen;
        uint32_t ref = (vk == IV_STR ? b + 1u : v.vpos) | (n_val << 16);
        if ((vk == IV_STR || vk == IV_SCALAR) && n_val >= 0x8000u) slow = true;
        if (!good && !null) {
          const uint32_t at = vk == IV_STR ? b : v.vpos, x = win[at];
          if ((a.opts & PJ_OPT_COERCE_SCALARS) && ((vk == IV_STR && (kind == K_I64 || kind == K_I32 || kind == K_BOOL)) || (vk == IV_SCALAR && kind == K_STR))) {
            if (vk == IV_STR) ref |= 0x80000000u;
            else if (!item_plain_scalar(win, at, vlen)) item_error(row, at, IE_REFUSED);
            good = true;
          } else if ((kind == K_LIST_STR && vk == IV_ELEM) || (kind == K_LIST_OBJ && vk == IV_LIST) || (vk == IV_SCALAR && !(x == '-' || x - (uint32_t)'0' <= 9u || x == 't' || x == 'f')))
            item_error(row, close, IE_REFUSED);
          else if (SCHEMA == PJ_SCHEMA_MIXED && s == IS_ROOT && ItField::models(f) != 7u) item_error(row, close, IE_REFUSED); /* another model's property has no type */
          else item_error(row, at, PJ_E_TYPE);
        }
        if (truncs && vk == IV_STR && vclose == (sh.line[ln + 1u] & 0xFFFFu) - 1u) good = false; /* cut off: it reports that itself */
        const uint32_t bit = 1u << ItField::bit(f), word = ItField::word(f);
        const bool keep = good && !null;
        if (s == IS_ELEM) {
          /* integers are decoded here, a string's reference is kept (twelve bits of length) */
          uint32_t w2 = bit << 30 | (keep ? bit << 28 : 0u);
          if (keep && kind == K_STR) {
            if (n_val >= 0x1000u) slow = true;
            w2 |= ref & 0x0FFFFFFFu;
            atomicAdd(&row[LW + 1u], n_val << 16);
          } else if (keep) {
            int64_t val = 0;
            const uint32_t at = ref & 0xFFFFu;
            if (!item_int(win, at, n_val, kind == K_I64, &val)) {
              const uint32_t x = win[at];
              item_error(row, ref >> 31 ? at - 1u : at, (!(ref >> 31) && item_other_type(x)) ? (uint32_t)PJ_E_TYPE : IE_REFUSED);
            }
            if (!slow) { pairs[erow] = (uint32_t)(uint64_t)val; pairs[erow + 1u] = (uint32_t)((uint64_t)val >> 32); }
          }
          if (!slow) { if ((atomicOr(&pairs[erow + 2u], w2) >> 30) & bit) item_error(row, close, IE_REFUSED); } /* repeated key */
        } else {
          const uint32_t nm = SCHEMA == PJ_SCHEMA_MIXED && s == IS_ROOT ? (~ItField::models(f) & 7u) << IF_NOTMODEL : 0u;
          const uint32_t old = atomicOr(&row[IW_FLAGS], bit | nm | (keep ? bit << IF_PRESENT : 0u));
          if (old & bit) item_error(row, close, IE_REFUSED);
          /* of a key given twice the first value is judged (a failure there comes before the repetition) */
          if (keep && kind <= K_DATETIME && !(old & (bit << IF_PRESENT))) row[word] = ref;
        }
      }
    }
    nT += (uint32_t)__popc(NE);
    st = NI ? __shfl_sync(0xFFFFFFFFu, out, 31 - __clz((int)NI)) : st;
    pk = (PK >> 31) & 1u;
    if (__any_sync(0xFFFFFFFFu, slow)) {
      __syncwarp(); /* every lane is through with the rows */
      if (lane < n) {
        uint32_t* row = rows + (i0 + lane) * STRIDE;
        const uint32_t at = sh.line[i0 + lane] & 0xFFFFu;
        row[IW_FLAGS] = IF_RECORD; row[IW_ERR] = (at << 8) | IE_REFUSED;
        if constexpr (ItemSlots<SCHEMA>::lists) { row[IW_LIST] = 0; row[LW] = 0; row[LW + 1u] = 0; }
      }
      __syncwarp();
      return;
    }
  }
  if constexpr (ItemSlots<SCHEMA>::lists) {
    if (single && lane == 0) { uint32_t* row = rows + i0 * STRIDE; row[IW_LIST] |= nP << 16; row[LW] |= nT << 16; }
  }
  __syncwarp();
}
/* The lines the walk did not recognise: each by a warp when they are few, otherwise runs of them, several to a step. */
template <int SCHEMA, bool ARR>
__device__ __forceinline__ void item_packs(const ItemArgs& a, const StreamGeom& g, ItemShared& sh, const uint8_t* win, uint32_t* pairs, uint32_t* rows, uint32_t nodd) {
  const uint32_t lane = threadIdx.x & 31u, nline = sh.nline;
  const bool few = nodd * 4u <= nline;
  for (;;) {
    uint32_t x = 0;
    if (lane == 0) x = atomicAdd(&sh.next, few ? 1u : 4u);
    x = __shfl_sync(0xFFFFFFFFu, x, 0);
    if (x >= (few ? nodd : nline)) return;
    uint32_t i = x, end = x + 4u < nline ? x + 4u : nline;
    if (few) { /* line number x of the odd ones */
      uint32_t at = 0;
      i = 0;
#pragma unroll
      for (uint32_t k = 0; k < IT_WARPS; ++k) {
        const uint32_t m = sh.oddmask[k], n = (uint32_t)__popc(m);
        if (x >= at && x < at + n) {
          const bool hit = (uint32_t)__popc(m & ((1u << lane) - 1u)) == x - at && ((m >> lane) & 1u);
          i = 32u * k + (uint32_t)__ffs((int)__ballot_sync(0xFFFFFFFFu, hit)) - 1u;
        }
        at += n;
      }
      end = i + 1u;
    }
    while (i < end) {
      const uint32_t k0 = sh.line[i] >> 16;
      if (!((sh.oddmask[i >> 5] >> (i & 31u)) & 1u)) { ++i; continue; }
      uint32_t n = 1;
      while (i + n < end && ((sh.oddmask[(i + n) >> 5] >> ((i + n) & 31u)) & 1u) && (sh.line[i + n + 1u] >> 16) - k0 <= 32u && sh.line[i + n + 1u] >> 16 != sh.line[i + n] >> 16) ++n;
      item_pack<SCHEMA, ARR>(a, g, sh, win, pairs, rows, i, n);
      i += n;
    }
  }
}

/* ---- 4. values ------------------------------------------------------------------------------------------------ */
/* The integers, of any model, one after the other: word | bit << 8 | int64 << 16; 0 = no more. */
template <int OBJ>
PJ_CX uint32_t it_int_field(uint32_t nth) {
  uint32_t at = 0;
  for (int i = 0; i < CObj<OBJ>::N; ++i) {
    const uint32_t kind = CObj<OBJ>::f[i].kind;
    if (kind != K_I64 && kind != K_I32) continue;
    if (at++ == nth) return it_root_word<OBJ>(i) | ((uint32_t)i << 8) | ((kind == K_I64 ? 1u : 0u) << 16);
  }
  return 0;
}
template <int OBJ, int CH>
PJ_CX uint32_t it_int_all(uint32_t nth) { /* the embedded object's come after the root's */
  const uint32_t r = it_int_field<OBJ>(nth);
  if (r) return r;
  if constexpr (CH >= 0) {
    uint32_t own = 0;
    for (int i = 0; i < CObj<OBJ>::N; ++i) own += CObj<OBJ>::f[i].kind == K_I64 || CObj<OBJ>::f[i].kind == K_I32;
    uint32_t at = own;
    for (int i = 0; i < CObj<CH>::N; ++i) {
      const uint32_t kind = CObj<CH>::f[i].kind;
      if (kind != K_I64 && kind != K_I32) continue;
      if (at++ == nth) return (ItModel<OBJ>::child_word + it_flat_word<CH>(i)) | ((IB_CHILD + (uint32_t)i) << 8) | ((kind == K_I64 ? 1u : 0u) << 16);
    }
  }
  return 0;
}
template <int OBJ, uint32_t NTH> struct ItInt { static constexpr uint32_t v = it_int_all<OBJ, ItModel<OBJ>::child>(NTH); };

/* Model of a row: PJ_TYPE_*, 0 when the keys do not tell (mixed streams). */
template <int SCHEMA>
__device__ __forceinline__ uint32_t item_type(uint32_t flags) {
  if constexpr (SCHEMA != PJ_SCHEMA_MIXED) return (uint32_t)SCHEMA;
  else {
    const uint32_t m = ~(flags >> IF_NOTMODEL) & 7u;
    return m == 1u ? (uint32_t)PJ_TYPE_PET : (m == 2u ? (uint32_t)PJ_TYPE_ORDER : (m == 4u ? (uint32_t)PJ_TYPE_USER : (uint32_t)PJ_TYPE_NONE));
  }
}
/* The values of one field (or of the integer number V) of 32 lines, a line per lane. */
enum { VU_INT0 = 0, VU_INT1 = 1, VU_INT2 = 2, VU_ENUM = 3, VU_BOOL = 4, VU_DATE = 5, VU_ELEM = 6, VU_COUNT = 7 };
template <int SCHEMA> struct ItemValueUnits {
  static constexpr uint32_t mask = SCHEMA == PJ_SCHEMA_PET ? (1u << VU_ELEM) | (1u << VU_INT0) | (1u << VU_INT1) | (1u << VU_ENUM)
                                   : (SCHEMA == PJ_SCHEMA_ORDER ? 0x3Fu : (SCHEMA == PJ_SCHEMA_USER ? (1u << VU_INT0) | (1u << VU_INT1) : 0x7Fu));
};
static_assert(ItInt<OBJ_PET, 2>::v == 0 && ItInt<OBJ_ORDER, 3>::v == 0 && ItInt<OBJ_USER, 2>::v == 0, "integers per model");
template <int OBJ, uint32_t KIND>
__device__ __forceinline__ uint32_t item_kind_field() { /* word | bit << 8 of the property of this kind */
  constexpr int i = it_find<OBJ>(KIND);
  if constexpr (i < 0) return 0;
  else return it_root_word<OBJ>(i) | ((uint32_t)i << 8);
}
template <int SCHEMA, uint32_t KIND>
__device__ __forceinline__ uint32_t item_field_of(uint32_t type) {
  if constexpr (SCHEMA == PJ_SCHEMA_PET) return item_kind_field<OBJ_PET, KIND>();
  else if constexpr (SCHEMA == PJ_SCHEMA_ORDER) return item_kind_field<OBJ_ORDER, KIND>();
  else if constexpr (SCHEMA == PJ_SCHEMA_USER) return item_kind_field<OBJ_USER, KIND>();
  else return type == PJ_TYPE_PET ? item_kind_field<OBJ_PET, KIND>() : (type == PJ_TYPE_ORDER ? item_kind_field<OBJ_ORDER, KIND>() : item_kind_field<OBJ_USER, KIND>());
}
template <int SCHEMA, uint32_t NTH>
__device__ __forceinline__ uint32_t item_int_of(uint32_t type) {
  if constexpr (SCHEMA == PJ_SCHEMA_PET) return ItInt<OBJ_PET, NTH>::v;
  else if constexpr (SCHEMA == PJ_SCHEMA_ORDER) return ItInt<OBJ_ORDER, NTH>::v;
  else if constexpr (SCHEMA == PJ_SCHEMA_USER) return ItInt<OBJ_USER, NTH>::v;
  else return type == PJ_TYPE_PET ? ItInt<OBJ_PET, NTH>::v : (type == PJ_TYPE_ORDER ? ItInt<OBJ_ORDER, NTH>::v : ItInt<OBJ_USER, NTH>::v);
}
/* Element j of a list of objects as the walk left it (three strings: a key, a key, a value) into its row of three words. */
__device__ __forceinline__ void item_elem_row(const uint8_t* win, const uint32_t* moved, uint32_t* pairs, uint32_t k, uint32_t* row) {
  uint32_t* e = pairs + k;
  const uint32_t p0 = e[0], p1 = e[1], p2 = e[2];
  uint32_t at = (p0 >> 16) + 1u, end = (p1 & 0xFFFFu) - 1u; /* at the colon and at the comma, but for blanks */
  const uint32_t from = at, to = end;
  while (at < to && win[at] != ':') ++at;
  ++at;
  while (at < to && item_blank(win[at])) ++at;
  while (end > from && win[end] != ',') --end;
  while (end > at && item_blank(win[end - 1u])) --end;
  int64_t val = 0;
  if (end <= at || !item_int(win, at, end - at, true, &val)) { const uint32_t x = win[at]; item_error(row, at, item_other_type(x) ? (uint32_t)PJ_E_TYPE : IE_REFUSED); }
  const uint32_t open = p2 & 0xFFFFu, n = (p2 >> 16) - open - 1u - item_freed(win, moved, k + 2u, p2 >> 16);
  e[0] = (uint32_t)(uint64_t)val; e[1] = (uint32_t)((uint64_t)val >> 32);
  e[2] = (open + 1u) | (n << 16) | 0xF0000000u;
}
/* The elements of the lists of 32 lines (n of a lane's), 32 at a time: f(line's lane, element of the line's list, live). */
template <class F>
__device__ __forceinline__ void item_each_element(uint8_t* owner, uint32_t n, F f) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t inc = warp_incl_scan(n), e = inc - n, total = __shfl_sync(0xFFFFFFFFu, inc, 31);
  const uint32_t some = __ballot_sync(0xFFFFFFFFu, n != 0);
  if (n) owner[__popc(some & ((1u << lane) - 1u))] = (uint8_t)lane;
  __syncwarp();
  for (uint32_t r = 0; r < total; r += 32) {
    const uint32_t before = (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, n != 0 && e < r));
    const uint32_t starts = __reduce_or_sync(0xFFFFFFFFu, n != 0 && e - r < 32u ? 1u << (e - r) : 0u);
    const uint32_t src = owner[before + (uint32_t)__popc(starts & ((2u << lane) - 1u)) - 1u]; /* lane 31: 2 << 31 wraps to 0, so all ones */
    const uint32_t se = __shfl_sync(0xFFFFFFFFu, e, (int)src);
    f(src, r + lane - se, r + lane < total);
  }
  __syncwarp();
}
template <int SCHEMA>
__device__ __forceinline__ void item_value(const ItemArgs& a, uint8_t* owner, const uint32_t* moved, const uint8_t* win, uint32_t* pairs, uint32_t* rows, uint32_t* row, bool live, uint32_t unit) {
  const uint32_t flags = live ? row[IW_FLAGS] : 0u;
  const bool rec = (flags & IF_RECORD) != 0; /* refused ones too: an earlier failure may be found here, and every value present has its reference */
  const uint32_t type = item_type<SCHEMA>(flags);
  Win w;
  w.s = win; w.w0 = 0;
  if (unit <= VU_INT2) {
    const uint32_t desc = unit == VU_INT0 ? item_int_of<SCHEMA, 0>(type) : (unit == VU_INT1 ? item_int_of<SCHEMA, 1>(type) : item_int_of<SCHEMA, 2>(type));
    const uint32_t word = desc & 255u, bit = (desc >> 8) & 255u;
    if (rec && desc && ((flags >> (IF_PRESENT + bit)) & 1u)) {
      const bool is64 = (desc >> 16) & 1u;
      const uint32_t ref = row[word], pos = ref & 0xFFFFu;
      int64_t v = 0;
      if (!item_int(win, pos, (ref >> 16) & 0x7FFFu, is64, &v)) {
        const uint32_t x = win[pos];
        item_error(row, ref >> 31 ? pos - 1u : pos, (!(ref >> 31) && item_other_type(x)) ? (uint32_t)PJ_E_TYPE : IE_REFUSED);
      }
      row[word] = (uint32_t)(uint64_t)v;
      if (is64) row[word + 1] = (uint32_t)((uint64_t)v >> 32);
    }
  } else if (unit == VU_ENUM) {
    uint32_t desc = item_field_of<SCHEMA, K_ENUM>(type), bit = desc >> 8;
    if (SCHEMA == PJ_SCHEMA_MIXED && (flags & IF_ROWS)) { /* its key is one of two models' */
      bit = IB_SHARED;
      if (rec && type != PJ_TYPE_NONE && ((flags >> (IF_PRESENT + IB_SHARED)) & 1u)) atomicOr(&row[IW_FLAGS], 1u << (IF_PRESENT + (desc >> 8)));
    }
    if (rec && desc && ((flags >> (IF_PRESENT + bit)) & 1u)) {
      const uint32_t word = desc & 255u, ref = row[word], pos = ref & 0xFFFFu, n = (ref >> 16) & 0x7FFFu;
      int e = -1;
      if (n <= 14) {
        const uint64_t x = wpeek8(w, pos), y = wpeek8(w, pos + 8);
        const uint64_t lo = n >= 8 ? x : (n ? x & (~0ull >> (64 - 8 * n)) : 0);
        const uint64_t hi = n > 8 ? y & (~0ull >> (64 - 8 * (n - 8))) : 0;
        if (SCHEMA == PJ_SCHEMA_PET || (SCHEMA == PJ_SCHEMA_MIXED && type == PJ_TYPE_PET)) e = match_enum<0>(n, lo, hi);
        else e = match_enum<1>(n, lo, hi);
      }
      if (e >= 0) row[word] = (uint32_t)e;
      else if (a.opts & PJ_OPT_ENUM_UNKNOWN_AS_NULL) atomicAnd(&row[IW_FLAGS], ~(1u << (IF_PRESENT + (desc >> 8))));
      else item_error(row, pos - 1u, PJ_E_ENUM);
    }
  } else if (unit == VU_BOOL) {
    const uint32_t desc = item_field_of<SCHEMA, K_BOOL>(type);
    if (rec && desc && ((flags >> (IF_PRESENT + (desc >> 8))) & 1u)) {
      const uint32_t word = desc & 255u, ref = row[word], pos = ref & 0xFFFFu, n = (ref >> 16) & 0x7FFFu;
      if (item_true(win, pos, n)) row[word] = 1;
      else if (item_false(win, pos, n)) row[word] = 0;
      else { const uint32_t x = win[pos]; item_error(row, pos, (!(ref >> 31) && (x == '-' || x - (uint32_t)'0' <= 9u)) ? (uint32_t)PJ_E_TYPE : IE_REFUSED); }
    }
  } else if (unit == VU_DATE) {
    const uint32_t desc = item_field_of<SCHEMA, K_DATETIME>(type);
    if (rec && desc && ((flags >> (IF_PRESENT + (desc >> 8))) & 1u)) {
      const uint32_t word = desc & 255u, ref = row[word], pos = ref & 0xFFFFu;
      int64_t ep = 0; int32_t ns = 0, of = 0;
      if (fast_datetime(w, pos, (ref >> 16) & 0x7FFFu, &ep, &ns, &of)) {
        row[word] = (uint32_t)(uint64_t)ep; row[word + 1] = (uint32_t)((uint64_t)ep >> 32); row[word + 2] = (uint32_t)ns; row[word + 3] = (uint32_t)of;
      } else item_error(row, pos - 1u, PJ_E_DATETIME);
    }
  } else if constexpr (ItemSlots<SCHEMA>::lists) { /* elements of lists of objects that the walk found */
    const bool mine = rec && type == PJ_TYPE_PET && !(flags & IF_ROWS);
    const uint32_t l = mine ? row[ItWords<OBJ_PET>::n] : 0u, n = l >> 16;
    const uint32_t at = (uint32_t)(row - rows);
    item_each_element(owner, n, [&](uint32_t src, uint32_t j, bool has) {
      const uint32_t k = __shfl_sync(0xFFFFFFFFu, l, (int)src) & 0xFFFFu, r = __shfl_sync(0xFFFFFFFFu, at, (int)src);
      if (has) item_elem_row(win, moved, pairs, k + 3u * j, rows + r);
    });
  }
}

/* ---- 5. emission ------------------------------------------------------------------------------------------------ */
/* n bytes at window offset pos to dst (any alignment): whole words of dst, odd bytes at both ends */
__device__ __forceinline__ void item_copy(uint8_t* dst, const uint8_t* win, uint32_t pos, uint32_t n) {
  uint32_t h = (0u - (uint32_t)reinterpret_cast<uintptr_t>(dst)) & 3u;
  if (h > n) h = n;
  if (h > 0) dst[0] = win[pos];
  if (h > 1) dst[1] = win[pos + 1];
  if (h > 2) dst[2] = win[pos + 2];
  dst += h; pos += h; n -= h;
  const uint32_t* p = reinterpret_cast<const uint32_t*>(win) + (pos >> 2);
  const uint32_t sh = (pos & 3u) * 8u, nw = n >> 2;
  uint32_t x0 = p[0];
  uint32_t* d4 = reinterpret_cast<uint32_t*>(dst);
  for (uint32_t i = 0; i < nw; ++i) {
    const uint32_t x1 = p[i + 1];
    d4[i] = __funnelshift_r(x0, x1, sh);
    x0 = x1;
  }
  const uint32_t t = n & 3u;
  if (t) {
    const uint32_t last = __funnelshift_r(x0, p[nw + 1], sh);
    uint8_t* e = dst + 4u * nw;
    e[0] = (uint8_t)last;
    if (t > 1) e[1] = (uint8_t)(last >> 8);
    if (t > 2) e[2] = (uint8_t)(last >> 16);
  }
}
/* The strings of a warp's lanes (n bytes at window offset pos), one behind the other from dst on: put together in shared
 * memory, so that they leave in whole words side by side. Returns their bytes. rel: bytes of the lanes before. */
__device__ __forceinline__ void item_emit_run(uint32_t* stage, uint8_t* dst, const uint8_t* win, uint32_t pos, uint32_t n, uint32_t rel, uint32_t total) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t d0 = (uint32_t)reinterpret_cast<uintptr_t>(dst) & 3u, end = d0 + total;
  if (end > IT_STAGE * 4u) { if (n) item_copy(dst + rel, win, pos, n); return; }
  const uint32_t nw = (end + 3u) >> 2;
  for (uint32_t j = lane; j < nw; j += 32) stage[j] = 0;
  __syncwarp();
  if (n) {
    const uint32_t b = d0 + rel, lead = b & 3u, k1 = (lead + n - 1u) >> 2; /* last word */
    const int32_t from = (int32_t)pos - (int32_t)lead;
    const uint32_t* p = reinterpret_cast<const uint32_t*>(win) + (from >> 2);
    const uint32_t sh = ((uint32_t)from & 3u) * 8u;
    uint32_t* d = stage + (b >> 2);
    uint32_t x0 = p[0], keep = 0xFFFFFFFFu << (8u * lead), k = 0;
    if (k1) { /* the first word may be shared with the string before */
      const uint32_t x1 = p[1];
      atomicOr(d, __funnelshift_r(x0, x1, sh) & keep);
      keep = 0xFFFFFFFFu;
      x0 = x1; k = 1;
    }
    for (; k + 4u <= k1; k += 4u) { /* four loads on their way at a time: 2 M mixed records 2.02 -> 1.97 ms */
      const uint32_t x1 = p[k + 1], x2 = p[k + 2], x3 = p[k + 3], x4 = p[k + 4];
      d[k] = __funnelshift_r(x0, x1, sh); d[k + 1] = __funnelshift_r(x1, x2, sh); d[k + 2] = __funnelshift_r(x2, x3, sh); d[k + 3] = __funnelshift_r(x3, x4, sh);
      x0 = x4;
    }
    for (; k < k1; ++k) {
      const uint32_t x1 = p[k + 1];
      d[k] = __funnelshift_r(x0, x1, sh);
      x0 = x1;
    }
    const uint32_t v = __funnelshift_r(x0, p[k1 + 1], sh) & keep & (0xFFFFFFFFu >> (8u * (3u - ((lead + n - 1u) & 3u))));
    atomicOr(d + k1, v);
  }
  __syncwarp();
  uint32_t* out = reinterpret_cast<uint32_t*>(dst - d0);
  for (uint32_t j = lane; j < nw; j += 32) {
    const uint32_t v = stage[j];
    if ((j > 0 || d0 == 0) && 4u * j + 4u <= end) out[j] = v;
    else for (uint32_t b = 0; b < 4; ++b) if (4u * j + b >= d0 && 4u * j + b < end) reinterpret_cast<uint8_t*>(out + j)[b] = (uint8_t)(v >> (8u * b));
  }
  __syncwarp();
}
/* The place of a model root's row among 32 lines and what a lane needs to write it. */
struct ItemOut {
  const uint8_t* win;
  const uint32_t* row;
  uint32_t* stage;
  uint8_t* owner;
  const uint32_t* moved;
  uint32_t flags, chunk;
  uint32_t apart; /* lanes of this model whose record stands apart */
  bool has_row;
  uint64_t at; /* row of the model's table */
};
/* first counter of a model; its row of a record that stands apart holds them in order */
template <int OBJ> struct ItSlot0 { static constexpr uint32_t n = OBJ == OBJ_USER ? (uint32_t)SLOT_USR_STR0 : (uint32_t)SLOT_PET_CAT_NAME; };
static constexpr uint32_t IT_APART = 6; /* counters of a model */
static_assert((uint32_t)SLOT_USR_STR0 - (uint32_t)SLOT_PET_CAT_NAME == IT_APART && NSLOT - (uint32_t)SLOT_USR_STR0 == IT_APART, "as many for Pets as for Users");
static_assert(ItWords<OBJ_PET>::n >= IW_FIELDS + IT_APART && ItStride<PJ_SCHEMA_USER>::n >= IW_FIELDS + IT_APART, "room for them");
/* Lanes side by side, without those apart, one run of them after the other: f(first lane, behind the last one). Nearly always one. */
template <class F>
__device__ __forceinline__ void item_each_run(uint32_t apart, F f) {
  for (uint32_t lo = 0; lo < 32;) {
    const uint32_t rest = apart >> lo, end = rest ? lo + (uint32_t)__ffs((int)rest) - 1u : 32u;
    if (end > lo) f(lo, end);
    lo = end + 1u;
  }
}
/* fixed-width columns of root or embedded object OBJ */
template <int OBJ, bool ROOT, uint32_t WORD0, uint32_t BIT0, int I = 0>
__device__ __forceinline__ void item_emit_fixed(const ItemArgs& a, const ItemOut& o) {
  if constexpr (I == 0) colp<uint8_t>(&a.cols, CObj<OBJ>::present_col)[o.at] = (uint8_t)((o.flags >> (IF_PRESENT + BIT0)) & ((1u << CObj<OBJ>::N) - 1u));
  if constexpr (I < CObj<OBJ>::N) {
    constexpr uint32_t kind = CObj<OBJ>::f[I].kind, col = CObj<OBJ>::f[I].col;
    constexpr uint32_t word = ROOT ? it_root_word<OBJ>(I) : WORD0 + it_flat_word<OBJ>(I);
    const bool pr = (o.flags >> (IF_PRESENT + BIT0 + I)) & 1u;
    const uint32_t* row = o.row;
    if constexpr (kind == K_I64) colp<int64_t>(&a.cols, col)[o.at] = pr ? (int64_t)((uint64_t)row[word] | ((uint64_t)row[word + 1] << 32)) : 0;
    else if constexpr (kind == K_I32) colp<int32_t>(&a.cols, col)[o.at] = pr ? (int32_t)row[word] : 0;
    else if constexpr (kind == K_BOOL || kind == K_ENUM) colp<uint8_t>(&a.cols, col)[o.at] = pr ? (uint8_t)row[word] : (kind == K_ENUM ? 255 : 0);
    else if constexpr (kind == K_DATETIME) {
      colp<int64_t>(&a.cols, col)[o.at] = pr ? (int64_t)((uint64_t)row[word] | ((uint64_t)row[word + 1] << 32)) : 0;
      colp<int32_t>(&a.cols, col + 1)[o.at] = pr ? (int32_t)row[word + 2] : 0;
      colp<int32_t>(&a.cols, col + 2)[o.at] = pr ? (int32_t)row[word + 3] : 0;
    } else if constexpr (kind == K_OBJ) item_emit_fixed<CObj<OBJ>::f[I].child, false, ItModel<OBJ>::child_word, IB_CHILD>(a, o);
    item_emit_fixed<OBJ, ROOT, WORD0, BIT0, I + 1>(a, o);
  }
}
/* string columns of root or embedded object OBJ (every lane of the warp calls this). APART: some of the tile's records stand apart */
template <bool APART, int MODEL, int OBJ, bool ROOT, uint32_t WORD0, uint32_t BIT0, int I = 0>
__device__ __forceinline__ void item_emit_strings(const ItemArgs& a, const ItemShared& sh, const ItemOut& o) {
  if constexpr (I < CObj<OBJ>::N) {
    constexpr uint32_t kind = CObj<OBJ>::f[I].kind, col = CObj<OBJ>::f[I].col, slot = CObj<OBJ>::f[I].cnt;
    constexpr uint32_t word = ROOT ? it_root_word<OBJ>(I) : WORD0 + it_flat_word<OBJ>(I);
    if constexpr (kind == K_STR) {
      const bool pr = o.has_row && ((o.flags >> (IF_PRESENT + BIT0 + I)) & 1u);
      const uint32_t ref = o.row[word], n = pr ? (ref >> 16) & 0x7FFFu : 0u, at = sh.base[slot] + sh.csum[slot][o.chunk];
      if constexpr (!APART) {
        const uint32_t inc = warp_incl_scan(n);
        if (o.has_row) colp<uint32_t>(&a.cols, col)[o.at] = at + inc - n;
        item_emit_run(o.stage, colp<uint8_t>(&a.cols, col + 1) + at, o.win, ref & 0xFFFFu, n, inc - n, __shfl_sync(0xFFFFFFFFu, inc, 31));
      } else {
        const uint32_t lane = threadIdx.x & 31u, all = (o.apart >> lane) & 1u ? o.row[IW_FIELDS + slot - ItSlot0<MODEL>::n] : n, inc = warp_incl_scan(all);
        if (o.has_row) colp<uint32_t>(&a.cols, col)[o.at] = at + inc - all;
        item_each_run(o.apart, [&](uint32_t lo, uint32_t end) {
          const uint32_t from = __shfl_sync(0xFFFFFFFFu, inc - all, (int)lo), to = __shfl_sync(0xFFFFFFFFu, inc, (int)end - 1);
          item_emit_run(o.stage, colp<uint8_t>(&a.cols, col + 1) + at + from, o.win, ref & 0xFFFFu, lane >= lo && lane < end ? n : 0u, inc - all - from, to - from);
        });
      }
    } else if constexpr (kind == K_OBJ) item_emit_strings<APART, MODEL, CObj<OBJ>::f[I].child, false, ItModel<OBJ>::child_word, IB_CHILD>(a, sh, o);
    item_emit_strings<APART, MODEL, OBJ, ROOT, WORD0, BIT0, I + 1>(a, sh, o);
  }
}
/* bytes of the lines' strings per slot, added up over the warp into csum[slot][chunk] */
template <int OBJ, bool ROOT, uint32_t WORD0, uint32_t BIT0, int I = 0>
__device__ __forceinline__ void item_sum_strings(ItemShared& sh, const uint32_t* row, bool mine, uint32_t flags, uint32_t chunk, uint32_t lane) {
  if constexpr (I < CObj<OBJ>::N) {
    constexpr uint32_t kind = CObj<OBJ>::f[I].kind, slot = CObj<OBJ>::f[I].cnt;
    if constexpr (kind == K_STR) {
      constexpr uint32_t word = ROOT ? it_root_word<OBJ>(I) : WORD0 + it_flat_word<OBJ>(I);
      const uint32_t s = __reduce_add_sync(0xFFFFFFFFu, mine && ((flags >> (IF_PRESENT + BIT0 + I)) & 1u) ? (row[word] >> 16) & 0x7FFFu : 0u);
      if (lane == 0) sh.csum[slot][chunk] = s;
    } else if constexpr (kind == K_OBJ) item_sum_strings<CObj<OBJ>::f[I].child, false, ItModel<OBJ>::child_word, IB_CHILD>(sh, row, mine, flags, chunk, lane);
    item_sum_strings<OBJ, ROOT, WORD0, BIT0, I + 1>(sh, row, mine, flags, chunk, lane);
  }
}
/* the lists of 32 lines, an element per lane */
template <bool APART, bool OBJS>
__device__ __forceinline__ void item_emit_lists(const ItemArgs& a, const ItemShared& sh, const ItemOut& o, const uint32_t* pairs, bool mine) {
  constexpr int F = OBJS ? ItModel<OBJ_PET>::ei : ItModel<OBJ_PET>::li;
  constexpr int E = OBJ_TAG;
  constexpr uint32_t col = CObj<OBJ_PET>::f[F].col, slot = CObj<OBJ_PET>::f[F].cnt;
  constexpr uint32_t bslot = OBJS ? CObj<E>::f[it_string_field<E>()].cnt : slot + 1u;
  static_assert(CObj<E>::f[0].kind == K_I64 && CObj<E>::f[1].kind == K_STR, "list elements: an integer and a string");
  constexpr uint32_t off_col = OBJS ? CObj<E>::f[1].col : col + 1u;
  const uint32_t l = mine ? o.row[OBJS ? ItWords<OBJ_PET>::n : (uint32_t)IW_LIST] : 0u, n = l >> 16;
  const uint64_t r0 = (uint64_t)sh.base[slot] + sh.csum[slot][o.chunk];
  const uint32_t lane = threadIdx.x & 31u;
  const bool apart = APART && ((o.apart >> lane) & 1u);
  const uint32_t all = apart ? o.row[IW_FIELDS + slot - ItSlot0<OBJ_PET>::n] : n, inc = warp_incl_scan(all);
  if (o.has_row) colp<uint32_t>(&a.cols, col)[o.at] = (uint32_t)r0 + inc - all;
  const uint32_t at0 = sh.base[bslot] + sh.csum[bslot][o.chunk];
  uint32_t at = at0, done = 0;
  auto element = [&](uint32_t src, uint32_t j, bool has) {
    const uint32_t k = __shfl_sync(0xFFFFFFFFu, l, (int)src) & 0xFFFFu;
    const uint64_t r = r0 + done + lane;
    uint32_t pos = 0, len = 0;
    if constexpr (OBJS) {
      if (has) {
        const uint32_t* e = pairs + k + 3u * j;
        const uint32_t x = e[2];
        colp<uint8_t>(&a.cols, CObj<E>::present_col)[r] = (uint8_t)((x >> 28) & 3u);
        colp<int64_t>(&a.cols, CObj<E>::f[0].col)[r] = (x >> 28) & 1u ? (int64_t)((uint64_t)e[0] | ((uint64_t)e[1] << 32)) : 0;
        pos = x & 0xFFFFu; len = (x >> 29) & 1u ? (x >> 16) & 0xFFFu : 0u;
      }
    } else if (has) { const uint32_t pr = pairs[k + j]; pos = (pr & 0xFFFFu) + 1u; len = (pr >> 16) - pos - item_freed(o.win, o.moved, k + j, pr >> 16); }
    const uint32_t sc = warp_incl_scan(len), total = __shfl_sync(0xFFFFFFFFu, sc, 31);
    if (has) colp<uint32_t>(&a.cols, off_col)[r] = at + sc - len;
    item_emit_run(o.stage, colp<uint8_t>(&a.cols, off_col + 1u) + at, o.win, pos, len, sc - len, total);
    at += total; done += 32;
  };
  if constexpr (!APART) item_each_element(o.owner, n, element);
  else {
    const uint32_t w = mine ? o.row[ItWords<OBJ_PET>::n + 1u] : 0u, own = apart ? o.row[IW_FIELDS + bslot - ItSlot0<OBJ_PET>::n] : (OBJS ? w >> 16 : w & 0xFFFFu);
    const uint32_t bytes = warp_incl_scan(own) - own; /* of the lists of the lanes before */
    item_each_run(o.apart, [&](uint32_t lo, uint32_t end) {
      at = at0 + __shfl_sync(0xFFFFFFFFu, bytes, (int)lo); done = __shfl_sync(0xFFFFFFFFu, inc - all, (int)lo);
      item_each_element(o.owner, lane >= lo && lane < end ? n : 0u, element);
    });
  }
}
/* ---- the exact parser -------------------------------------------------------------------------------------------- */

__device__ __forceinline__ Rd item_reader(const ItemArgs& a, const uint8_t* in, uint64_t limit) {
  Rd rd;
  rd.in = in; rd.lf_ws = a.sep ? 1u : 0u; rd.open_end = (a.is_last || a.sep) ? 0u : 1u; rd.limit = limit; rd.opts = a.opts; rd.rec_end = limit;
  return rd;
}
/* Line ln for the exact parser, in shared memory when what is there is what the input says and the whole line, else where it lies. */
struct ItemText { const uint8_t* in; uint64_t start, limit; };
__device__ __forceinline__ ItemText item_text(const ItemArgs& a, const StreamGeom& g, const ItemShared& sh, const uint8_t* win, uint32_t ln) {
  const uint32_t at = sh.line[ln] & 0xFFFFu, sep = (sh.line[ln + 1u] & 0xFFFFu) - 1u;
  if (sep < g.hi_valid && !((sh.movedline[ln >> 5] >> (ln & 31u)) & 1u)) return ItemText{win, at, a.sep ? sep : sep + 1u};
  const uint64_t s0 = g.v0 + at - g.mis;
  if (!a.sep) return ItemText{a.in, s0, a.limit}; /* (it looks for the line feed itself) */
  if (sh.open_end && ln + 1u == sh.nline) return ItemText{a.in, s0, arr_extent(a.in, a.len, a.sep, s0 - 1u, a.res->first_opener).end};
  return ItemText{a.in, s0, g.v0 + sep - g.mis};
}
/* A line where it lies, for the word-at-a-time tokeniser: positions from an aligned word on. It looks ahead, so 32 readable bytes have to
 * follow the line: in array framing behind its end, in NDJSON behind a limit that no line which uses the tokeniser's answer reaches. */
struct ItemDirect { Win w; uint32_t start, limit; };
__device__ __forceinline__ bool item_direct(const ItemArgs& a, const ItemText& t, ItemDirect& d) {
  if (t.in != a.in || t.limit + (a.sep ? 32u : 0u) > a.limit) return false;
  const uint64_t end = a.sep ? t.limit : (a.limit < 32u ? 0u : a.limit - 32u);
  const uint32_t mis = (uint32_t)(reinterpret_cast<uintptr_t>(a.in + t.start) & 3u);
  if (end <= t.start || end - t.start > 0x7FFF0000u) return false;
  d.w.s = a.in + t.start - mis; d.w.w0 = (int64_t)t.start - mis;
  d.start = mis; d.limit = (uint32_t)(end - t.start) + mis;
  return true;
}
/* A record's model, what it adds to every counter and whether the word-at-a-time tokeniser took it (else the exact parser did), or
 * PJ_TYPE_NONE and kind and offset of its failure. */
struct ItemSize { uint32_t type, err, off, fast, cnt[NSLOT]; };
template <int SCHEMA>
__device__ __noinline__ void item_size(const ItemArgs& a, const ItemText t, ItemSize* r) {
  ItemDirect d;
  r->type = PJ_TYPE_NONE; r->err = 0; r->off = 0; r->fast = 0;
  if (item_direct(a, t, d)) {
    uint32_t tape[TAPE_MIN_CAP], pos = 0;
    Tape tp;
    tp.e = tape; tp.stride = 1; tp.cap = TAPE_MIN_CAP; tp.n = 0;
    uint32_t v = fast_outline<SCHEMA>(d.w, d.start, d.limit, a.sep ? 1u : 0u, a.sep ? 0u : 1u, nullptr, nullptr, 0, tp, r->cnt, &r->type, &r->err, &pos);
    if (v == FAST_FAILED && ((!a.sep && pos >= d.limit) || ((a.opts & PJ_OPT_ENUM_UNKNOWN_AS_NULL) && r->err == PJ_E_ENUM) || ((a.opts & PJ_OPT_COERCE_SCALARS) && r->err == PJ_E_TYPE))) v = FAST_REFUSED;
    if (v == FAST_ACCEPTED) { r->err = 0; r->fast = 1; return; }
    r->type = PJ_TYPE_NONE;
    if (v == FAST_FAILED) { r->off = pos - d.start; return; }
    r->err = 0;
  }
  PS s;
  s.p = t.start; s.err = 0; s.err_pos = 0;
  Out<false> so;
  so.cols = &a.cols;
  uint64_t p = t.start;
  if (a.sep) while (p < t.limit && (item_blank(t.in[p]) || t.in[p] == '\n')) ++p;
  if (p < t.limit || !a.sep) r->type = parse_record<false>(c_schema, item_reader(a, t.in, t.limit), s, (uint32_t)SCHEMA, so, 0);
  else fail(s, PJ_E_SYNTAX, t.limit); /* an extent without a value */
  for (uint32_t k = 0; k < NSLOT; ++k) r->cnt[k] = so.cnt[k];
  if (s.err) { r->type = PJ_TYPE_NONE; r->err = s.err; r->off = (uint32_t)(s.err_pos - t.start); }
  else if (t.in == a.in && s.p - t.start > *(volatile uint32_t*)&a.res->max_rec) atomicMax(&a.res->max_rec, (uint32_t)(s.p - t.start < 0x7FFFFFFFu ? s.p - t.start : 0x7FFFFFFFu));
}
/* its columns, from the places o gives on; by the parser that sized it */
template <int SCHEMA>
__device__ __noinline__ void item_place(const ItemArgs& a, const ItemText t, uint32_t fast, Out<true>& o, uint64_t n) {
  if (fast) {
    ItemDirect d;
    uint32_t tape[TAPE_MIN_CAP], x[3];
    Tape tp;
    tp.e = tape; tp.stride = 1; tp.cap = TAPE_MIN_CAP; tp.n = 0;
    if (item_direct(a, t, d)) fast_outline<SCHEMA>(d.w, d.start, d.limit, a.sep ? 1u : 0u, a.sep ? 0u : 1u, &a.cols, o.base, n, tp, nullptr, &x[0], &x[1], &x[2]);
    return;
  }
  PS s;
  s.p = t.start; s.err = 0; s.err_pos = 0;
  parse_record<true>(c_schema, item_reader(a, t.in, t.limit), s, (uint32_t)SCHEMA, o, n);
}
/* Line ln, a record the own steps refused: its row says how it failed or, if it is a valid one after all, that it stands apart (IF_ROWS: by the
 * word-at-a-time tokeniser), and what it adds to its model's counters. */
template <int SCHEMA>
__device__ __noinline__ void item_judge(const ItemArgs& a, const StreamGeom& g, ItemShared& sh, const uint8_t* win, uint32_t* row, uint32_t ln) {
  ItemSize r;
  item_size<SCHEMA>(a, item_text(a, g, sh, win, ln), &r);
  row[IW_ERR] = r.err;
  if (r.err) { row[IW_FLAGS] = IF_BAD | IF_RECORD; row[IW_LIST] = r.off; return; }
  const uint32_t slot0 = r.type == PJ_TYPE_USER ? ItSlot0<OBJ_USER>::n : ItSlot0<OBJ_PET>::n;
  if (r.type != PJ_TYPE_ORDER) for (uint32_t j = 0; j < IT_APART; ++j) row[IW_FIELDS + j] = r.cnt[slot0 + j];
  if constexpr (ItemSlots<SCHEMA>::lists) { row[IW_LIST] = 0; row[ItWords<OBJ_PET>::n] = 0; row[ItWords<OBJ_PET>::n + 1u] = 0; }
  row[IW_FLAGS] = IF_APART | IF_RECORD | (r.fast ? IF_ROWS : 0u) | (SCHEMA == PJ_SCHEMA_MIXED ? (~(1u << (r.type - 1u)) & 7u) << IF_NOTMODEL : 0u);
  sh.apart = 1;
}
/* what the records of a warp's lines that stand apart add to the sums of its group */
template <int SCHEMA>
__device__ __noinline__ void item_sum_apart(ItemShared& sh, const uint32_t* row, bool apart, uint32_t type) {
#pragma unroll 1
  for (uint32_t j = 0; j < 2u * IT_APART; ++j) {
    const uint32_t slot = (uint32_t)SLOT_PET_CAT_NAME + j;
    const bool pet = j < IT_APART;
    if (!((ItemSlots<SCHEMA>::mask >> slot) & 1u)) continue;
    const uint32_t s = __reduce_add_sync(0xFFFFFFFFu, apart && type == (pet ? (uint32_t)PJ_TYPE_PET : (uint32_t)PJ_TYPE_USER) ? row[IW_FIELDS + (pet ? j : j - IT_APART)] : 0u);
    if ((threadIdx.x & 31u) == 0) sh.csum[slot][threadIdx.x >> 5] += s;
  }
}
/* what a record that does not stand apart adds to its model's counters */
template <int MODEL, int OBJ, bool ROOT, uint32_t WORD0, uint32_t BIT0, int I = 0>
__device__ __forceinline__ void item_counts(const uint32_t* row, uint32_t flags, uint32_t* cnt) {
  if constexpr (I < CObj<OBJ>::N) {
    constexpr uint32_t kind = CObj<OBJ>::f[I].kind, at = CObj<OBJ>::f[I].cnt - ItSlot0<MODEL>::n;
    constexpr uint32_t word = ROOT ? it_root_word<OBJ>(I) : WORD0 + it_flat_word<OBJ>(I), LW = ItWords<OBJ_PET>::n;
    if constexpr (kind == K_STR) cnt[at] = (flags >> (IF_PRESENT + BIT0 + I)) & 1u ? (row[word] >> 16) & 0x7FFFu : 0u;
    else if constexpr (kind == K_OBJ) item_counts<MODEL, CObj<OBJ>::f[I].child, false, ItModel<OBJ>::child_word, IB_CHILD>(row, flags, cnt);
    else if constexpr (kind == K_LIST_STR) { cnt[at] = row[IW_LIST] >> 16; cnt[at + 1u] = row[LW + 1u] & 0xFFFFu; }
    else if constexpr (kind == K_LIST_OBJ) {
      constexpr int E = CObj<OBJ>::f[I].child;
      cnt[at] = row[LW] >> 16; cnt[CObj<E>::f[it_string_field<E>()].cnt - ItSlot0<MODEL>::n] = row[LW + 1u] >> 16;
    }
    item_counts<MODEL, OBJ, ROOT, WORD0, BIT0, I + 1>(row, flags, cnt);
  }
}
/* The columns of the records among 32 lines that stand apart (every lane of the warp calls this): by the exact parser once more, at the
 * place the records of their model before them leave. n: the lane's record, at: its row in its model's table. */
template <int SCHEMA>
__device__ __noinline__ void item_emit_apart(const ItemArgs& a, const StreamGeom& g, const ItemShared& sh, const uint8_t* win, const uint32_t* row, uint32_t flags, uint32_t type, uint32_t ln, uint32_t c, uint64_t n, uint64_t at) {
  const bool apart = (flags & IF_APART) != 0;
  Out<true> o;
  o.cols = &a.cols;
#pragma unroll 1
  for (uint32_t k = 0; k < NSLOT; ++k) { o.base[k] = (uint32_t)at; o.room[k] = 1; o.cnt[k] = 0; } /* (counters of rows) */
  auto model = [&](auto obj) {
    constexpr int OBJ = decltype(obj)::value;
    const bool mine = type == (OBJ == OBJ_PET ? (uint32_t)PJ_TYPE_PET : (uint32_t)PJ_TYPE_USER);
    uint32_t cnt[IT_APART];
#pragma unroll
    for (uint32_t j = 0; j < IT_APART; ++j) cnt[j] = 0;
    if (mine && apart) for (uint32_t j = 0; j < IT_APART; ++j) cnt[j] = row[IW_FIELDS + j];
    else if (mine) item_counts<OBJ, OBJ, true, 0u, 0u>(row, flags, cnt);
#pragma unroll
    for (uint32_t j = 0; j < IT_APART; ++j) {
      const uint32_t slot = ItSlot0<OBJ>::n + j, before = warp_incl_scan(cnt[j]) - cnt[j];
      o.base[slot] = sh.base[slot] + sh.csum[slot][c] + before; o.room[slot] = cnt[j];
    }
  };
  if constexpr (SCHEMA == PJ_SCHEMA_PET || SCHEMA == PJ_SCHEMA_MIXED) model(ItInteger<OBJ_PET>());
  if constexpr (SCHEMA == PJ_SCHEMA_USER || SCHEMA == PJ_SCHEMA_MIXED) model(ItInteger<OBJ_USER>());
  if (apart) {
    item_place<SCHEMA>(a, item_text(a, g, sh, win, ln), flags & IF_ROWS, o, n);
  }
}

/* The lines whose preceding separator lies in [lo, hi) of the input, one after the other (head: and before them the one at
 * byte 0): f(start, limit). */
template <class F>
__device__ __forceinline__ void item_each_line(const ItemArgs& a, uint64_t lo, uint64_t hi, bool head, F f) {
  if (a.sep) {
    for (uint64_t p = lo; p < hi; ++p) {
      if (!((a.sep[p >> 6] >> (p & 63)) & 1u)) continue;
      const ExtentOut x = arr_extent(a.in, a.len, a.sep, p, a.res->first_opener);
      if (x.second_opener) atomicMin(&a.res->doc_err_off, (unsigned long long)p); /* a second document */
      if (x.is_record) f(x.start, x.end);
    }
  } else {
    if (head && nd_is_record(a.in, 0, a.limit, (int)a.is_last)) f((uint64_t)0, a.limit);
    for (uint64_t p = lo; p < hi; ++p)
      if (a.in[p] == '\n' && nd_is_record(a.in, p + 1, a.limit, (int)a.is_last)) f(p + 1, a.limit);
  }
}
/* A tile of many more lines or strings than its shared memory has room for, read where it lies: every thread walks the lines that begin in its
 * share of the tile's bytes, once to size them and once to size and emit them, with the word-at-a-time tokeniser and, for what that one
 * refuses, the exact parser. */
template <int SCHEMA>
__device__ __noinline__ void item_slow_tile(const ItemArgs& a, const StreamGeom& g, ItemShared& sh, uint32_t tile, uint32_t tid) {
  using SL = ItemSlots<SCHEMA>;
  __shared__ uint32_t sh_scan[33];
  const uint32_t lane = tid & 31, warp = tid >> 5;
  const uint64_t share = (g.own_end + IT_THREADS - 1) / IT_THREADS, v_hi = g.v0 + g.own_end; /* v: offsets from the aligned base */
  uint64_t lo = g.v0 + share * tid, hi = lo + share;
  if (hi > v_hi) hi = v_hi;
  lo = lo > g.mis ? lo - g.mis : 0; hi = hi > g.mis ? hi - g.mis : 0;
  const bool head = tile == 0 && tid == 0 && !a.sep && a.is_first && a.limit > 0; /* also the line at byte 0 */
  uint32_t sum[IT_NLB], nerr = 0;
#pragma unroll
  for (uint32_t k = 0; k < IT_NLB; ++k) sum[k] = 0;
  uint32_t my_base[IT_NLB];
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    if (head || lo < hi)
      item_each_line(a, lo, hi, head, [&](uint64_t s0, uint64_t limit) {
        const ItemText t = ItemText{a.in, s0, limit};
        ItemSize r;
        item_size<SCHEMA>(a, t, &r);
        if (pass == 0) {
          sum[IT_REC]++;
          nerr += r.err != 0;
          if (!r.err) for (uint32_t k = SL::lo; k < SL::hi; ++k) sum[k] += r.cnt[k];
        } else {
          const uint64_t i = my_base[IT_REC];
          colp<uint64_t>(&a.cols, PJ_COL_REC_START)[i] = a.goff + s0;
          colp<uint8_t>(&a.cols, PJ_COL_ERR_KIND)[i] = (uint8_t)r.err;
          colp<uint32_t>(&a.cols, PJ_COL_ERR_OFF)[i] = r.off;
          if (SCHEMA == PJ_SCHEMA_MIXED) {
            colp<uint8_t>(&a.cols, PJ_COL_REC_TYPE)[i] = (uint8_t)r.type;
            colp<uint32_t>(&a.cols, PJ_COL_REC_ROW)[i] = r.type == PJ_TYPE_NONE ? 0xFFFFFFFFu : my_base[r.type - 1];
          }
          Out<true> o;
          o.cols = &a.cols;
          for (uint32_t k = 0; k < NSLOT; ++k) { o.base[k] = my_base[k]; o.room[k] = (k >= SL::lo && k < SL::hi && !r.err) ? r.cnt[k] : 0u; }
          if (r.err) { if (SCHEMA != PJ_SCHEMA_MIXED) store_absent<true>(c_schema, (uint32_t)SCHEMA, o, i); }
          else {
            item_place<SCHEMA>(a, t, r.fast, o, i);
            for (uint32_t k = SL::lo; k < SL::hi; ++k) my_base[k] += r.cnt[k];
          }
          my_base[IT_REC]++;
        }
      });
    if (pass == 0) {
#pragma unroll
      for (uint32_t k = 0; k < IT_NLB; ++k) {
        my_base[k] = 0;
        if (!((SL::mask >> k) & 1u)) continue;
        uint32_t total;
        my_base[k] = block_excl_scan(sum[k], &total, sh_scan);
        if (tid == 0) sh.tot[k] = total;
      }
      __syncthreads();
      if (warp == 0) item_resolve<SCHEMA>(a, sh, tile, lane);
      __syncthreads();
      if (!sh.ok) return;
#pragma unroll
      for (uint32_t k = 0; k < IT_NLB; ++k) if ((SL::mask >> k) & 1u) my_base[k] += sh.base[k];
      for (int d = 16; d; d >>= 1) nerr += __shfl_xor_sync(0xFFFFFFFFu, nerr, d);
      if (lane == 0 && nerr) atomicAdd(&a.res->n_errors, (unsigned long long)nerr);
    }
  }
  if (tile == a.ntiles - 1) item_close_offsets(a, sh, tid);
}

/* The columns of a tile that knows its place: four kinds of them x groups of 32 lines. APART: records stand apart; a version of its own, out of
 * line, because tiles without one paid for it: with one version for both the kernel spilled 1140 bytes per thread instead of 120 and 200k Users
 * with blanks took 140 us instead of 129, 100k Users in an array 70 instead of 61. */
template <int SCHEMA, bool APART>
__device__ __forceinline__ void item_emit_tile(const ItemArgs& a, const StreamGeom& g, ItemShared& sh, const uint8_t* win, const uint32_t* pairs, const uint32_t* rows) {
  using SL = ItemSlots<SCHEMA>;
  constexpr uint32_t STRIDE = ItStride<SCHEMA>::n;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nline = sh.nline, nchunk = (nline + 31u) >> 5;
  for (uint32_t u = warp; u < 4u * nchunk; u += IT_WARPS) {
    /* groups differ in cost (mixed streams: by model) as well as kinds: a warp gets another group of each kind */
    const uint32_t what = u / nchunk, c = (u + what) % nchunk, i = c * 32u + lane;
    const uint32_t ln = i < nline ? (SCHEMA == PJ_SCHEMA_MIXED ? (uint32_t)sh.perm[i] : i) : 0u;
    const uint32_t* r = rows + ln * STRIDE;
    ItemOut o;
    o.win = win; o.row = r; o.chunk = c; o.stage = sh.stage[warp]; o.owner = sh.owner[warp]; o.moved = sh.nspecial ? sh.special : nullptr;
    const uint32_t f = i < nline ? r[IW_FLAGS] : 0u;
    const bool rec = (f & IF_RECORD) != 0, good = rec && !(f & IF_BAD);
    const uint32_t lt = (1u << lane) - 1u;
    const uint64_t n = (uint64_t)sh.base[IT_REC] + sh.csum[IT_REC][ln >> 5] + (uint32_t)__popc(sh.recs[ln >> 5] & ((1u << (ln & 31u)) - 1u));
    const uint32_t type = good ? item_type<SCHEMA>(f) : (uint32_t)PJ_TYPE_NONE;
    const bool apart = APART && good && (f & IF_APART);
    o.flags = good && !apart ? f : 0u;
    o.apart = APART ? __ballot_sync(0xFFFFFFFFu, apart) : 0u;
    o.at = n;
    uint32_t bp = 0, bo = 0, bu = 0;
    if constexpr (SCHEMA == PJ_SCHEMA_MIXED) {
      bp = __ballot_sync(0xFFFFFFFFu, type == PJ_TYPE_PET); bo = __ballot_sync(0xFFFFFFFFu, type == PJ_TYPE_ORDER); bu = __ballot_sync(0xFFFFFFFFu, type == PJ_TYPE_USER);
      const uint32_t mine = type == PJ_TYPE_PET ? bp : (type == PJ_TYPE_ORDER ? bo : bu);
      const uint32_t slot = type == PJ_TYPE_PET ? SLOT_ROWS_PET : (type == PJ_TYPE_ORDER ? SLOT_ROWS_ORD : SLOT_ROWS_USR);
      o.at = sh.base[slot] + sh.csum[slot][c] + (uint32_t)__popc(mine & lt);
    }
    if (what == 3u) {
      const uint32_t bg = __ballot_sync(0xFFFFFFFFu, good), br = __ballot_sync(0xFFFFFFFFu, rec);
      if (lane == 0) {
        if (br != bg) atomicAdd(&a.res->n_errors, (unsigned long long)__popc(br & ~bg));
        if (bg & ~o.apart) atomicAdd(&a.res->n_fast, (unsigned long long)__popc(bg & ~o.apart));
      }
      if (APART && o.apart) item_emit_apart<SCHEMA>(a, g, sh, win, r, f, type, ln, c, n, o.at);
      if (rec) {
        colp<uint64_t>(&a.cols, PJ_COL_REC_START)[n] = a.goff + g.v0 + (r[IW_POS] & 0xFFFFu) - g.mis;
        colp<uint8_t>(&a.cols, PJ_COL_ERR_KIND)[n] = good ? 0 : (uint8_t)r[IW_ERR];
        colp<uint32_t>(&a.cols, PJ_COL_ERR_OFF)[n] = good ? 0u : r[IW_LIST];
        if constexpr (SCHEMA == PJ_SCHEMA_MIXED) {
          colp<uint8_t>(&a.cols, PJ_COL_REC_TYPE)[n] = (uint8_t)type;
          colp<uint32_t>(&a.cols, PJ_COL_REC_ROW)[n] = type == PJ_TYPE_NONE ? 0xFFFFFFFFu : (uint32_t)o.at;
        }
      }
      if (rec && !apart) {
        if constexpr (SCHEMA == PJ_SCHEMA_PET) item_emit_fixed<OBJ_PET, true, 0u, 0u>(a, o);
        else if constexpr (SCHEMA == PJ_SCHEMA_ORDER) item_emit_fixed<OBJ_ORDER, true, 0u, 0u>(a, o);
        else if constexpr (SCHEMA == PJ_SCHEMA_USER) item_emit_fixed<OBJ_USER, true, 0u, 0u>(a, o);
        else {
          if (type == PJ_TYPE_PET) item_emit_fixed<OBJ_PET, true, 0u, 0u>(a, o);
          else if (type == PJ_TYPE_ORDER) item_emit_fixed<OBJ_ORDER, true, 0u, 0u>(a, o);
          else if (type == PJ_TYPE_USER) item_emit_fixed<OBJ_USER, true, 0u, 0u>(a, o);
        }
      }
    } else if (what == 2u) {
      if constexpr (SCHEMA == PJ_SCHEMA_PET) { o.has_row = rec; item_emit_strings<APART, OBJ_PET, OBJ_PET, true, 0u, 0u>(a, sh, o); }
      else if constexpr (SCHEMA == PJ_SCHEMA_USER) { o.has_row = rec; item_emit_strings<APART, OBJ_USER, OBJ_USER, true, 0u, 0u>(a, sh, o); }
      else if constexpr (SCHEMA == PJ_SCHEMA_MIXED) {
        const uint32_t apart_all = o.apart;
        o.has_row = type == PJ_TYPE_PET; o.apart = apart_all & bp;
        if (bp) item_emit_strings<APART, OBJ_PET, OBJ_PET, true, 0u, 0u>(a, sh, o);
        o.has_row = type == PJ_TYPE_USER; o.apart = apart_all & bu;
        if (bu) item_emit_strings<APART, OBJ_USER, OBJ_USER, true, 0u, 0u>(a, sh, o);
      }
    } else if constexpr (SL::lists) {
      const bool pet = type == PJ_TYPE_PET;
      o.has_row = SCHEMA == PJ_SCHEMA_PET ? rec : pet;
      if constexpr (SCHEMA == PJ_SCHEMA_MIXED) o.apart &= bp;
      if (SCHEMA == PJ_SCHEMA_PET || bp) { if (what == 0u) item_emit_lists<APART, false>(a, sh, o, pairs, pet); else item_emit_lists<APART, true>(a, sh, o, pairs, pet); }
    }
  }
}
template <int SCHEMA>
__device__ __noinline__ void item_emit_tile_apart(const ItemArgs& a, const StreamGeom& g, ItemShared& sh, const uint8_t* win, const uint32_t* pairs, const uint32_t* rows) {
  item_emit_tile<SCHEMA, true>(a, g, sh, win, pairs, rows);
}

/* ---- a tile ------------------------------------------------------------------------------------------------------ */
/* Steps 2 to 5 of a tile whose index stands. False (for every thread): the other road; nothing was published. */
template <int SCHEMA, bool ARR>
__device__ __forceinline__ bool item_tile(const ItemArgs& a, const StreamGeom& g, ItemShared& sh, uint8_t* win, uint32_t* pairs, uint32_t* rows, uint32_t tile, uint32_t tid, long long* ck) {
  using SL = ItemSlots<SCHEMA>;
  constexpr uint32_t STRIDE = ItStride<SCHEMA>::n;
  constexpr uint32_t LW = ItWords<OBJ_PET>::n;
  constexpr int E = OBJ_TAG;
  constexpr uint32_t PCNT = CObj<OBJ_PET>::f[ItModel<OBJ_PET>::li].cnt, TCNT = CObj<OBJ_PET>::f[ItModel<OBJ_PET>::ei].cnt;
  constexpr uint32_t TBYTES = CObj<E>::f[it_string_field<E>()].cnt;
  static_assert(ItModel<OBJ_PET>::elem == OBJ_TAG && ItModel<OBJ_ORDER>::elem < 0 && ItModel<OBJ_USER>::elem < 0 && ItModel<OBJ_ORDER>::li < 0 && ItModel<OBJ_USER>::li < 0, "lists are Pet's");
  const uint32_t lane = tid & 31, warp = tid >> 5;
  const uint32_t nline = sh.nline, nchunk = (nline + 31u) >> 5;
  if (sh.nspecial) {
    item_specials(a, sh, win, pairs, tid);
    __syncthreads();
  }
  const uint32_t mine = item_walk<SCHEMA, ARR>(a, g, sh, win, pairs, rows, tid); /* line, model */
  if (SCHEMA == PJ_SCHEMA_MIXED) __syncthreads(); /* the lines were walked in another order */
  uint32_t* row = rows + (tid < nline ? tid : 0u) * STRIDE; /* from here on a thread has the line of its number */
  {
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, tid < nline && (row[IW_FLAGS] & IF_ODD));
    if (lane == 0) sh.oddmask[warp] = m;
  }
  if (__syncthreads_or((int)sh.slow)) return false;
  {
    uint32_t nodd = 0, nmoved = 0;
#pragma unroll
    for (uint32_t k = 0; k < IT_WARPS; ++k) { nodd += (uint32_t)__popc(sh.oddmask[k]); nmoved += (uint32_t)__popc(sh.movedline[k] & ~sh.oddmask[k]); }
    if (tid == 0) sh.ndense = nline - nodd - nmoved; /* in one spelling, nothing decoded */
    if (nodd) {
      /* the second walk takes 1000 cycles a string, however few lines are left; a line or two per warp go to the packs at once (300 k mixed
         records, 1 % malformed: 328 -> 278 us) */
      if (nodd > 2u * IT_WARPS) {
        __syncthreads(); /* oddmask[] is read */
        item_walk_again<SCHEMA, ARR>(a, g, sh, win, pairs, rows, tid, mine);
        nodd = 0;
#pragma unroll
        for (uint32_t k = 0; k < IT_WARPS; ++k) nodd += (uint32_t)__popc(sh.oddmask[k]);
      }
      if (nodd) item_packs<SCHEMA, ARR>(a, g, sh, win, pairs, rows, nodd);
      __syncthreads();
    }
  }

  /* ---- values: fields x groups of 32 lines ---- */
  {
    uint32_t u = 0;
#pragma unroll 1
    for (int v = VU_COUNT - 1; v >= 0; --v) {
      if (!((ItemValueUnits<SCHEMA>::mask >> v) & 1u)) continue;
      for (uint32_t c = 0; c < nchunk; ++c, ++u) {
        if ((u & (IT_WARPS - 1u)) != warp) continue;
        const uint32_t i = c * 32u + lane;
        const bool live = i < nline;
        const uint32_t ln = live ? (SCHEMA == PJ_SCHEMA_MIXED ? (uint32_t)sh.perm[i] : i) : 0u; /* several models: lines of one side by side */
        item_value<SCHEMA>(a, sh.owner[warp], sh.nspecial ? sh.special : nullptr, win, pairs, rows, rows + ln * STRIDE, live, (uint32_t)v);
      }
    }
  }
  __syncthreads();

  /* ---- verdicts and sums ---- */
  uint32_t flags = 0, type = PJ_TYPE_NONE;
  if (warp < nchunk) {
    flags = tid < nline ? row[IW_FLAGS] : 0u;
    const bool rec = (flags & IF_RECORD) != 0;
    uint32_t e = rec ? row[IW_ERR] : IE_NONE;
    type = item_type<SCHEMA>(flags);
    if (rec && e == IE_NONE) { /* required properties; is the model known? */
      if (SCHEMA == PJ_SCHEMA_MIXED && type == PJ_TYPE_NONE) e = IE_REFUSED;
      else {
        const uint32_t req = type == PJ_TYPE_PET ? (uint32_t)CObj<OBJ_PET>::required : (type == PJ_TYPE_ORDER ? (uint32_t)CObj<OBJ_ORDER>::required : (uint32_t)CObj<OBJ_USER>::required);
        if (((flags >> IF_PRESENT) & req) != req) e = ((row[IW_POS] >> 16) << 8) | (uint32_t)PJ_E_REQUIRED;
      }
    }
    if (rec && e != IE_NONE) {
      const uint32_t kind = e & 0xFFu;
      if ((flags & IF_MOVED) || kind == IE_REFUSED || ((a.opts & PJ_OPT_COERCE_SCALARS) && kind == PJ_E_TYPE)) item_judge<SCHEMA>(a, g, sh, win, row, tid);
      else { row[IW_FLAGS] = IF_BAD | IF_RECORD; row[IW_ERR] = kind; row[IW_LIST] = (e >> 8) - (row[IW_POS] & 0xFFFFu); }
      flags = row[IW_FLAGS];
      type = flags & IF_BAD ? (uint32_t)PJ_TYPE_NONE : item_type<SCHEMA>(flags);
    } else if (!rec) type = PJ_TYPE_NONE;
    const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, rec ? (sh.line[tid + 1u] & 0xFFFFu) - (row[IW_POS] & 0xFFFFu) : 0u);
    if (lane == 0 && most > *(volatile uint32_t*)&a.res->max_rec) atomicMax(&a.res->max_rec, most); /* (seldom more than a few times) */
    const uint32_t br = __ballot_sync(0xFFFFFFFFu, rec);
    if (lane == 0) { sh.csum[IT_REC][warp] = (uint32_t)__popc(br); sh.recs[warp] = br; }
  }
  if constexpr (SCHEMA == PJ_SCHEMA_MIXED) { /* from here on the lines of a model lie side by side, in order */
    uint32_t ends[4];
    __syncthreads(); /* perm[] is read */
    item_sort(sh, tid, tid >= nline ? 4u : (type == PJ_TYPE_NONE ? 3u : type - 1u), ends);
    if (tid < nline) {
      row = rows + sh.perm[tid] * STRIDE;
      flags = row[IW_FLAGS];
      type = tid < ends[0] ? (uint32_t)PJ_TYPE_PET : (tid < ends[1] ? (uint32_t)PJ_TYPE_ORDER : (tid < ends[2] ? (uint32_t)PJ_TYPE_USER : (uint32_t)PJ_TYPE_NONE));
    }
  }
  if (warp < nchunk) {
    if constexpr (SCHEMA == PJ_SCHEMA_MIXED) {
      const uint32_t bp = __ballot_sync(0xFFFFFFFFu, type == PJ_TYPE_PET), bo = __ballot_sync(0xFFFFFFFFu, type == PJ_TYPE_ORDER), bu = __ballot_sync(0xFFFFFFFFu, type == PJ_TYPE_USER);
      if (lane == 0) { sh.csum[SLOT_ROWS_PET][warp] = (uint32_t)__popc(bp); sh.csum[SLOT_ROWS_ORD][warp] = (uint32_t)__popc(bo); sh.csum[SLOT_ROWS_USR][warp] = (uint32_t)__popc(bu); }
    }
    if constexpr (SL::lists) {
      const bool pet = type == PJ_TYPE_PET;
      item_sum_strings<OBJ_PET, true, 0u, 0u>(sh, row, pet, flags, warp, lane);
      const uint32_t n0 = __reduce_add_sync(0xFFFFFFFFu, pet ? row[IW_LIST] >> 16 : 0u), n1 = __reduce_add_sync(0xFFFFFFFFu, pet ? row[LW] >> 16 : 0u);
      const uint32_t b0 = __reduce_add_sync(0xFFFFFFFFu, pet ? row[LW + 1u] & 0xFFFFu : 0u), b1 = __reduce_add_sync(0xFFFFFFFFu, pet ? row[LW + 1u] >> 16 : 0u);
      if (lane == 0) { sh.csum[PCNT][warp] = n0; sh.csum[TCNT][warp] = n1; sh.csum[PCNT + 1u][warp] = b0; sh.csum[TBYTES][warp] = b1; }
    }
    if constexpr (SCHEMA == PJ_SCHEMA_USER || SCHEMA == PJ_SCHEMA_MIXED) item_sum_strings<OBJ_USER, true, 0u, 0u>(sh, row, type == PJ_TYPE_USER, flags, warp, lane);
    const bool apart = tid < nline && (flags & IF_APART);
    if (__any_sync(0xFFFFFFFFu, apart)) item_sum_apart<SCHEMA>(sh, row, apart, type);
  }
  __syncthreads();
  ck[3] = clock64();

  /* ---- where everything of the tile goes ---- */
  if (warp == 0) {
#pragma unroll
    for (uint32_t k0 = 0; k0 < IT_NLB; k0 += 32 / IT_WARPS) { /* as many counters a time as the warp's lanes hold groups of lines */
      constexpr uint32_t some = (1u << (32 / IT_WARPS)) - 1u;
      if (!((SL::mask >> k0) & some)) continue;
      const uint32_t k = k0 + lane / IT_WARPS, c = lane % IT_WARPS;
      const bool used = (SL::mask >> k) & 1u;
      const uint32_t v = used && c < nchunk ? sh.csum[k][c] : 0u;
      uint32_t inc = v;
#pragma unroll
      for (uint32_t d = 1; d < IT_WARPS; d <<= 1) { const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, d, IT_WARPS); if (c >= d) inc += x; }
      if (used) { sh.csum[k][c] = inc - v; if (c == IT_WARPS - 1u) sh.tot[k] = inc; }
    }
    __syncwarp();
    item_resolve<SCHEMA>(a, sh, tile, lane);
    if (lane == 0) sh.next = 0;
  }
  __syncthreads();
  ck[4] = clock64();
  if (!sh.ok) return true;

  /* ---- emission: four kinds of columns x groups of 32 lines ---- */
  if (sh.apart) item_emit_tile_apart<SCHEMA>(a, g, sh, win, pairs, rows); else item_emit_tile<SCHEMA, false>(a, g, sh, win, pairs, rows);
  if (tile == a.ntiles - 1) item_close_offsets(a, sh, tid);
  return true;
}

template <int SCHEMA> struct ItTablesOf { static constexpr ItTables t = it_tables(SCHEMA); };
template <int SCHEMA> __device__ const ItTables d_item_tables = ItTablesOf<SCHEMA>::t;
struct ItGapTableOf { static constexpr ItGapTable t = it_gap_table(); };
static __device__ const ItGapTable d_gap_table = ItGapTableOf::t;

template <int SCHEMA, bool ARR>
__device__ __forceinline__ bool item_try(const ItemArgs& a, const StreamGeom& g, ItemShared& sh, uint8_t* win, uint32_t* strs, uint32_t* rows, uint32_t tile, uint32_t tid, long long* ck) {
  const bool fine = item_index<ARR>(a, g, sh, win, strs, tid, tile);
  if (__syncthreads_or(!fine || sh.slow)) return false; /* (decided together: what a warp that goes on may set there comes too late) */
  return item_tile<SCHEMA, ARR>(a, g, sh, win, strs, rows, tile, tid, ck);
}

template <int SCHEMA>
__global__ void __launch_bounds__(IT_THREADS, IT_BLOCKS) k_parse_items(const __grid_constant__ ItemArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ __align__(16) ItemShared sh;
  const uint32_t tid = threadIdx.x;
  const ItemLayout lay = item_layout(a.win_bytes, a.str_words, a.row_cap, ItStride<SCHEMA>::n);
  uint8_t* win = smem + lay.win;
  uint32_t* strs = reinterpret_cast<uint32_t*>(smem + lay.strs);
  uint32_t* rows = reinterpret_cast<uint32_t*>(smem + lay.rows);

  if (tid == 0) { sh.tile = atomicAdd(a.ticket, 1u); mbar_init(&sh.mbar, 1); sh.slow = 0; sh.next = 0; sh.odd = 0; sh.nspecial = 0; sh.apart = 0; }
  if constexpr (SCHEMA == PJ_SCHEMA_MIXED) {
    if (a.looks && (tid >> 5) == 1u) { /* (beside the ticket's way to memory and back) */
      static_assert(ND_LOOKS == 64, "two each");
      const uint32_t n = __reduce_add_sync(0xFFFFFFFFu, a.looks[tid & 31u] + a.looks[tid]);
      if (tid == 32u) sh.aside = nd_looks_long(n);
    } else if (tid == 32u) sh.aside = 0;
  }
  __syncthreads();
  const uint32_t tile = sh.tile;
  if (tile >= a.ntiles) return;
  if constexpr (SCHEMA == PJ_SCHEMA_MIXED) {
    if (sh.aside) { if (tile == 0 && tid == 0) a.res->aside = 1u; return; }
  }
  long long ck[5];
  ck[0] = clock64();
  const uint32_t mis = (uint32_t)(reinterpret_cast<uintptr_t>(a.in) & 15u);
  const StreamGeom g = stream_geom(mis, a.len, a.limit, a.tile_bytes, tile, a.win_bytes);

  /* ---- stage the window: one bulk copy of whole 16-byte blocks (the first and the last one may hold bytes that are not
     input: they lie in the same aligned 16 bytes as input bytes, so they are readable; they are masked) ---- */
  if (g.copy_bytes && tid == 0) { mbar_expect_tx(&sh.mbar, g.copy_bytes); bulk_g2s(win, a.in - mis + g.v0, g.copy_bytes, &sh.mbar); }
  for (uint32_t k = tid; k < IT_SLOTS * 8; k += IT_THREADS) (&sh.key[0][0])[k] = (&d_item_tables<SCHEMA>.key[0][0])[k];
  for (uint32_t k = tid; k < IT_SLOTS * 3; k += IT_THREADS) (&sh.field[0][0])[k] = (&d_item_tables<SCHEMA>.field[0][0])[k];
  for (uint32_t k = tid; k < IG_SLOTS * 4; k += IT_THREADS) reinterpret_cast<uint32_t*>(sh.gap)[k] = reinterpret_cast<const uint32_t*>(d_gap_table.e)[k];
  for (uint32_t k = tid; k < IT_MAX_STRS / 32; k += IT_THREADS) { sh.special[k] = 0; sh.broken[k] = 0; }
  if (tid < IT_MAX_LINES / 32) { sh.oddline[tid] = 0; sh.movedline[tid] = 0; }
  int stage_failed = 0;
  if (g.copy_bytes) stage_failed = !mbar_wait_bounded(&sh.mbar, 0, a.spin_limit_ns);
  if (__syncthreads_or(stage_failed)) { /* the block gives up together: the results of the call are void */
    if (tid == 0) {
      atomicExch(&a.res->timeout, 1u);
      /* the copy may still be in flight, and the block's shared memory must not pass to another block before it has
         landed: one thread stays and waits for it, again with a limit */
      mbar_wait_bounded(&sh.mbar, 0, a.spin_limit_ns);
    }
    return;
  }
  if (tid < 48) win[g.hi_valid + tid] = '\n';
  __syncthreads();
  ck[1] = clock64();

  bool done = false;
  if (a.sep) done = item_try<SCHEMA, true>(a, g, sh, win, strs, rows, tile, tid, ck);
  else done = item_try<SCHEMA, false>(a, g, sh, win, strs, rows, tile, tid, ck);
  if (!done) {
    __syncthreads();
    item_slow_tile<SCHEMA>(a, g, sh, tile, tid);
    return;
  }
  __syncthreads();
  if (tid == 0) {
    const long long c5 = clock64();
    atomicAdd(&a.res->phase_cycles[0], (unsigned long long)(ck[1] - ck[0]));
    if (sh.ndense) atomicAdd(&a.res->n_dense, (unsigned long long)sh.ndense);
    if (sh.nline) item_note_strings(a, sh.nstr, sh.stop - (sh.line[0] & 0xFFFFu));
    atomicAdd(&a.res->phase_cycles[1], (unsigned long long)(ck[3] - ck[1]));
    atomicAdd(&a.res->phase_cycles[2], (unsigned long long)(ck[4] - ck[3]));
    atomicAdd(&a.res->phase_cycles[3], (unsigned long long)(c5 - ck[4]));
  }
}

}  // namespace pj
#endif

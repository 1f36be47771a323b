/*
 * pj_item.cuh — k_parse_items<SCHEMA>: JSON records to typed columns in one kernel and one pass over HBM, with the work
 * spread over STRINGS instead of records.
 *
 * One thread block = one tile of the input, staged in shared memory by one bulk copy. Its warps take equal byte ranges
 * of the tile; a warp owns the records whose preceding separator (the line feed; in array framing a bit of the
 * separator bitmap) lies in its range, and follows its last one to its end.
 *
 *  1. item_index: 32 bytes per lane and step. Byte-parallel masks of quotes and control characters give the positions
 *     of all quotes of the warp's records in order: string k = (open, close). Backslashes, bytes beyond ASCII and control
 *     characters take extra work only in the steps that hold one; strings with escapes are decoded in place.
 *  2. item_tokens: 32 strings per step, one per lane: a string and the gap behind it, up to the next string. The
 *     punctuation of a gap alone tells where in the record it stands (`}],` closes an element, its list and is
 *     followed by a key of the root; `,` and `:` leave the place as it is), so the object a string lies in is the one
 *     the nearest telling gap before it left: one ballot and one shuffle instead of a walk. Keys are looked up in a
 *     hash table, and the REFERENCE to the key's value goes to its place in the record's row. Nothing is parsed here and
 *     no lane waits for a longer record.
 *  3. item_values: one record (or list element) per lane: the references of a property are decoded by 32 lanes that all
 *     do the same (integers, enums, date-times), then what is required is checked.
 *  4. Counts per record are added up, ONE decoupled look-back over the earlier tiles gives the tile's place in every
 *     column and arena, and the columns are written.
 *
 * The steps detect every deviation from a valid record of the model; the common failures (wrong JSON type, unknown
 * literal, bad date-time, missing property, record ending inside a string) are reported with the exact parser's kind
 * and offset, because the smallest offset of a record's deviations is its first failure. Any other deviation sends the
 * record to the exact parser (pj_core.cuh); should that one accept the record (unknown keys with nested values, repeated keys,
 * ...), or does the tile not fit the shared memory laid out for it (a record longer than the window, many more records
 * or strings than its bytes suggest), the block walks the tile with the exact parser alone (item_slow_tile).
 */
#ifndef PJ_ITEM_CUH
#define PJ_ITEM_CUH

#include "pj_dev.cuh"
#include "pj_fast.cuh"
#include "pj_index.cuh"
#include "pj_array.cuh"
#include "pj_item_tables.h"
#include "pj_result.h"
#include "pj_stream.cuh"

namespace pj {

static constexpr uint32_t IT_THREADS = 256;
static constexpr uint32_t IT_WARPS = IT_THREADS / 32;
static constexpr uint32_t IT_STEP = 1024;        /* bytes a warp indexes per step */
static constexpr uint32_t IT_FRONT = 32;         /* bytes before the window that may be read (and mean nothing) */
static constexpr uint32_t IT_PAD = IT_STEP + 64; /* ... and behind it */
static constexpr uint32_t IT_MAX_RECS = 256;     /* records per tile */
static constexpr uint32_t IT_RCHUNKS = IT_MAX_RECS / 32;
static constexpr uint32_t IT_MAX_UNITS = 64;     /* groups of 32 list elements per tile and list */
static constexpr uint32_t IT_MAX_STRS = 1024;    /* strings per warp */
static constexpr uint32_t IT_MAX_WIN = 65536 - 64; /* window offsets are 16-bit */
static constexpr uint32_t IT_ARR_SEP = 0x1E;     /* what the separators of array framing are replaced with in the window */

static constexpr uint32_t IT_MAX_DYN_SMEM = 200 * 1024; /* dynamic shared memory of a block */
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
  uint32_t win_bytes;  /* bytes staged per tile: the tile and what its last records may need behind it */
  uint32_t str_ratio;  /* 32-bit words for strings per 256 bytes of text */
  uint32_t row_cap;    /* record rows in shared memory */
  uint32_t opts;       /* PJ_OPT_* bits that change a rule */
  unsigned long long spin_limit_ns;
  const uint64_t* sep; /* array framing: one bit per input byte, set for `[`, the commas and `]` that delimit records; else null */
  ItemTile* tiles;
  uint32_t* ticket;
  DevResult* res;
  const DevResult* prev;    /* totals of the pieces of the same call parsed by earlier launches (null: none) */
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
  /* position of slot k among the used ones */
  static PJ_CX uint32_t pos(uint32_t k) { return k == IT_REC ? count - 1u : k - lo; }
  static constexpr bool lists = SCHEMA == PJ_SCHEMA_PET || SCHEMA == PJ_SCHEMA_MIXED;
};
static_assert((ItemSlots<PJ_SCHEMA_MIXED>::nagg) <= 6, "packed totals fit");

/* shared memory of a tile: what the dynamic part holds, from a 16-byte aligned base */
struct ItemLayout { uint32_t win, strs, rows, total; };
PJ_HD ItemLayout item_layout(uint32_t win_bytes, uint32_t str_ratio, uint32_t row_cap, uint32_t stride) {
  ItemLayout l;
  l.win = IT_FRONT;
  l.strs = (l.win + win_bytes + IT_PAD + 15u) & ~15u;
  l.rows = l.strs + ((((win_bytes + 64u) * str_ratio) >> 8) + 2u * IT_WARPS + 4u) * 4u;
  l.rows = (l.rows + 15u) & ~15u;
  l.total = l.rows + row_cap * stride * 4u;
  return l;
}

/* what a warp leaves about its range */
struct ItemWarp {
  uint32_t nstr, nterm, start, stop; /* strings, separators that end a line, first line, last separator */
  uint32_t str0, words;              /* first of its words for strings, how many there are */
  uint32_t nrec, nphoto, ntag;
  uint32_t odd;                      /* bit 0: special strings, bit 1: records that end inside a string */
  uint32_t row0;                     /* first row */
};
struct ItemShared {
  __align__(16) uint32_t key[IT_SLOTS][8];
  uint32_t field[3][IT_SLOTS];
  __align__(16) ItGapEntry gap[IG_SLOTS];
  ItemWarp w[IT_WARPS];
  uint32_t special[IT_WARPS][IT_MAX_STRS / 32]; /* per string: it holds a backslash, a control character or a byte beyond ASCII ... */
  uint32_t broken[IT_WARPS][IT_MAX_STRS / 32];  /* ... and is not a valid one */
  uint16_t todo[IT_WARPS][64];
  uint32_t csum[IT_NLB][IT_RCHUNKS]; /* record-level counters: sums per 32 records, then exclusive prefixes */
  uint32_t usum[2][IT_MAX_UNITS];    /* string bytes per 32 list elements (list of strings, list of objects), then exclusive prefixes */
  uint32_t tot[IT_NLB], base[IT_NLB];
  uint32_t ok, slow, bad, tile, next;
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
/* the eight flags (0x80 per byte) of two words as bits, times 128, added to acc */
__device__ __forceinline__ uint32_t item_gather(uint32_t f0, uint32_t f1) { return __dp4a(f1, 0x80402010u, __dp4a(f0, 0x08040201u, 0u)) >> 7; }
template <class F>
__device__ __forceinline__ uint32_t item_mask32(const uint32_t* w, F f) {
  uint32_t m = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) m |= item_gather(f(w[2 * k]), f(w[2 * k + 1])) << (8 * k);
  return m;
}
__device__ __forceinline__ uint32_t item_prefix_xor(uint32_t x) {
  x ^= x << 1; x ^= x << 2; x ^= x << 4; x ^= x << 8; x ^= x << 16;
  return x;
}
/* bytes escaped by an odd run of backslashes (32 bytes; carry: the first byte is escaped) */
__device__ __forceinline__ uint32_t item_escaped(uint32_t bs, uint32_t carry) {
  const uint32_t even = 0x55555555u;
  bs &= ~carry;
  const uint32_t follows = (bs << 1) | carry;
  const uint32_t odd_starts = bs & ~even & ~follows;
  const uint32_t sum = odd_starts + bs;
  return (even ^ (sum << 1)) & follows;
}

/* Positions of the quotes of the records this warp owns. False: the tile does not fit (or cannot be told apart this
 * way), the block has to take the other road. */
template <bool ARR>
__device__ __forceinline__ bool item_index(const ItemArgs& a, const StreamGeom& g, ItemShared& sh, uint8_t* win, uint32_t* strs, uint32_t warp, uint32_t lane, uint32_t tile) {
  const uint32_t span = (((a.tile_bytes + IT_WARPS - 1) / IT_WARPS) + 31u) & ~31u;
  const uint32_t lo = warp * span;
  uint32_t hi = lo + span;
  if (hi > g.own_end) hi = g.own_end;
  bool started = !ARR && tile == 0 && warp == 0 && a.is_first && a.limit > 0;
  uint32_t start = g.mis, stop = 0, nq = 0, nterm = 0, ecarry = 0;
  bool done = false, fine = true;
  uint32_t odd_bits = 0;
  ItemWarp& W = sh.w[warp];
  if (lane == 0) { W.nstr = 0; W.nterm = 0; W.start = 0; W.stop = 0; W.str0 = 0; W.words = 0; W.row0 = 0; W.nrec = 0; W.nphoto = 0; W.ntag = 0; W.odd = 0; }
  if (!started && lo >= hi) return true;
  const int32_t end_valid = (int32_t)g.hi_valid + (g.to_limit ? 1 : 0); /* the end of the input counts as a separator */
  const uint32_t lt = (1u << lane) - 1u;
  uint16_t* q16 = nullptr;
  uint32_t str0 = 0, words = 0;
  for (uint32_t o = lo; !done; o += IT_STEP) {
    if ((int32_t)o >= end_valid) { fine = !started; break; } /* its last record runs out of the window */
    if (!started && o >= hi) break;
    const int32_t p0 = (int32_t)(o + 32u * lane);
    uint32_t w[8];
    {
      const uint4* src = reinterpret_cast<const uint4*>(win + p0);
      const uint4 x = src[0], y = src[1];
      w[0] = x.x; w[1] = x.y; w[2] = x.z; w[3] = x.w; w[4] = y.x; w[5] = y.y; w[6] = y.z; w[7] = y.w;
    }
    const uint32_t vm = item_low(end_valid - p0) & ~item_low((int32_t)g.lo_valid - p0);
    uint32_t q = item_mask32(w, [](uint32_t x) { return ~((((x ^ 0x22222222u) & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x) & 0x80808080u; }) & vm;
    uint32_t c = item_mask32(w, [](uint32_t x) { return ~(((x & 0x7F7F7F7Fu) + 0x60606060u) | x) & 0x80808080u; }) & vm;
    uint32_t sp = 0; /* bit 7 of a byte set: some word has a backslash or a byte beyond ASCII there */
#pragma unroll
    for (int k = 0; k < 8; ++k) sp |= ~(((w[k] ^ 0x5C5C5C5Cu) & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | w[k];
    const bool has_sp = (sp & 0x80808080u) != 0;
    /* separators */
    uint32_t t = 0;
    if (ARR) {
      const int64_t bit = (int64_t)g.v0 + p0 - (int64_t)g.mis; /* input offset of the lane's first byte */
      const int64_t nwords32 = (int64_t)((a.len + 31) >> 5);
      const uint32_t* sw = reinterpret_cast<const uint32_t*>(a.sep);
      const int64_t i0 = bit >> 5; /* floor: the first tile may begin a few bytes before the input */
      const uint32_t b0 = i0 >= 0 && i0 < nwords32 ? sw[i0] : 0u, b1 = i0 + 1 >= 0 && i0 + 1 < nwords32 ? sw[i0 + 1] : 0u;
      t = __funnelshift_r(b0, b1, (uint32_t)(bit & 31)) & vm;
      if (g.to_limit && (int32_t)g.hi_valid >= p0 && (int32_t)g.hi_valid < p0 + 32) t |= 1u << (g.hi_valid - (uint32_t)p0);
      for (uint32_t m = t; m; m &= m - 1u) win[p0 + __ffs((int)m) - 1] = (uint8_t)IT_ARR_SEP;
      c |= t; /* all of them count as control characters from here on */
    } else {
      for (uint32_t m = c; m; m &= m - 1u) {
        const uint32_t b = (uint32_t)__ffs((int)m) - 1u;
        if (win[p0 + b] == '\n') t |= 1u << b;
      }
    }
    if (!started) {
      const uint32_t cand = t & item_low((int32_t)hi - p0);
      const uint32_t bal = __ballot_sync(0xFFFFFFFFu, cand != 0);
      if (!bal) continue;
      start = __shfl_sync(0xFFFFFFFFu, (uint32_t)p0 + (uint32_t)__ffs((int)cand), __ffs((int)bal) - 1); /* behind the separator */
      started = true;
    }
    if (!q16) {
      str0 = ((start * a.str_ratio) >> 8) + 2u * warp;
      q16 = reinterpret_cast<uint16_t*>(strs + str0);
    }
    uint32_t act = ~item_low((int32_t)start - p0);
    {
      const uint32_t cand = t & act & ~item_low((int32_t)hi - p0);
      const uint32_t bal = __ballot_sync(0xFFFFFFFFu, cand != 0);
      if (bal) {
        stop = __shfl_sync(0xFFFFFFFFu, (uint32_t)p0 + (uint32_t)__ffs((int)cand) - 1u, __ffs((int)bal) - 1);
        done = true;
        act &= item_low((int32_t)stop + 1 - p0);
      }
    }
    t &= act; q &= act;
    const uint32_t ctl = c & act & ~t;
    uint32_t B = 0, H = 0;
    const bool any_sp = __any_sync(0xFFFFFFFFu, has_sp);
    if (any_sp) {
      B = item_mask32(w, [](uint32_t x) { return item_eq4(x, 0x5C5C5C5Cu); }) & vm;
      H = item_mask32(w, [](uint32_t x) { return x & 0x80808080u; }) & act;
      if (__any_sync(0xFFFFFFFFu, B != 0) || ecarry) {
        if (__any_sync(0xFFFFFFFFu, B == 0xFFFFFFFFu)) { fine = false; break; }
        const uint32_t cout = (uint32_t)__clz((int)~B) & 1u; /* parity of the run of backslashes that ends the 32 bytes */
        uint32_t cin = __shfl_up_sync(0xFFFFFFFFu, cout, 1);
        if (lane == 0) cin = ecarry;
        q &= ~item_escaped(B, cin);
        ecarry = __shfl_sync(0xFFFFFFFFu, cout, 31);
      }
      B &= act;
    } else if (ecarry) { if (lane == 0) q &= ~1u; ecarry = 0; }
    /* order of the quotes; a record that ends inside a string gets its separator as the closing quote */
    uint32_t ex, total;
    for (;;) {
      const uint32_t n = (uint32_t)__popc(q);
      const uint32_t inc = warp_incl_scan(n);
      ex = inc - n;
      total = __shfl_sync(0xFFFFFFFFu, inc, 31);
      uint32_t odd = 0;
      for (uint32_t m = t & ~q; m; m &= m - 1u) { /* separators this lane sees with a string open */
        const uint32_t low = (m & (0u - m)) - 1u;
        if ((nq + ex + (uint32_t)__popc(q & low)) & 1u) { odd = m & (0u - m); break; }
      }
      const uint32_t bal = __ballot_sync(0xFFFFFFFFu, odd != 0);
      if (!bal) break;
      if ((int)lane == __ffs((int)bal) - 1) q |= odd;
      odd_bits |= 2u;
    }
    /* strings that need a closer look */
    if (__any_sync(0xFFFFFFFFu, (B | H | ctl) != 0)) {
      odd_bits |= 1u;
      const uint32_t instr = item_prefix_xor(q) ^ (((nq + ex) & 1u) ? 0xFFFFFFFFu : 0u);
      for (uint32_t m = (B | H | ctl) & instr; m; m &= m - 1u) {
        const uint32_t k = (nq + ex + (uint32_t)__popc(q & ((m & (0u - m)) - 1u))) >> 1;
        if (k < IT_MAX_STRS) atomicOr(&sh.special[warp][k >> 5], 1u << (k & 31u));
      }
      if (ARR) { /* a raw separator byte of our own choice in the text */
        bool raw = false;
        for (uint32_t m = ctl; m; m &= m - 1u) raw = raw || win[p0 + __ffs((int)m) - 1] == IT_ARR_SEP;
        if (__any_sync(0xFFFFFFFFu, raw)) { fine = false; break; }
      }
    }
    {
      const uint32_t upto = done ? stop + 1u : o + IT_STEP; /* the words of the bytes seen so far: ranges never share one */
      words = ((upto * a.str_ratio) >> 8) + 2u * warp + 2u - str0;
      if ((nq + total) / 2u + 1u > words || (nq + total) / 2u >= IT_MAX_STRS) { fine = false; break; }
      uint32_t i = nq + ex;
      for (uint32_t m = q; m; m &= m - 1u) q16[i++] = (uint16_t)((uint32_t)p0 + (uint32_t)__ffs((int)m) - 1u);
    }
    nq += total;
    nterm += __reduce_add_sync(0xFFFFFFFFu, (uint32_t)__popc(t));
  }
  if (!fine) return false;
  if (started && done) {
    if (lane == 0) {
      W.nstr = nq >> 1; W.nterm = nterm; W.start = start; W.stop = stop; W.str0 = str0; W.words = words; W.odd = odd_bits;
      strs[str0 + (nq >> 1)] = (stop + 1u) | ((stop + 1u) << 16);
    }
  }
  return true;
}

/* One string that holds a backslash, a control character or a byte beyond ASCII: decoded in place (the decoded text is
 * never longer); what is left over up to the old closing quote becomes blanks. False: not a valid string. */
static __device__ __noinline__ bool item_decode_string(uint8_t* win, uint32_t open, uint32_t close, uint32_t opts, uint32_t* new_close, uint32_t* moved) {
  uint32_t p = open + 1u, d = p;
  *moved = 0; *new_close = close;
  if (win[close] != '"') return false; /* the record ends inside it */
  while (p < close) {
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
  if (d != close) {
    win[d] = '"';
    for (uint32_t k = d + 1; k <= close; ++k) win[k] = ' ';
    *new_close = d;
  }
  return true;
}
/* the strings of a warp that item_index() marked, 32 at a time */
__device__ __forceinline__ void item_specials(const ItemArgs& a, ItemShared& sh, uint8_t* win, uint32_t* strs, uint32_t warp, uint32_t lane) {
  if (!(sh.w[warp].odd & 1u)) return;
  const uint32_t nstr = sh.w[warp].nstr;
  uint32_t* pairs = strs + sh.w[warp].str0;
  const uint32_t nw = (nstr + 31u) >> 5; /* <= 32 */
  const uint32_t mine = lane < nw ? sh.special[warp][lane] : 0u;
  if (!__any_sync(0xFFFFFFFFu, mine != 0)) return;
  uint32_t have = 0;
  for (uint32_t k = 0; k < nw; ++k) {
    const uint32_t bits = __shfl_sync(0xFFFFFFFFu, mine, (int)k);
    if ((bits >> lane) & 1u) sh.todo[warp][have + (uint32_t)__popc(bits & ((1u << lane) - 1u))] = (uint16_t)(32u * k + lane);
    have += (uint32_t)__popc(bits);
    __syncwarp();
    if (have >= 32u || k + 1 == nw) {
      uint32_t at = 0;
      while (have - at >= 32u || (k + 1 == nw && at < have)) {
        const uint32_t n = have - at < 32u ? have - at : 32u;
        if (lane < n) {
          const uint32_t s = sh.todo[warp][at + lane];
          const uint32_t pr = pairs[s];
          uint32_t nc, moved;
          if (!item_decode_string(win, pr & 0xFFFFu, pr >> 16, a.opts, &nc, &moved)) atomicOr(&sh.broken[warp][s >> 5], 1u << (s & 31u));
          else pairs[s] = (pr & 0xFFFFu) | (nc << 16);
          if (!moved) atomicAnd(&sh.special[warp][s >> 5], ~(1u << (s & 31u))); /* plain after all: positions are the input's */
        }
        at += n;
      }
      __syncwarp();
      const uint32_t rest = have - at;
      const uint32_t keep = lane < rest ? sh.todo[warp][at + lane] : 0u;
      __syncwarp();
      if (lane < rest) sh.todo[warp][lane] = (uint16_t)keep;
      have = rest;
      __syncwarp();
    }
  }
}

/* ---- 2. tokens ------------------------------------------------------------------------------------------------ */
__device__ __forceinline__ uint32_t item_peek4(const uint8_t* win, uint32_t p) {
  Win w;
  w.s = win; w.w0 = 0;
  return wpeek4(w, p);
}
__device__ __forceinline__ void item_error(uint32_t* row, uint32_t pos, uint32_t kind) { atomicMin(&row[IW_ERR], (pos << 8) | kind); }
/* A scalar token that belongs to no property: only what is cheap to see as valid (integers, literals) passes. */
static __device__ __noinline__ bool item_plain_scalar(const uint8_t* win, uint32_t s, uint32_t n) {
  if (n == 4 && (item_peek4(win, s) == 0x65757274u || item_peek4(win, s) == 0x6C6C756Eu)) return true;
  if (n == 5 && win[s] == 'f' && item_peek4(win, s + 1) == 0x65736C61u) return true;
  uint32_t i = win[s] == '-' ? 1u : 0u;
  if (i >= n || (win[s + i] == '0' && i + 1 < n)) return false;
  for (; i < n; ++i) if (win[s + i] - (uint32_t)'0' > 9u) return false;
  return true;
}

/* A gap as the tables know it, and the places in it that matter. */
struct ItemView {
  uint32_t desc;              /* ItGap, 0: not one of the texts */
  uint32_t vpos, vend;        /* first byte of the value behind the colon, end of a number or literal */
  uint32_t last_sep, nsep;    /* the separator that ends the record: its last byte, how many there are (blank lines) */
  uint32_t clpos;             /* the record's closing brace */
};
template <bool ARR>
__device__ __forceinline__ bool item_blank(uint32_t x) { return x == ' ' || x == '\t' || x == '\r' || (ARR && x == '\n'); }
template <bool ARR>
__device__ __forceinline__ uint32_t item_gap_find(const ItemShared& sh, uint32_t lo, uint32_t hi, uint32_t len) {
  const ItGapEntry e = sh.gap[it_gap_hash(lo, hi, ARR)];
  return e.lo == lo && e.hi == hi && e.len == len ? e.desc : 0u;
}
/* A gap with blanks: its text is put together byte by byte, numbers and literals are skipped. */
template <bool ARR>
__device__ __forceinline__ void item_gap_spaced(const ItemShared& sh, const uint8_t* win, uint32_t from, uint32_t b, ItemView& v) {
  constexpr uint32_t T = ARR ? IT_ARR_SEP : (uint32_t)'\n';
  Win w;
  w.s = win; w.w0 = 0;
  uint64_t text = 0;
  uint32_t n = 0, p = from, brace = 0, last = 0;
  v.nsep = 0; v.vpos = b; v.vend = 0; v.last_sep = 0; v.clpos = 0;
  while (p < b && n <= 8) {
    uint32_t c = win[p];
    if (item_blank<ARR>(c)) { ++p; continue; }
    if (n == 1) v.vpos = p;
    if (c - (uint32_t)'0' <= 9u || c == '-' || (c | 0x20u) - (uint32_t)'a' <= 25u) {
      ++p;
      for (;;) {
        const uint64_t m = swar_nondigit(wpeek8(w, p));
        if (!m) { p += 8; continue; }
        p += ctz64(m) >> 3;
        const uint32_t x = win[p];
        if ((x | 0x20u) - (uint32_t)'a' <= 25u || x == '.' || x == '+' || x == '-') { ++p; continue; }
        break;
      }
      v.vend = p;
      c = '0';
    } else {
      if (c == '}') brace = p;
      if (c == T) {
        v.last_sep = p; ++v.nsep;
        if (last == T) { ++p; continue; } /* a blank line */
        v.clpos = brace;
      }
      ++p;
    }
    last = c;
    if (n < 8) text |= (uint64_t)c << (8 * n);
    ++n;
  }
  v.desc = n <= 8 && p == b ? item_gap_find<ARR>(sh, (uint32_t)text, (uint32_t)(text >> 32), n) : 0u;
}
template <int SCHEMA, bool ARR>
__device__ __forceinline__ bool item_tokens(const ItemArgs& a, const StreamGeom& g, ItemShared& sh, const uint8_t* win, uint32_t* strs, uint32_t* rows, uint32_t warp, uint32_t lane) {
  constexpr uint32_t STRIDE = ItStride<SCHEMA>::n;
  constexpr uint32_t T = ARR ? IT_ARR_SEP : (uint32_t)'\n';
  ItemWarp& W = sh.w[warp];
  const uint32_t nstr = W.nstr, start = W.start, stop = W.stop, row0 = W.row0, odd = W.odd;
  uint32_t* pairs = strs + W.str0;
  uint32_t* photo_end = pairs + W.words; /* list strings are kept from the end of the warp's words downwards */
  const uint32_t lt = (1u << lane) - 1u, le = (2u << lane) - 1u; /* lane 31: 2 << 31 wraps to 0, so all ones */
  if (W.nterm == 0) return true;
  for (uint32_t k = lane; k < W.nterm; k += 32) { rows[(row0 + k) * STRIDE + IW_FLAGS] = 0; rows[(row0 + k) * STRIDE + IW_ERR] = IE_NONE; }
  bool slow = false;
  if (nstr == 0) { /* no string at all: blank lines, or records for the other road */
    uint32_t seen = 0, seps = 0;
    for (uint32_t p = start + lane; p <= stop; p += 32) {
      const uint32_t x = win[p];
      if (x == T) seps += p < g.hi_valid; else if (!item_blank<ARR>(x)) seen = 1;
    }
    seps = __reduce_add_sync(0xFFFFFFFFu, seps);
    return !__any_sync(0xFFFFFFFFu, seen != 0) && !(ARR && seps) && (ARR || a.is_last || stop < g.hi_valid);
  }
  uint32_t seps = 0; /* separators met */
  __syncwarp();
  /* what precedes the first string: blank lines and an opening brace */
  {
    uint32_t err = 0, first = start, bad = 0, n = 0;
    if (lane == 0) {
      uint32_t p = start, brace = 0;
      const uint32_t e = pairs[0] & 0xFFFFu;
      for (; p < e; ++p) {
        const uint32_t x = win[p];
        if (x == T && !ARR && !brace) { if (err) bad = 1; first = p + 1u; ++n; }
        else if (x == T) bad = 1;
        else if (x == '{' && !brace && !err) brace = 1;
        else if (!item_blank<ARR>(x)) err = 1;
      }
      if (!brace) err = 1;
      reinterpret_cast<uint16_t*>(&rows[row0 * STRIDE + IW_POS])[0] = (uint16_t)first;
      if (err) item_error(&rows[row0 * STRIDE], first, IE_REFUSED);
    }
    slow = __any_sync(0xFFFFFFFFu, bad != 0);
    seps = n; /* of lane 0 */
  }
  uint32_t st = IS_ROOT, rec = 0, nP = 0, nT = 0, pk = 0;
  for (uint32_t k0 = 0; k0 < nstr; k0 += 32) {
    const uint32_t k = k0 + lane;
    const bool live = k < nstr;
    const uint32_t pr = pairs[live ? k : nstr], nx = pairs[live ? k + 1u : nstr];
    const uint32_t open = pr & 0xFFFFu, close = pr >> 16, b = nx & 0xFFFFu;
    const bool trunc = (odd & 2u) && live && win[close] == T;
    const uint32_t from = trunc ? close : close + 1u;
    __syncwarp(); /* every lane has its pairs: what lies before k0 + 32 may be overwritten */

    /* ---- the gap behind the string ---- */
    ItemView v;
    v.vpos = b; v.vend = 0;
    {
      /* without blanks: the bytes themselves, or `:0` and what follows the number (found from the gap's end) */
      Win w;
      w.s = win; w.w0 = 0;
      const uint32_t n = b - from;
      const uint64_t h = wpeek8(w, from);
      uint32_t lo = (uint32_t)h, hi = (uint32_t)(h >> 32);
      const uint32_t c0 = lo & 0xFFu, c1 = (lo >> 8) & 0xFFu;
      if (n < 8u) {
        const uint64_t m = (1ull << (8u * n)) - 1ull;
        lo &= (uint32_t)m; hi &= (uint32_t)(m >> 32);
      }
      uint32_t len = n;
      bool fits = n <= 8u;
      if (c0 == ':' && n > 1u) v.vpos = from + 1u;
      if (c0 == ':' && n > 2u && (c1 - (uint32_t)'0' <= 9u || c1 == '-' || c1 - (uint32_t)'a' <= 25u)) {
        const uint64_t t = wpeek8(w, b - 8u);
        const uint32_t tl = (uint32_t)t, th = (uint32_t)(t >> 32);
        /* bytes 0x30-0x3F and 0x60-0x6F: digits, and the letters a literal ends with */
        const uint32_t ah = (th ^ 0x30303030u) & 0xF0F0F0F0u, bh = (th ^ 0x60606060u) & 0xF0F0F0F0u;
        const uint32_t al = (tl ^ 0x30303030u) & 0xF0F0F0F0u, bl = (tl ^ 0x60606060u) & 0xF0F0F0F0u;
        const uint32_t zh = (~((ah & 0x7F7F7F7Fu) + 0x7F7F7F7Fu | ah) | ~((bh & 0x7F7F7F7Fu) + 0x7F7F7F7Fu | bh)) & 0x80808080u;
        const uint32_t zl = (~((al & 0x7F7F7F7Fu) + 0x7F7F7F7Fu | al) | ~((bl & 0x7F7F7F7Fu) + 0x7F7F7F7Fu | bl)) & 0x80808080u;
        const uint32_t tail = zh ? (uint32_t)__clz((int)zh) >> 3 : 4u + ((uint32_t)__clz((int)zl) >> 3); /* bytes behind the last of them */
        v.vend = b - tail;
        fits = tail >= 1u && tail <= 6u;
        len = tail + 2u;
        const uint64_t x = (t >> (8u * (8u - (fits ? tail : 1u)))) << 16;
        lo = (uint32_t)x | (uint32_t)':' | ((uint32_t)'0' << 8); hi = (uint32_t)(x >> 32);
      }
      v.desc = fits ? item_gap_find<ARR>(sh, lo, hi, len) : 0u;
      const uint32_t brace = (v.desc & ItGap::BRACE) ? 1u : 0u;
      v.last_sep = b - 1u - brace; v.clpos = v.last_sep - 1u;
      v.nsep = (v.desc & ItGap::ENDS) ? 1u : 0u;
    }
    bool next_bad = false;
    if (live && v.desc == 0 && !trunc) {
      item_gap_spaced<ARR>(sh, win, from, b, v);
      /* Blank lines between records are none. But in array framing an extent without a value is a record (only the end of the
         input follows the closing bracket), and so is a blank line that the readable bytes cut off. */
      if (v.desc && v.nsep > 1u) slow = slow || (ARR ? !(v.nsep == 2u && v.last_sep >= g.hi_valid) : (v.last_sep >= g.hi_valid && !a.is_last));
    }
    if (live && v.desc && (v.desc & ItGap::ENDS)) {
      if (!(v.desc & ItGap::BRACE) != (k + 1u == nstr)) v.desc = 0; /* a brace opens the next record, if there is one */
      if (!a.is_last && v.last_sep >= g.hi_valid) v.desc = 0;       /* the readable bytes end here, the stream does not */
    }
    const bool ok = live && v.desc != 0;
    if (live && !ok) { /* a record that ends inside this string, or no valid record: they have to be kept apart all the same */
      uint32_t n = 0;
      for (uint32_t p = from; p < b; ++p) if (win[p] == T) { ++n; v.last_sep = p; }
      if (n > 1u) slow = true;
      v.nsep = n; v.vend = 0; v.clpos = 0;
      if (n && k + 1u != nstr) { /* does the next record begin as it should? */
        uint32_t p = v.last_sep + 1u;
        while (p < b && item_blank<ARR>(win[p])) ++p;
        next_bad = true;
        if (win[p] == '{') { ++p; while (p < b && item_blank<ARR>(win[p])) ++p; next_bad = p != b; }
      }
      /* trunc: nothing may stand between the string and its separator; the gap begins with it */
      v.desc = ItGap::make(IV_NONE, 15, IS_ROOT, n != 0, n != 0, false, false, false);
    }
    const uint32_t d = v.desc, vk = ItGap::vk(d);
    const bool telling = live && (d & ItGap::TELLS), ends = live && (d & ItGap::ENDS), newelem = live && (d & ItGap::ELEM);
    bool iskey = live && (d & ItGap::KEY);

    /* ---- the object the string lies in: what the nearest telling gap before it left ---- */
    const uint32_t NI = __ballot_sync(0xFFFFFFFFu, telling);
    const uint32_t pm = NI & lt;
    const uint32_t from_lane = __shfl_sync(0xFFFFFFFFu, ItGap::out(d), pm ? 31 - __clz((int)pm) : 0);
    const uint32_t s = pm ? from_lane : st;
    const uint32_t RN = __ballot_sync(0xFFFFFFFFu, ends);
    const uint32_t myrec = rec + (uint32_t)__popc(RN & lt);
    const uint32_t PK = __ballot_sync(0xFFFFFFFFu, iskey && vk == IV_STR);
    const bool isval = lane ? (PK >> (lane - 1)) & 1u : pk != 0;
    const bool iselem = live && !isval && s == IS_LIST && !iskey;
    const uint32_t EL = __ballot_sync(0xFFFFFFFFu, iselem);
    const uint32_t NE = __ballot_sync(0xFFFFFFFFu, newelem);
    const bool inrow = live && myrec < W.nterm; /* always: every record ends at a separator of its own */
    uint32_t* row = rows + (row0 + (inrow ? myrec : 0u)) * STRIDE;
    const uint32_t need = ItGap::need(d);
    const bool role_ok = isval ? !iskey : (s == IS_LIST ? !iskey : (iskey || trunc));
    if (inrow) {
      if (trunc) { item_error(row, close, (!a.is_last && close >= g.hi_valid) ? IE_REFUSED : (uint32_t)PJ_E_EOF); if (!role_ok) item_error(row, open, IE_REFUSED); }
      else if (!ok || !role_ok || !(need == 15u || need == s)) { item_error(row, close, IE_REFUSED); iskey = false; }
      if (odd & 1u) {
        if (((sh.special[warp][k >> 5] | sh.broken[warp][k >> 5]) >> (k & 31u)) & 1u) {
          atomicOr(&row[IW_FLAGS], IF_MOVED);
          if ((sh.broken[warp][k >> 5] >> (k & 31u)) & 1u) item_error(row, open - 1u, IE_REFUSED); /* before anything its text is judged by */
        }
      }
      if (ends) { /* the record's last string */
        reinterpret_cast<uint16_t*>(&row[IW_POS])[1] = (uint16_t)v.clpos;
        row[IW_CUM] = (nP + (uint32_t)__popc(EL & le)) | ((nT + (uint32_t)__popc(NE & le)) << 16);
        if (k + 1u != nstr && myrec + 1u < W.nterm) {
          reinterpret_cast<uint16_t*>(&row[STRIDE + IW_POS])[0] = (uint16_t)(v.last_sep + 1u);
          if (next_bad) item_error(row + STRIDE, v.last_sep + 1u, IE_REFUSED);
        }
      }
      if (iselem) {
        const uint32_t i = nP + (uint32_t)__popc(EL & lt);
        if (nstr + 1u + i < W.words) photo_end[-(int32_t)i - 1] = (open + 1u) | ((close - open - 1u) << 16);
        else slow = true;
      }
    } else iskey = false;
    if (NE) {
      if (newelem) {
        const uint32_t t = nT + (uint32_t)__popc(NE & lt);
        if (3u * t + 3u <= k0 + 32u && 3u * t + 3u <= nstr) {
          pairs[3u * t] = 0; pairs[3u * t + 1] = 0; pairs[3u * t + 2] = (row0 + myrec) << 16;
        } else slow = true;
      }
      __syncwarp();
    }
    /* ---- keys ---- */
    if (iskey && !slow) {
      const uint32_t n = close - open - 1u;
      const uint32_t* kw = reinterpret_cast<const uint32_t*>(win) + ((open + 1u) >> 2);
      const uint32_t ksh = ((open + 1u) & 3u) * 8u;
      const uint32_t y0 = kw[0], y1 = kw[1], y2 = kw[2], y3 = kw[3], y4 = kw[4];
      const uint32_t x0 = __funnelshift_r(y0, y1, ksh), x1 = __funnelshift_r(y1, y2, ksh), x2 = __funnelshift_r(y2, y3, ksh), x3 = __funnelshift_r(y3, y4, ksh);
      const uint32_t slot = it_hash(x0 & 0xFFFFu, n, IT_MUL);
      const uint4 kt = *reinterpret_cast<const uint4*>(&sh.key[slot][0]), km = *reinterpret_cast<const uint4*>(&sh.key[slot][4]);
      uint32_t f = sh.field[s == IS_ROOT ? 0 : (s == IS_CHILD ? 1 : 2)][slot];
      if ((((x0 ^ kt.x) & km.x) | ((x1 ^ kt.y) & km.y) | ((x2 ^ kt.z) & km.z) | ((x3 ^ kt.w) & km.w)) != 0 || n < 2u || n > 15u) f = 0;
      const uint32_t vlen = v.vend - v.vpos;
      if (!f) {
        if (!(vk == IV_STR || (vk == IV_SCALAR && item_plain_scalar(win, v.vpos, vlen)))) item_error(row, close, IE_REFUSED);
      } else {
        const uint32_t kind = ItField::kind(f), vclose = nx >> 16;
        const bool null = vk == IV_SCALAR && vlen == 4u && item_peek4(win, v.vpos) == 0x6C6C756Eu;
        bool good = ((ItField::allowed(f) >> vk) & 1u) != 0;
        const uint32_t len = vk == IV_STR ? vclose - b - 1u : vlen;
        uint32_t ref = (vk == IV_STR ? b + 1u : v.vpos) | (len << 16);
        if ((vk == IV_STR || vk == IV_SCALAR) && len >= 0x8000u) slow = true;
        if (!good && !null) {
          const uint32_t at = vk == IV_STR ? b : v.vpos, x = win[at];
          if ((a.opts & PJ_OPT_COERCE_SCALARS) && ((vk == IV_STR && (kind == K_I64 || kind == K_I32 || kind == K_BOOL)) || (vk == IV_SCALAR && kind == K_STR))) {
            if (vk == IV_STR) ref |= 0x80000000u;
            else if (!item_plain_scalar(win, at, vlen)) item_error(row, at, IE_REFUSED);
            good = true;
          } else if ((kind == K_LIST_STR && vk == IV_ELEM) || (kind == K_LIST_OBJ && vk == IV_LIST) || (vk == IV_SCALAR && !(x == '-' || x - (uint32_t)'0' <= 9u || x == 't' || x == 'f')))
            item_error(row, close, IE_REFUSED);
          else item_error(row, at, PJ_E_TYPE);
        }
        if ((odd & 2u) && vk == IV_STR && win[vclose] == T) good = false; /* cut off: it reports that itself */
        const uint32_t bit = 1u << ItField::bit(f), word = ItField::word(f);
        if (s == IS_ELEM) {
          const uint32_t t = nT + (uint32_t)__popc(NE & lt) - 1u;
          const uint32_t old = atomicOr(&pairs[3u * t + 2u], bit | (good && !null ? bit << 4 : 0u));
          if (old & bit) item_error(row, close, IE_REFUSED); /* repeated key */
          if (good && !null) pairs[3u * t + word] = ref;
        } else {
          const uint32_t nm = SCHEMA == PJ_SCHEMA_MIXED && s == IS_ROOT ? (~ItField::models(f) & 7u) << IF_NOTMODEL : 0u;
          const uint32_t old = atomicOr(&row[IW_FLAGS], bit | nm | (good && !null ? bit << IF_PRESENT : 0u));
          if (old & bit) item_error(row, close, IE_REFUSED);
          if (good && !null && kind <= K_DATETIME) row[word] = ref;
        }
      }
    }
    seps += v.nsep;
    st = NI ? __shfl_sync(0xFFFFFFFFu, ItGap::out(d), 31 - __clz((int)NI)) : st;
    rec += (uint32_t)__popc(RN); nP += (uint32_t)__popc(EL); nT += (uint32_t)__popc(NE);
    pk = (PK >> 31) & 1u;
    if (__any_sync(0xFFFFFFFFu, slow)) return false;
  }
  if (lane == 0) { W.nrec = rec; W.nphoto = nP; W.ntag = nT; }
  return __reduce_add_sync(0xFFFFFFFFu, seps) == W.nterm; /* none was taken for part of a number */
}

/* ---- 3. values ------------------------------------------------------------------------------------------------ */
/* -?(0|[1-9][0-9]*) in the n bytes at pos, within int64 / int32. Read from its end, eight digits at a time. */
__device__ __forceinline__ bool item_int(const uint8_t* win, uint32_t pos, uint32_t n, bool is64, int64_t* out) {
  Win w;
  w.s = win; w.w0 = 0;
  const bool neg = n && win[pos] == '-';
  pos += neg; n -= neg;
  if (n == 0 || n > 19) return false;
  if (win[pos] == '0' && n > 1) return false;
  const uint32_t e = pos + n;
  uint64_t mag, bad;
  {
    uint64_t x = wpeek8(w, e - 8u);
    const uint32_t k = n < 8 ? n : 8u;
    if (k < 8) x = (x & (~0ull << (64 - 8 * k))) | (0x3030303030303030ull >> (8 * k));
    bad = swar_nondigit(x);
    mag = swar_parse8(x);
  }
  if (n > 8) {
    uint64_t x = wpeek8(w, e - 16u);
    const uint32_t k = n - 8 < 8 ? n - 8 : 8u;
    if (k < 8) x = (x & (~0ull << (64 - 8 * k))) | (0x3030303030303030ull >> (8 * k));
    bad |= swar_nondigit(x);
    mag += (uint64_t)swar_parse8(x) * 100000000ull;
  }
  if (n > 16) {
    const uint32_t k = n - 16; /* 1..3 */
    uint32_t x = item_peek4(win, e - 20u);
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

/* the properties of OBJ that are neither integers nor plain strings */
template <int OBJ, int I = 0>
__device__ __forceinline__ void item_other_values(const ItemArgs& a, const uint8_t* win, uint32_t* row, uint32_t& flags) {
  if constexpr (I < CObj<OBJ>::N) {
    constexpr uint32_t kind = CObj<OBJ>::f[I].kind, word = it_root_word<OBJ>(I), bit = 1u << (IF_PRESENT + I);
    if constexpr (kind == K_ENUM || kind == K_BOOL || kind == K_DATETIME) {
      if (flags & bit) {
        const uint32_t ref = row[word], pos = ref & 0xFFFFu, n = (ref >> 16) & 0x7FFFu;
        Win w;
        w.s = win; w.w0 = 0;
        if constexpr (kind == K_ENUM) {
          int e = -1;
          if (n <= 14) {
            const uint64_t x = wpeek8(w, pos), y = wpeek8(w, pos + 8);
            const uint64_t lo = n >= 8 ? x : (n ? x & (~0ull >> (64 - 8 * n)) : 0);
            const uint64_t hi = n > 8 ? y & (~0ull >> (64 - 8 * (n - 8))) : 0;
            e = match_enum<CObj<OBJ>::f[I].child>(n, lo, hi);
          }
          if (e >= 0) row[word] = (uint32_t)e;
          else if (a.opts & PJ_OPT_ENUM_UNKNOWN_AS_NULL) flags &= ~bit;
          else item_error(row, pos - 1u, PJ_E_ENUM);
        } else if constexpr (kind == K_BOOL) {
          if (item_true(win, pos, n)) row[word] = 1;
          else if (item_false(win, pos, n)) row[word] = 0;
          else {
            const uint32_t x = win[pos];
            item_error(row, pos, (!(ref >> 31) && (x == '-' || x - (uint32_t)'0' <= 9u)) ? (uint32_t)PJ_E_TYPE : IE_REFUSED);
          }
        } else {
          int64_t ep = 0; int32_t ns = 0, of = 0;
          if (fast_datetime(w, pos, n, &ep, &ns, &of)) { row[word] = (uint32_t)(uint64_t)ep; row[word + 1] = (uint32_t)((uint64_t)ep >> 32); row[word + 2] = (uint32_t)ns; row[word + 3] = (uint32_t)of; }
          else item_error(row, pos - 1u, PJ_E_DATETIME);
        }
      }
    }
    item_other_values<OBJ, I + 1>(a, win, row, flags);
  }
}
__device__ __forceinline__ void item_int_value(const ItemArgs& a, const uint8_t* win, uint32_t* row, uint32_t flags, uint32_t desc) {
  const uint32_t word = desc & 255u, bit = (desc >> 8) & 255u;
  if (desc && ((flags >> (IF_PRESENT + bit)) & 1u)) {
    const bool is64 = (desc >> 16) & 1u;
    const uint32_t ref = row[word], pos = ref & 0xFFFFu, n = (ref >> 16) & 0x7FFFu;
    int64_t v;
    if (item_int(win, pos, n, is64, &v)) {
      row[word] = (uint32_t)(uint64_t)v;
      if (is64) row[word + 1] = (uint32_t)((uint64_t)v >> 32);
    } else {
      const uint32_t x = win[pos];
      item_error(row, ref >> 31 ? pos - 1u : pos, (!(ref >> 31) && (x == 't' || x == 'f')) ? (uint32_t)PJ_E_TYPE : IE_REFUSED);
    }
  }
}
/* Model of a row: PJ_TYPE_*, 0 when the keys do not tell (mixed streams). */
template <int SCHEMA>
__device__ __forceinline__ uint32_t item_type(uint32_t flags) {
  if constexpr (SCHEMA != PJ_SCHEMA_MIXED) return (uint32_t)SCHEMA;
  else {
    const uint32_t m = ~(flags >> IF_NOTMODEL) & 7u;
    return m == 1u ? (uint32_t)PJ_TYPE_PET : (m == 2u ? (uint32_t)PJ_TYPE_ORDER : (m == 4u ? (uint32_t)PJ_TYPE_USER : (uint32_t)PJ_TYPE_NONE));
  }
}
template <int OBJ>
__device__ __forceinline__ void item_finish_values(const ItemArgs& a, const uint8_t* win, uint32_t* row, uint32_t& flags) {
  item_other_values<OBJ>(a, win, row, flags);
  if (row[IW_ERR] == IE_NONE && ((flags >> IF_PRESENT) & CObj<OBJ>::required) != (uint32_t)CObj<OBJ>::required) item_error(row, row[IW_POS] >> 16, PJ_E_REQUIRED);
}
/* one record per lane (live: it has one) */
template <int SCHEMA>
__device__ __forceinline__ void item_record_values(const ItemArgs& a, const uint8_t* win, uint32_t* row, bool live) {
  if (!live || (row[IW_ERR] != IE_NONE && (row[IW_ERR] & 0xFFu) == IE_REFUSED)) return; /* the exact parser will look at it */
  uint32_t flags = row[IW_FLAGS];
  const uint32_t type = item_type<SCHEMA>(flags);
  if (SCHEMA == PJ_SCHEMA_MIXED) {
    if (type == PJ_TYPE_NONE) { item_error(row, 0, IE_REFUSED); return; }
    if (flags & (1u << (IF_PRESENT + IB_SHARED))) flags |= type == PJ_TYPE_PET ? 1u << (IF_PRESENT + it_find<OBJ_PET>(K_ENUM)) : 1u << (IF_PRESENT + it_find<OBJ_ORDER>(K_ENUM));
  }
#pragma unroll
  for (uint32_t s = 0; s < 3; ++s) {
    uint32_t desc;
    const uint32_t dp = s == 0 ? ItInt<OBJ_PET, 0>::v : (s == 1 ? ItInt<OBJ_PET, 1>::v : ItInt<OBJ_PET, 2>::v);
    const uint32_t dn = s == 0 ? ItInt<OBJ_ORDER, 0>::v : (s == 1 ? ItInt<OBJ_ORDER, 1>::v : ItInt<OBJ_ORDER, 2>::v);
    const uint32_t du = s == 0 ? ItInt<OBJ_USER, 0>::v : (s == 1 ? ItInt<OBJ_USER, 1>::v : ItInt<OBJ_USER, 2>::v);
    if constexpr (SCHEMA == PJ_SCHEMA_PET) desc = dp;
    else if constexpr (SCHEMA == PJ_SCHEMA_ORDER) desc = dn;
    else if constexpr (SCHEMA == PJ_SCHEMA_USER) desc = du;
    else desc = type == PJ_TYPE_PET ? dp : (type == PJ_TYPE_ORDER ? dn : du);
    item_int_value(a, win, row, flags, desc);
  }
  static_assert(ItInt<OBJ_PET, 3>::v == 0 && ItInt<OBJ_ORDER, 3>::v == 0 && ItInt<OBJ_USER, 3>::v == 0, "three integers at most");
  if constexpr (SCHEMA == PJ_SCHEMA_PET) item_finish_values<OBJ_PET>(a, win, row, flags);
  else if constexpr (SCHEMA == PJ_SCHEMA_ORDER) item_finish_values<OBJ_ORDER>(a, win, row, flags);
  else if constexpr (SCHEMA == PJ_SCHEMA_USER) item_finish_values<OBJ_USER>(a, win, row, flags);
  else {
    if (type == PJ_TYPE_PET) item_finish_values<OBJ_PET>(a, win, row, flags);
    else if (type == PJ_TYPE_ORDER) item_finish_values<OBJ_ORDER>(a, win, row, flags);
    else item_finish_values<OBJ_USER>(a, win, row, flags);
  }
  row[IW_FLAGS] = flags;
}
/* one list element (three words at e) per lane: are its integers integers? */
template <int E, int I = 0>
__device__ __forceinline__ void item_element_values(const ItemArgs& a, const uint8_t* win, const uint32_t* e, uint32_t* row) {
  if constexpr (I < CObj<E>::N) {
    static_assert(CObj<E>::N <= 2 && (CObj<E>::f[I].kind == K_I64 || CObj<E>::f[I].kind == K_I32 || CObj<E>::f[I].kind == K_STR), "elements: two integers or strings");
    if constexpr (CObj<E>::f[I].kind != K_STR) {
      if ((e[2] >> (4 + I)) & 1u) {
        const uint32_t ref = e[I], pos = ref & 0xFFFFu;
        int64_t v;
        if (!item_int(win, pos, (ref >> 16) & 0x7FFFu, CObj<E>::f[I].kind == K_I64, &v)) {
          const uint32_t x = win[pos];
          item_error(row, ref >> 31 ? pos - 1u : pos, (!(ref >> 31) && (x == 't' || x == 'f')) ? (uint32_t)PJ_E_TYPE : IE_REFUSED);
        }
      }
    }
    item_element_values<E, I + 1>(a, win, e, row);
  }
}

/* Group u of 32 list elements: which warp's (*w) and its first element (*j0). counts: elements per warp. */
template <class C>
__device__ __forceinline__ void item_unit(uint32_t u, C count_of, uint32_t* w, uint32_t* j0) {
  uint32_t at = 0, ww = 0, jj = 0;
#pragma unroll
  for (uint32_t k = 0; k < IT_WARPS; ++k) {
    const uint32_t n = (count_of(k) + 31u) >> 5;
    if (u >= at && u < at + n) { ww = k; jj = (u - at) * 32u; }
    at += n;
  }
  *w = ww; *j0 = jj;
}

/* ---- 4. emission ------------------------------------------------------------------------------------------------ */
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
/* string column (offsets at col, bytes at col + 1) of 32 rows: lane = row; start0: where the 32 rows' bytes start */
__device__ __forceinline__ void item_emit_string(const ItemArgs& a, uint32_t col, const uint8_t* win, bool has_row, uint64_t row_out, uint32_t ref, bool present, uint32_t start0) {
  const uint32_t n = present ? (ref >> 16) & 0x7FFFu : 0u;
  const uint32_t at = start0 + warp_incl_scan(n) - n;
  if (has_row) colp<uint32_t>(&a.cols, col)[row_out] = at;
  if (n) item_copy(colp<uint8_t>(&a.cols, col + 1) + at, win, ref & 0xFFFFu, n);
}
/* the columns of flat object or root OBJ at row_out: WORD0 / BIT0 = where its properties stand in the row */
template <int OBJ, bool ROOT, uint32_t WORD0, uint32_t BIT0, int I = 0>
__device__ __forceinline__ void item_emit_fields(const ItemArgs& a, ItemShared& sh, const uint8_t* win, const uint32_t* row, bool has_row, uint32_t flags, uint64_t row_out, uint32_t chunk,
                                                 uint32_t nP, uint32_t nT) {
  if constexpr (I == 0) {
    if (has_row) colp<uint8_t>(&a.cols, CObj<OBJ>::present_col)[row_out] = (uint8_t)((flags >> (IF_PRESENT + BIT0)) & ((1u << CObj<OBJ>::N) - 1u));
  }
  if constexpr (I < CObj<OBJ>::N) {
    constexpr uint32_t kind = CObj<OBJ>::f[I].kind, col = CObj<OBJ>::f[I].col, slot = CObj<OBJ>::f[I].cnt;
    constexpr uint32_t word = ROOT ? it_root_word<OBJ>(I) : WORD0 + it_flat_word<OBJ>(I);
    const bool pr = (flags >> (IF_PRESENT + BIT0 + I)) & 1u;
    if constexpr (kind == K_I64) {
      if (has_row) colp<int64_t>(&a.cols, col)[row_out] = pr ? (int64_t)((uint64_t)row[word] | ((uint64_t)row[word + 1] << 32)) : 0;
    } else if constexpr (kind == K_I32) {
      if (has_row) colp<int32_t>(&a.cols, col)[row_out] = pr ? (int32_t)row[word] : 0;
    } else if constexpr (kind == K_BOOL || kind == K_ENUM) {
      if (has_row) colp<uint8_t>(&a.cols, col)[row_out] = pr ? (uint8_t)row[word] : (kind == K_ENUM ? 255 : 0);
    } else if constexpr (kind == K_DATETIME) {
      if (has_row) {
        colp<int64_t>(&a.cols, col)[row_out] = pr ? (int64_t)((uint64_t)row[word] | ((uint64_t)row[word + 1] << 32)) : 0;
        colp<int32_t>(&a.cols, col + 1)[row_out] = pr ? (int32_t)row[word + 2] : 0;
        colp<int32_t>(&a.cols, col + 2)[row_out] = pr ? (int32_t)row[word + 3] : 0;
      }
    } else if constexpr (kind == K_STR) {
      item_emit_string(a, col, win, has_row, row_out, row[word], pr && has_row, sh.base[slot] + sh.csum[slot][chunk]);
    } else if constexpr (kind == K_OBJ) {
      /* absent: its own bits are clear as well */
      item_emit_fields<CObj<OBJ>::f[I].child, false, ItModel<OBJ>::child_word, IB_CHILD>(a, sh, win, row, has_row, flags, row_out, chunk, nP, nT);
    } else {
      const uint32_t n = kind == K_LIST_STR ? nP : nT;
      const uint32_t at = sh.base[slot] + sh.csum[slot][chunk] + warp_incl_scan(n) - n;
      if (has_row) colp<uint32_t>(&a.cols, col)[row_out] = at;
    }
    item_emit_fields<OBJ, ROOT, WORD0, BIT0, I + 1>(a, sh, win, row, has_row, flags, row_out, chunk, nP, nT);
  }
}

/* bytes of the row's strings per slot, added up over the warp into csum[slot][chunk] */
template <int OBJ, bool ROOT, uint32_t WORD0, uint32_t BIT0, int I = 0>
__device__ __forceinline__ void item_sum_fields(ItemShared& sh, const uint32_t* row, bool mine, uint32_t flags, uint32_t chunk, uint32_t lane, uint32_t nP, uint32_t nT) {
  if constexpr (I < CObj<OBJ>::N) {
    constexpr uint32_t kind = CObj<OBJ>::f[I].kind, slot = CObj<OBJ>::f[I].cnt;
    if constexpr (kind == K_STR) {
      constexpr uint32_t word = ROOT ? it_root_word<OBJ>(I) : WORD0 + it_flat_word<OBJ>(I);
      const uint32_t s = __reduce_add_sync(0xFFFFFFFFu, mine && ((flags >> (IF_PRESENT + BIT0 + I)) & 1u) ? (row[word] >> 16) & 0x7FFFu : 0u);
      if (lane == 0) sh.csum[slot][chunk] = s;
    } else if constexpr (kind == K_OBJ) item_sum_fields<CObj<OBJ>::f[I].child, false, ItModel<OBJ>::child_word, IB_CHILD>(sh, row, mine, flags, chunk, lane, nP, nT);
    else if constexpr (kind == K_LIST_STR || kind == K_LIST_OBJ) {
      const uint32_t s = __reduce_add_sync(0xFFFFFFFFu, mine ? (kind == K_LIST_STR ? nP : nT) : 0u);
      if (lane == 0) sh.csum[slot][chunk] = s;
    }
    item_sum_fields<OBJ, ROOT, WORD0, BIT0, I + 1>(sh, row, mine, flags, chunk, lane, nP, nT);
  }
}

/* ---- the exact parser -------------------------------------------------------------------------------------------- */
static __constant__ Schema c_schema; /* one copy per translation unit that includes this header (each sets its own) */

/* A record the fast steps refused, from its first byte at input offset s up to `limit`: kind and offset of its failure in *err,
 * *off, or *err = 0 when it is a valid one after all. */
template <int SCHEMA>
__device__ __noinline__ void item_exact(const ItemArgs& a, uint64_t s0, uint64_t limit, uint32_t* err, uint32_t* off) {
  Rd rd;
  rd.in = a.in; rd.lf_ws = a.sep ? 1u : 0u; rd.open_end = (a.is_last || a.sep) ? 0u : 1u; rd.limit = limit; rd.opts = a.opts; rd.rec_end = limit;
  PS s;
  s.p = s0; s.err = 0; s.err_pos = 0;
  Out<false> so;
  so.cols = &a.cols;
  parse_record<false>(c_schema, rd, s, (uint32_t)SCHEMA, so, 0);
  *err = s.err; *off = (uint32_t)(s.err_pos - s0);
}

/* The lines whose preceding separator lies in [lo, hi) of the input, one after the other (head: and before them the one at
 * byte 0): f(start, limit, blank). */
template <class F>
__device__ __forceinline__ void item_each_line(const ItemArgs& a, uint64_t lo, uint64_t hi, bool head, F f) {
  if (a.sep) {
    for (uint64_t p = lo; p < hi; ++p) {
      if (!((a.sep[p >> 6] >> (p & 63)) & 1u)) continue;
      const ExtentOut x = arr_extent(a.in, a.len, a.sep, p, a.res->first_opener);
      if (x.second_opener) atomicMin(&a.res->doc_err_off, (unsigned long long)p); /* a second document */
      if (x.is_record) f(x.start, x.end, x.blank != 0);
    }
  } else {
    if (head && nd_is_record(a.in, 0, a.limit, (int)a.is_last)) f((uint64_t)0, a.limit, false);
    for (uint64_t p = lo; p < hi; ++p)
      if (a.in[p] == '\n' && nd_is_record(a.in, p + 1, a.limit, (int)a.is_last)) f(p + 1, a.limit, false);
  }
}
/* A tile with the exact parser alone, read where it lies: every thread walks the lines that begin in its share of the
 * tile's bytes, once to size them and once to emit them. */
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
      item_each_line(a, lo, hi, head, [&](uint64_t s0, uint64_t limit, bool blank) {
        Rd rd;
        rd.in = a.in; rd.lf_ws = a.sep ? 1u : 0u; rd.open_end = (a.is_last || a.sep) ? 0u : 1u; rd.limit = limit; rd.opts = a.opts; rd.rec_end = limit;
        PS s;
        s.p = s0; s.err = 0; s.err_pos = 0;
        Out<false> so;
        so.cols = &a.cols;
        uint32_t type = PJ_TYPE_NONE;
        if (blank) fail(s, PJ_E_SYNTAX, limit);
        else type = parse_record<false>(c_schema, rd, s, (uint32_t)SCHEMA, so, 0);
        if (s.err) type = PJ_TYPE_NONE;
        if (pass == 0) {
          sum[IT_REC]++;
          nerr += s.err != 0;
          if (!s.err) for (uint32_t k = SL::lo; k < SL::hi; ++k) sum[k] += so.cnt[k];
        } else {
          const uint64_t i = my_base[IT_REC];
          colp<uint64_t>(&a.cols, PJ_COL_REC_START)[i] = a.goff + s0;
          colp<uint8_t>(&a.cols, PJ_COL_ERR_KIND)[i] = (uint8_t)s.err;
          colp<uint32_t>(&a.cols, PJ_COL_ERR_OFF)[i] = s.err ? (uint32_t)(s.err_pos - s0) : 0u;
          if (SCHEMA == PJ_SCHEMA_MIXED) {
            colp<uint8_t>(&a.cols, PJ_COL_REC_TYPE)[i] = (uint8_t)type;
            colp<uint32_t>(&a.cols, PJ_COL_REC_ROW)[i] = type == PJ_TYPE_NONE ? 0xFFFFFFFFu : my_base[type - 1];
          }
          Out<true> o;
          o.cols = &a.cols;
          for (uint32_t k = 0; k < NSLOT; ++k) { o.base[k] = my_base[k]; o.room[k] = (k >= SL::lo && k < SL::hi && !s.err) ? so.cnt[k] : 0u; }
          if (s.err) { if (SCHEMA != PJ_SCHEMA_MIXED) store_absent<true>(c_schema, (uint32_t)SCHEMA, o, i); }
          else {
            PS s2;
            s2.p = s0; s2.err = 0; s2.err_pos = 0;
            parse_record<true>(c_schema, rd, s2, (uint32_t)SCHEMA, o, i);
            for (uint32_t k = SL::lo; k < SL::hi; ++k) my_base[k] += so.cnt[k];
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

/* ---- a tile ------------------------------------------------------------------------------------------------------ */
/* Record i of the tile: which warp's (its first record is *first) and its row. */
__device__ __forceinline__ uint32_t item_row_of(const ItemShared& sh, uint32_t i, uint32_t* first) {
  uint32_t at = 0, row = 0;
  *first = 0;
#pragma unroll
  for (uint32_t k = 0; k < IT_WARPS; ++k) {
    const uint32_t n = sh.w[k].nrec;
    if (i >= at && i < at + n) { row = sh.w[k].row0 + (i - at); *first = at; }
    at += n;
  }
  return row;
}
/* The place in the tile's part of a child table of list element j of warp w, whose record has the row `row`: the elements of
 * failed records take none. T: the list of objects. */
template <bool TAGS>
__device__ __forceinline__ uint32_t item_child_place(const ItemShared& sh, const uint32_t* rows, uint32_t stride, uint32_t w, uint32_t row, uint32_t j, uint32_t slot) {
  uint32_t rec = row - sh.w[w].row0;
#pragma unroll
  for (uint32_t k = 0; k < IT_WARPS; ++k) if (k < w) rec += sh.w[k].nrec;
  const uint32_t d = rows[row * stride + IW_ERR];
  return sh.csum[slot][rec >> 5] + j + (uint32_t)(int32_t)(int16_t)(TAGS ? d >> 16 : d & 0xFFFFu);
}
/* row of the record that holds list string j of warp w: the first whose running count is above j */
__device__ __forceinline__ uint32_t item_photo_row(const ItemShared& sh, const uint32_t* rows, uint32_t stride, uint32_t w, uint32_t j) {
  uint32_t lo = 0, hi = sh.w[w].nrec - 1u;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if ((rows[(sh.w[w].row0 + mid) * stride + IW_CUM] & 0xFFFFu) > j) hi = mid; else lo = mid + 1u;
  }
  return sh.w[w].row0 + lo;
}
static constexpr uint32_t IF_BAD = 1u << 31; /* IW_FLAGS of a failed record: the rest is its error offset */

/* one list element (three words at e) per lane: its columns at row `at` of the child table */
template <int E, int I = 0>
__device__ __forceinline__ void item_emit_element(const ItemArgs& a, const uint8_t* win, const uint32_t* e, bool good, uint64_t at, uint32_t start0) {
  if constexpr (I == 0) { if (good) colp<uint8_t>(&a.cols, CObj<E>::present_col)[at] = (uint8_t)((e[2] >> 4) & ((1u << CObj<E>::N) - 1u)); }
  if constexpr (I < CObj<E>::N) {
    constexpr uint32_t kind = CObj<E>::f[I].kind, col = CObj<E>::f[I].col;
    const bool pr = good && ((e[2] >> (4 + I)) & 1u);
    if constexpr (kind == K_STR) item_emit_string(a, col, win, good, at, e[I], pr, start0);
    else {
      int64_t v = 0;
      if (pr) item_int(win, e[I] & 0xFFFFu, (e[I] >> 16) & 0x7FFFu, kind == K_I64, &v);
      if (good) { if constexpr (kind == K_I64) colp<int64_t>(&a.cols, col)[at] = v; else colp<int32_t>(&a.cols, col)[at] = (int32_t)v; }
    }
    item_emit_element<E, I + 1>(a, win, e, good, at, start0);
  }
}
template <int E>
PJ_CX int it_string_field() {
  int at = -1;
  for (int i = 0; i < CObj<E>::N; ++i) if (CObj<E>::f[i].kind == K_STR) at = i;
  return at;
}

/* Steps 2 to 4 of a tile whose index stands. False: the other road (no barrier is left open, nothing was published). */
template <int SCHEMA, bool ARR>
__device__ __forceinline__ bool item_tile(const ItemArgs& a, const StreamGeom& g, ItemShared& sh, uint8_t* win, uint32_t* strs, uint32_t* rows, uint32_t tile, uint32_t tid, long long* ck) {
  using SL = ItemSlots<SCHEMA>;
  constexpr uint32_t STRIDE = ItStride<SCHEMA>::n;
  static_assert(IT_RCHUNKS == IT_WARPS, "one group of 32 records per warp");
  const uint32_t lane = tid & 31, warp = tid >> 5;
  /* rows are handed out by the separators each warp met */
  {
    uint32_t at = 0, all = 0;
#pragma unroll
    for (uint32_t k = 0; k < IT_WARPS; ++k) { const uint32_t n = sh.w[k].nterm; if (k < warp) at += n; all += n; }
    if (all > a.row_cap) return false; /* the same for every thread */
    if (lane == 0) sh.w[warp].row0 = at;
    __syncwarp();
  }
  item_specials(a, sh, win, strs, warp, lane);
  __syncwarp();
  if (!item_tokens<SCHEMA, ARR>(a, g, sh, win, strs, rows, warp, lane)) sh.slow = 1;
  __syncthreads();
  if (sh.slow) return false;
  ck[2] = clock64();
  uint32_t nrec = 0, nu0 = 0, nu1 = 0;
#pragma unroll
  for (uint32_t k = 0; k < IT_WARPS; ++k) { nrec += sh.w[k].nrec; nu0 += (sh.w[k].nphoto + 31u) >> 5; nu1 += (sh.w[k].ntag + 31u) >> 5; }
  if (nrec > IT_MAX_RECS || nu0 > IT_MAX_UNITS || nu1 > IT_MAX_UNITS) return false;
  const uint32_t nchunk = (nrec + 31u) >> 5;
  constexpr int E = OBJ_TAG;
  constexpr uint32_t PCNT = CObj<OBJ_PET>::f[ItModel<OBJ_PET>::li].cnt, TCNT = CObj<OBJ_PET>::f[ItModel<OBJ_PET>::ei].cnt;
  constexpr uint32_t PCOL = CObj<OBJ_PET>::f[ItModel<OBJ_PET>::li].col;
  static_assert(ItModel<OBJ_PET>::elem == OBJ_TAG && ItModel<OBJ_ORDER>::elem < 0 && ItModel<OBJ_USER>::elem < 0 && ItModel<OBJ_ORDER>::li < 0 && ItModel<OBJ_USER>::li < 0, "lists are Pet's");
  constexpr int ES = it_string_field<E>();
  constexpr uint32_t ESLOT = CObj<E>::f[ES].cnt; /* arena of the elements' strings */
  auto photos = [&](uint32_t k) { return sh.w[k].nphoto; };
  auto tags = [&](uint32_t k) { return sh.w[k].ntag; };
  auto photo_ref = [&](uint32_t w, uint32_t j) { return strs[sh.w[w].str0 + sh.w[w].words - 1u - j]; };
  auto tag_row = [&](uint32_t w, uint32_t j) { return strs + sh.w[w].str0 + 3u * j; };

  /* this warp's 32 records */
  const uint32_t i = warp * 32u + lane;
  const bool live = i < nrec;
  uint32_t first_of_warp;
  const uint32_t r = item_row_of(sh, i, &first_of_warp);
  uint32_t* row = rows + r * STRIDE;

  /* ---- values; list elements are taken from the last warp on, the records from the first ---- */
  if (warp < nchunk) item_record_values<SCHEMA>(a, win, row, live);
  if constexpr (SL::lists) {
    for (uint32_t u = IT_WARPS - 1u - warp; u < nu1 + nu0; u += IT_WARPS) {
      uint32_t w, j0, n = 0;
      if (u < nu1) {
        item_unit(u, tags, &w, &j0);
        const uint32_t j = j0 + lane;
        if (j < sh.w[w].ntag) {
          const uint32_t* e = tag_row(w, j);
          item_element_values<E>(a, win, e, rows + (e[2] >> 16) * STRIDE);
          if ((e[2] >> (4 + ES)) & 1u) n = (e[ES] >> 16) & 0x7FFFu;
        }
      } else {
        item_unit(u - nu1, photos, &w, &j0);
        const uint32_t j = j0 + lane;
        if (j < sh.w[w].nphoto) n = photo_ref(w, j) >> 16;
      }
      n = __reduce_add_sync(0xFFFFFFFFu, n);
      if (lane == 0) { if (u < nu1) sh.usum[1][u] = n; else sh.usum[0][u - nu1] = n; }
    }
  }
  __syncthreads();

  ck[7] = clock64();
  /* ---- verdicts and sums ---- */
  uint32_t nP = 0, nT = 0, type = PJ_TYPE_NONE;
  bool good = false;
  if (warp < nchunk) {
    const uint32_t e = live ? row[IW_ERR] : IE_NONE;
    uint32_t flags = live ? row[IW_FLAGS] : 0u;
    good = live && e == IE_NONE;
    if constexpr (SL::lists) { /* list lengths: the running counts less those of the warp's record before */
      if (live) {
        const uint32_t cum = row[IW_CUM], prev = i != first_of_warp ? rows[(r - 1u) * STRIDE + IW_CUM] : 0u;
        nP = (cum & 0xFFFFu) - (prev & 0xFFFFu); nT = (cum >> 16) - (prev >> 16);
        if (!good && (nP | nT)) { /* the elements of a failed record count for nothing */
          uint32_t w = 0, u0 = 0, u1 = 0, at = 0;
#pragma unroll
          for (uint32_t k = 0; k < IT_WARPS; ++k) if (r >= sh.w[k].row0 && sh.w[k].nrec && r < sh.w[k].row0 + sh.w[k].nrec) w = k;
          for (uint32_t k = 0; k < w; ++k) { u0 += (sh.w[k].nphoto + 31u) >> 5; u1 += (sh.w[k].ntag + 31u) >> 5; }
          for (at = prev & 0xFFFFu; at < (cum & 0xFFFFu); ++at) atomicSub(&sh.usum[0][u0 + (at >> 5)], photo_ref(w, at) >> 16);
          for (at = prev >> 16; at < (cum >> 16); ++at) {
            const uint32_t* t = tag_row(w, at);
            if ((t[2] >> (4 + ES)) & 1u) atomicSub(&sh.usum[1][u1 + (at >> 5)], (t[ES] >> 16) & 0x7FFFu);
          }
          nP = 0; nT = 0;
        }
      }
    }
    if (live && !good) {
      sh.bad = 1;
      uint32_t kind = e & 0xFFu, off = (e >> 8) - (row[IW_POS] & 0xFFFFu);
      if ((flags & IF_MOVED) || kind == IE_REFUSED || ((a.opts & PJ_OPT_COERCE_SCALARS) && kind == PJ_E_TYPE)) {
        const uint64_t s0 = g.v0 + (row[IW_POS] & 0xFFFFu) - g.mis;
        uint64_t limit = a.limit;
        if (ARR) { uint64_t p = s0; while (p < a.len && !((a.sep[p >> 6] >> (p & 63)) & 1u)) ++p; limit = p; }
        item_exact<SCHEMA>(a, s0, limit, &kind, &off);
        if (!kind) sh.slow = 1; /* a valid record of a kind the fast steps do not know */
      }
      row[IW_ERR] = kind; row[IW_FLAGS] = IF_BAD | off;
      flags = 0;
    }
    if (good) type = item_type<SCHEMA>(flags);
    const uint32_t bl = __ballot_sync(0xFFFFFFFFu, live);
    if (lane == 0) sh.csum[IT_REC][warp] = (uint32_t)__popc(bl);
    if constexpr (SCHEMA == PJ_SCHEMA_MIXED) {
      const uint32_t bp = __ballot_sync(0xFFFFFFFFu, type == PJ_TYPE_PET), bo = __ballot_sync(0xFFFFFFFFu, type == PJ_TYPE_ORDER), bu = __ballot_sync(0xFFFFFFFFu, type == PJ_TYPE_USER);
      if (lane == 0) { sh.csum[SLOT_ROWS_PET][warp] = (uint32_t)__popc(bp); sh.csum[SLOT_ROWS_ORD][warp] = (uint32_t)__popc(bo); sh.csum[SLOT_ROWS_USR][warp] = (uint32_t)__popc(bu); }
    }
    if constexpr (SL::lists) {
      item_sum_fields<OBJ_PET, true, 0u, 0u>(sh, row, type == PJ_TYPE_PET, flags, warp, lane, nP, nT);
      /* from an element's number in its warp to its place behind the group's first */
      const uint32_t exP = warp_incl_scan(nP) - nP, exT = warp_incl_scan(nT) - nT;
      if (good) {
        const uint32_t prev = i != first_of_warp ? rows[(r - 1u) * STRIDE + IW_CUM] : 0u;
        row[IW_ERR] = ((exP - (prev & 0xFFFFu)) & 0xFFFFu) | ((exT - (prev >> 16)) << 16);
      }
    }
    if constexpr (SCHEMA == PJ_SCHEMA_USER || SCHEMA == PJ_SCHEMA_MIXED) item_sum_fields<OBJ_USER, true, 0u, 0u>(sh, row, type == PJ_TYPE_USER, flags, warp, lane, 0u, 0u);
  }
  __syncthreads();
  if (sh.slow) return false;
  ck[3] = clock64();

  /* ---- where everything of the tile goes ---- */
  if (warp == 0) {
#pragma unroll
    for (uint32_t k0 = 0; k0 < IT_NLB; k0 += 4) { /* four counters a time, eight groups of records each */
      if (!((SL::mask >> k0) & 15u)) continue;
      const uint32_t k = k0 + (lane >> 3), c = lane & 7u;
      const bool bytes = SL::lists && (k == PCNT + 1u || k == ESLOT); /* come from the groups of list elements */
      uint32_t v = (((SL::mask >> k) & 1u) && !bytes && c < nchunk) ? sh.csum[k][c] : 0u;
      uint32_t inc = v;
#pragma unroll
      for (int d = 1; d < 8; d <<= 1) { const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, d, 8); if (c >= (uint32_t)d) inc += x; }
      if (((SL::mask >> k) & 1u) && !bytes) { sh.csum[k][c] = inc - v; if (c == 7) sh.tot[k] = inc; }
    }
    if constexpr (SL::lists) {
#pragma unroll
      for (uint32_t l = 0; l < 2; ++l) {
        const uint32_t n = l ? nu1 : nu0;
        const uint32_t v0 = 2 * lane < n ? sh.usum[l][2 * lane] : 0u, v1 = 2 * lane + 1 < n ? sh.usum[l][2 * lane + 1] : 0u;
        const uint32_t inc = warp_incl_scan(v0 + v1);
        __syncwarp();
        sh.usum[l][2 * lane] = inc - v0 - v1; sh.usum[l][2 * lane + 1] = inc - v1;
        if (lane == 31) sh.tot[l ? ESLOT : PCNT + 1u] = inc;
      }
    }
    __syncwarp();
    item_resolve<SCHEMA>(a, sh, tile, lane);
  }
  __syncthreads();
  ck[4] = clock64();
  if (!sh.ok) return true;

  /* ---- emission ---- */
  if (warp < nchunk) {
    const uint64_t rec = (uint64_t)sh.base[IT_REC] + i; /* chunk starts are multiples of 32 records */
    const uint32_t flags = good ? row[IW_FLAGS] : 0u;
    const uint32_t bg = __ballot_sync(0xFFFFFFFFu, good), bl = __ballot_sync(0xFFFFFFFFu, live);
    if (lane == 0) {
      if (bl != bg) atomicAdd(&a.res->n_errors, (unsigned long long)__popc(bl & ~bg));
      if (bg) atomicAdd(&a.res->n_fast, (unsigned long long)__popc(bg));
    }
    if (live) {
      colp<uint64_t>(&a.cols, PJ_COL_REC_START)[rec] = a.goff + g.v0 + (row[IW_POS] & 0xFFFFu) - g.mis;
      colp<uint8_t>(&a.cols, PJ_COL_ERR_KIND)[rec] = good ? 0 : (uint8_t)row[IW_ERR];
      colp<uint32_t>(&a.cols, PJ_COL_ERR_OFF)[rec] = good ? 0u : row[IW_FLAGS] & ~IF_BAD;
    }
    if constexpr (SCHEMA == PJ_SCHEMA_PET) item_emit_fields<OBJ_PET, true, 0u, 0u>(a, sh, win, row, live, flags, rec, warp, nP, nT);
    else if constexpr (SCHEMA == PJ_SCHEMA_ORDER) item_emit_fields<OBJ_ORDER, true, 0u, 0u>(a, sh, win, row, live, flags, rec, warp, 0u, 0u);
    else if constexpr (SCHEMA == PJ_SCHEMA_USER) item_emit_fields<OBJ_USER, true, 0u, 0u>(a, sh, win, row, live, flags, rec, warp, 0u, 0u);
    else {
      const uint32_t lt = (1u << lane) - 1u;
      const uint32_t bp = __ballot_sync(0xFFFFFFFFu, type == PJ_TYPE_PET), bo = __ballot_sync(0xFFFFFFFFu, type == PJ_TYPE_ORDER), bu = __ballot_sync(0xFFFFFFFFu, type == PJ_TYPE_USER);
      const uint32_t mine = type == PJ_TYPE_PET ? bp : (type == PJ_TYPE_ORDER ? bo : bu);
      const uint32_t slot = type == PJ_TYPE_PET ? SLOT_ROWS_PET : (type == PJ_TYPE_ORDER ? SLOT_ROWS_ORD : SLOT_ROWS_USR);
      const uint32_t out = sh.base[slot] + sh.csum[slot][warp] + (uint32_t)__popc(mine & lt);
      if (live) {
        colp<uint8_t>(&a.cols, PJ_COL_REC_TYPE)[rec] = (uint8_t)type;
        colp<uint32_t>(&a.cols, PJ_COL_REC_ROW)[rec] = type == PJ_TYPE_NONE ? 0xFFFFFFFFu : out;
      }
      if (bp) item_emit_fields<OBJ_PET, true, 0u, 0u>(a, sh, win, row, type == PJ_TYPE_PET, type == PJ_TYPE_PET ? flags : 0u, out, warp, type == PJ_TYPE_PET ? nP : 0u, type == PJ_TYPE_PET ? nT : 0u);
      if (bo) item_emit_fields<OBJ_ORDER, true, 0u, 0u>(a, sh, win, row, type == PJ_TYPE_ORDER, type == PJ_TYPE_ORDER ? flags : 0u, out, warp, 0u, 0u);
      if (bu) item_emit_fields<OBJ_USER, true, 0u, 0u>(a, sh, win, row, type == PJ_TYPE_USER, type == PJ_TYPE_USER ? flags : 0u, out, warp, 0u, 0u);
    }
  }
  if constexpr (SL::lists) {
    const bool bad = sh.bad != 0;
    for (;;) { /* groups of list elements go to whoever is free */
      uint32_t u = 0;
      if (lane == 0) u = atomicAdd(&sh.next, 1u);
      u = __shfl_sync(0xFFFFFFFFu, u, 0);
      if (u >= nu0 + nu1) break;
      uint32_t w, j0;
      if (u < nu0) {
        item_unit(u, photos, &w, &j0);
        const uint32_t j = j0 + lane;
        const bool has = j < sh.w[w].nphoto;
        bool ok = has;
        uint32_t at = 0, ref = 0;
        if (has) {
          ref = photo_ref(w, j);
          if (bad) {
            const uint32_t pr = item_photo_row(sh, rows, STRIDE, w, j);
            ok = !(rows[pr * STRIDE + IW_FLAGS] & IF_BAD);
            if (ok) at = item_child_place<false>(sh, rows, STRIDE, w, pr, j, PCNT);
          } else {
            at = j;
#pragma unroll
            for (uint32_t k = 0; k < IT_WARPS; ++k) if (k < w) at += sh.w[k].nphoto;
          }
        }
        item_emit_string(a, PCOL + 1u, win, ok, (uint64_t)sh.base[PCNT] + at, ref, ok, sh.base[PCNT + 1u] + sh.usum[0][u]);
      } else {
        item_unit(u - nu0, tags, &w, &j0);
        const uint32_t j = j0 + lane;
        const bool has = j < sh.w[w].ntag;
        bool ok = has;
        uint32_t at = 0;
        const uint32_t* e = tag_row(w, has ? j : j0);
        if (has) {
          const uint32_t pr = e[2] >> 16;
          if (bad) {
            ok = !(rows[pr * STRIDE + IW_FLAGS] & IF_BAD);
            if (ok) at = item_child_place<true>(sh, rows, STRIDE, w, pr, j, TCNT);
          } else {
            at = j;
#pragma unroll
            for (uint32_t k = 0; k < IT_WARPS; ++k) if (k < w) at += sh.w[k].ntag;
          }
        }
        item_emit_element<E>(a, win, e, ok, (uint64_t)sh.base[TCNT] + at, sh.base[ESLOT] + sh.usum[1][u - nu0]);
      }
    }
  }
  if (tile == a.ntiles - 1) item_close_offsets(a, sh, tid);
  return true;
}

template <int SCHEMA> struct ItTablesOf { static constexpr ItTables t = it_tables(SCHEMA); };
template <int SCHEMA> __device__ const ItTables d_item_tables = ItTablesOf<SCHEMA>::t;
template <bool ARR> struct ItGapTableOf { static constexpr ItGapTable t = it_gap_table(ARR ? IT_ARR_SEP : (uint32_t)'\n'); };
template <bool ARR> __device__ const ItGapTable d_gap_table = ItGapTableOf<ARR>::t;

template <int SCHEMA>
__global__ void __launch_bounds__(IT_THREADS, 3) k_parse_items(const __grid_constant__ ItemArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ __align__(16) ItemShared sh;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const ItemLayout lay = item_layout(a.win_bytes, a.str_ratio, a.row_cap, ItStride<SCHEMA>::n);
  uint8_t* win = smem + lay.win;
  uint32_t* strs = reinterpret_cast<uint32_t*>(smem + lay.strs);
  uint32_t* rows = reinterpret_cast<uint32_t*>(smem + lay.rows);

  if (tid == 0) { sh.tile = atomicAdd(a.ticket, 1u); mbar_init(&sh.mbar, 1); sh.slow = 0; sh.bad = 0; sh.next = 0; }
  __syncthreads();
  const uint32_t tile = sh.tile;
  if (tile >= a.ntiles) return;
  long long ck[8];
  ck[0] = clock64();
  const uint32_t mis = (uint32_t)(reinterpret_cast<uintptr_t>(a.in) & 15u);
  const StreamGeom g = stream_geom(mis, a.len, a.limit, a.tile_bytes, tile, a.win_bytes);

  /* ---- stage the window: one bulk copy of whole 16-byte blocks (the first and the last one may hold bytes that are not
     input: they lie in the same aligned 16 bytes as input bytes, so they are readable; they are masked) ---- */
  if (g.copy_bytes && tid == 0) { mbar_expect_tx(&sh.mbar, g.copy_bytes); bulk_g2s(win, a.in - mis + g.v0, g.copy_bytes, &sh.mbar); }
  for (uint32_t k = tid; k < IT_SLOTS * 8; k += IT_THREADS) (&sh.key[0][0])[k] = (&d_item_tables<SCHEMA>.key[0][0])[k];
  for (uint32_t k = tid; k < IT_SLOTS * 3; k += IT_THREADS) (&sh.field[0][0])[k] = (&d_item_tables<SCHEMA>.field[0][0])[k];
  {
    const uint32_t* gt = reinterpret_cast<const uint32_t*>(a.sep ? d_gap_table<true>.e : d_gap_table<false>.e);
    for (uint32_t k = tid; k < IG_SLOTS * 4; k += IT_THREADS) reinterpret_cast<uint32_t*>(sh.gap)[k] = gt[k];
  }
  for (uint32_t k = tid; k < IT_WARPS * IT_MAX_STRS / 32; k += IT_THREADS) { (&sh.special[0][0])[k] = 0; (&sh.broken[0][0])[k] = 0; }
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
  if (tid < 64) win[g.hi_valid + tid] = '\n';
  __syncthreads();
  ck[1] = clock64();

  bool done = false;
  if (a.sep) {
    /* a document that is not one clean array is left to the other road */
    const bool clean = a.res->doc_err_off == ~0ull && a.res->n_openers == 1u && !a.res->arr_final_s && a.res->arr_final_d == 0;
    if (clean) {
      if (!item_index<true>(a, g, sh, win, strs, warp, lane, tile)) sh.slow = 1;
      __syncthreads();
      ck[6] = clock64();
      if (!sh.slow) done = item_tile<SCHEMA, true>(a, g, sh, win, strs, rows, tile, tid, ck);
    }
  } else {
    if (!item_index<false>(a, g, sh, win, strs, warp, lane, tile)) sh.slow = 1;
    __syncthreads();
    ck[6] = clock64();
    if (!sh.slow) done = item_tile<SCHEMA, false>(a, g, sh, win, strs, rows, tile, tid, ck);
  }
  if (!done) {
    __syncthreads();
    item_slow_tile<SCHEMA>(a, g, sh, tile, tid);
    return;
  }
  __syncthreads();
  if (tid == 0) {
    const long long c5 = clock64();
    atomicAdd(&a.res->phase_cycles[0], (unsigned long long)(ck[1] - ck[0]));
    atomicAdd(&a.res->n_wide, (unsigned long long)(ck[6] - ck[1])); atomicAdd(&a.res->n_wide_fast, (unsigned long long)(ck[2] - ck[6])); atomicAdd(&a.res->wide_cycles[0], (unsigned long long)(ck[7] - ck[2])); atomicAdd(&a.res->wide_cycles[1], (unsigned long long)(ck[3] - ck[7]));
    atomicAdd(&a.res->phase_cycles[1], (unsigned long long)(ck[3] - ck[1]));
    atomicAdd(&a.res->phase_cycles[2], (unsigned long long)(ck[4] - ck[3]));
    atomicAdd(&a.res->phase_cycles[3], (unsigned long long)(c5 - ck[4]));
  }
}

}  // namespace pj
#endif

/*
 * pj_index_emu.cpp — TEST INFRASTRUCTURE. k_arr_index (pj_array_index.cuh), k_nd_records (pj_kernels.cuh) and k_arr_records
 * (pj_array_kernels.cuh), unchanged, on the host, block after block, under pj_block_emu.h; the separators word after word by
 * pj_array_ref.h; and the look-backs alone, on states that blocks running side by side would leave. tests/test_index_emulation.py drives it.
 */
#include <algorithm>
#include <vector>

#include "pj_block_emu.h"

/* what the kernels beside it use */
static struct { uint32_t x, y; } blockIdx, gridDim;
template <class T> static inline T __ldg(const T* p) { return *p; }
static inline uint32_t __vcmpeq4(uint32_t a, uint32_t b) {
  uint32_t r = 0;
  for (int k = 0; k < 4; ++k) if (((a ^ b) >> (8 * k) & 255u) == 0) r |= 255u << (8 * k);
  return r;
}
static inline int __popcll(unsigned long long x) { return __builtin_popcountll(x); }
static inline int __ffsll(long long x) { return __builtin_ffsll(x); }
static inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t s) { return (uint32_t)(((((uint64_t)hi << 32) | lo) << (s & 31u)) >> 32); }
namespace pj {
inline void bulk_s2g(void*, const void*, uint32_t) {}
inline void bulk_s2g_wait_read() {}
inline void fence_async_smem() {}
}  // namespace pj

#include "pj_array_kernels.cuh"
#include "pj_array_ref.h"

using namespace pj;

namespace {
ArrIndexArgs g_args;
void one_thread_1(void*) { k_arr_index<1>(g_args); }
void one_thread_4(void*) { k_arr_index<4>(g_args); }
IndexArgs g_index;
ArrArgs g_arr;
RecordTiles g_tiles;
void nd_thread_1(void*) { k_nd_records<1>(g_index, g_tiles); }
void nd_thread_4(void*) { k_nd_records<4>(g_index, g_tiles); }
void arr_thread(void*) { k_arr_records(g_arr, g_tiles); }
/* a look-back by one warp; every lane's answer */
struct Back { uint32_t tile; bool ok[32]; ArrState state[32]; unsigned long long excl[32]; uint32_t* flag; } g_back;
void arr_back(void*) { const uint32_t l = threadIdx.x; g_back.ok[l] = arr_lookback(g_args, g_back.tile, l, &g_back.state[l]); }
void sum_back(void*) { const uint32_t l = threadIdx.x; g_back.ok[l] = lookback_u64(g_tiles.agg, g_tiles.inc, g_back.flag, 1, g_back.tile, l, &g_back.excl[l]); }
}  // namespace

extern "C" const char* emu_index_error() { return emu_block::error; }
/* Returns 0, or what differs: 1 separators, 2 first byte outside the array, 3 first opener, 4 final state; -1: a rule of the block was broken. */
extern "C" int emu_arr_index(const uint8_t* in, uint64_t len, uint32_t words, uint32_t order) {
  const uint64_t nwords = (len + 63) >> 6;
  std::vector<uint64_t> want(nwords + 1, 0), got(nwords + 1, 0);
  DevResult res;
  memset((void*)&res, 0, sizeof res);
  res.doc_err_off = res.first_opener = ~0ull;
  unsigned long long doc = ~0ull, first = ~0ull;
  ArrState st;
  st.c = 0; st.s = 0; st.d = 0;
  for (uint64_t w = 0; w < nwords; ++w) {
    const WordMasks m = word_masks(in + w * 64, (uint32_t)std::min<uint64_t>(64, len - w * 64));
    const WordEval e = eval_word(m, st);
    const WordMarks k = mark_word(m, e, st.d);
    want[w] = k.sep;
    if (k.doc_bit < 64) doc = std::min<unsigned long long>(doc, w * 64 + k.doc_bit);
    if (k.opener_bit < 64) first = std::min<unsigned long long>(first, w * 64 + k.opener_bit);
    st = e.out;
  }
  emu_block::error[0] = 0; emu_block::steps = 0;
  ArrIndexArgs& a = g_args;
  memset((void*)&a, 0, sizeof a);
  const uint32_t mis = (uint32_t)((uintptr_t)in & 15u);
  if (!mis) std::fill(got.begin(), got.end(), ~0ull); /* (stored, not or-ed) */
  a.in = in; a.len = len; a.sep = got.data(); a.ntiles = arr_tiles(mis, len, words);
  std::vector<unsigned long long> state(3 * (size_t)a.ntiles, 0);
  uint32_t ticket = 0;
  a.ticket = &ticket; a.fn0 = state.data(); a.fn1 = a.fn0 + a.ntiles; a.inc = a.fn1 + a.ntiles;
  a.spin_limit_ns = 1; a.res = &res;
  for (uint32_t t = 0; t < a.ntiles; ++t)
    if (!emu_block::run(AI_THREADS, words == 4 ? one_thread_4 : one_thread_1, nullptr, order + t)) return -1;
  if (res.timeout) return -1;
  if (memcmp(want.data(), got.data(), nwords * 8)) return 1;
  if (res.doc_err_off != doc) return 2;
  if (res.first_opener != first) return 3;
  return res.arr_final_s == st.s && res.arr_final_d == st.d ? 0 : 4;
}

/* The record index: words 1 or 4, or 0 for an array, whose separators are taken from pj_array_ref.h. Returns the number of records or -1. */
extern "C" int64_t emu_index_records(const uint8_t* in, uint64_t len, uint32_t words, uint64_t* starts, uint64_t cap, uint32_t order) {
  emu_block::error[0] = 0; emu_block::steps = 0;
  DevResult res;
  memset((void*)&res, 0, sizeof res);
  res.doc_err_off = res.first_opener = ~0ull;
  const uint64_t nwords = (len + 63) >> 6, per = (uint64_t)INDEX_TILE * (words ? words : 1);
  std::vector<uint64_t> sep(nwords + 1, 0);
  if (!words) {
    ArrState st;
    st.c = 0; st.s = 0; st.d = 0;
    for (uint64_t w = 0; w < nwords; ++w) {
      const WordMasks m = word_masks(in + w * 64, (uint32_t)std::min<uint64_t>(64, len - w * 64));
      const WordEval e = eval_word(m, st);
      const WordMarks k = mark_word(m, e, st.d);
      sep[w] = k.sep;
      if (k.opener_bit < 64) res.first_opener = std::min<unsigned long long>(res.first_opener, w * 64 + k.opener_bit);
      st = e.out;
    }
  }
  memset((void*)&g_index, 0, sizeof g_index);
  g_index.in = in; g_index.len = g_index.limit = len; g_index.is_first = g_index.is_last = 1; g_index.rec_start = starts; g_index.cap = cap;
  g_arr.in = in; g_arr.len = len; g_arr.nwords = nwords; g_arr.sep = sep.data(); g_arr.rec_start = starts; g_arr.cap = cap; g_arr.goff = 0; g_arr.res = &res;
  const uint64_t ntiles = words ? (len + 15 + per) / per : (nwords ? (nwords + ARR_THREADS - 1) / ARR_THREADS : 1);
  std::vector<unsigned long long> state(2 * ntiles, 0);
  uint32_t ticket = 0;
  g_tiles.ticket = &ticket; g_tiles.agg = state.data(); g_tiles.inc = state.data() + ntiles; g_tiles.ntiles = (uint32_t)ntiles; g_tiles.spin_limit_ns = 1; g_tiles.res = &res;
  for (uint64_t t = 0; t < ntiles; ++t)
    if (!emu_block::run(words ? INDEX_THREADS : ARR_THREADS, words == 4 ? nd_thread_4 : (words ? nd_thread_1 : arr_thread), nullptr, order + (uint32_t)t)) return -1;
  return res.timeout ? -1 : (int64_t)res.n_records;
}

/* The state before `tile` of n tiles: functions d[4 n], st[n] of all of them, the state behind tile `known` (c | s << 1, depth), which is the newest that is
 * known. missing: a tile that has published nothing yet (n: none). Returns 0, 1 (lanes differ, or not the serial fold's state), 2 (gave up) or -1. */
extern "C" int emu_arr_lookback(uint32_t n, uint32_t tile, const uint8_t* st, const int32_t* d, int32_t known, uint32_t known_state, int32_t known_depth, uint32_t missing) {
  emu_block::error[0] = 0; emu_block::steps = 0;
  DevResult res;
  memset((void*)&res, 0, sizeof res);
  std::vector<unsigned long long> fn0(n, 0), fn1(n, 0), inc(n, 0);
  for (uint32_t t = 0; t < tile; ++t) {
    if (t == missing) continue;
    fn0[t] = fn_pack(d[4 * t], d[4 * t + 1]) | ((unsigned long long)st[t] << 40);
    fn1[t] = fn_pack(d[4 * t + 2], d[4 * t + 3]);
  }
  ArrState s;
  s.c = s.s = 0; s.d = 0;
  if (known >= 0) { s.c = known_state & 1u; s.s = known_state >> 1; s.d = known_depth; inc[known] = state_pack(s); fn0[known] = 0; }
  for (uint32_t t = (uint32_t)(known + 1); t < tile; ++t) { /* one after the other */
    const uint32_t x = s.c | (s.s << 1), o = (st[t] >> (2 * x)) & 3u;
    s.d += d[4 * t + x]; s.c = o & 1u; s.s = o >> 1;
  }
  memset((void*)&g_args, 0, sizeof g_args);
  g_args.fn0 = fn0.data(); g_args.fn1 = fn1.data(); g_args.inc = inc.data(); g_args.spin_limit_ns = 1; g_args.res = &res;
  if (missing < n) res.timeout = 1; /* (another tile has run out of patience; time stands still here) */
  g_back.tile = tile;
  if (!emu_block::run(32, arr_back, nullptr, tile)) return -1;
  for (int l = 0; l < 32; ++l) {
    if (!g_back.ok[l]) return 2;
    if (g_back.state[l].c != s.c || g_back.state[l].s != s.s || g_back.state[l].d != s.d) return 1;
  }
  return 0;
}
/* The same of running totals: agg[n] of the tiles, the total up to and including tile `known`. */
extern "C" int emu_sum_lookback(uint32_t n, uint32_t tile, const uint64_t* agg, int32_t known, uint64_t upto, uint32_t missing) {
  emu_block::error[0] = 0; emu_block::steps = 0;
  std::vector<unsigned long long> a(n, 0), inc(n, 0);
  unsigned long long want = known >= 0 ? upto : 0;
  for (uint32_t t = 0; t < tile; ++t) {
    if (t != missing && (int32_t)t != known) a[t] = TS_VALID | agg[t];
    if ((int32_t)t > known) want += agg[t];
  }
  if (known >= 0) inc[known] = TS_VALID | upto;
  g_tiles.agg = a.data(); g_tiles.inc = inc.data();
  uint32_t flag = missing < n;
  g_back.flag = &flag; g_back.tile = tile;
  if (!emu_block::run(32, sum_back, nullptr, tile)) return -1;
  for (int l = 0; l < 32; ++l) {
    if (!g_back.ok[l]) return 2;
    if (g_back.excl[l] != want) return 1;
  }
  return 0;
}

/*
 * pj_index_emu.cpp — TEST INFRASTRUCTURE. k_arr_index (pj_array_index.cuh, unchanged) on the host, block after block, under
 * pj_block_emu.h, and the same separators word after word by the functions of pj_array.cuh. tests/test_index_emulation.py drives it.
 */
#include <algorithm>
#include <vector>

#include "pj_block_emu.h"
#include "pj_array_index.cuh"

using namespace pj;

namespace {
ArrIndexArgs g_args;
void one_thread_1(void*) { k_arr_index<1>(g_args); }
void one_thread_4(void*) { k_arr_index<4>(g_args); }
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

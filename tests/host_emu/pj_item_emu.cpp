/*
 * pj_item_emu.cpp — TEST INFRASTRUCTURE. k_parse_items (pj_item.cuh, unchanged) on the host, block after block, under
 * pj_block_emu.h. Compiled once per model set with -DEMU_SCHEMA=1..4; tests/test_item_emulation.py drives it.
 */
#include <algorithm>
#include <vector>

#include "pj_block_emu.h"
#include "pj_item.cuh"
#include "pj_item_shape.h"
#include "pj_choice.h"
#include "pj_array_ref.h"

using namespace pj;

namespace pj {
thread_local __attribute__((aligned(16))) uint8_t smem[228 * 1024];
}

#define CAT2(a, b) a##b
#define CAT(a, b) CAT2(a, b)

namespace {
ItemArgs g_args;
void one_thread(void*) { k_parse_items<EMU_SCHEMA>(g_args); }

struct Opts { /* mirrored in tests/test_item_emulation.py */
  uint64_t len, slack, goff;
  uint32_t array, is_first, is_last, opts, tile_bytes, win_bytes, str_words, row_cap, order;
  uint64_t rec_cap;
};
/* separators of an array, word after word as the index kernels evaluate them */
void array_index(const uint8_t* in, uint64_t len, std::vector<uint64_t>& sep, DevResult& res) {
  const uint64_t nwords = (len + 63) >> 6;
  sep.assign(nwords + 1, 0);
  ArrState st;
  st.c = 0; st.s = 0; st.d = 0;
  res.doc_err_off = res.first_opener = ~0ull;
  for (uint64_t w = 0; w < nwords; ++w) {
    const WordMasks m = word_masks(in + w * 64, (uint32_t)std::min<uint64_t>(64, len - w * 64));
    const WordEval e = eval_word(m, st);
    const WordMarks k = mark_word(m, e, st.d);
    sep[w] = k.sep;
    if (k.doc_bit < 64) res.doc_err_off = std::min<unsigned long long>(res.doc_err_off, w * 64 + k.doc_bit);
    if (k.opener_bit < 64) res.first_opener = std::min<unsigned long long>(res.first_opener, w * 64 + k.opener_bit);
    st = e.out;
  }
  res.arr_final_s = st.s; res.arr_final_d = st.d;
}
}  // namespace

extern "C" const char* emu_item_error() { return emu_block::error; }
extern "C" uint64_t emu_item_barriers() { return emu_block::n_barriers; }
static NdChoice g_choice;
extern "C" void emu_choice_reset() { g_choice = NdChoice(); }
/* the call just made; returns whether the next one takes k_parse_items */
extern "C" int emu_choice_note(uint64_t len, float ms, uint64_t records, uint64_t errors, uint64_t fast, uint64_t dense, uint32_t max_rec) {
  note_call(g_choice, len, ms, records, errors, fast, dense, max_rec);
  return g_choice.items;
}
/* out: tile, window, words for strings, rows, bytes of dynamic shared memory, the most that may be, blocks an SM holds */
extern "C" void emu_item_shape(uint64_t len, double avg, double guess, uint32_t longest, uint32_t strs_per_kb, uint32_t tile_opt, uint32_t* out) {
  const ItemShape s = item_shape(ItemShapeIn{len, avg, guess, longest, strs_per_kb, tile_opt, ItStride<EMU_SCHEMA>::n, 148});
  const uint32_t total = item_layout(s.win_bytes, s.str_words, s.row_cap, ItStride<EMU_SCHEMA>::n).total;
  uint32_t blocks = IT_BLOCKS;
  while (blocks > 1 && total > item_room(blocks)) --blocks;
  const uint32_t v[7] = {s.tile_bytes, s.win_bytes, s.str_words, s.row_cap, total, IT_MAX_DYN_SMEM, blocks};
  for (int k = 0; k < 7; ++k) out[k] = v[k];
}

/* in: 16-byte aligned base + the caller's misalignment, readable in whole 16-byte blocks. stats[5]: fast records, lines the strict
 * walk took, longest record, tiles, strings per 1024 bytes. Returns 0, 1 (some buffer is too small) or -1 (see emu_item_error). */
extern "C" int emu_item_parse(const Opts* o, const uint8_t* in, pj_columns* out, uint64_t* stats) {
  Schema S;
  build_schema(&S);
  memcpy((void*)&c_schema, &S, sizeof S);
  emu_block::error[0] = 0; emu_block::n_barriers = 0; emu_block::steps = 0;
  ItemArgs& a = g_args;
  memset((void*)&a, 0, sizeof a);
  DevResult res;
  memset(&res, 0, sizeof res);
  std::vector<uint64_t> sep;
  if (o->array) array_index(in, o->len, sep, res);
  a.in = in; a.len = o->len; a.limit = o->len + o->slack; a.goff = o->goff;
  a.is_first = o->is_first; a.is_last = o->is_last;
  a.tile_bytes = o->tile_bytes; a.win_bytes = o->win_bytes; a.str_words = o->str_words; a.row_cap = o->row_cap;
  a.ntiles = (uint32_t)stream_tiles((uint32_t)((uintptr_t)in & 15u), o->len, 1u, o->tile_bytes);
  a.opts = o->opts; a.spin_limit_ns = 1;
  a.sep = o->array ? sep.data() : nullptr;
  std::vector<ItemTile> tiles(a.ntiles);
  memset((void*)tiles.data(), 0, tiles.size() * sizeof(ItemTile));
  uint32_t ticket = 0;
  a.tiles = tiles.data(); a.ticket = &ticket; a.res = &res;
  build_finalize_plan(S, EMU_SCHEMA, &a.plan);
  for (int i = 0; i < PJ_MAX_COLS; ++i) a.cols.ptr[i] = out->col[i].ptr;
  for (uint32_t k = 0; k < NSLOT; ++k) a.slot_cap[k] = 0xFFFFFFFFull;
  a.rec_cap = o->rec_cap;
  const uint32_t total = item_layout(a.win_bytes, a.str_words, a.row_cap, ItStride<EMU_SCHEMA>::n).total;
  if (total > sizeof smem) { snprintf(emu_block::error, sizeof emu_block::error, "shared memory: %u bytes", total); return -1; }
  bool fine = true;
  for (uint32_t t = 0; t < a.ntiles && fine; ++t) {
    memset(smem, 0xC3, total);
    EMU_POISON(smem + total, sizeof smem - total);
    fine = emu_block::run(IT_THREADS, one_thread, nullptr, o->order + t);
    EMU_UNPOISON(smem + total, sizeof smem - total);
  }
  if (fine && res.timeout) { snprintf(emu_block::error, sizeof emu_block::error, "a bounded wait ran out"); fine = false; }
  if (!fine) return -1;
  stats[0] = res.n_fast; stats[1] = res.n_dense; stats[2] = res.max_rec; stats[3] = a.ntiles; stats[4] = res.strs_per_kb;
  const uint64_t N = res.n_records;
  for (int c = 0; c < PJ_MAX_COLS; ++c) out->col[c].count = 0;
  out->col[PJ_COL_REC_START].count = out->col[PJ_COL_ERR_KIND].count = out->col[PJ_COL_ERR_OFF].count = N;
  if (EMU_SCHEMA == PJ_SCHEMA_MIXED) out->col[PJ_COL_REC_TYPE].count = out->col[PJ_COL_REC_ROW].count = N;
  for (uint32_t k = 0; k < a.plan.n; ++k) {
    const FinalizeItem& it = a.plan.item[k];
    out->col[it.col].count = (it.rows_slot == 0xFF ? N : res.total[it.rows_slot]) + (it.sentinel_slot != 0xFF ? 1 : 0);
  }
  out->schema = EMU_SCHEMA; out->n_records = N; out->n_errors = res.n_errors;
  for (int t = 0; t < 4; ++t) out->n_rows[t] = 0;
  if (EMU_SCHEMA == PJ_SCHEMA_MIXED) { out->n_rows[1] = res.total[SLOT_ROWS_PET]; out->n_rows[2] = res.total[SLOT_ROWS_ORD]; out->n_rows[3] = res.total[SLOT_ROWS_USR]; }
  else out->n_rows[EMU_SCHEMA] = N;
  out->doc_err_kind = 0; out->doc_err_off = 0;
  if (o->array) {
    if (res.doc_err_off != ~0ull) { out->doc_err_kind = PJ_E_SYNTAX; out->doc_err_off = res.doc_err_off; }
    else if (res.first_opener == ~0ull || res.arr_final_s || res.arr_final_d != 0) { out->doc_err_kind = PJ_E_EOF; out->doc_err_off = o->len; }
  }
  return res.over ? 1 : 0;
}

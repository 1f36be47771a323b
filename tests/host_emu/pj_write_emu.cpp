/*
 * pj_write_emu.cpp — TEST INFRASTRUCTURE. k_write_tile (pj_write_tile.cuh, unchanged) on the host, block after block, under
 * pj_block_emu.h. tests/test_write_emulation.py drives it.
 */
#include <vector>

#include "pj_block_emu.h"

/* what the writer uses besides */
static inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t s) { return (uint32_t)(((((uint64_t)hi << 32) | lo) << (s & 31u)) >> 32); }
namespace pj {
inline void bulk_s2g(void* dst, const void* src, uint32_t bytes) {
  if (((uintptr_t)dst | (uintptr_t)src | bytes) & 15u) emu_block::fail("a bulk copy that is not aligned", __LINE__);
  memcpy(dst, src, bytes);
}
inline void bulk_s2g_wait_read() {}
inline void fence_async_smem() {}
}  // namespace pj

#include "pj_write_tile.cuh"
#include "pj_write_shape.h"

using namespace pj;

namespace pj {
thread_local __attribute__((aligned(16))) uint8_t smem[228 * 1024];
}

namespace {
static bool g_short = false;
WTileArgs g_args;
uint32_t g_schema;
void one_thread(void*) {
  switch (g_schema) {
    case PJ_SCHEMA_PET: if (g_short) k_write_tile<PJ_SCHEMA_PET, WT_SHORT_THREADS>(g_args); else k_write_tile<PJ_SCHEMA_PET>(g_args); break;
    case PJ_SCHEMA_ORDER: k_write_tile<PJ_SCHEMA_ORDER>(g_args); break;
    case PJ_SCHEMA_USER: k_write_tile<PJ_SCHEMA_USER>(g_args); break;
    default: k_write_tile<PJ_SCHEMA_MIXED>(g_args); break;
  }
}
}  // namespace

/* Pets by blocks of WT_SHORT_THREADS, from now on. */
extern "C" void emu_write_short(int on) { g_short = on != 0; }
extern "C" const char* emu_write_error() { return emu_block::error; }
/* The records' text without the brackets of an array. recs, shared: records per tile, bytes of shared memory. Returns 0, 1 (no room) or -1. */
extern "C" int emu_write_tiles(uint32_t schema, uint32_t array, int inclusion, uint32_t lower, const pj_columns* cols, uint8_t* out, uint64_t cap, uint32_t recs, uint32_t shared,
                               uint32_t order, uint64_t* out_len) {
  emu_block::error[0] = 0; emu_block::steps = 0;
  DevResult res;
  memset((void*)&res, 0, sizeof res);
  res.ok = 1;
  WTileArgs& a = g_args;
  memset((void*)&a, 0, sizeof a);
  g_schema = schema;
  a.w.n = schema == PJ_SCHEMA_MIXED ? cols->n_records : cols->n_rows[schema];
  a.w.schema = schema; a.w.array = array; a.w.inclusion = inclusion; a.w.hexa = lower ? 'a' : 'A';
  a.w.out = out; a.w.cap = cap; a.w.res = &res;
  for (int i = 0; i < PJ_MAX_COLS; ++i) a.w.cols.ptr[i] = cols->col[i].ptr;
  Schema S;
  build_schema(&S);
  wt_columns(S, schema, a.w.cols, &a);
  a.recs = recs; a.smem = shared; a.spin_limit_ns = 1;
  a.ntiles = a.w.n ? (uint32_t)((a.w.n + recs - 1) / recs) : 1u;
  std::vector<unsigned long long> state(2 * (size_t)a.ntiles, 0);
  uint32_t ticket = 0;
  a.ticket = &ticket; a.agg = state.data(); a.inc = state.data() + a.ntiles;
  bool fine = true;
  for (uint32_t t = 0; t < a.ntiles && fine; ++t) {
    memset(smem, 0xC3, shared);
    EMU_POISON(smem + shared, sizeof smem - shared);
    fine = emu_block::run(g_short && schema == PJ_SCHEMA_PET ? WT_SHORT_THREADS : wt_threads(schema), one_thread, nullptr, order + t);
    EMU_UNPOISON(smem + shared, sizeof smem - shared);
  }
  if (fine && res.timeout) { snprintf(emu_block::error, sizeof emu_block::error, "a bounded wait ran out"); fine = false; }
  if (!fine) return -1;
  *out_len = res.out_bytes;
  return res.ok ? 0 : 1;
}
/* Columns of a stream of several models, as the tiles stage them and as the limits count them: with an element per row, others, the same two. */
extern "C" void emu_write_columns(uint32_t* out) {
  Schema S;
  build_schema(&S);
  WTileArgs a;
  memset((void*)&a, 0, sizeof a);
  wt_columns(S, PJ_SCHEMA_MIXED, a.w.cols, &a);
  out[0] = a.nrow; out[1] = a.ncol - a.nrow; out[2] = WT_ROW_COLS; out[3] = WT_OTHER_COLS;
}
extern "C" void emu_write_shape(uint64_t n, const uint64_t* rows, uint64_t arena, uint64_t strs, uint64_t objs, uint32_t* out) {
  WriteShapeIn in{n, {rows[0], rows[1], rows[2]}, arena, strs, objs, 148};
  const WriteShape s = write_shape(in, WT_MAX_RECS, WT_MAX_SMEM);
  out[0] = s.recs; out[1] = s.smem;
}

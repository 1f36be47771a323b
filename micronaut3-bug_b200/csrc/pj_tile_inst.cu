/*
 * pj_tile_inst.cu — one instantiation of the parse kernel, compiled once per model set with -DPJ_TILE_SCHEMA=1..4 (Pet,
 * Order, User, mixed) so that the four build in parallel. Each object carries its own copy of the constant model
 * tables, set by its init function.
 */
#include <cuda_runtime.h>

#include "petjson.h"
#include "pj_item.cuh"

#ifndef PJ_TILE_SCHEMA
#error "compile with -DPJ_TILE_SCHEMA=<PJ_SCHEMA_* value>"
#endif
#define PJ_CAT2(a, b) a##b
#define PJ_CAT(a, b) PJ_CAT2(a, b)

namespace pj {

cudaError_t PJ_CAT(item_init_, PJ_TILE_SCHEMA)(const Schema* s) {
  cudaError_t e = cudaFuncSetAttribute(k_parse_items<PJ_TILE_SCHEMA>, cudaFuncAttributeMaxDynamicSharedMemorySize, IT_MAX_DYN_SMEM);
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_schema, s, sizeof(Schema));
  return e;
}
cudaError_t PJ_CAT(item_launch_, PJ_TILE_SCHEMA)(const ItemArgs* a, cudaStream_t stream) {
  const ItemLayout l = item_layout(a->win_bytes, a->str_words, a->row_cap, ItStride<PJ_TILE_SCHEMA>::n);
  k_parse_items<PJ_TILE_SCHEMA><<<a->ntiles, IT_THREADS, l.total, stream>>>(*a);
  return cudaGetLastError();
}

}  // namespace pj

/*
 * pj_stream_inst.cu — one instantiation of k_parse_stream (a record per thread), compiled once per model set with
 * -DPJ_TILE_SCHEMA=1..4 like pj_tile_inst.cu. Each object carries its own copy of the constant model tables.
 */
#include <cuda_runtime.h>

#include "petjson.h"
#include "pj_kernels.cuh"
#include "pj_stream_kernel.cuh"

#ifndef PJ_TILE_SCHEMA
#error "compile with -DPJ_TILE_SCHEMA=<PJ_SCHEMA_* value>"
#endif
#define PJ_CAT2(a, b) a##b
#define PJ_CAT(a, b) PJ_CAT2(a, b)

namespace pj {

cudaError_t PJ_CAT(stream_init_, PJ_TILE_SCHEMA)(const Schema* s) {
  cudaError_t e = cudaFuncSetAttribute(k_parse_stream<PJ_TILE_SCHEMA>, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_SMEM_BYTES);
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_schema, s, sizeof(Schema));
  return e;
}
cudaError_t PJ_CAT(stream_launch_, PJ_TILE_SCHEMA)(const StreamArgs* a, unsigned grid, cudaStream_t stream) {
  k_parse_stream<PJ_TILE_SCHEMA><<<grid, ST_THREADS, ST_SMEM_BYTES, stream>>>(*a);
  return cudaGetLastError();
}

}  // namespace pj

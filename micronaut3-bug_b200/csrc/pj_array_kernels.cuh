/*
 * pj_array_kernels.cuh — the record index of array framing on its own (pj_index_records), behind the separators of k_arr_index.
 *
 *   k_arr_records<>   one candidate per separator: extent, blank test, keep / drop; count per tile, then (after a scan) store rec_start
 */
#ifndef PJ_ARRAY_KERNELS_CUH
#define PJ_ARRAY_KERNELS_CUH

#include "pj_array.cuh"
#include "pj_array_index.cuh"
#include "pj_kernels.cuh"

namespace pj {

static constexpr int ARR_THREADS = 256; /* words per block: one block covers 16 KiB, like the NDJSON index */

struct ArrArgs {
  const uint8_t* in;
  uint64_t len, nwords;
  const uint64_t* sep; /* [nwords] separator bitmap */
  uint32_t* tile_cnt;  /* [tiles + 1] */
  uint64_t* rec_start; /* outputs of k_arr_records<true> */
  uint64_t cap, goff;
  DevResult* res;
};

template <bool WRITE>
__global__ void __launch_bounds__(ARR_THREADS) k_arr_records(const __grid_constant__ ArrArgs a) {
  __shared__ uint32_t sh[33];
  const uint64_t w = (uint64_t)blockIdx.x * ARR_THREADS + threadIdx.x;
  const unsigned long long first_opener = a.res->first_opener;
  uint64_t seps = w < a.nwords ? a.sep[w] : 0;
  uint32_t cnt = 0;
  for (uint64_t t = seps; t; t &= t - 1) {
    const uint64_t p = (w << 6) + ctz64a(t);
    const ExtentOut x = arr_extent(a.in, a.len, a.sep, p, first_opener);
    if (!WRITE && x.second_opener) atomicMin(&a.res->doc_err_off, (unsigned long long)p);
    cnt += x.is_record;
  }
  uint32_t total;
  const uint32_t ex = block_excl_scan(cnt, &total, sh);
  if (!WRITE) {
    if (threadIdx.x == 0) a.tile_cnt[blockIdx.x] = total;
    return;
  }
  uint64_t at = (uint64_t)a.tile_cnt[blockIdx.x] + ex;
  for (uint64_t t = seps; t; t &= t - 1) {
    const uint64_t p = (w << 6) + ctz64a(t);
    const ExtentOut x = arr_extent(a.in, a.len, a.sep, p, first_opener);
    if (!x.is_record) continue;
    if (at < a.cap) {
      a.rec_start[at] = x.start + a.goff;
    }
    at++;
  }
}

}  // namespace pj
#endif

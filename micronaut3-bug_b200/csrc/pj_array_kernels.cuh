/*
 * pj_array_kernels.cuh — the record index of array framing on its own (pj_index_records), behind the separators of k_arr_index.
 *
 *   k_arr_records   one candidate per separator: extent, blank test, keep / drop; a tile's place by look-back, then rec_start
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
  uint64_t* rec_start;
  uint64_t cap, goff;
  DevResult* res;
};

static __global__ void __launch_bounds__(ARR_THREADS) k_arr_records(const __grid_constant__ ArrArgs a, const __grid_constant__ RecordTiles t) {
  __shared__ uint32_t sh[33], sh_tile;
  __shared__ unsigned long long sh_before[2];
  if (threadIdx.x == 0) sh_tile = atomicAdd(t.ticket, 1u);
  __syncthreads();
  const uint32_t tile = sh_tile;
  if (tile >= t.ntiles) return;
  const uint64_t w = (uint64_t)tile * ARR_THREADS + threadIdx.x;
  const unsigned long long first_opener = a.res->first_opener;
  uint64_t keep = w < a.nwords ? a.sep[w] : 0;
  for (uint64_t m = keep; m; m &= m - 1) {
    const uint64_t p = (w << 6) + ctz64a(m);
    const ExtentOut x = arr_extent(a.in, a.len, a.sep, p, first_opener);
    if (x.second_opener) atomicMin(&a.res->doc_err_off, (unsigned long long)p);
    if (!x.is_record) keep &= ~(m & (0ull - m));
  }
  uint32_t total;
  const uint32_t mine = block_excl_scan((uint32_t)popc64(keep), &total, sh);
  unsigned long long at;
  if (!records_before(t, tile, total, &at, sh_before)) return;
  at += mine;
  for (uint64_t m = keep; m; m &= m - 1, ++at)
    if (at < a.cap) a.rec_start[at] = (w << 6) + ctz64a(m) + 1u + a.goff; /* an extent begins behind its separator */
}

}  // namespace pj
#endif

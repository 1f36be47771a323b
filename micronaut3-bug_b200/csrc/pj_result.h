/*
 * pj_result.h — the block of counters and flags the kernels leave for the host.
 */
#ifndef PJ_RESULT_H
#define PJ_RESULT_H

#include "pj_schema.h"

namespace pj {

/* Written by the kernels, read back by the host once per call. */
struct DevResult {
  unsigned long long n_records;
  unsigned long long n_errors;
  unsigned long long total[NSLOT];
  unsigned long long out_bytes; /* writer: JSON bytes */
  unsigned long long doc_err_off;
  uint32_t doc_err_kind;
  uint32_t ok;      /* every output fits its buffer */
  uint32_t over;    /* stream kernel: some output does not fit its buffer */
  uint32_t timeout; /* a bounded wait ran out */
  uint32_t aside;   /* k_parse_items: left to k_parse_stream, nothing done */
  unsigned long long n_fast;  /* records decoded by the speculative pass alone; k_parse_stream: low half, in the high half those its warps took in step */
  unsigned long long phase_cycles[4]; /* tile kernel, summed over blocks: staging, tokenising, look-back, emit */
  unsigned long long lookback_polls, lookback_rounds;
  unsigned long long n_wide;       /* records walked by a whole warp */
  unsigned long long n_wide_fast;  /* of those, finished by the word-at-a-time tokeniser (the rest: the exact parser) */
  unsigned long long wide_cycles[2]; /* cycles the blocks spent in the warps' size pass / emit pass, summed over blocks */
  unsigned long long n_dense; /* k_parse_items: lines that hold no blank between tokens and no null */
  uint32_t max_rec;  /* bytes of the longest record, as far as the tiles saw its end */
  uint32_t strs_per_kb; /* k_parse_items: strings per 1024 bytes, of the tile with the most */
  unsigned long long first_opener; /* array framing: offset of the first `[` at depth 0 */
  uint32_t arr_final_s;            /* array framing: the input ends inside a string */
  int32_t arr_final_d;             /* array framing: nesting depth at the end of the input */
};

}  // namespace pj
#endif

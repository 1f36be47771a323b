/*
 * pj_kernels.cuh — sm_100a kernels of the record index, the writer and the checksums.
 *
 * JSON is parsed by k_parse_stream (pj_stream_kernel.cuh) and k_parse_items (pj_item.cuh), which build their own line index. This
 * header holds
 *   - the NDJSON record index on its own: k_nd_records (pj_index_records), and k_nd_index<false> / k_scan_single / k_nd_index<true> (the
 *     same for inputs that L2 holds, and its allocation-free variant);
 *   - what runs before and behind a call's kernels: k_reset, k_fetch, and k_write_close behind the writer's tiles (pj_write_tile.cuh);
 *   - the checksums of columns.
 *
 * Kernels that wait on other blocks (the look-backs) take their tile from an atomic ticket, so every block they
 * wait for is running or done, and every wait is bounded (the spin limit of the kernel's arguments ->
 * DevResult.timeout -> PJ_ERR_TIMEOUT).
 */
#ifndef PJ_KERNELS_CUH
#define PJ_KERNELS_CUH

#if defined(__CUDACC__)
#include <cuda_runtime.h>
#endif
#include <stddef.h>

#include "pj_core.cuh"
#include "pj_dev.cuh"
#include "pj_fast.cuh"
#include "pj_index.cuh"
#include "pj_result.h"
#include "pj_write_tile.cuh"

namespace pj {

static constexpr int INDEX_THREADS = 256;
static constexpr int INDEX_BYTES_PER_THREAD = 64;
static constexpr int INDEX_TILE = INDEX_THREADS * INDEX_BYTES_PER_THREAD; /* 16 KiB */

/* ---- NDJSON record index ---------------------------------------------------------------------- */
/* 64-bit mask of the LF bytes among the 64 bytes at the 16-byte aligned address a, of which the
 * first `valid` (>= 1) belong to the input. */
__device__ __forceinline__ uint64_t lf_mask64(const uint8_t* a, uint64_t valid) {
  const uint4* q = reinterpret_cast<const uint4*>(a);
  uint64_t m = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if ((uint64_t)(k * 16) >= valid) break; /* never touch a 16-byte block that holds no input byte */
    uint4 v = __ldg(q + k);
    uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t e = __vcmpeq4(w[j], 0x0A0A0A0Au) & 0x01010101u; /* 1 per matching byte */
      uint32_t nib = (e * 0x01020408u) >> 24;                  /* gather the four flags */
      m |= (uint64_t)(nib & 0xF) << (k * 16 + j * 4);
    }
  }
  return m;
}

struct IndexArgs {
  const uint8_t* in;
  uint64_t len, limit;
  int is_first, is_last;
  uint32_t* tile; /* [tiles + 1]: counts, then (after the scan) exclusive bases */
  uint64_t* rec_start;
  uint64_t cap, goff;
};

/* One thread looks at 64 input bytes. Every LF inside [0, len) makes the following byte a candidate
 * line start; byte 0 is one too when the shard is the first of its stream. WRITE = false counts the
 * candidates that are records per tile; WRITE = true stores their offsets at the scanned positions. */
template <bool WRITE>
__global__ void __launch_bounds__(INDEX_THREADS) k_nd_index(const __grid_constant__ IndexArgs a) {
  __shared__ uint32_t sh[33];
  const uint32_t mis = (uint32_t)(reinterpret_cast<uintptr_t>(a.in) & 15u);
  const uint8_t* base = a.in - mis; /* 16-byte aligned */
  const uint64_t v0 = (uint64_t)blockIdx.x * INDEX_TILE + (uint64_t)threadIdx.x * INDEX_BYTES_PER_THREAD; /* offset from base */
  const uint64_t vend = a.len ? a.len + mis : 0; /* an empty input is never dereferenced */
  uint64_t m = 0;
  if (v0 < vend) {
    m = lf_mask64(base + v0, vend - v0);
    if (v0 < mis) m &= ~0ull << (mis - v0);               /* bytes before in[0] */
    if (vend - v0 < 64) m &= ~(~0ull << (vend - v0));      /* bytes at or after in[len] */
  }
  const bool head = a.is_first && blockIdx.x == 0 && threadIdx.x == 0; /* candidate at byte 0 */
  uint32_t cnt = 0;
  if (!WRITE) {
    if (head && nd_is_record(a.in, 0, a.limit, a.is_last)) cnt++;
    for (uint64_t t = m; t; t &= t - 1) {
      uint64_t p = v0 + (uint64_t)(__ffsll((long long)t) - 1) - mis + 1;
      if (nd_is_record(a.in, p, a.limit, a.is_last)) cnt++;
    }
    uint32_t total;
    block_excl_scan(cnt, &total, sh);
    if (threadIdx.x == 0) a.tile[blockIdx.x] = total;
  } else {
    /* recount, then place */
    uint64_t keep = 0;
    bool head_keep = head && nd_is_record(a.in, 0, a.limit, a.is_last);
    cnt = head_keep ? 1u : 0u;
    for (uint64_t t = m; t; t &= t - 1) {
      int b = __ffsll((long long)t) - 1;
      uint64_t p = v0 + (uint64_t)b - mis + 1;
      if (nd_is_record(a.in, p, a.limit, a.is_last)) { keep |= 1ull << b; cnt++; }
    }
    uint32_t total;
    uint64_t at = (uint64_t)a.tile[blockIdx.x] + block_excl_scan(cnt, &total, sh);
    if (head_keep) { if (at < a.cap) a.rec_start[at] = a.goff; at++; }
    for (uint64_t t = keep; t; t &= t - 1) {
      uint64_t p = v0 + (uint64_t)(__ffsll((long long)t) - 1) - mis + 1;
      if (at < a.cap) a.rec_start[at] = p + a.goff;
      at++;
    }
  }
}

/* What a tile's position among the records needs: its number, and the totals of the tiles before it. */
struct RecordTiles {
  uint32_t* ticket;
  unsigned long long *agg, *inc; /* [ntiles] records of the tile / up to and including it | TS_VALID */
  uint32_t ntiles;
  unsigned long long spin_limit_ns;
  DevResult* res;
};
/* Records of the tiles before `tile`, which has `total`; the last tile leaves them all. Every thread of the block calls it; false when a bounded
 * wait ran out. sh: two words. */
__device__ __forceinline__ bool records_before(const RecordTiles& t, uint32_t tile, uint32_t total, unsigned long long* before, unsigned long long* sh) {
  if (threadIdx.x < 32u) {
    const uint32_t lane = threadIdx.x;
    if (lane == 0) {
      st_relaxed_u64(&t.agg[tile], TS_VALID | total);
      if (tile == 0) st_relaxed_u64(&t.inc[tile], TS_VALID | total);
    }
    unsigned long long excl = 0;
    const bool ok = lookback_u64(t.agg, t.inc, &t.res->timeout, t.spin_limit_ns, tile, lane, &excl);
    if (lane == 0) {
      if (tile && ok) st_relaxed_u64(&t.inc[tile], TS_VALID | (excl + total));
      if (tile == t.ntiles - 1u) t.res->n_records = excl + total;
      sh[0] = excl; sh[1] = ok;
    }
  }
  __syncthreads();
  *before = sh[0];
  return sh[1] != 0;
}
/* The NDJSON record index in one pass: W words of 64 bytes per thread, a tile's place by look-back. (In two passes and
 * three launches: 1000 Pets 38 -> 31 us a call; 1 M Pets 157 -> 147, where the look-back takes a third.)
 * k_nd_index stays for inputs that it reads from L2 the second time, and for callers without memory for the tiles' states. */
template <int W>
__global__ void __launch_bounds__(INDEX_THREADS) k_nd_records(const __grid_constant__ IndexArgs a, const __grid_constant__ RecordTiles t) {
  __shared__ uint32_t sh[33], sh_tile;
  __shared__ unsigned long long sh_before[2];
  if (threadIdx.x == 0) sh_tile = atomicAdd(t.ticket, 1u);
  __syncthreads();
  const uint32_t tile = sh_tile;
  if (tile >= t.ntiles) return;
  const uint32_t mis = (uint32_t)(reinterpret_cast<uintptr_t>(a.in) & 15u);
  const uint8_t* base = a.in - mis; /* 16-byte aligned */
  const uint64_t v0 = ((uint64_t)tile * INDEX_THREADS + threadIdx.x) * (64u * W), vend = a.len ? a.len + mis : 0; /* an empty input is never dereferenced */
  const bool head = a.is_first && tile == 0 && threadIdx.x == 0 && nd_is_record(a.in, 0, a.limit, a.is_last); /* byte 0 begins a line, too */
  uint64_t keep[W];
  uint32_t cnt = head ? 1u : 0u;
#pragma unroll
  for (int k = 0; k < W; ++k) keep[k] = v0 + 64u * k < vend ? lf_mask64(base + v0 + 64u * k, vend - v0 - 64u * k) : 0ull;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    const uint64_t v = v0 + 64u * k;
    if (v < mis) keep[k] &= ~0ull << (mis - v);                        /* bytes before in[0] */
    if (v < vend && vend - v < 64) keep[k] &= ~(~0ull << (vend - v)); /* bytes at or after in[len] */
    for (uint64_t m = keep[k]; m; m &= m - 1u) {
      const uint64_t bit = m & (0ull - m);
      const uint32_t b = (uint32_t)__ffsll((long long)m); /* behind the line feed */
      if (b < 64u && v + b < vend && base[v + b] > ' ') { cnt++; continue; }
      if (nd_is_record(a.in, v + (uint64_t)(__ffsll((long long)m) - 1) - mis + 1, a.limit, a.is_last)) cnt++; else keep[k] &= ~bit;
    }
  }
  uint32_t total;
  const uint32_t mine = block_excl_scan(cnt, &total, sh);
  unsigned long long at;
  if (!records_before(t, tile, total, &at, sh_before)) return;
  at += mine;
  if (head) { if (at < a.cap) a.rec_start[at] = a.goff; at++; }
#pragma unroll
  for (int k = 0; k < W; ++k)
    for (uint64_t m = keep[k]; m; m &= m - 1u, ++at)
      if (at < a.cap) a.rec_start[at] = v0 + 64u * k + (uint64_t)(__ffsll((long long)m) - 1) - mis + 1 + a.goff;
}

/* ---- scans over device-resident lengths -------------------------------------------------------- */
/* Single block: exclusive scan of data[0..n) in place, data[n] = total; also *total_out. */
template <class T>
__global__ void __launch_bounds__(1024) k_scan_single(T* data, uint64_t n, unsigned long long* total_out) {
  __shared__ T sh[33];
  T carry = 0;
  for (uint64_t b = 0; b < n; b += blockDim.x) {
    uint64_t i = b + threadIdx.x;
    T v = i < n ? data[i] : T(0), tot;
    T ex = block_excl_scan(v, &tot, sh);
    if (i < n) data[i] = carry + ex;
    carry += tot;
  }
  if (threadIdx.x == 0) { data[n] = carry; if (total_out) *total_out = (unsigned long long)carry; }
}

/* ---- the state of a call --------------------------------------------------------------------------------------------- */
struct ResetArgs {
  unsigned long long *state, *more; /* tickets, look-back words; a bitmap that is or-ed into (or null) */
  uint64_t words, more_words;
  DevResult* res;
  const uint8_t* in; /* the input and where the line feeds in pieces of it go (or null), see nd_look_at() */
  uint64_t len;
  uint32_t* looks;
};
/* line feeds of piece k; a block of ND_LOOK_BYTES / 16 threads */
__device__ __forceinline__ uint32_t nd_look(const uint8_t* in, uint64_t len, uint32_t k, uint32_t* sh) {
  const uint8_t* p = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(in + nd_look_at(len, k)) & ~(uintptr_t)15) + 16u * threadIdx.x;
  uint32_t n = 0;
  if (p >= in && p + 16 <= in + len) n = (uint32_t)__popcll(lf_mask64(p, 16));
  if (threadIdx.x == 0) *sh = 0;
  __syncthreads();
  if (n) atomicAdd(sh, n);
  __syncthreads();
  return *sh;
}
/* no ticket taken, no tile's totals known, nothing counted */
static __global__ void __launch_bounds__(256) k_reset(const __grid_constant__ ResetArgs a) {
  const uint64_t first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t k = first; k < a.words; k += step) a.state[k] = 0;
  for (uint64_t k = first; k < a.more_words; k += step) a.more[k] = 0;
  if (blockIdx.x == 0) {
    uint32_t* r = reinterpret_cast<uint32_t*>(a.res);
    for (uint32_t k = threadIdx.x; k < sizeof(DevResult) / 4; k += blockDim.x) {
      const uint32_t at = 4u * k;
      const bool none = at - (uint32_t)offsetof(DevResult, doc_err_off) < 8u || at - (uint32_t)offsetof(DevResult, first_opener) < 8u; /* running minima */
      r[k] = none ? 0xFFFFFFFFu : (at == offsetof(DevResult, ok) ? 1u : 0u);
    }
  }
  if (a.looks && blockIdx.x < ND_LOOKS) {
    __shared__ uint32_t sh;
    const uint32_t n = nd_look(a.in, a.len, blockIdx.x, &sh);
    if (threadIdx.x == 0) a.looks[blockIdx.x] = n;
  }
}
static_assert(ND_LOOK_BYTES == 16 * 256, "16 bytes a thread");
/* closes the text: brackets of array framing, the total, the verdict; the result goes to host memory (one warp) */
static __global__ void k_write_close(const __grid_constant__ WriteArgs a, DevResult* host) {
  if (threadIdx.x == 0) {
    const uint64_t body = a.res->out_bytes;
    const uint64_t total = a.array ? (body ? body + 1 : 2) : body;
    a.res->out_bytes = total;
    const bool ok = a.res->ok && total <= a.cap;
    a.res->ok = ok;
    if (a.array && ok) { a.out[0] = '['; a.out[total - 1] = ']'; }
  }
  __syncwarp();
  for (uint32_t k = threadIdx.x; k < sizeof(DevResult) / 4; k += 32u) reinterpret_cast<uint32_t*>(host)[k] = reinterpret_cast<const uint32_t*>(a.res)[k];
}

/* ---- what a small call gives back ------------------------------------------------------------------------------------- */
/* The result block, and columns or text, to host memory the device writes to: one launch behind the call's last kernel instead of a copy per
 * column that waits for the totals first. (20 Pets from host memory and back: 17 copies and two waits, 308 us; 80 with it. Up to 1 MB: beyond, the
 * copies' bytes take longer than their number.) */
struct FetchCol { const uint8_t* p; uint8_t shift, slot, plus, pad[5]; }; /* slot: the total that counts its elements (plus more); FETCH_* */
enum { FETCH_RECORDS = 0xFF, FETCH_TEXT = 0xFE };
static constexpr uint64_t FETCH_ROOM = 1u << 20; /* bytes */
struct FetchArgs {
  const DevResult* res;
  DevResult* host_res;
  uint8_t* host; /* FETCH_ROOM bytes */
  uint32_t n;    /* columns */
  FetchCol col[PJ_MAX_COLS];
};
PJ_HD uint64_t fetch_bytes(const FetchCol& c, const DevResult& r) {
  return ((c.slot == FETCH_RECORDS ? r.n_records : (c.slot == FETCH_TEXT ? r.out_bytes : r.total[c.slot])) + c.plus) << c.shift;
}
/* does everything fit? (decided alike on both sides) */
PJ_HD uint64_t fetch_place(uint64_t at, uint64_t bytes) { return at + ((bytes + 15u) & ~15ull); }
static __global__ void __launch_bounds__(256) k_fetch(const __grid_constant__ FetchArgs a) {
  __shared__ uint64_t sh_at[PJ_MAX_COLS + 1];
  const uint32_t tid = threadIdx.x;
  if (blockIdx.x == 0)
    for (uint32_t k = tid; k < sizeof(DevResult) / 4; k += 256u) reinterpret_cast<uint32_t*>(a.host_res)[k] = reinterpret_cast<const uint32_t*>(a.res)[k];
  if (a.n == 0) return;
  if (tid < a.n) sh_at[tid] = fetch_bytes(a.col[tid], *a.res);
  __syncthreads();
  uint64_t at = 0;
  for (uint32_t k = 0; k < a.n && at <= FETCH_ROOM; ++k) at = fetch_place(at, sh_at[k]);
  if (at > FETCH_ROOM || a.res->timeout || a.res->over || !a.res->ok) return;
  at = 0;
  for (uint32_t k = 0; k < a.n; ++k) { /* (staged columns and text start at 256-byte multiples, and their room ends at one) */
    const uint64_t blocks = (sh_at[k] + 15u) >> 4;
    const uint4* src = reinterpret_cast<const uint4*>(a.col[k].p);
    uint4* dst = reinterpret_cast<uint4*>(a.host + at);
    for (uint64_t b = (uint64_t)blockIdx.x * 256u + tid; b < blocks; b += (uint64_t)gridDim.x * 256u) dst[b] = src[b];
    at = fetch_place(at, sh_at[k]);
  }
}

/* ---- column checksums --------------------------------------------------------------------------------- */
PJ_HD uint64_t checksum_mix(uint64_t x) {
  x ^= x >> 30; x *= 0xBF58476D1CE4E5B9ull;
  x ^= x >> 27; x *= 0x94D049BB133111EBull;
  x ^= x >> 31;
  return x;
}
PJ_HD uint64_t checksum_term(uint64_t word, uint64_t j) { return checksum_mix(word + 0x9E3779B97F4A7C15ull * (j + 1)); }
struct ChecksumArgs {
  const uint8_t* p[PJ_MAX_COLS];
  uint64_t n[PJ_MAX_COLS]; /* bytes */
  unsigned long long* out; /* [PJ_MAX_COLS], zeroed */
};
/* blockIdx.y = column; the blocks of a column stride over its 8-byte words */
static __global__ void __launch_bounds__(256) k_checksum(const __grid_constant__ ChecksumArgs a) {
  const uint32_t col = blockIdx.y;
  const uint8_t* p = a.p[col];
  const uint64_t n = a.n[col];
  const uint64_t nwords = (n + 7) / 8;
  const bool aligned = (reinterpret_cast<uintptr_t>(p) & 7u) == 0;
  unsigned long long s = 0;
  for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < nwords; j += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t w = 0;
    if (aligned && 8 * j + 8 <= n) w = *reinterpret_cast<const uint64_t*>(p + 8 * j);
    else for (uint32_t b = 0; b < 8 && 8 * j + b < n; ++b) w |= (uint64_t)p[8 * j + b] << (8 * b);
    s += checksum_term(w, j);
  }
  for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, d);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(&a.out[col], s);
}

}  // namespace pj
#endif

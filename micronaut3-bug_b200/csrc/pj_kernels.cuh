/*
 * pj_kernels.cuh — sm_100a kernels of the record index, the writer and the checksums.
 *
 * JSON is parsed by k_parse_stream (pj_stream_kernel.cuh) and k_parse_items (pj_item.cuh), which build their own line index. This
 * header holds
 *   - the NDJSON record index on its own (k_nd_index<false> / k_scan_single / k_nd_index<true>: pj_index_records and
 *     its allocation-free variant);
 *   - the writer: columns --k_arena_flags--> "any byte to escape?" --k_write_tile--> text --k_write_close--> brackets, total.
 *
 * Kernels that wait on other blocks (the look-backs) take their tile from an atomic ticket, so every block they
 * wait for is running or done, and every wait is bounded (the spin limit of the kernel's arguments ->
 * DevResult.timeout -> PJ_ERR_TIMEOUT).
 */
#ifndef PJ_KERNELS_CUH
#define PJ_KERNELS_CUH

#include <cuda_runtime.h>

#include "pj_core.cuh"
#include "pj_dev.cuh"
#include "pj_fast.cuh"
#include "pj_index.cuh"
#include "pj_result.h"
#include "pj_write_core.cuh"
#include "pj_write_fast.cuh"

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

/* ---- writer arguments ------------------------------------------------------------------------- */
struct WriteArgs {
  uint64_t n;             /* records (mixed) or rows */
  uint32_t schema, array; /* array: wrap as [r,r,...] */
  int inclusion;
  uint32_t hexa;          /* 'A' or 'a': hex letters of \u00xx escapes */
  uint8_t* out;
  uint64_t cap;
  DevResult* res;
  DevCols cols;
};


/* ================================================================================================
 * Single-pass tile writer (columns -> JSON text)
 *
 * One block takes TILE_THREADS consecutive records. Every thread measures its record (size pass of
 * pj_write_fast.cuh), the lengths are scanned inside the block, the tile's start in the output comes
 * from a decoupled look-back over the tiles before it (one 64-bit running total; the protocol of the
 * parse kernel), every thread then writes its record into a window in shared memory, and the block
 * copies the window to the output with 16-byte stores. A tile whose text does not fit the window is
 * written to global memory directly. Text is produced once and written to HBM once.
 * ================================================================================================ */
#ifndef PJ_WT_THREADS
#define PJ_WT_THREADS 128 /* records (= threads) per writer tile */
#endif
#ifndef PJ_WT_WIN_KB
#define PJ_WT_WIN_KB 40 /* text window per tile in shared memory */
#endif
#ifndef PJ_WT_BLOCKS
#define PJ_WT_BLOCKS 5 /* resident blocks per SM the kernel is compiled for */
#endif
static constexpr uint32_t WT_THREADS = PJ_WT_THREADS;
static_assert(WT_THREADS % 32 == 0 && WT_THREADS >= 96, "the copy-out of the window's odd ends uses threads 32.. and 64..");
static constexpr uint32_t WTILE_WIN_BYTES = PJ_WT_WIN_KB * 1024;
static constexpr uint32_t WTILE_SMEM_BYTES = WTILE_WIN_BYTES + 32;

struct WTileArgs {
  WriteArgs w;
  unsigned long long* agg; /* [ntiles] text bytes of the tile | TS_VALID */
  unsigned long long* inc; /* [ntiles] text bytes of all tiles up to and including it | TS_VALID */
  uint32_t* ticket;
  uint32_t ntiles;
  unsigned long long spin_limit_ns;
};

/* Exclusive prefix of `tile` over all earlier tiles. Warp 0 only, all lanes; false when the bounded wait ran out. */
__device__ __forceinline__ bool lookback_u64(const unsigned long long* agg, const unsigned long long* inc, uint32_t* timeout_flag, unsigned long long limit_ns,
                                             uint32_t tile, uint32_t lane, unsigned long long* excl_out) {
  unsigned long long excl = 0;
  int64_t j = (int64_t)tile - 1;
  const unsigned long long t0 = global_ns();
  while (j >= 0) {
    const int64_t mine = j - lane;
    unsigned long long wa, wi;
    uint32_t first_inc;
    for (;;) {
      wa = TS_VALID; wi = TS_VALID; /* tiles before the first: inclusive total 0 */
      if (mine >= 0) { wi = ld_relaxed_u64(&inc[mine]); wa = ld_relaxed_u64(&agg[mine]); }
      const bool has_inc = wi & TS_VALID, has_agg = wa & TS_VALID;
      const uint32_t inc_mask = __ballot_sync(0xFFFFFFFFu, has_inc);
      const uint32_t ready_mask = __ballot_sync(0xFFFFFFFFu, has_inc || has_agg);
      first_inc = inc_mask ? (uint32_t)(__ffs((int)inc_mask) - 1) : 32u;
      const uint32_t need = first_inc >= 31 ? 0xFFFFFFFFu : ((2u << first_inc) - 1u);
      if ((ready_mask & need) == need) break;
      uint32_t give_up = 0;
      if (lane == 0) give_up = (global_ns() - t0 > limit_ns) || *(volatile uint32_t*)timeout_flag;
      give_up = __shfl_sync(0xFFFFFFFFu, give_up, 0);
      if (give_up) { if (lane == 0) atomicExch(timeout_flag, 1u); return false; }
      __nanosleep(100);
    }
    unsigned long long c = lane < first_inc ? (wa & ~TS_VALID) : (lane == first_inc ? (wi & ~TS_VALID) : 0ull);
#pragma unroll
    for (int d = 16; d; d >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, d);
    excl += c;
    if (first_inc < 32) break;
    j -= 32;
  }
  *excl_out = excl;
  return true;
}

/* Does any byte of the string arenas need a JSON escape (below 0x20, '"', '\\')? Text is mostly free of
 * them, and knowing so lets the tile writer take string lengths from the offset columns alone. */
struct ArenaArgs {
  const uint8_t* p[12];
  uint64_t n[12];
  uint32_t count;
  DevResult* res;
};
__device__ __forceinline__ uint32_t word_needs_escape(uint32_t x) {
  const uint32_t xq = x ^ 0x22222222u, xb = x ^ 0x5C5C5C5Cu;
  return (((x - 0x20202020u) & ~x) | ((xq - 0x01010101u) & ~xq) | ((xb - 0x01010101u) & ~xb)) & 0x80808080u;
}
static __global__ void __launch_bounds__(256) k_arena_flags(const __grid_constant__ ArenaArgs a) {
  const uint64_t gtid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, gsize = (uint64_t)gridDim.x * blockDim.x;
  uint32_t any = 0;
  for (uint32_t r = 0; r < a.count; ++r) {
    const uint8_t* p = a.p[r];
    const uint64_t n = a.n[r];
    uint64_t head = (16 - (reinterpret_cast<uintptr_t>(p) & 15u)) & 15u;
    if (head > n) head = n;
    const uint64_t nvec = (n - head) >> 4, tail = head + (nvec << 4);
    const uint4* v = reinterpret_cast<const uint4*>(p + head);
    for (uint64_t k = gtid; k < nvec; k += gsize) {
      const uint4 x = __ldg(v + k);
      any |= word_needs_escape(x.x) | word_needs_escape(x.y) | word_needs_escape(x.z) | word_needs_escape(x.w);
    }
    if (gtid < head) any |= escape_extra_byte(p[gtid]);
    if (gtid < n - tail) any |= escape_extra_byte(p[tail + gtid]);
  }
  if (__syncthreads_or((int)any) && threadIdx.x == 0) a.res->needs_escape = 1u;
}

/* The writer is bound by the latency of its column loads (one dependent chain per property). Asking for all the
 * row-indexed values of a record at once, before the first is needed, lets those latencies overlap. */
__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
template <int OBJ, int I = 0>
__device__ __forceinline__ void prefetch_row(const DevCols* c, uint64_t row) {
  if constexpr (I == 0) prefetch_l1(colp<uint8_t>(c, CObj<OBJ>::present_col) + row);
  if constexpr (I < CObj<OBJ>::N) {
    constexpr uint32_t kind = FK<OBJ, I>::kind, col = FK<OBJ, I>::col;
    if constexpr (kind == K_I64) prefetch_l1(colp<int64_t>(c, col) + row);
    else if constexpr (kind == K_I32) prefetch_l1(colp<int32_t>(c, col) + row);
    else if constexpr (kind == K_BOOL || kind == K_ENUM) prefetch_l1(colp<uint8_t>(c, col) + row);
    else if constexpr (kind == K_DATETIME) { prefetch_l1(colp<int64_t>(c, col) + row); prefetch_l1(colp<int32_t>(c, col + 1) + row); prefetch_l1(colp<int32_t>(c, col + 2) + row); }
    else if constexpr (kind == K_STR || kind == K_LIST_STR || kind == K_LIST_OBJ) prefetch_l1(colp<uint32_t>(c, col) + row + 1);
    else if constexpr (kind == K_OBJ) prefetch_row<FK<OBJ, I>::child>(c, row);
    prefetch_row<OBJ, I + 1>(c, row);
  }
}

static __global__ void __launch_bounds__(WT_THREADS, PJ_WT_BLOCKS) k_write_tile(const __grid_constant__ WTileArgs a) {
  constexpr uint32_t NWARPS = WT_THREADS / 32;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ uint32_t sh_warp[NWARPS];
  __shared__ uint32_t sh_tile, sh_ok;
  __shared__ unsigned long long sh_base;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) sh_tile = atomicAdd(a.ticket, 1u);
  __syncthreads();
  const uint32_t tile = sh_tile;
  if (tile >= a.ntiles) return;
  const uint64_t i = (uint64_t)tile * WT_THREADS + tid;
  uint32_t type = PJ_TYPE_NONE;
  uint64_t row = 0;
  const bool plain = !a.w.res->needs_escape; /* no string of the columns holds a byte to escape */
  const long long c0 = clock64();
  const bool located = i < a.w.n && write_locate(a.w.schema, &a.w.cols, i, &type, &row);
  uint32_t len = 0;
  if (located) {
    if (type == PJ_TYPE_PET) prefetch_row<OBJ_PET>(&a.w.cols, row);
    else if (type == PJ_TYPE_ORDER) prefetch_row<OBJ_ORDER>(&a.w.cols, row);
    else prefetch_row<OBJ_USER>(&a.w.cols, row);
    WOut w; w.dst = nullptr; w.n = 0; w.hexa = a.w.hexa;
    if (plain) fwrite_record<false, true>(&a.w.cols, type, row, a.w.inclusion, w); else fwrite_record<false, false>(&a.w.cols, type, row, a.w.inclusion, w);
    len = (uint32_t)w.n + 1; /* LF, or the comma / closing bracket that follows the record */
  }
  const uint32_t incl = warp_incl_scan(len);
  if (lane == 31) sh_warp[warp] = incl;
  uint32_t loc = incl - len;
  __syncthreads();
  const long long c1 = clock64();
  uint32_t tile_total = 0;
#pragma unroll
  for (uint32_t q = 0; q < NWARPS; ++q) { if (q < warp) loc += sh_warp[q]; tile_total += sh_warp[q]; }
  const uint64_t lead = a.w.array ? 1 : 0; /* the opening bracket */
  if (warp == 0) {
    if (lane == 0) {
      st_relaxed_u64(&a.agg[tile], TS_VALID | tile_total);
      if (tile == 0) st_relaxed_u64(&a.inc[tile], TS_VALID | tile_total);
    }
    unsigned long long excl = 0;
    const bool ok = lookback_u64(a.agg, a.inc, &a.w.res->timeout, a.spin_limit_ns, tile, lane, &excl);
    if (lane == 0) {
      if (tile != 0 && ok) st_relaxed_u64(&a.inc[tile], TS_VALID | (excl + tile_total));
      const bool room = lead + excl + tile_total <= a.w.cap;
      if (ok && !room) a.w.res->ok = 0;
      if (tile == a.ntiles - 1) a.w.res->out_bytes = excl + tile_total; /* text bytes of all records */
      sh_base = excl;
      sh_ok = ok && room;
    }
  }
  __syncthreads();
  const long long c2 = clock64();
  long long c3 = c2;
  if (!sh_ok) return;
  uint8_t* dst0 = a.w.out + lead + sh_base; /* where the tile's text starts */
  const uint8_t sep = a.w.array ? (uint8_t)',' : (uint8_t)'\n';
  if (tile_total + 16 <= WTILE_WIN_BYTES) {
    /* the window mirrors the output's alignment: window byte k goes to (dst0 - pad)[k] */
    const uint32_t pad = (uint32_t)(reinterpret_cast<uintptr_t>(dst0) & 15u);
    if (located) {
      WOut w; w.dst = smem + pad + loc; w.n = 0; w.hexa = a.w.hexa;
      if (plain) fwrite_record<true, true>(&a.w.cols, type, row, a.w.inclusion, w); else fwrite_record<true, false>(&a.w.cols, type, row, a.w.inclusion, w);
      smem[pad + loc + w.n] = sep;
    }
    fence_async_smem();
    __syncthreads();
    c3 = clock64();
    /* the 16-byte multiples in the middle leave with one bulk copy (cp.async.bulk shared -> global), the odd
       bytes at both ends with plain stores */
    uint8_t* gbase = dst0 - pad;
    const uint32_t end = pad + tile_total;
    const uint32_t lo16 = (pad + 15u) & ~15u, hi16 = end & ~15u;
    if (hi16 > lo16) {
      if (tid == 0) { bulk_s2g(gbase + lo16, smem + lo16, hi16 - lo16); bulk_s2g_wait_read(); }
      if (tid >= 32 && tid < 32 + (lo16 - pad)) gbase[pad + tid - 32] = smem[pad + tid - 32];
      if (tid >= 64 && tid < 64 + (end - hi16)) gbase[hi16 + tid - 64] = smem[hi16 + tid - 64];
    } else {
      for (uint32_t b = pad + tid; b < end; b += WT_THREADS) gbase[b] = smem[b];
    }
  } else if (located) {
    WOut w; w.dst = dst0 + loc; w.n = 0; w.hexa = a.w.hexa;
    if (plain) fwrite_record<true, true>(&a.w.cols, type, row, a.w.inclusion, w); else fwrite_record<true, false>(&a.w.cols, type, row, a.w.inclusion, w);
    dst0[loc + w.n] = sep;
  }
  __syncthreads();
  if (tid == 0) { /* cycles per phase: size pass, look-back, text into the window, copy-out */
    const long long c4 = clock64();
    atomicAdd(&a.w.res->phase_cycles[0], (unsigned long long)(c1 - c0));
    atomicAdd(&a.w.res->phase_cycles[1], (unsigned long long)(c2 - c1));
    atomicAdd(&a.w.res->phase_cycles[2], (unsigned long long)(c3 - c2));
    atomicAdd(&a.w.res->phase_cycles[3], (unsigned long long)(c4 - c3));
  }
}
/* closes the text: brackets of array framing, the total, the verdict */
static __global__ void k_write_close(const __grid_constant__ WriteArgs a) {
  if (threadIdx.x || blockIdx.x) return;
  const uint64_t body = a.res->out_bytes;
  const uint64_t total = a.array ? (body ? body + 1 : 2) : body;
  a.res->out_bytes = total;
  const bool ok = a.res->ok && total <= a.cap;
  a.res->ok = ok;
  if (a.array && ok) { a.out[0] = '['; a.out[total - 1] = ']'; }
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

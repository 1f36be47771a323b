/*
 * pj_block_emu.h — TEST INFRASTRUCTURE. The part of CUDA that k_parse_items uses, on the host: the threads of one block are
 * fibers of one OS thread, warp collectives and block barriers are rendezvous, blocks run one after the other.
 *
 * What it checks besides results: that all lanes of a warp meet in the SAME collective (source line), that all threads
 * of the block meet at the same barrier, that a block ends with all of its threads, that bulk copies are aligned, and that the
 * device-side spin loops end. A rule that is broken ends the run with a message in emu_block::error. With AddressSanitizer, shared
 * memory behind the launch's size is poisoned.
 * It stands in for pj_dev.cuh (whose include guard it takes), so the kernel's source is compiled unchanged.
 */
#ifndef PJ_BLOCK_EMU_H
#define PJ_BLOCK_EMU_H

#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <type_traits>
#include <vector>

#if defined(__SANITIZE_ADDRESS__)
#include <sanitizer/asan_interface.h>
#include <sanitizer/common_interface_defs.h>
#define EMU_POISON(p, n) ASAN_POISON_MEMORY_REGION(p, n)
#define EMU_UNPOISON(p, n) ASAN_UNPOISON_MEMORY_REGION(p, n)
#else
#define EMU_POISON(p, n) ((void)0)
#define EMU_UNPOISON(p, n) ((void)0)
#endif

namespace emu_block {

enum Kind { RUN = 0, BALLOT, ANY, ALL, SHFL, SHFL_UP, SHFL_DOWN, SHFL_XOR, RADD, RMIN, RMAX, ROR, SYNCWARP, SYNC, SYNC_OR, DONE };
#if !defined(__x86_64__)
#error "the switch between fibers is written for x86-64"
#endif
/* callee-saved registers on the old stack, stack pointer to *save, on with the other stack (swapcontext() makes a system call each time, and
 * AddressSanitizer clears a whole stack's shadow in it) */
extern "C" void pj_emu_switch(void** save, void* load);
asm(".weak pj_emu_switch\n.type pj_emu_switch, @function\npj_emu_switch:\n"
    "  push %rbx\n  push %rbp\n  push %r12\n  push %r13\n  push %r14\n  push %r15\n"
    "  mov %rsp, (%rdi)\n  mov %rsi, %rsp\n"
    "  pop %r15\n  pop %r14\n  pop %r13\n  pop %r12\n  pop %rbp\n  pop %rbx\n  ret\n");
struct Fiber {
  void* sp = nullptr;
  void* fake = nullptr; /* of AddressSanitizer */
  uint32_t tid = 0;
  int kind = DONE, site = 0;
  uint32_t mask = 0, width = 32;
  int arg = 0;
  uint64_t val = 0, res = 0;
};
static constexpr uint32_t MAX_THREADS = 1024;
static constexpr size_t STACK = 512 * 1024;

inline char error[512];
inline uint64_t n_barriers; /* block barriers passed since the last run began */
inline uint32_t n_threads;
inline Fiber fiber[MAX_THREADS];
inline Fiber* cur;
inline void* scheduler;
inline std::vector<uint8_t*> stacks;
inline const void* sched_stack; inline size_t sched_size;
struct Body { void (*call)(void*); void* arg; };
inline Body body;
inline bool dirty;
inline uint64_t steps, step_limit = 400000000ull;

inline void fail(const char* what, int a = 0, int b = 0) {
  if (!error[0]) snprintf(error, sizeof error, "%s (thread %u, lines %d and %d)", what, cur ? cur->tid : 0u, a, b);
}
inline void to_scheduler(bool leaving) {
  Fiber* me = cur;
#if defined(__SANITIZE_ADDRESS__)
  __sanitizer_start_switch_fiber(leaving ? nullptr : &me->fake, sched_stack, sched_size);
#endif
  (void)leaving;
  pj_emu_switch(&me->sp, scheduler);
#if defined(__SANITIZE_ADDRESS__)
  __sanitizer_finish_switch_fiber(me->fake, &sched_stack, &sched_size);
#endif
}
inline void enter() {
#if defined(__SANITIZE_ADDRESS__)
  __sanitizer_finish_switch_fiber(nullptr, &sched_stack, &sched_size);
#endif
  body.call(body.arg);
  cur->kind = DONE;
  to_scheduler(true);
}
inline uint64_t meet(int kind, int site, uint32_t mask, uint64_t val, int arg = 0, uint32_t width = 32) {
  Fiber* f = cur;
  f->kind = kind; f->site = site; f->mask = mask; f->val = val; f->arg = arg; f->width = width;
  to_scheduler(false);
  return f->res;
}
inline bool resolve_warp(uint32_t w) {
  Fiber* f = fiber + 32 * w;
  for (int i = 1; i < 32; ++i)
    if (f[i].kind != f[0].kind || f[i].site != f[0].site) { cur = f + i; fail("lanes of a warp meet in different places", f[0].site, f[i].site); return false; }
  uint64_t acc = f[0].kind == ALL ? 1 : (f[0].kind == RMIN ? 0xFFFFFFFFull : 0);
  for (int i = 0; i < 32; ++i) {
    const uint32_t v = (uint32_t)f[i].val;
    if (f[i].mask != 0xFFFFFFFFu) { cur = f + i; fail("a collective of part of a warp", f[i].site); return false; }
    switch (f[0].kind) {
      case BALLOT: acc |= (uint64_t)(f[i].val != 0) << i; break;
      case ANY: acc |= f[i].val != 0; break;
      case ALL: acc &= f[i].val != 0; break;
      case RADD: acc = (uint32_t)(acc + v); break;
      case RMIN: acc = v < acc ? v : acc; break;
      case RMAX: acc = v > acc ? v : acc; break;
      case ROR: acc |= v; break;
      default: break;
    }
  }
  for (int i = 0; i < 32; ++i) {
    const int lo = i / (int)f[i].width * (int)f[i].width, hi = lo + (int)f[i].width;
    int src = i;
    switch (f[0].kind) {
      case SHFL: src = lo + (f[i].arg & ((int)f[i].width - 1)); break;
      case SHFL_UP: src = i - f[i].arg < lo ? i : i - f[i].arg; break;
      case SHFL_DOWN: src = i + f[i].arg >= hi ? i : i + f[i].arg; break;
      case SHFL_XOR: src = (i ^ f[i].arg) >= hi ? i : (i ^ f[i].arg); break;
      default: src = -1;
    }
    f[i].res = src < 0 ? acc : f[src].val;
  }
  for (int i = 0; i < 32; ++i) f[i].kind = RUN;
  return true;
}
/* One block of n threads, all of which run call(arg). False: a rule was broken, see error. order: which warp goes first. */
inline bool run(uint32_t n, void (*call)(void*), void* arg, uint32_t order) {
  n_threads = n;
  body.call = call; body.arg = arg;
  while (stacks.size() < n) stacks.push_back((uint8_t*)aligned_alloc(64, STACK));
  for (uint32_t i = 0; i < n; ++i) {
    Fiber& f = fiber[i];
    f.tid = i; f.kind = RUN; f.fake = nullptr;
    if (dirty) EMU_UNPOISON(stacks[i], STACK); else EMU_UNPOISON(stacks[i] + STACK - 4096, 4096); /* (what enter() left) */
    void** top = (void**)(stacks[i] + STACK) - 2; /* the address enter() starts at, as if called from nowhere */
    top[0] = (void*)enter; top[1] = nullptr;
    f.sp = top - 6;
  }
  dirty = true; /* until the block has ended */
  const uint32_t nw = n / 32;
  for (;;) {
    bool ran = false;
    for (uint32_t k = 0; k < nw; ++k) {
      const uint32_t w = (k * (2 * (order % 16) + 1) + order) % nw; /* (nw is a power of two: every warp once) */
      for (;;) {
        bool any = false;
        uint32_t collective = 0;
        for (uint32_t i = 0; i < 32; ++i) {
          const uint32_t lane = order & 1 ? 31 - i : i;
          Fiber* f = fiber + 32 * w + lane;
          if (f->kind == RUN) {
            cur = f;
            if (++steps > step_limit) { fail("the block does not end"); return false; }
#if defined(__SANITIZE_ADDRESS__)
            void* keep = nullptr;
            __sanitizer_start_switch_fiber(&keep, stacks[f->tid], STACK);
#endif
            pj_emu_switch(&scheduler, f->sp);
#if defined(__SANITIZE_ADDRESS__)
            __sanitizer_finish_switch_fiber(keep, nullptr, nullptr);
#endif
            any = ran = true;
            if (error[0]) return false;
          }
          collective += f->kind > RUN && f->kind < SYNC;
        }
        if (collective == 32) { if (!resolve_warp(w)) return false; any = true; }
        if (!any) break;
      }
    }
    uint32_t at_barrier = 0, done = 0;
    for (uint32_t i = 0; i < n; ++i) { at_barrier += fiber[i].kind == SYNC || fiber[i].kind == SYNC_OR; done += fiber[i].kind == DONE; }
    if (done == n) { dirty = false; return true; }
    if (at_barrier == n) {
      uint64_t acc = 0;
      for (uint32_t i = 0; i < n; ++i) {
        if (fiber[i].kind != fiber[0].kind || fiber[i].site != fiber[0].site) { cur = fiber + i; fail("threads of a block meet at different barriers", fiber[0].site, fiber[i].site); return false; }
        acc |= fiber[i].val != 0;
      }
      for (uint32_t i = 0; i < n; ++i) { fiber[i].res = acc; fiber[i].kind = RUN; }
      ++n_barriers;
      continue;
    }
    if (!ran) {
      for (uint32_t i = 0; i < n; ++i) if (fiber[i].kind != SYNC && fiber[i].kind != SYNC_OR) { cur = fiber + i; break; }
      fail("threads wait for others that do not come", cur->site, cur->kind);
      return false;
    }
  }
}

template <class T> uint64_t bits(T v) { return (uint64_t)(typename std::conditional<sizeof(T) == 8, uint64_t, uint32_t>::type)v; }
template <class T> T shfl(int kind, int site, uint32_t mask, T v, int arg, int width = 32) { return (T)meet(kind, site, mask, bits(v), arg, (uint32_t)width); }
template <class T> T fetch_add(T* p, T v) { const T o = *p; *p = (T)(o + v); return o; }
template <class T> T fetch_min(T* p, T v) { const T o = *p; if (v < o) *p = v; return o; }
template <class T> T fetch_max(T* p, T v) { const T o = *p; if (v > o) *p = v; return o; }
template <class T> T fetch_or(T* p, T v) { const T o = *p; *p = o | v; return o; }
template <class T> T fetch_and(T* p, T v) { const T o = *p; *p = o & v; return o; }
template <class T> T swap(T* p, T v) { const T o = *p; *p = v; return o; }
struct Idx { uint32_t x; };
inline Idx thread_idx() { return Idx{cur->tid}; }
inline Idx block_dim() { return Idx{n_threads}; }

}  // namespace emu_block

struct uint4 { uint32_t x, y, z, w; };
typedef int cudaError_t;

#define threadIdx (emu_block::thread_idx())
#define blockDim (emu_block::block_dim())
#define __device__
#define __host__
#define __global__
#define __constant__
#define __grid_constant__
#define __launch_bounds__(...)
#define __shared__ thread_local
#define __align__(n) __attribute__((aligned(n)))
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline)) /* (no system header may come after this one) */

#define __ballot_sync(m, p) ((uint32_t)emu_block::meet(emu_block::BALLOT, __LINE__, m, (p) != 0))
#define __any_sync(m, p) ((int)emu_block::meet(emu_block::ANY, __LINE__, m, (p) != 0))
#define __all_sync(m, p) ((int)emu_block::meet(emu_block::ALL, __LINE__, m, (p) != 0))
#define __shfl_sync(m, v, ...) emu_block::shfl(emu_block::SHFL, __LINE__, m, v, __VA_ARGS__)
#define __shfl_up_sync(m, v, ...) emu_block::shfl(emu_block::SHFL_UP, __LINE__, m, v, __VA_ARGS__)
#define __shfl_down_sync(m, v, ...) emu_block::shfl(emu_block::SHFL_DOWN, __LINE__, m, v, __VA_ARGS__)
#define __shfl_xor_sync(m, v, ...) emu_block::shfl(emu_block::SHFL_XOR, __LINE__, m, v, __VA_ARGS__)
#define __reduce_add_sync(m, v) ((uint32_t)emu_block::meet(emu_block::RADD, __LINE__, m, (uint32_t)(v)))
#define __reduce_min_sync(m, v) ((uint32_t)emu_block::meet(emu_block::RMIN, __LINE__, m, (uint32_t)(v)))
#define __reduce_max_sync(m, v) ((uint32_t)emu_block::meet(emu_block::RMAX, __LINE__, m, (uint32_t)(v)))
#define __reduce_or_sync(m, v) ((uint32_t)emu_block::meet(emu_block::ROR, __LINE__, m, (uint32_t)(v)))
#define __syncwarp() ((void)emu_block::meet(emu_block::SYNCWARP, __LINE__, 0xFFFFFFFFu, 0))
#define __syncthreads() ((void)emu_block::meet(emu_block::SYNC, __LINE__, 0xFFFFFFFFu, 0))
#define __syncthreads_or(v) ((int)emu_block::meet(emu_block::SYNC_OR, __LINE__, 0xFFFFFFFFu, (v) != 0))

static inline int __popc(uint32_t x) { return __builtin_popcount(x); }
static inline int __ffs(int x) { return __builtin_ffs(x); }
static inline int __clz(int x) { return x ? __builtin_clz((unsigned)x) : 32; }
static inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) { return (uint32_t)((((uint64_t)hi << 32) | lo) >> (s & 31u)); }
static inline uint32_t __dp4a(uint32_t a, uint32_t b, uint32_t c) {
  for (int k = 0; k < 4; ++k) c += ((a >> (8 * k)) & 255u) * ((b >> (8 * k)) & 255u);
  return c;
}
static inline long long clock64() { return 0; }
static inline void __nanosleep(unsigned) { if (++emu_block::steps > emu_block::step_limit) { emu_block::fail("a wait does not end"); emu_block::to_scheduler(false); } }
template <class T, class U> T atomicAdd(T* p, U v) { return emu_block::fetch_add(p, (T)v); }
template <class T, class U> T atomicMin(T* p, U v) { return emu_block::fetch_min(p, (T)v); }
template <class T, class U> T atomicMax(T* p, U v) { return emu_block::fetch_max(p, (T)v); }
template <class T, class U> T atomicOr(T* p, U v) { return emu_block::fetch_or(p, (T)v); }
template <class T, class U> T atomicAnd(T* p, U v) { return emu_block::fetch_and(p, (T)v); }
template <class T, class U> T atomicExch(T* p, U v) { return emu_block::swap(p, (T)v); }

/* ---- pj_dev.cuh ---- */
#define PJ_DEV_CUH
namespace pj {
template <class T>
T warp_incl_scan(T v) {
  const unsigned lane = threadIdx.x & 31;
  for (int d = 1; d < 32; d <<= 1) {
    const T u = __shfl_up_sync(0xFFFFFFFFu, v, d);
    if (lane >= (unsigned)d) v += u;
  }
  return v;
}
template <class T>
T block_excl_scan(T v, T* total, T* sh) {
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const T inc = warp_incl_scan(v);
  __syncthreads();
  if (lane == 31) sh[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const T w = lane < nwarps ? sh[lane] : T(0);
    const T wi = warp_incl_scan(w);
    if (lane < nwarps) sh[lane] = wi - w;
    if (lane == nwarps - 1) sh[32] = wi;
  }
  __syncthreads();
  *total = sh[32];
  return sh[warp] + inc - v;
}
static constexpr unsigned long long TS_VALID = 1ull << 63;
inline unsigned long long ld_relaxed_u64(const unsigned long long* p) { return *p; }
inline void st_relaxed_u64(unsigned long long* p, unsigned long long v) { *p = v; }
inline unsigned long long global_ns() { return 0; }
inline void mbar_init(unsigned long long* bar, uint32_t) { *bar = 0; }
inline void mbar_expect_tx(unsigned long long* bar, uint32_t bytes) { *bar += bytes; }
inline void bulk_g2s(void* dst, const void* src, uint32_t bytes, unsigned long long* bar) {
  if (((uintptr_t)dst | (uintptr_t)src | bytes) & 15u) emu_block::fail("a bulk copy that is not aligned", __LINE__);
  memcpy(dst, src, bytes);
  *bar -= bytes;
}
inline bool mbar_wait_bounded(unsigned long long* bar, uint32_t, unsigned long long) { return *bar == 0; }
}  // namespace pj

#endif

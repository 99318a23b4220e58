#pragma once
// Persistent task-graph executor for the multifrontal sweeps (sm_100a).
//
// One kernel launch runs a whole sweep, in one of two schedules.  Static
// (the default): each CTA (128 threads) claims the next task index in list
// order with an atomic counter, waits until the counters the task depends on
// reach their targets (bounded spin; on timeout the CTA records DE_TIMEOUT
// and leaves, so a planning error can never hang the GPU), executes the task,
// then publishes its counter with release semantics; the claim of the next
// task goes out before that, in a GEMM task during its epilogue (in the build
// of the solves and products beside the release).  Dynamic: a
// finished task releases its waiters itself and keeps one of them; idle CTAs
// claim the others from a ready bitmap (bounded polling, same timeout rule).
//
// Dense FP64 tile arithmetic uses the double-precision tensor-core MMA
// (mma.sync m16n8k4 f64): a 64x64 C tile is split over 4 warps, 32x32 each.
// GEMM operand tiles are staged through a ring of shared-memory K chunks by
// cp.async; tiles produced by other CTAs in the same launch are read only
// after an acquire that ordered their writes before the read.  The other
// tasks read with L2-coherent loads (__ldcg).
#include <cuda_runtime.h>
#include <cstdint>

#include "engine.h"

namespace chb {

// ------------------------------------------------------------------ sync
__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Publication of a counter: every caller runs it from one thread right
// after a __syncthreads(), and the release is cumulative, so the CTA's
// writes before the barrier are visible (gpu scope) before the increment
// without a separate fence (measured: cholesky 6.48 -> 6.38 ms at 40^3
// without the __threadfence() that preceded it).
__device__ __forceinline__ void red_release_add(int* p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ int ld_volatile(const int* p) { return *((const volatile int*)p); }

__device__ __forceinline__ int ld_acquire_sys(const int* p) {
  int v;
  asm volatile("ld.acquire.sys.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Waits until the copy of incoming chunk j has raised its flag (the host
// stream copies the chunk, then the flag).  Bounded like every wait: on
// timeout DE_TIMEOUT is recorded and the sweep leaves.
static __device__ void wait_arrival(const RunArgs& ra, int j) {
  if (j < 0 || j >= ra.nio_in) {
    atomicCAS(&ra.ctl[1], 0, DE_BAD_TASK);
    return;
  }
  int64_t spins = 0;
  unsigned ns = 64;
  while (ld_acquire_sys(ra.io_in + j) == 0) {
    if (++spins > ra.spin_limit) {
      atomicCAS(&ra.ctl[1], 0, DE_TIMEOUT);
      atomicAdd(&ra.ctl[3], 1);
      return;
    }
    if ((spins & 15) == 0 && ld_volatile(&ra.ctl[1]) != 0) return;
    __nanosleep(ns);
    if (ns < 1024) ns <<= 1;
  }
}

// Host-visible flag: the CTA's earlier writes (ordered by the caller's
// __syncthreads) become visible to the copy engines before the flag.
__device__ __forceinline__ void raise_io_flag(int* p) {
  __threadfence_system();
  asm volatile("st.release.sys.global.b32 [%0], %1;" ::"l"(p), "r"(1) : "memory");
}

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// ------------------------------------------------------ dynamic schedule
// Ready tasks are bits of a bitmap (64 tasks per word, bit = list position)
// with a summary bitmap of the nonzero words.  ctl[5] is the finished
// frontier: every task in the words below it has finished, so no ready bit
// can appear there again; ctl[4] counts finished tasks.
//
// A finished task decrements the pending counts of its waiters (one lane of
// warp 0 per waiter, acq_rel).  Of the waiters it makes ready, the CTA keeps
// the one of lowest list position and runs it next, so a chain of dependent
// tasks never passes through the bitmap; the others are published with a
// release OR into the bitmap and claimed by idle CTAs with an acquire AND.
//
// Summary invariant: a word that turns nonzero has its summary bit set after
// it; a claimer that clears a summary bit re-reads the word after the clear
// and sets the bit again if the word is nonzero.  The fences between the word
// and summary accesses on both sides keep a nonzero word from ever losing its
// summary bit.
__device__ __forceinline__ int atom_add_acq_rel(int* p, int v) {
  int old;
  asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}

__device__ __forceinline__ void red_or_release(unsigned long long* p, unsigned long long v) {
  asm volatile("red.release.gpu.global.or.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ unsigned long long atom_and_acquire(unsigned long long* p, unsigned long long v) {
  unsigned long long old;
  asm volatile("atom.acquire.gpu.global.and.b64 %0, [%1], %2;" : "=l"(old) : "l"(p), "l"(v) : "memory");
  return old;
}

__device__ __forceinline__ unsigned long long atom_and_acq_rel(unsigned long long* p, unsigned long long v) {
  unsigned long long old;
  asm volatile("atom.acq_rel.gpu.global.and.b64 %0, [%1], %2;" : "=l"(old) : "l"(p), "l"(v) : "memory");
  return old;
}

// Publishes ready task s: its bit (release: the waiter's inputs are visible
// to whoever acquires the bit), then its word's summary bit (release: after
// the word).  Neither waits for a reply.
__device__ __forceinline__ void publish_ready(const RunArgs& ra, int s) {
  red_or_release(ra.ready + (s >> 6), 1ull << (s & 63));
  red_or_release(ra.summ + (s >> 12), 1ull << ((s >> 6) & 63));
}

// Clears the summary bit of a word seen empty.  The acq_rel AND reads the
// summary after any publish that set the bit, so the word re-read below
// shows that publish's task (unless it was claimed since).
__device__ __forceinline__ void clear_summary(const RunArgs& ra, int wi) {
  const unsigned long long bit = 1ull << (wi & 63);
  atom_and_acq_rel(ra.summ + (wi >> 6), ~bit);
  if (ld_relaxed_u64(ra.ready + wi) != 0) red_or_release(ra.summ + (wi >> 6), bit);
}

__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gmem_src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(gmem_src) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Releases the waiters listed in succ[b, e) (warp 0); the first 32 come
// from pre (shared memory) when it is given.  With handoff, the released
// waiter of lowest list position (below *next, the earlier candidate)
// becomes *next and is not published; the displaced candidate is.
__device__ __forceinline__ void release_list(const RunArgs& ra, int b, int e, const int* pre, bool handoff,
                                             int* next) {
  const int lane = threadIdx.x & 31;
  for (int i0 = b; i0 < e; i0 += 32) {
    int s = -1;
    if (i0 + lane < e) {
      s = (pre && i0 == b) ? pre[lane] : __ldg(ra.succ + i0 + lane);
      if (atom_add_acq_rel(ra.pend + s, -1) != 1) s = -1;
    }
    __syncwarp();  // orders every lane's acquire before the other lanes' publishes
    if (!handoff) {
      if (s >= 0) publish_ready(ra, s);
      continue;
    }
    int m = (s >= 0) ? s : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = min(m, __shfl_xor_sync(0xffffffffu, m, o));
    const int prev = *next;
    const int keep = min(m, prev);
    if (s >= 0 && s != keep) publish_ready(ra, s);
    if (lane == 0 && prev != 0x7fffffff && prev != keep) publish_ready(ra, prev);
    *next = keep;
  }
}

// Advances the finished frontier over every word whose tasks have all
// finished.
__device__ __forceinline__ void advance_frontier(const RunArgs& ra) {
  __threadfence();
  int cur = ld_volatile(&ra.ctl[5]);
  while (cur < ra.nwords) {
    const int cnt = min(64, ra.ntasks - 64 * cur);
    if (ld_volatile(ra.wclaimed + cur) < cnt) break;
    const int prev = atomicCAS(&ra.ctl[5], cur, cur + 1);
    cur = (prev == cur) ? cur + 1 : prev;
  }
}

// Claims the word's set bit of rank (blockIdx.x mod its popcount), so that
// CTAs claiming at once spread over the word (lane 0).  Returns the task, or
// -1 when the word has emptied (then, for a word found through the summary,
// its summary bit is cleared).
__device__ __forceinline__ int claim_in_word(const RunArgs& ra, int wi, unsigned long long w, bool from_summary) {
  while (w) {
    const unsigned lo = (unsigned)w, hi = (unsigned)(w >> 32);
    const int plo = __popc(lo), r = (int)(blockIdx.x % (unsigned)(plo + __popc(hi)));
    const int pos = r < plo ? (int)__fns(lo, 0, r + 1) : 32 + (int)__fns(hi, 0, r - plo + 1);
    const unsigned long long bit = 1ull << pos;
    const unsigned long long old = atom_and_acquire(ra.ready + wi, ~bit);
    if (old & bit) return wi * 64 + pos;
    w = old;
  }
  if (from_summary) clear_summary(ra, wi);
  return -1;
}

// Claims a ready task for this CTA (warp 0; every lane returns it): first in
// the 32 bitmap words from the cached frontier *lo, then through the summary
// beyond them.  Returns ntasks when every task has finished, when a device
// error is set, or when nothing became ready within the spin limit
// (DE_TIMEOUT).
__device__ __forceinline__ int claim_task(const RunArgs& ra, int* lo) {
  const int lane = threadIdx.x & 31;
  int64_t spins = 0;
  unsigned ns = 64;
  for (;;) {
    const int wi = *lo + lane;
    const unsigned long long w = (wi < ra.nwords) ? ld_relaxed_u64(ra.ready + wi) : 0ull;
    int stop = 0, front = 0;
    if (lane == 0) {
      stop = ld_volatile(&ra.ctl[4]) >= ra.ntasks || ld_volatile(&ra.ctl[1]) != 0;
      front = ld_volatile(&ra.ctl[5]);
    }
    if (__shfl_sync(0xffffffffu, stop, 0)) return ra.ntasks;
    front = __shfl_sync(0xffffffffu, front, 0);
    unsigned bal = __ballot_sync(0xffffffffu, w != 0);
    while (bal) {
      const int src = __ffs(bal) - 1;
      bal &= bal - 1;
      const unsigned long long ww = __shfl_sync(0xffffffffu, w, src);
      int got = -1;
      if (lane == 0) got = claim_in_word(ra, *lo + src, ww, false);
      got = __shfl_sync(0xffffffffu, got, 0);
      if (got >= 0) return got;
    }
    if (front > *lo) {
      *lo = front;
      continue;
    }
    // beyond the window: summary words from the one holding word *lo + 32
    const int first = *lo + 32;
    for (int s0 = first >> 6; s0 < ra.nsumm; s0 += 32) {
      unsigned long long sw = (s0 + lane < ra.nsumm) ? ld_relaxed_u64(ra.summ + s0 + lane) : 0ull;
      if (s0 + lane == (first >> 6)) sw &= ~0ull << (first & 63);
      unsigned sb = __ballot_sync(0xffffffffu, sw != 0);
      while (sb) {
        const int src = __ffs(sb) - 1;
        sb &= sb - 1;
        unsigned long long bits = __shfl_sync(0xffffffffu, sw, src);
        int got = -1;
        if (lane == 0) {
          while (bits && got < 0) {
            const int wj = (s0 + src) * 64 + __ffsll((long long)bits) - 1;
            bits &= bits - 1;
            got = claim_in_word(ra, wj, ld_relaxed_u64(ra.ready + wj), true);
          }
        }
        got = __shfl_sync(0xffffffffu, got, 0);
        if (got >= 0) return got;
      }
    }
    if (++spins > ra.spin_limit) {
      if (lane == 0) {
        atomicCAS(&ra.ctl[1], 0, DE_TIMEOUT);
        atomicAdd(&ra.ctl[3], 1);
      }
      return ra.ntasks;
    }
    __nanosleep(ns);
    if (ns < 512) ns <<= 1;
  }
}

// After task ti (warp 0, the CTA's writes ordered before by __syncthreads):
// releases the waiters of the task (the first 32 prefetched into pre;
// already done mid task by a split task: own_released) and,
// when the task completes its group, of the group; counts the task into its
// bitmap word's finished tasks and the finished count.  Returns the released
// waiter this CTA runs next, or -1 (also when a device error is set).
__device__ __forceinline__ int finish_task(const RunArgs& ra, int ti, int group, int sb, int se, const int* pre,
                                           bool own_released) {
  const int lane = threadIdx.x & 31;
  int next = 0x7fffffff;
  int gdone = 0, filled = 0, err = 0;
  if (lane == 0 && group >= 0) gdone = atom_add_acq_rel(ra.counters + group, 1) + 1 == __ldg(ra.ctarget + group);
  if (lane == 1) filled = atomicAdd(ra.wclaimed + (ti >> 6), 1) + 1 == min(64, ra.ntasks - (ti & ~63));
  if (lane == 2) err = ld_volatile(&ra.ctl[1]);
  if (lane == 3) red_release_add(ra.counters + ti, 1);  // for the mid waits of split tasks
  cp_async_wait_all();
  if (!own_released) release_list(ra, sb, se, pre, true, &next);
  if (__shfl_sync(0xffffffffu, gdone, 0))
    release_list(ra, __ldg(ra.succ_off + group), __ldg(ra.succ_off + group + 1), nullptr, true, &next);
  if (lane == 1 && filled) advance_frontier(ra);
  if (lane == 0) red_release_add(&ra.ctl[4], 1);
  if (__shfl_sync(0xffffffffu, err, 2) != 0 && next != 0x7fffffff) {
    if (lane == 0) publish_ready(ra, next);  // left for the exit path; nothing runs after an error
    next = 0x7fffffff;
  }
  return next == 0x7fffffff ? -1 : next;
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned sm_id() {
  unsigned r;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(r));
  return r;
}

// ------------------------------------------------------------- operands
struct SmemLayout {
  double* A;   // [TILE][LDS]: A(r, k) stored at A[k*LDS + r]
  double* B;   // [TILE][LDS]
};

constexpr int PER_THREAD = (TILE * KC) / NTHREADS;  // staged elements per thread

// Address of element (r, k) of an operand; ok is cleared outside the
// triangle of OM_TRI_* operands (the caller sets it from the bounds).
template <int MODE>
__device__ __forceinline__ const double* op_addr(const double* X, int ld, int diag, int koff, int r, int k, bool& ok) {
  if (MODE == OM_N) return X + (int64_t)k * ld + r;
  if (MODE == OM_T) return X + (int64_t)r * ld + k;
  if (MODE == OM_TRI_N) {
    ok = ok && r + diag >= k;
    return X + (int64_t)k * ld + r;
  }
  if (MODE == OM_TRI_T) {
    ok = ok && k + diag >= r;
    return X + (int64_t)r * ld + k;
  }
  // OM_SYM: element (r + diag, k + koff) of a symmetric matrix stored lower
  const int gr = r + diag, gc = k + koff;
  return gr >= gc ? X + (int64_t)gc * ld + gr : X + (int64_t)gr * ld + gc;
}

// 8-byte asynchronous copy global -> shared; zeros when !ok (nothing is read).
// Tiles written by other CTAs of the launch are read only after an acquire
// that ordered their writes before this copy, so the L1-allocating form
// sees them.
__device__ __forceinline__ void cp_async8_zfill(double* dst, const double* src, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(ok ? 8 : 0) : "memory");
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Coordinates of the s-th staged element of this thread.  Operands read
// along k (OM_T, OM_TRI_T) give consecutive threads consecutive k so that
// global reads stay coalesced; the others give consecutive threads
// consecutive rows.
template <int MODE>
__device__ __forceinline__ void stage_coord(int s, int& r, int& kk) {
  const int idx = threadIdx.x + s * NTHREADS;
  if (MODE == OM_T || MODE == OM_TRI_T) {
    kk = idx % KC;
    r = idx / KC;
  } else {
    r = idx % TILE;
    kk = idx / TILE;
  }
}

// Issues the copies of the operand's K chunk [k0, k0 + KC) into a stage:
// S[kk*LDS + r] = op(r, k0 + kk), zero outside [0,rows) x [0,K).  For the
// plain and triangular modes a thread's elements lie at fixed strides from
// one base pointer (the coordinates of stage_coord with the thread count a
// multiple of TILE and of KC), which saves the per-element address
// arithmetic.
static_assert(NTHREADS % TILE == 0 && NTHREADS % KC == 0, "stage coordinates assume whole rows / columns");
template <int MODE>
__device__ __forceinline__ void issue_chunk_t(const double* __restrict__ X, int ld, int diag, int koff, int rows,
                                              int k0, int K, double* S) {
  const int tid = threadIdx.x;
  if (MODE == OM_N || MODE == OM_TRI_N) {
    constexpr int KSTEP = NTHREADS / TILE;  // k rows per element step
    const int r = tid % TILE, kb = tid / TILE;
    const double* p = X + (int64_t)(k0 + kb) * ld + r;
#pragma unroll
    for (int s = 0; s < PER_THREAD; s++) {
      const int kk = kb + KSTEP * s, k = k0 + kk;
      const bool ok = r < rows && k < K && (MODE == OM_N || r + diag >= k);
      cp_async8_zfill(S + kk * LDS + r, ok ? p + (int64_t)(KSTEP * s) * ld : X, ok);
    }
  } else if (MODE == OM_T || MODE == OM_TRI_T) {
    constexpr int RSTEP = NTHREADS / KC;  // rows per element step
    const int kk = tid % KC, rb = tid / KC, k = k0 + kk;
    const double* p = X + (int64_t)rb * ld + k;
#pragma unroll
    for (int s = 0; s < PER_THREAD; s++) {
      const int r = rb + RSTEP * s;
      const bool ok = r < rows && k < K && (MODE == OM_T || k + diag >= r);
      cp_async8_zfill(S + kk * LDS + r, ok ? p + (int64_t)(RSTEP * s) * ld : X, ok);
    }
  } else {
#pragma unroll
    for (int s = 0; s < PER_THREAD; s++) {
      int r, kk;
      stage_coord<MODE>(s, r, kk);
      const int k = k0 + kk;
      bool ok = r < rows && k < K;
      const double* src = op_addr<MODE>(X, ld, diag, koff, r, k, ok);
      cp_async8_zfill(S + kk * LDS + r, ok ? src : X, ok);
    }
  }
}

// Operand held in registers for the duration of a task.
struct Opnd {
  const double* X;
  int ld, diag, koff, mode;
};

__device__ __forceinline__ Opnd make_opnd(const RunArgs& ra, const Operand& o) {
  Opnd p;
  p.X = ra.bases[o.base] + o.off;
  p.ld = o.ld;
  p.diag = o.diag;
  p.koff = o.pad2;
  p.mode = o.mode;
  return p;
}

__device__ __forceinline__ void issue_chunk(const Opnd& o, int rows, int k0, int K, double* S) {
  switch (o.mode) {
    case OM_N: issue_chunk_t<OM_N>(o.X, o.ld, o.diag, o.koff, rows, k0, K, S); break;
    case OM_T: issue_chunk_t<OM_T>(o.X, o.ld, o.diag, o.koff, rows, k0, K, S); break;
    case OM_TRI_N: issue_chunk_t<OM_TRI_N>(o.X, o.ld, o.diag, o.koff, rows, k0, K, S); break;
    case OM_TRI_T: issue_chunk_t<OM_TRI_T>(o.X, o.ld, o.diag, o.koff, rows, k0, K, S); break;
    default: issue_chunk_t<OM_SYM>(o.X, o.ld, o.diag, o.koff, rows, k0, K, S); break;
  }
}

// Double-precision tensor-core MMA, m16n8k4 (sm_90+):
//   A 16x4 row-major: a0 = A(g, q), a1 = A(g + 8, q)
//   B 4x8 col-major:  b0 = B(q, g)
//   C 16x8:           c0,c1 = C(g, 2q + {0,1}), c2,c3 = C(g + 8, 2q + {0,1})
// with g = lane / 4, q = lane % 4.  A warp owns a 32x32 C sub-tile: two m16
// rows x four n8 columns.
__device__ __forceinline__ void dmma16(double (&c)[4], double a0, double a1, double b) {
  asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
               : "d"(a0), "d"(a1), "d"(b));
}

// Accumulator layout: acc[i][j][h] with i in 0..1 (m16 tile), j in 0..3 (n8
// tile), h in 0..3 (c0..c3).
typedef double Acc[2][4][4];

// Tile coordinates of acc[i][j][h] inside the 64x64 C tile.
__device__ __forceinline__ void acc_coord(int i, int j, int h, int& r, int& c) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, q = lane & 3;
  r = (warp >> 1) * 32 + 16 * i + g + ((h & 2) ? 8 : 0);
  c = (warp & 1) * 32 + 8 * j + 2 * q + (h & 1);
}

// acc += A(:, 0:kn) * B(:, 0:kn)^T from tiles in shared memory, A(r, k) at
// sA[k*LA + r] and B(c, k) at sB[k*LB + c] (kn multiple of 4).
template <int LA, int LB>
__device__ __forceinline__ void mma_block_ld(const double* sA, const double* sB, int kn, Acc& acc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, q = lane & 3;
  const int r0 = (warp >> 1) * 32 + g, c0 = (warp & 1) * 32 + g;
#pragma unroll 4
  for (int kk = 0; kk < kn; kk += 4) {
    double a[2][2], b[4];
    const double* ak = sA + (kk + q) * LA + r0;
    const double* bk = sB + (kk + q) * LB + c0;
#pragma unroll
    for (int i = 0; i < 2; i++) {
      a[i][0] = ak[16 * i];
      a[i][1] = ak[16 * i + 8];
    }
#pragma unroll
    for (int j = 0; j < 4; j++) b[j] = bk[8 * j];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) dmma16(acc[i][j], a[i][0], a[i][1], b[j]);
  }
}

// The GEMM stages (leading dimension LDS).
__device__ __forceinline__ void mma_block(const double* sA, const double* sB, int kn, Acc& acc) {
  mma_block_ld<LDS, LDS>(sA, sB, kn, acc);
}

// The m16 and n8 tiles of the calling warp's 32x32 sub-tile that meet an
// m x n product (warp-uniform): mi in 0..2, nj in 0..4.
__device__ __forceinline__ void warp_tiles(int m, int n, int& mi, int& nj) {
  const int warp = threadIdx.x >> 5;
  const int r = m - (warp >> 1) * 32, c = n - (warp & 1) * 32;
  mi = r <= 0 ? 0 : (r >= 32 ? 2 : (r + 15) >> 4);
  nj = c <= 0 ? 0 : (c >= 32 ? 4 : (c + 7) >> 3);
}

// mma_block for a partial tile: only the warp's first mi m16 and nj n8
// tiles are multiplied (the others hold rows or columns outside the
// product, which the epilogue does not store).  A narrow product (a few
// right-hand sides, the edge tiles of a front) then issues a fraction of
// the MMAs of a full 64x64 tile.
__device__ __forceinline__ void mma_block_part(const double* sA, const double* sB, int kn, Acc& acc, int mi,
                                               int nj) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, q = lane & 3;
  const int r0 = (warp >> 1) * 32 + g, c0 = (warp & 1) * 32 + g;
#pragma unroll 2
  for (int kk = 0; kk < kn; kk += 4) {
    double a[2][2], b[4];
    const double* ak = sA + (kk + q) * LDS + r0;
    const double* bk = sB + (kk + q) * LDS + c0;
#pragma unroll
    for (int i = 0; i < 2; i++) {
      a[i][0] = i < mi ? ak[16 * i] : 0.0;
      a[i][1] = i < mi ? ak[16 * i + 8] : 0.0;
    }
#pragma unroll
    for (int j = 0; j < 4; j++) b[j] = j < nj ? bk[8 * j] : 0.0;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (i < mi && j < nj) dmma16(acc[i][j], a[i][0], a[i][1], b[j]);
  }
}

__device__ __forceinline__ void zero_acc(Acc& acc) {
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int h = 0; h < 4; h++) acc[i][j][h] = 0.0;
}

// ------------------------------------------------------------ TF32 path
__device__ __forceinline__ uint32_t to_tf32(float f) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(f));
  return r;
}

// TF32 MMA m16n8k8 with FP32 accumulation:
//   A 16x8 row-major: a0 = A(g, q), a1 = A(g+8, q), a2 = A(g, q+4), a3 = A(g+8, q+4)
//   B 8x8 col-major:  b0 = B(q, g), b1 = B(q+4, g)
//   C 16x8: as the FP64 MMA (c0,c1 row g, c2,c3 row g+8; columns 2q, 2q+1)
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

typedef float AccF[2][4][4];

// High and low TF32 parts of an FP64 value (x ~ hi + lo to about 22 bits).
__device__ __forceinline__ void split_tf32(double x, uint32_t& hi, uint32_t& lo) {
  const float f = (float)x;
  hi = to_tf32(f);
  lo = to_tf32((float)(x - (double)__uint_as_float(hi)));
}

// accf += A(:, 0:kn) B(:, 0:kn)^T from FP64 stages (kn a multiple of 8; the
// stage is zero past K).  X3: three products (hi*hi + hi*lo + lo*hi).
template <bool X3>
__device__ __forceinline__ void mma_block_tf32(const double* sA, const double* sB, int kn, AccF& acc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, q = lane & 3;
  const int r0 = (warp >> 1) * 32 + g, c0 = (warp & 1) * 32 + g;
#pragma unroll 2
  for (int kk = 0; kk < kn; kk += 8) {
    uint32_t ah[2][4], al[2][4], bh[4][2], bl[4][2];
    const double* ak0 = sA + (kk + q) * LDS + r0;
    const double* ak4 = sA + (kk + q + 4) * LDS + r0;
    const double* bk0 = sB + (kk + q) * LDS + c0;
    const double* bk4 = sB + (kk + q + 4) * LDS + c0;
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const double v[4] = {ak0[16 * i], ak0[16 * i + 8], ak4[16 * i], ak4[16 * i + 8]};
#pragma unroll
      for (int e = 0; e < 4; e++) {
        if (X3) split_tf32(v[e], ah[i][e], al[i][e]);
        else ah[i][e] = to_tf32((float)v[e]);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const double v0 = bk0[8 * j], v1 = bk4[8 * j];
      if (X3) {
        split_tf32(v0, bh[j][0], bl[j][0]);
        split_tf32(v1, bh[j][1], bl[j][1]);
      } else {
        bh[j][0] = to_tf32((float)v0);
        bh[j][1] = to_tf32((float)v1);
      }
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (X3) {
          mma_tf32(acc[i][j], al[i], bh[j][0], bh[j][1]);
          mma_tf32(acc[i][j], ah[i], bl[j][0], bl[j][1]);
        }
        mma_tf32(acc[i][j], ah[i], bh[j][0], bh[j][1]);
      }
  }
}

// acc = opA * opB^T over K through a GEMM_STAGES-deep ring of K chunks in
// shared memory: the copies of chunk c + GEMM_STAGES - 1 are in flight while
// chunk c is multiplied; one barrier per chunk.
constexpr int GEMM_STAGES = 4;
constexpr int STAGE_DOUBLES = 2 * KC * LDS;  // A chunk, then B chunk

template <int PREC>
__device__ void gemm_acc_p(const Opnd& A, const Opnd& B, int m, int n, int K, const SmemLayout& sm, Acc& acc) {
  AccF accf;
  if (PREC != PREC_FP64) {
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int h = 0; h < 4; h++) accf[i][j][h] = 0.f;
  }
  zero_acc(acc);
  const int nch = (K + KC - 1) / KC;
  double* const ring = sm.A;
  int wmi, wnj;
  warp_tiles(m, n, wmi, wnj);
  const bool full = wmi == 2 && wnj == 4;
#pragma unroll
  for (int c = 0; c < GEMM_STAGES - 1; c++) {
    if (c < nch) {
      issue_chunk(A, m, c * KC, K, ring + c * STAGE_DOUBLES);
      issue_chunk(B, n, c * KC, K, ring + c * STAGE_DOUBLES + KC * LDS);
    }
    cp_async_commit();
  }
  for (int c = 0; c < nch; c++) {
    cp_async_wait_group<GEMM_STAGES - 2>();  // this thread's copies of chunk c
    __syncthreads();                         // everyone's; and chunk c - 1 is consumed
    const int cn = c + GEMM_STAGES - 1;
    if (cn < nch) {
      double* d = ring + (cn % GEMM_STAGES) * STAGE_DOUBLES;
      issue_chunk(A, m, cn * KC, K, d);
      issue_chunk(B, n, cn * KC, K, d + KC * LDS);
    }
    cp_async_commit();
    const double* st = ring + (c % GEMM_STAGES) * STAGE_DOUBLES;
    int kn = min(KC, K - c * KC);
    if (PREC == PREC_FP64) {
      kn = (kn + 3) & ~3;
      if (full) mma_block(st, st + KC * LDS, kn, acc);
      else if (wmi > 0 && wnj > 0) mma_block_part(st, st + KC * LDS, kn, acc, wmi, wnj);
    } else {
      kn = (kn + 7) & ~7;
      mma_block_tf32<PREC == PREC_TF32X3>(st, st + KC * LDS, kn, accf);
    }
  }
  cp_async_wait_group<0>();
  __syncthreads();
  if (PREC != PREC_FP64) {
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int h = 0; h < 4; h++) acc[i][j][h] = (double)accf[i][j][h];
  }
}

// ------------------------------------------------------ tcgen05 TF32 tiles
// TF32 GEMM tiles of the mixed-precision sweeps on the fifth-generation
// tensor cores: tcgen05.mma.cta_group::1.kind::tf32 with M = N = 64 and
// K = 8 per instruction, FP32 accumulators in tensor memory (64 columns per
// CTA, allocated once per launch when the program has such tiles).  K goes
// through the FP64 cp.async ring as for the other tiles (three stages here);
// per chunk of KC = 16 the 128 threads round the stage to TF32 (cvt.rna, as
// the mma.sync tiles do) into one of two shared-memory buffers in the
// canonical K-major layout without swizzle: core matrices of 8 rows x 16
// bytes, element (r, k) of the chunk at byte ((r/8)*4 + k/4)*128 + (r%8)*16 +
// (k%4)*4, so the next 4 columns start 128 bytes on (leading byte offset) and
// the next 8 rows 512 bytes on (stride byte offset).  One thread issues the
// chunk's two MMAs and commits them to the buffer's mbarrier; a buffer is
// refilled once its last commit has arrived.  The epilogue reads the
// accumulator with tcgen05.ld (for M = 64, row 16w + i lives in TMEM lane
// 32w + i, so warp w reads its own sub-partition's lanes 0..15) and adds
// alpha*acc + beta*C in FP64.
constexpr int TC_STAGES = 3;                       // FP64 ring stages of a tcgen05 tile
constexpr int TC_STAGE_FLOATS = 2 * TILE * KC;     // A then B of one chunk, TF32
// instruction descriptor: F32 accumulator (bits 4-5 = 1), A and B TF32
// (bits 7-9, 10-12 = 2), both K-major, N >> 3 (bits 17-22), M >> 4 (bits 24-28)
constexpr uint32_t TC_IDESC = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(TILE >> 3) << 17) |
                              ((uint32_t)(TILE >> 4) << 24);
static_assert(TC_STAGES * STAGE_DOUBLES * 8 + 2 * TC_STAGE_FLOATS * 4 <= ENGINE_SMEM_BASE_DOUBLES * 8,
              "tcgen05 staging exceeds the engine's shared memory");

struct TcState {
  uint32_t tmem;        // accumulator: TMEM lane 0, first allocated column
  uint64_t* mbar;       // two mbarriers in shared memory
  uint32_t ncommit[2];  // commits issued to each mbarrier (same in every thread)
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: start address >> 4 (bits 0-13), leading
// byte offset 128 >> 4 (bits 16-29), stride byte offset 512 >> 4 (bits
// 32-45), descriptor version 1 (bits 46-47), no swizzle (bits 61-63 = 0)
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(128u >> 4) << 16) | ((uint64_t)(512u >> 4) << 32) |
         (1ull << 46);
}

__device__ __forceinline__ void tc_mma(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
      "l"(adesc), "l"(bdesc), "r"(TC_IDESC), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t* mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(mbar))
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_init(uint64_t* m) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(m)) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* m, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(m)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait for the completion of the phase with the given parity (an
// MMA chunk takes well under a microsecond; each try_wait may suspend the
// thread for a while, so the bound is time, 2 s); a wait that runs out
// records DE_TIMEOUT and returns false.
static __device__ bool mbar_wait(const RunArgs& ra, uint64_t* m, uint32_t parity) {
  if (mbar_test(m, parity)) return true;
  const unsigned long long t0 = global_ns();
  while (!mbar_test(m, parity)) {
    if (global_ns() - t0 > 2000000000ull) {
      atomicCAS(&ra.ctl[1], 0, DE_TIMEOUT);
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// One FP64 stage (A(r, k) at st[k*LDS + r], B at st + KC*LDS) rounded to
// TF32 into a staging buffer in the canonical K-major layout; each thread
// writes 16-byte rows of core matrices.
__device__ __forceinline__ void tc_stage(const double* st, float* S) {
#pragma unroll
  for (int it = 0; it < 4; it++) {
    const int idx = threadIdx.x + it * NTHREADS;  // (operand, 4-column group, row)
    const int op = idx >> 8, q = (idx >> 6) & 3, r = idx & 63;
    const double* src = st + op * KC * LDS + 4 * q * LDS + r;
    float4 v;
    v.x = __uint_as_float(to_tf32((float)src[0]));
    v.y = __uint_as_float(to_tf32((float)src[LDS]));
    v.z = __uint_as_float(to_tf32((float)src[2 * LDS]));
    v.w = __uint_as_float(to_tf32((float)src[3 * LDS]));
    *reinterpret_cast<float4*>(S + op * TILE * KC + ((r >> 3) * 4 + q) * 32 + (r & 7) * 4) = v;
  }
}

// C = alpha * opA * opB^T + beta * C for an m x n tile (masked to r + cdiag
// >= c when lower) with TF32 products on tcgen05 and FP32 accumulation.
static __device__ void gemm_tc_tf32(const RunArgs& ra, const Opnd& A, const Opnd& B, int m, int n, int K,
                             const SmemLayout& sm, TcState& ts, double* __restrict__ C, int ldc, bool lower,
                             int cdiag, double alpha, double beta) {
  const int nch = (K + KC - 1) / KC;
  double* const ring = sm.A;
  float* const stg = reinterpret_cast<float*>(ring + TC_STAGES * STAGE_DOUBLES);
#pragma unroll
  for (int c = 0; c < TC_STAGES - 1; c++) {
    if (c < nch) {
      issue_chunk(A, m, c * KC, K, ring + c * STAGE_DOUBLES);
      issue_chunk(B, n, c * KC, K, ring + c * STAGE_DOUBLES + KC * LDS);
    }
    cp_async_commit();
  }
  for (int c = 0; c < nch; c++) {
    cp_async_wait_group<TC_STAGES - 2>();  // this thread's copies of chunk c
    __syncthreads();                       // everyone's; and chunk c - 1 is converted
    const int cn = c + TC_STAGES - 1;
    if (cn < nch) {
      double* d = ring + (cn % TC_STAGES) * STAGE_DOUBLES;
      issue_chunk(A, m, cn * KC, K, d);
      issue_chunk(B, n, cn * KC, K, d + KC * LDS);
    }
    cp_async_commit();
    const int buf = c & 1;
    if (c >= 2) mbar_wait(ra, ts.mbar + buf, (ts.ncommit[buf] - 1) & 1);  // chunk c - 2 has read it
    float* S = stg + buf * TC_STAGE_FLOATS;
    tc_stage(ring + (c % TC_STAGES) * STAGE_DOUBLES, S);
    fence_proxy_async();
    __syncthreads();
    if (threadIdx.x == 0) {
      tc_fence_after();
      const uint32_t sa = smem_u32(S), sb = smem_u32(S + TILE * KC);
      tc_mma(ts.tmem, tc_desc(sa), tc_desc(sb), c > 0 ? 1u : 0u);
      tc_mma(ts.tmem, tc_desc(sa + 256), tc_desc(sb + 256), 1u);
      tc_commit(ts.mbar + buf);
    }
    ts.ncommit[buf]++;
  }
  cp_async_wait_group<0>();
  // the last commit covers every MMA of the tile
  const int lb = (nch - 1) & 1;
  mbar_wait(ra, ts.mbar + lb, (ts.ncommit[lb] - 1) & 1);
  tc_fence_after();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = warp * 16 + lane;
  const uint32_t taddr = ts.tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
  for (int c0 = 0; c0 < TILE; c0 += 16) {
    uint32_t v[16];
    tmem_ld16(taddr + c0, v);
    if (lane < 16 && r < m) {
      double old[16];
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const int c = c0 + j;
        const bool ok = c < n && !(lower && r + cdiag < c);
        old[j] = (beta != 0.0 && ok) ? __ldcg(C + (int64_t)c * ldc + r) : 0.0;
      }
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const int c = c0 + j;
        if (c >= n || (lower && r + cdiag < c)) continue;
        double x = alpha * (double)__uint_as_float(v[j]);
        if (beta != 0.0) x += beta * old[j];
        C[(int64_t)c * ldc + r] = x;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
}

__device__ __forceinline__ void gemm_acc(const Opnd& A, const Opnd& B, int m, int n, int K, const SmemLayout& sm,
                                         Acc& acc) {
  gemm_acc_p<PREC_FP64>(A, B, m, n, K, sm, acc);
}

// C = alpha*acc + beta*C (masked to m x n and, for lower, to r + cdiag >= c).
// All old values are fetched before the first store so that the loads are
// in flight together (the compiler cannot reorder them across stores to C).
// C += alpha acc with atomic adds (CM_ATOMIC).
static __device__ void store_acc_atomic(double* __restrict__ C, int ldc, int m, int n, double alpha, const Acc& acc) {
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int h = 0; h < 4; h++) {
        int r, c;
        acc_coord(i, j, h, r, c);
        if (r < m && c < n) atomicAdd(C + (int64_t)c * ldc + r, alpha * acc[i][j][h]);
      }
}

static __device__ void store_acc(double* __restrict__ C, int ldc, int m, int n, bool lower, int cdiag, double alpha,
                          double beta, const Acc& acc) {
  double old[2][4][4];
  if (beta != 0.0) {
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int h = 0; h < 4; h++) {
          int r, c;
          acc_coord(i, j, h, r, c);
          const bool ok = r < m && c < n && !(lower && r + cdiag < c);
          old[i][j][h] = ok ? __ldcg(C + (int64_t)c * ldc + r) : 0.0;
        }
  }
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int h = 0; h < 4; h++) {
        int r, c;
        acc_coord(i, j, h, r, c);
        if (r >= m || c >= n) continue;
        if (lower && r + cdiag < c) continue;
        double v = alpha * acc[i][j][h];
        if (beta != 0.0) v += beta * old[i][j][h];
        C[(int64_t)c * ldc + r] = v;
      }
}

// ------------------------------------------------------------------ GEMM
// GEMM task (T_GEMM), and the look-ahead step of the blocked Cholesky
// (T_LA) as two passes through the same code.  T_LA, with the next diagonal
// tile D (operand c, m x m, lower part), the tile A below the current
// diagonal block (operand a, m x n, overwritten) and M = L_cc^{-1} (operand
// b, read as lower-triangular):
//   pass 0: L = A M^T -> A;  early signal (aux[3] - 1, when aux[3] > 0)
//   pass 1: D -= L L^T (lower part), L read back from L2
// Both passes share one inlined copy of the GEMM code: a second copy (or a
// call) makes the persistent kernel spill.
template <bool TC, bool EARLY>
__device__ void run_gemm_or_la(const RunArgs& ra, const Task& t, const SmemLayout& sm, TcState& ts, int& claim) {
  const bool la = t.op == T_LA;
  const int passes = la ? 2 : 1;
  for (int ph = 0; ph < passes; ph++) {
    const Operand& ob = (la && ph == 1) ? t.a : t.b;
    const Operand& oc = (la && ph == 0) ? t.a : t.c;
    const Opnd A = make_opnd(ra, t.a), B = make_opnd(ra, ob);
    const int m = t.m, n = (la && ph == 1) ? t.m : t.n, K = (la && ph == 1) ? t.n : t.k;
    const bool lower = la ? ph == 1 : t.cmode == CM_LOWER;
    const int cdiag = la ? 0 : t.cdiag;
    const double alpha = la ? (ph == 0 ? 1.0 : -1.0) : t.alpha;
    const double beta = la ? (ph == 0 ? 0.0 : 1.0) : t.beta;
    if (TC && !la && t.c.prec == PREC_TF32) {
      gemm_tc_tf32(ra, A, B, m, n, K, sm, ts, ra.bases[oc.base] + oc.off, oc.ld, lower, cdiag, alpha, beta);
      continue;
    }
    Acc acc;
    if (la || t.c.prec == PREC_FP64) gemm_acc_p<PREC_FP64>(A, B, m, n, K, sm, acc);
    else if (t.c.prec == PREC_TF32) gemm_acc_p<PREC_TF32>(A, B, m, n, K, sm, acc);
    else gemm_acc_p<PREC_TF32X3>(A, B, m, n, K, sm, acc);
    // static, EARLY: claim the next task, whose index comes back during the epilogue
    if (EARLY && !ra.dynamic && ph == passes - 1 && threadIdx.x == 32) claim = atomicAdd(&ra.ctl[0], 1);
    if (!la && t.cmode == CM_ATOMIC) store_acc_atomic(ra.bases[oc.base] + oc.off, oc.ld, m, n, alpha, acc);
    else store_acc(ra.bases[oc.base] + oc.off, oc.ld, m, n, lower, cdiag, alpha, beta, acc);
    if (la && ph == 0) {
      __syncthreads();
      if (t.aux[3] > 0) {
        if (ra.dynamic) {
          const int c = t.aux[3] - 1;
          if (threadIdx.x < 32)
            release_list(ra, __ldg(ra.succ_off + c), __ldg(ra.succ_off + c + 1), nullptr, false, nullptr);
        } else if (threadIdx.x == 0) {
          red_release_add(ra.counters + (t.aux[3] - 1), 1);
        }
      }
    }
  }
}

// Reduction of split-K partial products (T_SUM): C = alpha * sum_q P_q +
// beta * C over the m x n tile (masked to r + cdiag >= c when cmode is
// CM_LOWER), P_q at a.off + q * aux[1] (ld a.ld), q = 0 .. aux[0]-1 added in
// order, so the result does not depend on the schedule.
static __device__ void run_sum(const RunArgs& ra, const Task& t) {
  const double* __restrict__ P = ra.bases[t.a.base] + t.a.off;
  double* __restrict__ C = ra.bases[t.c.base] + t.c.off;
  const int ldp = t.a.ld, ldc = t.c.ld, m = t.m, n = t.n, np = t.aux[0];
  const int64_t stride = (int64_t)(uint32_t)t.aux[1];
  const bool lower = t.cmode == CM_LOWER;
  constexpr int NQ = 4;                            // quarters of the tile
  constexpr int E = TILE * TILE / NTHREADS / NQ;  // elements per thread and quarter
  constexpr int U = 4;                            // partials loaded together
  // a thread's elements of U partials are loaded together (up to U E loads
  // in flight), then added partial after partial in index order; quarters
  // keep the registers in check
#pragma unroll 1
  for (int qt = 0; qt < NQ; qt++) {
    if (qt * E * NTHREADS / TILE >= n) break;  // the quarter's columns start at or after n
    double acc[E];
#pragma unroll
    for (int e = 0; e < E; e++) acc[e] = 0.0;
    for (int q0 = 0; q0 < np; q0 += U) {
      double v[U][E];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const double* Pq = P + (q0 + u) * stride;
#pragma unroll
        for (int e = 0; e < E; e++) {
          const int idx = threadIdx.x + (qt * E + e) * NTHREADS, r = idx % TILE, c = idx / TILE;
          v[u][e] = (q0 + u < np && r < m && c < n) ? __ldcg(Pq + (int64_t)c * ldp + r) : 0.0;
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++)
#pragma unroll
        for (int e = 0; e < E; e++)
          if (q0 + u < np) acc[e] += v[u][e];
    }
#pragma unroll
    for (int e = 0; e < E; e++) {
      const int idx = threadIdx.x + (qt * E + e) * NTHREADS, r = idx % TILE, c = idx / TILE;
      if (r >= m || c >= n || (lower && r + t.cdiag < c)) continue;
      double v = t.alpha * acc[e];
      if (t.beta != 0.0) v += t.beta * __ldcg(C + (int64_t)c * ldc + r);
      C[(int64_t)c * ldc + r] = v;
    }
  }
}

// One step of a block substitution (the triangular solves):
// C (m x n) = alpha A (m x K) B (K x n) + beta C, m <= 64, K <= TRSV_KMAX,
// with A a step operand computed before the sweep's chain ([-G_c | M_c] or
// [M_c; -H_c] stored transposed) and B adjacent x tiles, C one of them; or a
// narrow product of the solves (T_GEMM with aux[0] = GEMM_NARROW, n <= 32,
// A in the factor, C possibly added into with atomics).
// A's copies into shared memory (sA[k*TRSV_LA + r], k in [K, K4) zero) are
// issued before the task's mid waits [cdiag, nwait) (the x tiles it reads,
// written by the chain; all waits of a narrow product under the static
// order, since the factor is there from the start), so that they overlap the
// wait.  Then B is read, 8 right-hand sides at a time, a group's up to 12
// loads a thread in flight together (sB[j*TRSV_LB + k]), and each warp
// multiplies its 16 rows with FP64 MMAs in four chains.  A wait that runs
// out sets the timeout status and returns once the copies have landed.
// Bound by the hops of the chain: a step is an L2 round trip for B, the
// product and the release.  With B in three dependent groups of loads, one
// chain of MMAs and the products of the factor as 64 x 64 tiles, a pair of
// 40^3 solves took 1604 us with 8 right-hand sides, 1474 with one; now 1096
// and 1008.
template <int BUILD>
__device__ __forceinline__ bool is_narrow(const Task& t) {
  return BUILD == EB_SOLVE && t.op == T_GEMM && t.aux[0] == GEMM_NARROW;
}

static __device__ void run_trsv(const RunArgs& ra, const Task& t, double* smem, int ti, int& claim) {
  __shared__ int s_trsv_abort;
  constexpr int LA = TRSV_LA, LB = TRSV_LB;
  double* sA = smem;
  double* sB = smem + TRSV_KMAX * LA;
  const int m = t.m, n = t.n, K = t.k, K4 = (K + 3) & ~3;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  {
    // (rows from m on stay as they are: they meet only rows of the product
    // that are not stored)
    const double* __restrict__ X = ra.bases[t.a.base] + t.a.off;
    const int ld = t.a.ld;
    if (t.a.mode == OM_T) {
      // A(r, k) = X[r*ld + k]: a row a warp, consecutive lanes take consecutive k
      for (int r = warp; r < m; r += NTHREADS / 32)
        for (int k = lane; k < K4; k += 32)
          cp_async8_zfill(sA + k * LA + r, k < K ? X + (int64_t)r * ld + k : X, k < K);
    } else {
      for (int k = warp; k < K4; k += NTHREADS / 32)
        for (int r = lane; r < m; r += 32)
          cp_async8_zfill(sA + k * LA + r, k < K ? X + (int64_t)k * ld + r : X, k < K);
    }
    cp_async_commit();
  }
  if (tid == 0) {
    int abort = 0;
    // (under the dynamic schedule a narrow product is released on all its waits)
    const int w0 = t.op == T_TRSV ? t.cdiag : (ra.dynamic ? t.nwait : 0);
    for (int w = w0; w < t.nwait && !abort; w++) {
      const int2 wt = ra.waits[t.wait_off + w];
      int64_t spins = 0;
      unsigned ns = 16;
      while (ld_acquire(ra.counters + wt.x) < wt.y) {
        if (++spins > ra.spin_limit) {
          atomicCAS(&ra.ctl[1], 0, DE_TIMEOUT);
          atomicAdd(&ra.ctl[3], 1);
          abort = 1;
          break;
        }
        if ((spins & 15) == 0 && ld_volatile(&ra.ctl[1]) != 0) { abort = 1; break; }
        __nanosleep(ns);
        if (ns < 128) ns <<= 1;
      }
    }
    s_trsv_abort = abort;
    // a narrow product's dependencies are met now, not when it was claimed
    if (ra.trace && t.op == T_GEMM && !ra.dynamic) ra.trace[4 * (int64_t)ti + 1] = global_ns();
  }
  __syncthreads();
  if (s_trsv_abort) {
    cp_async_wait_all();
    return;
  }
  const double* __restrict__ Xb = ra.bases[t.b.base] + t.b.off;
  const int ldb = t.b.ld;  // B(j, k) = Xb[j*ldb + k] (x tiles, operand mode OM_T)
  double* __restrict__ C = ra.bases[t.c.base] + t.c.off;
  const int ldc = t.c.ld;
  const int jb = tid >> 4, kb = tid & 15;  // 16 threads a column of B
  for (int j0 = 0; j0 < n; j0 += 8) {
    const int nb = min(8, n - j0);
    {
      double v[TRSV_KMAX / 16];
      const double* __restrict__ src = Xb + (int64_t)(j0 + jb) * ldb;
#pragma unroll
      for (int e = 0; e < TRSV_KMAX / 16; e++) v[e] = (kb + 16 * e < K && jb < nb) ? __ldcg(src + kb + 16 * e) : 0.0;
#pragma unroll
      for (int e = 0; e < TRSV_KMAX / 16; e++) sB[jb * LB + kb + 16 * e] = v[e];
    }
    if (j0 == 0) cp_async_wait_all();
    __syncthreads();
    if (!ra.dynamic && j0 + 8 >= n && tid == 32) claim = atomicAdd(&ra.ctl[0], 1);
    if (16 * warp < m) {
      double acc[4][4];
#pragma unroll
      for (int e = 0; e < 4; e++) acc[e][0] = acc[e][1] = acc[e][2] = acc[e][3] = 0.0;
      const double* ar = sA + 16 * warp + g;
      const double* br = sB + g * LB;
      for (int k0 = 0; k0 < K4; k0 += 16) {
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int k = k0 + 4 * e + q;
          if (k0 + 4 * e < K4) dmma16(acc[e], ar[k * LA], ar[k * LA + 8], br[k]);
        }
      }
#pragma unroll
      for (int h = 0; h < 4; h++) {
        const int r = 16 * warp + g + ((h & 2) ? 8 : 0), j = 2 * q + (h & 1);
        if (r < m && j < nb) {
          double* cp = C + (int64_t)(j0 + j) * ldc + r;
          double val = t.alpha * ((acc[0][h] + acc[1][h]) + (acc[2][h] + acc[3][h]));
          if (t.cmode == CM_ATOMIC) {
            atomicAdd(cp, val);
          } else {
            if (t.beta != 0.0) val += t.beta * __ldcg(cp);
            *cp = val;
          }
        }
      }
    }
    __syncthreads();
  }
}

// C = alpha * M2 * (opA * opB^T), M2 = lower-triangular m x m tile (operand
// `c` of the task holds C; M2 is described by aux: base aux[0], ld aux[1],
// offset (aux[2] | aux[3] << 32)).
static __device__ void run_mrow(const RunArgs& ra, const Task& t, const SmemLayout& sm) {
  const Opnd A = make_opnd(ra, t.a), B = make_opnd(ra, t.b);
  double* C = ra.bases[t.c.base] + t.c.off;
  const int ldc = t.c.ld, m = t.m, n = t.n, K = t.k;
  const double alpha = t.alpha;
  const int64_t moff = (int64_t)(uint32_t)t.aux[2] | ((int64_t)t.aux[3] << 32);
  const double* __restrict__ M2 = ra.bases[t.aux[0]] + moff;
  const int ldm = t.aux[1];
  Acc acc;
  gemm_acc(A, B, m, n, K, sm, acc);
  // T = acc (m x n) into sm.B in B-stage layout: sB[k*LDS + n] = T(k, n)
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int h = 0; h < 4; h++) {
        int r, c;
        acc_coord(i, j, h, r, c);
        sm.B[r * LDS + c] = acc[i][j][h];
      }
  // sA[k*LDS + r] = M2(r, k) (lower triangle, zero padded), 32 loads in
  // flight per thread
  {
    double v[TILE * TILE / NTHREADS];
#pragma unroll
    for (int s2 = 0; s2 < TILE * TILE / NTHREADS; s2++) {
      const int idx = threadIdx.x + s2 * NTHREADS;
      const int r = idx % TILE, k = idx / TILE;
      v[s2] = (r < m && k < m && r >= k) ? __ldcg(M2 + (int64_t)k * ldm + r) : 0.0;
    }
#pragma unroll
    for (int s2 = 0; s2 < TILE * TILE / NTHREADS; s2++) {
      const int idx = threadIdx.x + s2 * NTHREADS;
      sm.A[(idx / TILE) * LDS + idx % TILE] = v[s2];
    }
  }
  __syncthreads();
  zero_acc(acc);
  mma_block(sm.A, sm.B, (m + 3) & ~3, acc);
  __syncthreads();
  store_acc(C, ldc, m, n, false, 0, alpha, 0.0, acc);
}

// ----------------------------------------------------------------- POTRF
// Cholesky of the b x b diagonal tile (operand a, in place, lower part
// written back); if aux[1] != 0 also writes M = L^{-1} (full b x b with
// zeros above the diagonal) to operand c.  A non-positive pivot records the
// LAPACK-style info aux[0] + j + 1 in ctl[2] (first writer wins).
//
// The tile is padded to 64 x 64 with an identity block (which factors and
// inverts to itself and does not couple to the leading b x b part), then
// processed in four 16-column blocks J:
//   (a) the 16x16 diagonal block is factored and inverted by one warp
//       (potrf_block16);
//   (b) panel below: L(r, J) = A(r, J) Minv_JJ^T            (DMMA)
//   (c) trailing lower triangle: A(r, c) -= L(r, J) L(c, J)^T (DMMA)
// and the inverse of the whole tile block row by block row:
//   M(I, :I) = -Minv_II (L(I, :I) M(:I, :I))                (DMMA)
// Warp 0 carries the dependent chain: in step J it computes the panel rows
// of block J (from block J-1), updates the diagonal block J, factors and
// inverts it.  Warps 1-3 meanwhile compute the other panel rows, update the
// trailing rows below block J (after a named barrier on warp 0's panel
// rows) and assemble block row J-1 of the inverse.  One block-wide barrier
// per step.  Beside the last block they also form its row's products
// L(I, :I) M(:I, :I) and store what is final, so that only the product with
// Minv_II and the last stores follow (they took 10.6k cycles, now 2.2k).
// (leading dimension of the tiles: with 4 mod 16 the MMA fragments, read
// along either index, meet no bank twice; TILE + 1 put four lanes on a bank)
constexpr int POTRF_LD = TILE + 4;
// sL, sM, an 8 x 8 tile of potrf_block16
constexpr int POTRF_SMEM_DOUBLES = 2 * TILE * POTRF_LD + 64;

// Phase timing for development builds (-DCHB_PROFILE_POTRF); compiled out
// otherwise.  Cycles per phase summed over tasks (thread 0's view):
// diagonal task 0 tile load, 1 panel rows and diagonal-block update,
// 2 16x16 factor and inverse, 4 end-of-step barrier, 5 L store,
// 6 last inverse block row, 7 M store, 8 first-part publish; look-ahead
// 16 mid waits, 17 tile load, 18 L' product, 19 L' store, 20 early signal,
// 21 L'L'^T product, 22 D update.  Task counts at 12 and 24.
#ifdef CHB_PROFILE_POTRF
static __device__ unsigned long long g_potrf_phase[32];
#define POTRF_STAMP(i)                                                    \
  do {                                                                    \
    long long now_ = clock64();                                           \
    if (threadIdx.x == 0) atomicAdd(&g_potrf_phase[i], now_ - stamp_);    \
    stamp_ = now_;                                                        \
  } while (0)
#define POTRF_COUNT(i)                                        \
  do {                                                        \
    if (threadIdx.x == 0) atomicAdd(&g_potrf_phase[i], 1ull); \
  } while (0)
#define POTRF_CLOCK_START long long stamp_ = clock64()
#else
#define POTRF_STAMP(i) \
  do {                 \
  } while (0)
#define POTRF_COUNT(i) \
  do {                 \
  } while (0)
#define POTRF_CLOCK_START \
  do {                    \
  } while (0)
#endif

// acc += A(16 x K) B(K x 8) (NEG: -=) with A(r, k) = pa[r + k*lda] and
// B(k, n) = pb[k*ksb + n*nsb] in shared memory (K a multiple of 8), in two
// chains of MMAs.
template <bool NEG>
__device__ __forceinline__ void warp_mma_16x8(double (&acc)[4], const double* pa, int lda, const double* pb,
                                              int ksb, int nsb, int K) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  double odd[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
  for (int k = 0; k < K; k += 8) {
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const double a0 = pa[g + (k + 4 * e + q) * lda], a1 = pa[g + 8 + (k + 4 * e + q) * lda];
      const double b0 = pb[(k + 4 * e + q) * ksb + g * nsb];
      dmma16(e ? odd : acc, NEG ? -a0 : a0, NEG ? -a1 : a1, b0);
    }
  }
#pragma unroll
  for (int h = 0; h < 4; h++) acc[h] += odd[h];
}

// FP64 MMA m8n8k4: A 8x4, a = A(g, q); B 4x8, b = B(q, g); C 8x8,
// c = C(g, 2q + {0, 1}), with g = lane / 4, q = lane % 4.
__device__ __forceinline__ void dmma8(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// Named barriers (id 0 is __syncthreads): bar.arrive publishes the
// caller's shared-memory writes to the threads that bar.sync on the id.
__device__ __forceinline__ void named_bar_arrive(int id, int nthreads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// Panel rows [r0, r0 + 16) of a 16-column block, in place:
// L(r, n) = sum_k A(r, k) Minv(n, k), both 16x8 halves by the calling warp
// (the block's columns at Lc, leading dimension LDL, Minv at Mb, LDM).
template <int LDL, int LDM>
__device__ __forceinline__ void potrf_panel_rows(double* Lc, const double* Mb, int r0) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  double a0[4] = {0.0, 0.0, 0.0, 0.0}, a1[4] = {0.0, 0.0, 0.0, 0.0};
  warp_mma_16x8<false>(a0, Lc + r0, LDL, Mb, LDM, 1, 16);
  warp_mma_16x8<false>(a1, Lc + r0, LDL, Mb + 8, LDM, 1, 16);
  __syncwarp();
  double* d = Lc + 2 * q * LDL + r0 + g;
#pragma unroll
  for (int h = 0; h < 4; h++) {
    d[(h & 1) * LDL + (h & 2) * 4] = a0[h];
    d[(8 + (h & 1)) * LDL + (h & 2) * 4] = a1[h];
  }
  __syncwarp();
}

// Lower-triangle part of the 16x8 tile at (r0, c0) minus the rank-16
// product of the panel block at jp: A(r, c) -= sum_k L(r, jp + k) L(c, jp + k).
template <int LDL>
__device__ __forceinline__ void potrf_syrk_tile(double* sL, int jp, int r0, int c0) {
  constexpr int LD = LDL;
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int r = r0 + g, c = c0 + 2 * q;
  double ac[4] = {sL[c * LD + r], sL[(c + 1) * LD + r], sL[c * LD + r + 8], sL[(c + 1) * LD + r + 8]};
  warp_mma_16x8<true>(ac, sL + jp * LD + r0, LD, sL + jp * LD + c0, LD, 1, 16);
  if (r >= c) sL[c * LD + r] = ac[0];
  if (r >= c + 1) sL[(c + 1) * LD + r] = ac[1];
  if (r + 8 >= c) sL[c * LD + r + 8] = ac[2];
  if (r + 8 >= c + 1) sL[(c + 1) * LD + r + 8] = ac[3];
}

#include "block16.cuh"

// Block row I of the inverse, column tiles of 8 columns: first the products
// T = L(I, :I) M(:I, tile) (K = 16 I) in the tile's place in sM, then, once
// the diagonal block's inverse is there, M(I, tile) = -Minv_II T in place.
__device__ __forceinline__ void potrf_inv_products(const double* sL, double* sM, int I, int tj) {
  constexpr int LD = POTRF_LD;
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3, i0 = 16 * I;
  double ac[4] = {0.0, 0.0, 0.0, 0.0};
  warp_mma_16x8<false>(ac, sL + i0, LD, sM + (8 * tj) * LD, 1, LD, i0);
  double* d = sM + (8 * tj + 2 * q) * LD + i0 + g;
  d[0] = ac[0];
  d[LD] = ac[1];
  d[8] = ac[2];
  d[LD + 8] = ac[3];
}
__device__ __forceinline__ void potrf_inv_finish(double* sM, int I, int tj) {
  constexpr int LD = POTRF_LD;
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3, i0 = 16 * I;
  double am[4] = {0.0, 0.0, 0.0, 0.0};
  warp_mma_16x8<true>(am, sM + i0 * LD + i0, LD, sM + (8 * tj) * LD + i0, 1, LD, 16);
  __syncwarp();
  double* d = sM + (8 * tj + 2 * q) * LD + i0 + g;
  d[0] = am[0];
  d[LD] = am[1];
  d[8] = am[2];
  d[LD + 8] = am[3];
}

// Columns [c0, c1), rows [r0, b) of a tile in shared memory to global memory
// (lower: on and below the diagonal), by the warps first, first + 1, ... 3, a
// column a warp.
__device__ __forceinline__ void potrf_store(double* __restrict__ X, int64_t ldx, const double* sX, int b, int c0,
                                            int c1, int r0, bool lower, int first) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < first) return;
#pragma unroll 4
  for (int c = c0 + warp - first; c < c1; c += NTHREADS / 32 - first) {
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int r = lane + 32 * e;
      if (r >= r0 && r < b && (!lower || r >= c)) X[c * ldx + r] = sX[c * POTRF_LD + r];
    }
  }
}

// acc[j] += A(16w : 16w + 16, :) B(8j : 8j + 8, :)^T for the calling warp w
// (rows of the 64x64 product by 16-row block, all eight 8-column tiles),
// A(r, k) at sA[k * POTRF_LD + r], B(c, k) at sB[k * POTRF_LD + c], B lower
// triangular: tile j takes only k < 8 (j + 1), so every warp issues 72 of
// the 128 MMAs of a full 64-deep product.
__device__ __forceinline__ void mma_rows_lower_b(const double* sA, const double* sB, double (&acc)[8][4]) {
  constexpr int LD = POTRF_LD;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  const int r0 = 16 * warp + g;
  // (unrolled: with j >= kb a branch, every MMA waited for its own load)
#pragma unroll
  for (int kb = 0; kb < TILE / 8; kb++) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int k = 8 * kb + 4 * h + q;
      const double a0 = sA[k * LD + r0], a1 = sA[k * LD + r0 + 8];
#pragma unroll
      for (int j = 0; j < TILE / 8; j++)
        if (j >= kb) dmma16(acc[j], a0, a1, sB[k * LD + 8 * j + g]);
    }
  }
}

// The 20 16x8 tiles on or below the diagonal of a 64x64 product, five per
// warp: tile t lies in 16-row block rb and 8-column block j, listed by row
// block 3, 2, 1, 0 (8, 6, 4 and 2 tiles).
__device__ __forceinline__ void lower_tile(int t, int& rb, int& j) {
  rb = t < 8 ? 3 : (t < 14 ? 2 : (t < 18 ? 1 : 0));
  j = t - (t < 8 ? 0 : (t < 14 ? 8 : (t < 18 ? 14 : 18)));
}

// acc[i] += A(rows of tile i) A(columns of tile i)^T over k < kn for the
// calling warp's five lower tiles (tile 5 w + i), A(r, k) at
// sA[k * POTRF_LD + r]: 80 MMAs per warp instead of 128 for the full square.
__device__ __forceinline__ void mma_lower_tiles(const double* sA, int kn, double (&acc)[5][4]) {
  constexpr int LD = POTRF_LD;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  int ro[5], co[5];
#pragma unroll
  for (int i = 0; i < 5; i++) {
    int rb, j;
    lower_tile(5 * warp + i, rb, j);
    ro[i] = 16 * rb + g;
    co[i] = 8 * j + g;
  }
#pragma unroll 4
  for (int kk = 0; kk < kn; kk += 4) {
    const double* ak = sA + (kk + q) * LD;
#pragma unroll
    for (int i = 0; i < 5; i++) dmma16(acc[i], ak[ro[i]], ak[ro[i] + 8], ak[co[i]]);
  }
}

// Look-ahead part of a fused diagonal task (T_POTRF with k = m2 > 0, run
// after the factorisation of the b = 64 tile; sL holds L_cc and sM holds
// M = L_cc^{-1}, both with leading dimension POTRF_LD):
//   1. wait for the task's mid waits (waits [cdiag, nwait): the updates of
//      tiles (c+1, c) and (c+1, c+1) from the previous column block);
//   2. L' = A(c+1, c) M^T  (m2 x b; A staged into sL), stored in place and
//      kept in sL;
//   3. early signal aux[3] - 1 (the readers of L');
//   4. A(c+1, c+1) -= L' L'^T (lower part, m2 x m2).
// The tiles lie at a.off + b (panel) and a.off + b*lda + b (diagonal).
__device__ __forceinline__ void potrf_lookahead(const RunArgs& ra, const Task& t, double* smem) {
  __shared__ int s_la_abort;
  constexpr int LD = POTRF_LD;
  double* sL = smem;
  const double* sM = smem + TILE * LD;
  const int b = t.m, m2 = t.k, lda = t.a.ld;
  double* __restrict__ X = ra.bases[t.a.base] + t.a.off;
  double* __restrict__ P = X + b;
  double* __restrict__ D = X + (int64_t)b * lda + b;
  const int tid = threadIdx.x;
  POTRF_CLOCK_START;
  POTRF_COUNT(24);
  __syncthreads();
  if (tid == 0) {
    int abort = 0;
    for (int w = t.cdiag; w < t.nwait && !abort; w++) {
      const int2 wt = ra.waits[t.wait_off + w];
      int64_t spins = 0;
      unsigned ns = 16;
      while (ld_acquire(ra.counters + wt.x) < wt.y) {
        if (++spins > ra.spin_limit) {
          atomicCAS(&ra.ctl[1], 0, DE_TIMEOUT);
          atomicAdd(&ra.ctl[3], 1);
          abort = 1;
          break;
        }
        if ((spins & 15) == 0 && ld_volatile(&ra.ctl[1]) != 0) { abort = 1; break; }
        __nanosleep(ns);
        if (ns < 128) ns <<= 1;
      }
    }
    s_la_abort = abort;
  }
  __syncthreads();
  if (s_la_abort) return;
  POTRF_STAMP(16);
  // A(c+1, c) into sL (rows >= m2 zero)
  {
    double v[TILE * TILE / NTHREADS];
#pragma unroll
    for (int s2 = 0; s2 < TILE * TILE / NTHREADS; s2++) {
      const int idx = tid + s2 * NTHREADS;
      const int r = idx % TILE, c = idx / TILE;
      v[s2] = (r < m2 && c < b) ? __ldcg(P + (int64_t)c * lda + r) : 0.0;
    }
#pragma unroll
    for (int s2 = 0; s2 < TILE * TILE / NTHREADS; s2++) {
      const int idx = tid + s2 * NTHREADS;
      sL[(idx / TILE) * LD + idx % TILE] = v[s2];
    }
  }
  __syncthreads();
  POTRF_STAMP(17);
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  {
    double acc[TILE / 8][4];
#pragma unroll
    for (int j = 0; j < TILE / 8; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0;
    mma_rows_lower_b(sL, sM, acc);  // b = TILE: only the last block column of a front has b < TILE
    __syncthreads();
    POTRF_STAMP(18);
    // L' into sL and in place
#pragma unroll
    for (int j = 0; j < TILE / 8; j++)
#pragma unroll
      for (int h = 0; h < 4; h++) {
        const int r = 16 * warp + g + ((h & 2) ? 8 : 0), c = 8 * j + 2 * q + (h & 1);
        const double v = (r < m2) ? acc[j][h] : 0.0;
        sL[c * LD + r] = v;
        if (r < m2 && c < b) P[(int64_t)c * lda + r] = v;
      }
  }
  __syncthreads();
  POTRF_STAMP(19);
  if (t.aux[3] > 0) {
    if (ra.dynamic) {
      const int c = t.aux[3] - 1;
      if (tid < 32) release_list(ra, __ldg(ra.succ_off + c), __ldg(ra.succ_off + c + 1), nullptr, false, nullptr);
    } else if (tid == 0) {
      red_release_add(ra.counters + (t.aux[3] - 1), 1);
    }
  }
  POTRF_STAMP(20);
  // D -= L' L'^T on and below the diagonal; D is loaded beside the product
  double old[5][4];
#pragma unroll
  for (int i = 0; i < 5; i++) {
    int rb, j;
    lower_tile(5 * warp + i, rb, j);
#pragma unroll
    for (int h = 0; h < 4; h++) {
      const int r = 16 * rb + g + ((h & 2) ? 8 : 0), c = 8 * j + 2 * q + (h & 1);
      old[i][h] = (r < m2 && r >= c) ? __ldcg(D + (int64_t)c * lda + r) : 0.0;
    }
  }
  double acc[5][4];
#pragma unroll
  for (int i = 0; i < 5; i++) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0;
  mma_lower_tiles(sL, b, acc);
  POTRF_STAMP(21);
#pragma unroll
  for (int i = 0; i < 5; i++) {
    int rb, j;
    lower_tile(5 * warp + i, rb, j);
#pragma unroll
    for (int h = 0; h < 4; h++) {
      const int r = 16 * rb + g + ((h & 2) ? 8 : 0), c = 8 * j + 2 * q + (h & 1);
      if (r < m2 && r >= c) D[(int64_t)c * lda + r] = old[i][h] - acc[i][h];
    }
  }
  POTRF_STAMP(22);
}

static __device__ void run_potrf(const RunArgs& ra, const Task& t, double* smem, int ti) {
  const int b = t.m;
  constexpr int LD = POTRF_LD;
  double* sL = smem;               // [col][row], lower; upper part zero
  double* sM = sL + TILE * LD;     // inverse, upper part zero
  double* sT = sM + TILE * LD;     // staging of potrf_block16
  double* __restrict__ X = ra.bases[t.a.base] + t.a.off;
  const int lda = t.a.ld;
  const int info_base = t.aux[0];
  const bool want_inv = t.aux[1] != 0;
  const bool factor = t.aux[2] == 0;  // aux[2] != 0: the tile already holds L; invert only
  double* __restrict__ Mout = want_inv ? ra.bases[t.c.base] + t.c.off : nullptr;
  const int ldm = t.c.ld;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  POTRF_CLOCK_START;
  POTRF_COUNT(12);
  {
    double v[TILE * TILE / NTHREADS];
#pragma unroll
    for (int s2 = 0; s2 < TILE * TILE / NTHREADS; s2++) {
      const int idx = tid + s2 * NTHREADS;
      const int r = idx % TILE, c = idx / TILE;
      v[s2] = (r < b && c < b && r >= c) ? __ldcg(X + (int64_t)c * lda + r) : (r == c ? 1.0 : 0.0);
    }
#pragma unroll
    for (int s2 = 0; s2 < TILE * TILE / NTHREADS; s2++) {
      const int idx = tid + s2 * NTHREADS;
      sL[(idx / TILE) * LD + idx % TILE] = (idx % TILE >= idx / TILE) ? v[s2] : 0.0;
      sM[(idx / TILE) * LD + idx % TILE] = 0.0;
    }
  }
  __syncthreads();
  POTRF_STAMP(0);
  // only the 16-column blocks that meet the b x b tile (the padding is the
  // identity and is neither factored nor inverted)
  const int NJ = (b + 15) >> 4, NB = 16 * NJ;
#pragma unroll 1
  for (int J = 0; J < NJ; J++) {
    const int j0 = 16 * J, j1 = j0 + 16, jp = j0 - 16;
    const bool panel = factor && J > 0;     // panel of block J-1 and the updates it feeds
    const bool below = panel && J < NJ - 1; // rows below block J to update
    if (warp == 0) {
      if (panel) {
        potrf_panel_rows<LD, LD>(sL + jp * LD, sM + jp * LD + jp, j0);
        if (below) named_bar_arrive(1, NTHREADS);
        else if (want_inv) named_bar_arrive(3, NTHREADS);  // the last block
        potrf_syrk_tile<LD>(sL, jp, j0, j0);
        potrf_syrk_tile<LD>(sL, jp, j0, j0 + 8);
        __syncwarp();
      }
      POTRF_STAMP(1);
      const int bad = potrf_block16<POTRF_LD, POTRF_LD>(sL + j0 * LD + j0, sM + j0 * LD + j0, sT, factor);
      if (lane == 0 && bad >= 0 && j0 + bad < b) atomicCAS(&ra.ctl[2], 0, info_base + j0 + bad + 1);
      POTRF_STAMP(2);
    } else {
      if (below) {
        const int rb = j0 + 16 * warp;  // warps 1, 2: the panel rows below block J
        if (rb < NB) potrf_panel_rows<LD, LD>(sL + jp * LD, sM + jp * LD + jp, rb);
        named_bar_sync(1, NTHREADS);
        // rows >= j1, columns >= j0, lower part, from the panel of block J-1
        const int nti = (NB - j1) / 16, ntj = (NB - j0) / 8;
        for (int tt = warp - 1; tt < nti * ntj; tt += NTHREADS / 32 - 1) {
          const int r0 = j1 + 16 * (tt / ntj), c0 = j0 + 8 * (tt % ntj);
          if (c0 <= r0 + 15) potrf_syrk_tile<LD>(sL, jp, r0, c0);
        }
      }
      if (want_inv && J >= 2)
        for (int tj = warp - 1; tj < 2 * (J - 1); tj += NTHREADS / 32 - 1) {
          potrf_inv_products(sL, sM, J - 1, tj);
          __syncwarp();
          potrf_inv_finish(sM, J - 1, tj);
        }
      if (J == NJ - 1 && J > 0) {
        // beside the last block: its row's products, and the stores of what
        // is final (columns of L before block J - 1, rows of the inverse
        // before row J)
        if (want_inv) {
          named_bar_sync(2, NTHREADS - 32);  // the inverse's rows before J
          if (factor) named_bar_sync(3, NTHREADS);  // row J of L up to block J - 1 (warp 0)
          for (int tj = warp - 1; tj < 2 * J; tj += NTHREADS / 32 - 1) potrf_inv_products(sL, sM, J, tj);
        }
        if (factor) potrf_store(X, lda, sL, b, 0, jp, 0, true, 1);
        if (want_inv) potrf_store(Mout, ldm, sM, j0, 0, j0, 0, false, 1);
      }
    }
    __syncthreads();
    POTRF_STAMP(4);
  }
  // the last block row of the inverse, and what is left to store
  if (want_inv)
    for (int tj = warp; tj < 2 * (NJ - 1); tj += NTHREADS / 32) potrf_inv_finish(sM, NJ - 1, tj);
  POTRF_STAMP(6);
  const int jl = 16 * (NJ - 1);
  if (factor) potrf_store(X, lda, sL, b, max(jl - 16, 0), b, 0, true, 0);
  POTRF_STAMP(5);
  if (!want_inv) return;
  __syncthreads();
  potrf_store(Mout, ldm, sM, b, 0, jl, jl, false, 0);
  potrf_store(Mout, ldm, sM, b, jl, b, 0, false, 0);
  POTRF_STAMP(7);
  if (t.k > 0) {
    // first part done: L_cc and M_cc are stored; the task's own waiters go
    __syncthreads();
    if (ra.dynamic) {
      if (tid < 32) release_list(ra, __ldg(ra.succ_off + ti), __ldg(ra.succ_off + ti + 1), nullptr, false, nullptr);
    } else if (tid == 0) {
      red_release_add(ra.counters + ti, 1);
    }
    POTRF_STAMP(8);
    potrf_lookahead(ra, t, smem);
  }
}

// ------------------------------------------------------------ assembly
// Extend-add for front k = aux[0], front columns [aux[1], aux[2]):
//   * zero the columns of the update block U_k that fall in the range
//     (if aux[3] & 1);
//   * for each child, last to first (the order the reference pops its update
//     stack, cholesky.c:41-52), add U_child(i, q) into F(r[i], r[q]) for the
//     child columns q whose relative index r[q] lies in the range.
// F(i, j) is the front panel (operand a: nj rows, ld a.ld) for j < nn, else
// the update block U_k (operand c, ld c.ld).  One warp per child column;
// children are applied one after the other.
// A child's relative indices, staged in shared memory once per child when
// they fit (one coalesced pass), so that each scattered access costs one
// round trip instead of two; otherwise read from global memory.
constexpr int RIDX_SMEM_MAX = ENGINE_SMEM_BASE_DOUBLES * 2;  // int32 entries in the base shared memory
__device__ __forceinline__ const int32_t* stage_ridx(const int32_t* __restrict__ r, int N, double* smem) {
  if (N > RIDX_SMEM_MAX) return r;
  int32_t* sr = reinterpret_cast<int32_t*>(smem);
  for (int i = threadIdx.x; i < N; i += NTHREADS) sr[i] = __ldg(r + i);
  __syncthreads();
  return sr;
}

constexpr int GATHER_INFLIGHT = 8;  // scattered elements in flight per lane
// Columns of at most 64 rows (a batch of small matrices has little else)
// leave most of those eight empty, and a column is one L2 round trip: so four
// columns at a time, two elements of each.  256 uneven grids, an extend-add
// task 17.0 -> 14.0 us, an extraction 10.4 -> 6.4.
constexpr int ASM_COLS = 4, ASM_ROWS = 2;

static __device__ void run_asm(const RunArgs& ra, const Task& t, double* smem) {
  const FrontDesc f = ra.fronts[t.aux[0]];
  const int j0 = t.aux[1], j1 = t.aux[2];
  const bool zero_u = (t.aux[3] & 1) != 0;
  double* __restrict__ P = ra.bases[t.a.base] + t.a.off;
  const int ldp = t.a.ld;
  double* __restrict__ Uk = ra.bases[t.c.base] + t.c.off;
  const int ldu = t.c.ld;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (zero_u) {
    for (int j = max(j0, f.nn) + warp; j < j1; j += NTHREADS / 32) {
      const int jj = j - f.nn;
      for (int i = jj + lane; i < f.na; i += 32) Uk[(int64_t)jj * ldu + i] = 0.0;
    }
  }
  __syncthreads();
  for (int l = f.chend - 1; l >= f.chbeg; l--) {
    const FrontDesc ch = ra.fronts[ra.chidx[l]];
    const int N = ch.na;
    const int32_t* r = stage_ridx(ra.relidx + ch.relptr, N, smem);
    const double* __restrict__ Uc = ra.bases[B_WS] + t.off2 + ch.upd;
    // child columns with r[q] in [j0, j1): r is strictly increasing
    int lo = 0, hi = N;
    while (lo < hi) { int mid = (lo + hi) >> 1; if (r[mid] < j0) lo = mid + 1; else hi = mid; }
    const int q0 = lo;
    hi = N;
    while (lo < hi) { int mid = (lo + hi) >> 1; if (r[mid] < j1) lo = mid + 1; else hi = mid; }
    const int q1 = lo;
    // a warp takes ASM_COLS columns at once, the first 32 * ASM_ROWS rows of
    // each in one round of loads, then what is left of each column
    auto column = [&](int q) {
      const int col = r[q];
      return (col < f.nn) ? P + (int64_t)col * ldp : Uk + (int64_t)(col - f.nn) * ldu - f.nn;
    };
    for (int qb = q0 + warp; qb < q1; qb += ASM_COLS * (NTHREADS / 32)) {
      double u[ASM_COLS][ASM_ROWS], d[ASM_COLS][ASM_ROWS];
      double* at[ASM_COLS][ASM_ROWS];
#pragma unroll
      for (int v = 0; v < ASM_COLS; v++) {
        const int q = qb + v * (NTHREADS / 32);
        double* const dst = q < q1 ? column(q) : nullptr;
#pragma unroll
        for (int e = 0; e < ASM_ROWS; e++) {
          const int i = q + lane + 32 * e;
          const bool ok = q < q1 && i < N;
          at[v][e] = ok ? dst + r[i] : nullptr;
          u[v][e] = ok ? __ldcg(Uc + (int64_t)q * N + i) : 0.0;
          d[v][e] = ok ? __ldcg(at[v][e]) : 0.0;
        }
      }
#pragma unroll
      for (int v = 0; v < ASM_COLS; v++)
#pragma unroll
        for (int e = 0; e < ASM_ROWS; e++)
          if (at[v][e]) *at[v][e] = d[v][e] + u[v][e];
      for (int v = 0; v < ASM_COLS; v++) {
        const int q = qb + v * (NTHREADS / 32);
        if (q >= q1 || N - q <= 32 * ASM_ROWS) break;
        double* const dst = column(q);
        const double* __restrict__ src = Uc + (int64_t)q * N;
        for (int i0 = q + 32 * ASM_ROWS; i0 < N; i0 += GATHER_INFLIGHT * 32) {
          int ri[GATHER_INFLIGHT];
          double uu[GATHER_INFLIGHT], dd[GATHER_INFLIGHT];
#pragma unroll
          for (int e = 0; e < GATHER_INFLIGHT; e++) {
            const int i = i0 + lane + 32 * e;
            ri[e] = (i < N) ? r[i] : -1;
            uu[e] = (i < N) ? __ldcg(src + i) : 0.0;
            dd[e] = (i < N) ? __ldcg(dst + ri[e]) : 0.0;
          }
#pragma unroll
          for (int e = 0; e < GATHER_INFLIGHT; e++)
            if (ri[e] >= 0) dst[ri[e]] = dd[e] + uu[e];
        }
      }
    }
    __syncthreads();
  }
}

// A whole small cholesky front (T_FRONT, nj <= TILE; cholesky.c:33-72 for
// one node) in shared memory: F(r, c) at F[c * FRONT_LD + r], lower part, the
// nn pivot columns padded with an identity to NP, a multiple of 16, and the
// separators from row and column NP on.
//   1. F = the block's lower trapezoid, zero elsewhere;
//   2. the children's update matrices added, last child first;
//   3. the pivot columns eliminated in 16-column blocks, the separators as
//      further rows below them, which leaves L11, L21 and the Schur
//      complement F22 - L21 L21^T: a diagonal block by a warp
//      (potrf_block16), the rows below it by substitution, a lane per row,
//      the update of the rest by MMAs;
//   4. the rows below replaced by W = L21 L11^{-1} (the reference's layout
//      of the off-diagonal block): by 16-column blocks, last to first,
//      W_J = (L21_J - sum_{K > J} W_K L(K, J)) L(J, J)^{-1}, the sum by MMAs
//      and the rest by substitution, a warp per 16 rows;
//   5. the block and the update matrix (operand c) written back.
// A non-positive pivot records ctl[2] = j + 1 and continues with 1.
// Bound by its chain of steps: with a barrier a pivot and scalar updates a
// front of 2-D 30^2 (merged) took 34.2 us, in blocks 11.4.
// (Substitution, not products with the inverses of the blocks: those leave a
// residual that grows with the block's condition, 7e-15 at 4e3.)
constexpr int FRONT_LD = TILE + 20;             // up to 80 rows; 4 mod 16
constexpr int FRONT_D = (TILE + 16) * FRONT_LD; // 1 / L(j, j)
static_assert(FRONT_D + TILE + TILE / 2 <= ENGINE_SMEM_BASE_DOUBLES,
              "small fronts exceed the engine's shared memory");

// Up to this many pivots are eliminated one by one (a padded block of 16 costs
// about as much as six of them; 4 and 8 measured the same on 2-D grids, 12
// 4 % slower).
constexpr int FRONT_SCALAR_NN = 4;

// Steps 3 and 4 of run_front for a few pivots, column by column with one
// barrier a pivot: pivot j updates the trailing part with its unscaled
// column, F(i, c) -= F(i, j) F(c, j) / d_j, and the column itself is scaled by
// 1 / L(j, j) in the next pivot's phase (nobody reads it then);
// 1 / L(j, j) = rsqrt(d_j), kept (in w, with L(j, j)) for the solve.
__device__ __forceinline__ void front_scalar(const RunArgs& ra, double* F, double* w, int nn, int nj) {
  constexpr int LD = FRONT_LD, NW = NTHREADS / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* rl = w;
  double* lj = w + FRONT_SCALAR_NN;
  int first_bad = -1;
  for (int j = 0; j < nn; j++) {
    const double d = F[j * LD + j];
    const bool bad = !(d > 0.0);
    if (bad && first_bad < 0) first_bad = j;
    const double rs = rsqrt(bad ? 1.0 : d), rd = rs * rs;
    if (j > 0) {
      const double rp = rl[j - 1];
      for (int i = j + tid; i < nj; i += NTHREADS) F[(j - 1) * LD + i] *= rp;
    }
    if (tid == 0) {
      rl[j] = rs;  // read from the next phase on
      lj[j] = (bad ? 1.0 : d) * rs;
    }
    for (int c = j + 1 + warp; c < nj; c += NW) {
      const double fc = F[j * LD + c] * rd;
      for (int i = c + lane; i < nj; i += 32) F[c * LD + i] -= F[j * LD + i] * fc;
    }
    __syncthreads();
  }
  for (int i = nn + tid; i < nj; i += NTHREADS) F[(nn - 1) * LD + i] *= rl[nn - 1];
  for (int j = tid; j < nn; j += NTHREADS) F[j * LD + j] = lj[j];
  if (tid == 0 && first_bad >= 0) atomicCAS(&ra.ctl[2], 0, first_bad + 1);
  __syncthreads();
  // W = L21 L11^{-1}, one row per thread, right-looking: w_j = t_j / L(j, j),
  // then t_j' -= w_j L(j, j') for j' < j (independent updates)
  for (int i = nn + tid; i < nj; i += NTHREADS)
    for (int j = nn - 1; j >= 0; j--) {
      const double v = F[j * LD + i] * rl[j];
      F[j * LD + i] = v;
      for (int l2 = 0; l2 < j; l2++) F[l2 * LD + i] -= v * F[l2 * LD + j];
    }
  __syncthreads();
}

// Rows [r0, r0 + 16) below the diagonal block in columns and rows j0 .. j0 + 16
// of F, in place: x L(J, J)^T = A(r, J), lane mod 16 a row, rd = 1 / L(j, j).
// The padding (columns from cols on, rows nn .. NP) stays zero whatever the
// rows hold.
__device__ __forceinline__ void front_panel_rows(double* F, const double* rd, int j0, int r0, int cols, int nn,
                                                 int NP) {
  constexpr int LD = FRONT_LD;
  const int r = r0 + (threadIdx.x & 15);
  double* const f = F + j0 * LD + r;
  const double* const d = F + j0 * LD + j0;
  double x[16];
#pragma unroll
  for (int c = 0; c < 16; c++) x[c] = f[c * LD];
#pragma unroll
  for (int j = 0; j < 16; j++) {
    x[j] *= rd[j];
#pragma unroll
    for (int c = (j + 1) & ~1; c < 16; c += 2) {
      const double2 l = *reinterpret_cast<const double2*>(d + j * LD + c);
      if (c > j) x[c] = fma(-x[j], l.x, x[c]);
      x[c + 1] = fma(-x[j], l.y, x[c + 1]);
    }
  }
  const bool row = r < nn || r >= NP;
  __syncwarp();
  if ((threadIdx.x & 16) == 0) {
#pragma unroll
    for (int c = 0; c < 16; c++) f[c * LD] = (row && c < cols) ? x[c] : 0.0;
  }
  __syncwarp();
}

// x := x L^{-1} for a row x of 16 columns, last to first, L(j, c) = d[c * LD + j],
// rd = 1 / L(j, j); the columns from cols on are zero.
template <int LD>
__device__ __forceinline__ void solve_row16(double (&x)[16], const double* d, const double* rd, int cols) {
#pragma unroll
  for (int j = 15; j >= 0; j--) {
    x[j] = j < cols ? x[j] * rd[j] : 0.0;
#pragma unroll
    for (int c = 0; c < j; c++) x[c] = fma(-x[j], d[c * LD + j], x[c]);
  }
}

// The same rows' x L(J, J) = B(r, J).
__device__ __forceinline__ void front_solve_rows(double* F, const double* rd, int j0, int r0, int cols) {
  constexpr int LD = FRONT_LD;
  double* const f = F + j0 * LD + r0 + (threadIdx.x & 15);
  double x[16];
#pragma unroll
  for (int c = 0; c < 16; c++) x[c] = f[c * LD];
  solve_row16<LD>(x, F + j0 * LD + j0, rd, cols);
  __syncwarp();
  if ((threadIdx.x & 16) == 0) {
#pragma unroll
    for (int c = 0; c < 16; c++) f[c * LD] = x[c];
  }
  __syncwarp();
}

static __device__ void run_front(const RunArgs& ra, const Task& t, double* smem) {
  constexpr int LD = FRONT_LD, NW = NTHREADS / 32;
  const FrontDesc f = ra.fronts[t.aux[0]];
  const int nn = f.nn, na = f.na, nj = f.nj;
  const bool blocked = nn > FRONT_SCALAR_NN;
  const int NJ = blocked ? (nn + 15) >> 4 : 0, NP = blocked ? 16 * NJ : nn, pad = NP - nn;
  const int NB = (NP + na + 15) >> 4, NF = blocked ? 16 * NB : nj;  // order of F
  double* F = smem;
  double* rd = smem + FRONT_D;        // 1 / L(j, j)
  int* sr = reinterpret_cast<int*>(rd + TILE);
  double* __restrict__ X = ra.bases[t.a.base] + t.a.off;
  double* __restrict__ U = ra.bases[t.c.base] + t.c.off;
  const int ldu = t.c.ld;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // F by column: a pivot column's trapezoid, an identity column or zeros
  // (four columns' loads at a time: a load is not moved above a store to
  // shared memory)
  for (int c4 = warp; c4 < NF; c4 += 4 * NW) {
    double v[4][3];
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int e = 0; e < 3; e++) {
        const int c = c4 + u * NW, r = lane + 32 * e;  // row of F; of the block: r or r - pad
        const int rb = r < NP ? r : r - pad;
        const bool in = c < nn && r >= c && (r < nn || (r >= NP && rb < nj));
        v[u][e] = in ? __ldcg(X + (int64_t)c * nj + rb) : (r == c && c >= nn && c < NP ? 1.0 : 0.0);
      }
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int e = 0; e < 3; e++) {
        const int c = c4 + u * NW, r = lane + 32 * e;
        if (c < NF && r < NF) F[c * LD + r] = v[u][e];
      }
  }
  __syncthreads();
  // the children's update matrices, last child first: its relative indices
  // staged in shared memory, then the lower triangle of U_c flattened over
  // the threads with FRONT_E loads in flight per thread (a child's entries
  // land on distinct front entries)
  constexpr int FRONT_E = 8;
  for (int l = f.chend - 1; l >= f.chbeg; l--) {
    const FrontDesc ch = ra.fronts[ra.chidx[l]];
    const int Nc = ch.na, tot = Nc * Nc;
    const int32_t* __restrict__ rr = ra.relidx + ch.relptr;
    const double* __restrict__ Uc = ra.bases[B_WS] + t.off2 + ch.upd;
    if (tid < Nc) {
      const int r = __ldg(rr + tid);
      sr[tid] = r < nn ? r : r + pad;
    }
    __syncthreads();
    for (int base = 0; base < tot; base += FRONT_E * NTHREADS) {
      double v[FRONT_E];
      int dst[FRONT_E];
#pragma unroll
      for (int e = 0; e < FRONT_E; e++) {
        const int idx = base + tid + e * NTHREADS, q = idx / Nc, i = idx - q * Nc;
        const bool ok = idx < tot && i >= q;
        v[e] = ok ? __ldcg(Uc + idx) : 0.0;
        dst[e] = ok ? sr[q] * LD + sr[i] : -1;
      }
#pragma unroll
      for (int e = 0; e < FRONT_E; e++)
        if (dst[e] >= 0) F[dst[e]] += v[e];
    }
    __syncthreads();
  }
  if (!blocked) {
    front_scalar(ra, F, rd, nn, nj);
  }
  // step J: warp 0 the panel rows, the update and the factor of diagonal
  // block J, warps 1-3 the other panel rows of block J - 1 and the updates
  // below (one more step, of all warps, for the separators' rows and columns)
#pragma unroll 1
  for (int J = 0; J < NJ; J++) {
    const int j0 = 16 * J, jp = j0 - 16;
    if (warp == 0) {
      if (J > 0) {
        front_panel_rows(F, rd + jp, jp, j0, 16, nn, NP);
        named_bar_arrive(1, NTHREADS);
        potrf_syrk_tile<LD>(F, jp, j0, j0);
        potrf_syrk_tile<LD>(F, jp, j0, j0 + 8);
        __syncwarp();
      }
      const int cols = min(16, nn - j0);
      const int bad = potrf_block16<LD, LD, false>(F + j0 * LD + j0, rd + j0, nullptr, true, cols);
      if (lane == 0 && bad >= 0 && bad < cols) atomicCAS(&ra.ctl[2], 0, j0 + bad + 1);
      if (cols < 16) {  // the padded rows of the block, whatever the pivots left there
        __syncwarp();
        for (int i = lane; i < 256; i += 32)
          if ((i >> 4) < cols && (i & 15) >= cols) F[(j0 + (i >> 4)) * LD + j0 + (i & 15)] = 0.0;
      }
    } else if (J > 0) {
      for (int rb = J + warp; rb < NB; rb += NW - 1) front_panel_rows(F, rd + jp, jp, 16 * rb, 16, nn, NP);
      named_bar_sync(1, NTHREADS);
      int at = 0;
      for (int I = J + 1; I < NB; I++)
        for (int c0 = j0; c0 < 16 * I + 16; c0 += 8)
          if (at++ % (NW - 1) == warp - 1) potrf_syrk_tile<LD>(F, jp, 16 * I, c0);
    }
    __syncthreads();
  }
  if (blocked && na > 0) {
    const int jp = NP - 16;
    for (int rb = NJ + warp; rb < NB; rb += NW) front_panel_rows(F, rd + jp, jp, 16 * rb, nn - jp, nn, NP);
    __syncthreads();
    int at = 0;
    for (int I = NJ; I < NB; I++)
      for (int c0 = NP; c0 < 16 * I + 16; c0 += 8)
        if (at++ % NW == warp) potrf_syrk_tile<LD>(F, jp, 16 * I, c0);
    __syncthreads();
    const int g = lane >> 2, q = lane & 3;
    for (int rb = NJ + warp; rb < NB; rb += NW) {
      const int r0 = 16 * rb;
#pragma unroll 1
      for (int J = NJ - 1; J >= 0; J--) {
        double* const d = F + (16 * J + 2 * q) * LD + r0 + g;
        if (J < NJ - 1) {
          double acc[2][4];
#pragma unroll
          for (int e = 0; e < 2; e++) {
#pragma unroll
            for (int h = 0; h < 4; h++) acc[e][h] = d[(8 * e + (h & 1)) * LD + (h & 2) * 4];
            for (int K = J + 1; K < NJ; K++)
              warp_mma_16x8<true>(acc[e], F + 16 * K * LD + r0, LD, F + (16 * J + 8 * e) * LD + 16 * K, 1, LD, 16);
          }
          __syncwarp();
#pragma unroll
          for (int e = 0; e < 2; e++)
#pragma unroll
            for (int h = 0; h < 4; h++) d[(8 * e + (h & 1)) * LD + (h & 2) * 4] = acc[e][h];
          __syncwarp();
        }
        front_solve_rows(F, rd + 16 * J, 16 * J, r0, nn - 16 * J);
      }
    }
    __syncthreads();
  }
  for (int c = warp; c < nn; c += NW)
    for (int r = c + lane; r < nj; r += 32) X[(int64_t)c * nj + r] = F[c * LD + (r < nn ? r : r + pad)];
  for (int q = warp; q < na; q += NW)
    for (int i = q + lane; i < na; i += 32) U[(int64_t)q * ldu + i] = F[(NP + q) * LD + NP + i];
}

// acc += A(16 x K) B(K x 8) (NEG: -=) over k0 <= k < K with
// A(r, k) = pa[r * ras + k * kas] and B(k, n) = pb[k * kbs + n * nbs] in shared
// memory, in two chains of MMAs; k0 a multiple of 8, any K.
template <bool NEG>
__device__ __forceinline__ void warp_mma_any(double (&acc)[4], const double* pa, int ras, int kas, const double* pb,
                                             int kbs, int nbs, int k0, int K) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  double odd[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
  for (int k = k0; k < K; k += 8) {
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int kk = k + 4 * e + q;
      const bool ok = kk < K;
      const double a0 = ok ? pa[g * ras + kk * kas] : 0.0, a1 = ok ? pa[(g + 8) * ras + kk * kas] : 0.0;
      const double b0 = ok ? pb[kk * kbs + g * nbs] : 0.0;
      dmma16(e ? odd : acc, NEG ? -a0 : a0, NEG ? -a1 : a1, b0);
    }
  }
#pragma unroll
  for (int h = 0; h < 4; h++) acc[h] += odd[h];
}

// A whole small projected-inverse front (T_PFRONT, nj <= TILE;
// projected_inverse.c:33-73 for one node) in shared memory: G holds L11,
// padded with an identity to a multiple of 16 columns, then M = L11^{-1} in
// its place, then S21; M by block columns, last to first,
//   M(I, J) L(J, J) = -sum_{J < K <= I} M(I, K) L(K, J)   (the identity for I = J),
// the sum by MMAs and the rest by substitution, a lane per row (block rows
// times the diagonal blocks' inverses lost up to a third more digits on
// ill-conditioned fronts); F holds the front: W and V_k (operand c, both triangles)
// first, then [Y11; S21 | V_k].
//   Y11 = M^T M;  S21 = -V_k W;  Y11 -= S21^T W   (FP64 MMAs);
//   U_c = F(r_c, r_c) for every child c (lower parts);
//   the block <- [Y11 (strict upper part zeroed); S21].
// A zero diagonal entry records ctl[2] = j + 1 and is taken as 1.
// With scalar dots, two barriers a column of M, a front of 2-D 30^2 (merged)
// took 24.1 us, now 10.1.
constexpr int PF_LD = TILE + 4;
static_assert(2 * TILE * PF_LD + TILE + TILE / 2 + 8 <= ENGINE_SMEM_BASE_DOUBLES,
              "small fronts exceed the engine's shared memory");

// M = L11^{-1} in place in G, column by column from the last (as LAPACK's
// unblocked triangular inverse), and Y11 = M^T M into F, by scalar dots that
// touch no zero of the triangles: for an L11 with infinities or NaN, which the
// zeros in the MMAs' tiles would spread to entries that do not depend on them.
__device__ __forceinline__ void pfront_scalar(double* G, double* F, int nn) {
  constexpr int LD = PF_LD, NW = NTHREADS / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int j = nn - 1; j >= 0; j--) {
    const double d = G[j * LD + j], ajj = 1.0 / (d == 0.0 ? 1.0 : d);
    const int i = j + 1 + tid;
    double v = 0.0;
    if (i < nn)
      for (int l = j + 1; l <= i; l++) v = fma(G[l * LD + i], G[j * LD + l], v);
    __syncthreads();
    if (i < nn) G[j * LD + i] = -ajj * v;
    if (tid == 0) G[j * LD + j] = ajj;
    __syncthreads();
  }
  for (int j = warp; j < nn; j += NW)
    for (int i = j + lane; i < nn; i += 32) {
      double v = 0.0;
      for (int l = i; l < nn; l++) v = fma(G[i * LD + l], G[j * LD + l], v);
      F[j * LD + i] = v;
    }
  __syncthreads();
}

static __device__ void run_pfront(const RunArgs& ra, const Task& t, double* smem) {
  constexpr int LD = PF_LD, NW = NTHREADS / 32;
  const FrontDesc f = ra.fronts[t.aux[0]];
  const int nn = f.nn, na = f.na, nj = f.nj;
  const int NJ = (nn + 15) >> 4, NP = 16 * NJ;
  double* F = smem;
  double* G = smem + TILE * LD;
  double* rd = G + TILE * LD;         // 1 / L(j, j)
  int* sr = reinterpret_cast<int*>(rd + TILE);
  int* s_bad = sr + TILE;
  double* __restrict__ X = ra.bases[t.a.base] + t.a.off;
  const double* __restrict__ V = ra.bases[t.c.base] + t.c.off;
  const int ldv = t.c.ld;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  if (tid == 0) *s_bad = -1;
  bool finite = true;
  // (four columns' loads at a time: a load is not moved above a store to
  // shared memory)
  for (int c4 = warp; c4 < NP; c4 += 4 * NW) {
    double v[4][2];
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int c = c4 + u * NW, r = lane + 32 * e;
        v[u][e] = (c < nn && r < nj) ? __ldcg(X + (int64_t)c * nj + r) : 0.0;
      }
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int c = c4 + u * NW, r = lane + 32 * e;
        if (r < NP) G[c * LD + r] = (c < nn && r < nn) ? (r >= c ? v[u][e] : 0.0) : (r == c ? 1.0 : 0.0);
        if (c < nn && r >= nn && r < nj) F[c * LD + r] = v[u][e];
        finite = finite && (r < c || r >= nn || isfinite(v[u][e]));
      }
  }
  for (int c4 = warp; c4 < na; c4 += 4 * NW) {
    double v[4][2];
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int c = c4 + u * NW, i = lane + 32 * e;
        v[u][e] = (c < na && i >= c && i < na) ? __ldcg(V + (int64_t)c * ldv + i) : 0.0;
      }
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int c = c4 + u * NW, i = lane + 32 * e;
        if (c < na && i >= c && i < na) {
          F[(nn + c) * LD + nn + i] = v[u][e];
          F[(nn + i) * LD + nn + c] = v[u][e];
        }
      }
  }
  finite = __syncthreads_and(finite);
  if (tid < NP) {
    const double d = G[tid * LD + tid];
    if (d == 0.0) atomicMax(s_bad, tid);
    rd[tid] = 1.0 / (d == 0.0 ? 1.0 : d);
  }
  __syncthreads();
  if (tid == 0 && *s_bad >= 0) atomicCAS(&ra.ctl[2], 0, *s_bad + 1);
  int at = 0;
  if (!finite) {
    pfront_scalar(G, F, nn);
  } else {
    // M in place of L11: block row J + warp of block column J (F's rows < nn
    // are free and take the sums to their rows' lanes)
#pragma unroll 1
    for (int J = NJ - 1; J >= 0; J--) {
      const int I = J + warp, r = 16 * I + (lane & 15);
      double* const gj = G + 16 * J * LD;
      double x[16];
      if (I < NJ) {
        if (warp == 0) {
#pragma unroll
          for (int c = 0; c < 16; c++) x[c] = (lane & 15) == c ? 1.0 : 0.0;
        } else {
          double* const fj = F + 16 * J * LD;
#pragma unroll
          for (int e = 0; e < 2; e++) {
            double y[4] = {0.0, 0.0, 0.0, 0.0};
            warp_mma_any<true>(y, G + 16 * I, 1, LD, gj + 8 * e * LD, 1, LD, 16 * (J + 1), 16 * (I + 1));
#pragma unroll
            for (int h = 0; h < 4; h++) {
              const int row = 16 * I + g + (h & 2) * 4;
              if (row < nn) fj[(8 * e + 2 * q + (h & 1)) * LD + row] = y[h];
            }
          }
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 16; c++) x[c] = r < nn ? fj[c * LD + r] : 0.0;
        }
        solve_row16<LD>(x, gj + 16 * J, rd + 16 * J, 16);
      }
      __syncthreads();
      if (I < NJ && lane < 16) {
#pragma unroll
        for (int c = 0; c < 16; c++) gj[c * LD + r] = x[c];
      }
      __syncthreads();
    }
    // Y11 = M^T M: tiles of 16 x 8 on and below the diagonal
    at = 0;
    for (int I = 0; I < NJ; I++)
      for (int c0 = 0; c0 < min(16 * I + 16, nn); c0 += 8) {
        if (at++ % NW != warp) continue;
        double y[4] = {0.0, 0.0, 0.0, 0.0};
        warp_mma_any<false>(y, G + 16 * I * LD, LD, 1, G + c0 * LD, 1, LD, 16 * I, NP);
#pragma unroll
        for (int h = 0; h < 4; h++) {
          const int r = 16 * I + g + (h & 2) * 4, c = c0 + 2 * q + (h & 1);
          if (r < nn && c <= r) F[c * LD + r] = y[h];
        }
      }
    __syncthreads();
  }
  if (na > 0) {
    // S21 = -V W into G
    at = 0;
    for (int r0 = 0; r0 < na; r0 += 16)
      for (int c0 = 0; c0 < nn; c0 += 8) {
        if (at++ % NW != warp) continue;
        double y[4] = {0.0, 0.0, 0.0, 0.0};
        warp_mma_any<true>(y, F + nn * LD + nn + r0, 1, LD, F + c0 * LD + nn, 1, LD, 0, na);
#pragma unroll
        for (int h = 0; h < 4; h++) {
          const int r = r0 + g + (h & 2) * 4, c = c0 + 2 * q + (h & 1);
          if (r < na && c < nn) G[c * LD + r] = y[h];
        }
      }
    __syncthreads();
    // Y11 -= S21^T W (summed on its own: added one by one to the larger Y11
    // the products would be rounded to its size each)
    at = 0;
    for (int I = 0; I < NJ; I++)
      for (int c0 = 0; c0 < min(16 * I + 16, nn); c0 += 8) {
        if (at++ % NW != warp) continue;
        double y[4] = {0.0, 0.0, 0.0, 0.0};
        warp_mma_any<false>(y, G + 16 * I * LD, LD, 1, F + c0 * LD + nn, 1, LD, 0, na);
#pragma unroll
        for (int h = 0; h < 4; h++) {
          const int r = 16 * I + g + (h & 2) * 4, c = c0 + 2 * q + (h & 1);
          if (r < nn && c <= r) F[c * LD + r] -= y[h];
        }
      }
    __syncthreads();
    for (int j = warp; j < nn; j += NW)
      for (int i = lane; i < na; i += 32) F[j * LD + nn + i] = G[j * LD + i];
    __syncthreads();
  }
  // the children's updates V_c = F(r_c, r_c), lower triangle, the relative
  // indices staged in shared memory per child
  for (int l = f.chbeg; l < f.chend; l++) {
    const FrontDesc ch = ra.fronts[ra.chidx[l]];
    const int Nc = ch.na, tot = Nc * Nc;
    const int32_t* __restrict__ rr = ra.relidx + ch.relptr;
    double* __restrict__ Uc = ra.bases[B_WS] + t.off2 + ch.upd;
    if (tid < Nc) sr[tid] = __ldg(rr + tid);
    __syncthreads();
    for (int idx = tid; idx < tot; idx += NTHREADS) {
      const int c = idx / Nc, i = idx - c * Nc;
      if (i >= c) Uc[idx] = F[sr[c] * LD + sr[i]];
    }
    __syncthreads();
  }
  for (int c = warp; c < nn; c += NW)
    for (int r = lane; r < nj; r += 32)
      X[(int64_t)c * nj + r] = (r < nn && r < c) ? 0.0 : F[c * LD + r];
}

// Gather of a child's update matrix out of its parent's front
// (projected_inverse.c:62-71, completion.c:61-66): for child c = aux[0] and
// child columns q in [aux[1], aux[2]), U_c(i, q) = F(r[i], r[q]) for i >= q,
// where F(row, col) (col <= row) is read from
//   operand a (rows < nn, ld a.ld) when row < nn,
//   operand b (rows >= nn, row nn at offset 0, ld b.ld) when col < nn <= row,
//   operand c (update block, ld c.ld) when col >= nn.
static __device__ void run_extract(const RunArgs& ra, const Task& t, double* smem) {
  const FrontDesc ch = ra.fronts[t.aux[0]];
  const FrontDesc f = ra.fronts[ch.parent];
  const int q0 = t.aux[1], q1 = t.aux[2];
  const int N = ch.na, nn = f.nn;
  const int32_t* r = stage_ridx(ra.relidx + ch.relptr, N, smem);
  const double* __restrict__ F11 = ra.bases[t.a.base] + t.a.off;
  const double* __restrict__ F21 = ra.bases[t.b.base] + t.b.off;
  const double* __restrict__ F22 = ra.bases[t.c.base] + t.c.off;
  const int ld11 = t.a.ld, ld21 = t.b.ld, ld22 = t.c.ld;
  double* __restrict__ Uc = ra.bases[B_WS] + t.off2 + ch.upd;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto entry = [&](int col, int row) {
    if (col >= nn) return F22 + (int64_t)(col - nn) * ld22 + (row - nn);
    if (row >= nn) return F21 + (int64_t)col * ld21 + (row - nn);
    return F11 + (int64_t)col * ld11 + row;
  };
  for (int qb = q0 + warp; qb < q1; qb += ASM_COLS * (NTHREADS / 32)) {
    double v[ASM_COLS][ASM_ROWS];
#pragma unroll
    for (int c = 0; c < ASM_COLS; c++) {
      const int q = qb + c * (NTHREADS / 32), col = q < q1 ? r[q] : 0;
#pragma unroll
      for (int e = 0; e < ASM_ROWS; e++) {
        const int i = q + lane + 32 * e;
        v[c][e] = (q < q1 && i < N) ? __ldcg(entry(col, r[i])) : 0.0;
      }
    }
#pragma unroll
    for (int c = 0; c < ASM_COLS; c++)
#pragma unroll
      for (int e = 0; e < ASM_ROWS; e++) {
        const int q = qb + c * (NTHREADS / 32), i = q + lane + 32 * e;
        if (q < q1 && i < N) Uc[(int64_t)q * N + i] = v[c][e];
      }
    for (int c = 0; c < ASM_COLS; c++) {
      const int q = qb + c * (NTHREADS / 32);
      if (q >= q1 || N - q <= 32 * ASM_ROWS) break;
      const int col = r[q];
      for (int i0 = q + 32 * ASM_ROWS; i0 < N; i0 += GATHER_INFLIGHT * 32) {
        double w[GATHER_INFLIGHT];
#pragma unroll
        for (int e = 0; e < GATHER_INFLIGHT; e++) {
          const int i = i0 + lane + 32 * e;
          w[e] = (i < N) ? __ldcg(entry(col, r[i])) : 0.0;
        }
#pragma unroll
        for (int e = 0; e < GATHER_INFLIGHT; e++) {
          const int i = i0 + lane + 32 * e;
          if (i < N) Uc[(int64_t)q * N + i] = w[e];
        }
      }
    }
  }
}

// Tile copy C = alpha * A (m x n).  aux[0] bit 0: copy only the lower
// triangle (r >= c); bit 1: write zeros above the diagonal; bit 2: write
// zeros everywhere (A is not read).  Bit 3: anti-transpose inside an
// aux[1] x aux[1] matrix: operands a and c are the matrices' origins and the
// tile has origin (aux[2], aux[3]) in C; C(i, j) = A(n-1-j, n-1-i) for the
// lower entries i >= j (with J the order reversal, C = J A^T J).  Bit 4:
// transpose, C(r, c) = A(c, r); bit 5 with it: only entries above the
// diagonal of the tile (r < c), used to symmetrise a diagonal block.
static __device__ void run_copy(const RunArgs& ra, const Task& t) {
  if (t.aux[0] & 16) {
    const double* __restrict__ A = ra.bases[t.a.base] + t.a.off;
    double* __restrict__ C = ra.bases[t.c.base] + t.c.off;
    const int lda = t.a.ld, ldc = t.c.ld, m = t.m, n = t.n;
    const bool upper = (t.aux[0] & 32) != 0;
    for (int base = 0; base < m * n; base += 8 * NTHREADS) {
      double v[8];
#pragma unroll
      for (int e = 0; e < 8; e++) {
        const int idx = base + threadIdx.x + e * NTHREADS;
        const int r = idx % m, c = idx / m;
        v[e] = (idx < m * n && (!upper || r < c)) ? __ldcg(A + (int64_t)r * lda + c) : 0.0;
      }
#pragma unroll
      for (int e = 0; e < 8; e++) {
        const int idx = base + threadIdx.x + e * NTHREADS;
        const int r = idx % m, c = idx / m;
        if (idx < m * n && (!upper || r < c)) C[(int64_t)c * ldc + r] = t.alpha * v[e];
      }
    }
    return;
  }
  if (t.aux[0] & 8) {
    const double* __restrict__ A = ra.bases[t.a.base] + t.a.off;
    double* __restrict__ C = ra.bases[t.c.base] + t.c.off;
    const int lda = t.a.ld, ldc = t.c.ld, m = t.m, n = t.n, nn = t.aux[1], i0 = t.aux[2], j0 = t.aux[3];
    for (int base = 0; base < m * n; base += 8 * NTHREADS) {
      double v[8];
#pragma unroll
      for (int e = 0; e < 8; e++) {
        const int idx = base + threadIdx.x + e * NTHREADS;
        const int gi = i0 + idx % m, gj = j0 + idx / m;
        v[e] = (idx < m * n && gi >= gj) ? __ldcg(A + (int64_t)(nn - 1 - gi) * lda + (nn - 1 - gj)) : 0.0;
      }
#pragma unroll
      for (int e = 0; e < 8; e++) {
        const int idx = base + threadIdx.x + e * NTHREADS;
        const int gi = i0 + idx % m, gj = j0 + idx / m;
        if (idx < m * n && gi >= gj) C[(int64_t)gj * ldc + gi] = v[e];
      }
    }
    return;
  }
  const double* __restrict__ A = ra.bases[t.a.base] + t.a.off;
  double* __restrict__ C = ra.bases[t.c.base] + t.c.off;
  const int lda = t.a.ld, ldc = t.c.ld, m = t.m, n = t.n;
  const bool lower = (t.aux[0] & 1) != 0, zup = (t.aux[0] & 2) != 0, zall = (t.aux[0] & 4) != 0;
  const double alpha = t.alpha;
  for (int base = 0; base < m * n; base += 8 * NTHREADS) {
    double v[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
      const int idx = base + threadIdx.x + e * NTHREADS;
      const int r = idx % m, c = idx / m;
      v[e] = (!zall && idx < m * n && (!lower || r >= c)) ? __ldcg(A + (int64_t)c * lda + r) : 0.0;
    }
#pragma unroll
    for (int e = 0; e < 8; e++) {
      const int idx = base + threadIdx.x + e * NTHREADS;
      const int r = idx % m, c = idx / m;
      if (idx >= m * n) continue;
      if (r >= c || !lower) C[(int64_t)c * ldc + r] = alpha * v[e];
      else if (zup) C[(int64_t)c * ldc + r] = 0.0;
    }
  }
}

// ------------------------------------------------------ update_factor
// Sums of eight values over the warp: every lane returns the sum of u[c],
// c = the lane's bits 4, 3, 2 (halving the values kept at each exchange, so
// nine shuffles instead of forty).
__device__ __forceinline__ double warp_sum8(const double (&u)[8]) {
  const int lane = threadIdx.x & 31;
  const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
  double a[4], c[2];
#pragma unroll
  for (int e = 0; e < 4; e++)
    a[e] = (h4 ? u[4 + e] : u[e]) + __shfl_xor_sync(0xffffffffu, h4 ? u[e] : u[4 + e], 16);
#pragma unroll
  for (int e = 0; e < 2; e++)
    c[e] = (h3 ? a[2 + e] : a[e]) + __shfl_xor_sync(0xffffffffu, h3 ? a[e] : a[2 + e], 8);
  double v = (h2 ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, h2 ? c[0] : c[1], 4);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v;
}

// Shared memory of a Householder panel (ql_panel_doubles): the panel, its T
// factor, and the exchange buffers and scalars of the reflections.
struct QlSmem {
  double* P;      // panel, column pc at P + pc * ld
  int ld;
  double* T;      // T factor, T(a, b) at T[b * ldt + a]
  int ldt;
  double* scr;    // this warp's 8 x 8 tile, leading dimension QL_SLD
  double* wb;     // this warp's products tau v^T c, two groups of eight columns
  double* vb;     // three reflectors with their tau
  double* taus;   // tau of reflector i (application order)
  int* lo;        // support [lo, hi] of the reflection of panel column pc
  int* hi;
  int h, nb;
};

// The reflection [alpha; x] -> [beta; 0] with xn2 = ||x||^2 > 0: beta, tau,
// 1 / (alpha - beta).  The norm is scaled as in LAPACK's dlapy2 where the
// squares could leave the range.
__device__ __forceinline__ void ql_reflection(double alpha, double xn2, double& beta, double& tau, double& scal) {
  const double q2 = fma(alpha, alpha, xn2);
  double nrm;
  if (q2 > 1e-280 && q2 < 1e280) {
    nrm = sqrt(q2);
  } else {
    const double xa = fabs(alpha), xb = sqrt(xn2), w = fmax(xa, xb), z = fmin(xa, xb);
    nrm = (z == 0.0) ? w : w * sqrt(1.0 + (z / w) * (z / w));
  }
  beta = -copysign(nrm, alpha);
  const double d = alpha - beta;
  tau = -d / beta;
  scal = 1.0 / d;
}

// The reflections of a panel of at most 4 SL columns and 32 RR rows, from
// s.P and back to it, with the whole panel in registers: column nb - 1 - i
// (reflector i) belongs to warp i mod 4, row r to lane r mod 32, and a
// warp's next pivot column is always in slot 0.
// After reflector i the owner of the next pivot column applies it to that
// column first, forms reflector i + 1, passes v and tau on through shared
// memory and only then turns to its other columns, so that the chain from
// pivot to pivot is two dots and the reflection's scalars, and the updates
// run beside it.  The owner arrives at the reflector's barrier, the other
// warps wait there.  Two barriers alternate, and three buffers: buffer i is
// written again for reflector i + 3, whose owner has waited at the barrier
// of i + 2, which every warp reaches after its last use of reflector i.
// (A column on eight lanes, sixteen rows each, has shorter sums but took
// 2.6k cycles a reflection against 1.7k.)
// A column goes through the same reflections, in the same order and with v
// scaled before the dots, as in an unblocked reduction: applying the
// reflections of several columns at once would also change the signs that
// rounding gives to pivots which are zero in exact arithmetic.
template <int SL, int RR>
__device__ __forceinline__ void ql_factor(const QlSmem& s) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, h = s.h, nb = s.nb;
  constexpr int NG = (SL + 7) / 8;     // groups of eight slots
  constexpr int VS = 32 * RR + 4;      // a reflector, then its tau
  double x[SL][RR];
#pragma unroll
  for (int e = 0; e < SL; e++)
#pragma unroll
    for (int k = 0; k < RR; k++) {
      const int i = 4 * e + warp, row = lane + 32 * k;
      x[e][k] = (i < nb && row < h) ? s.P[(nb - 1 - i) * s.ld + row] : 0.0;
    }
  int next = warp;             // reflector of slot 0
  double* vb = s.vb + 2 * VS;  // reflector i
  for (int i = -1; i < nb; i++) {
    double* const vn = vb == s.vb + 2 * VS ? s.vb : vb + VS;  // reflector i + 1
    const double tau = i >= 0 ? vb[32 * RR] : 0.0;
    const double* const v = vb + lane;
    const bool mine = i + 1 < nb && next == i + 1;
    if (mine) {
      const int pc = nb - 1 - next, lo = s.lo[pc], hi = s.hi[pc];
      if (tau != 0.0) {
        double u = 0.0;
#pragma unroll
        for (int k = 0; k < RR; k++) u = fma(v[32 * k], x[0][k], u);
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) u += __shfl_xor_sync(0xffffffffu, u, m);
        u *= tau;
#pragma unroll
        for (int k = 0; k < RR; k++) x[0][k] = fma(-v[32 * k], u, x[0][k]);
      }
      double xn2 = 0.0, piv = 0.0;
#pragma unroll
      for (int k = 0; k < RR; k++) {
        const int row = lane + 32 * k;
        const double a = (row >= lo && row < hi) ? x[0][k] : 0.0;
        xn2 = fma(a, a, xn2);
        if (row == hi) piv = x[0][k];
      }
#pragma unroll
      for (int m = 16; m > 0; m >>= 1) xn2 += __shfl_xor_sync(0xffffffffu, xn2, m);
      const double alpha = __shfl_sync(0xffffffffu, piv, hi & 31);
      double beta = alpha, taun = 0.0, scal = 1.0;
      if (hi > lo && xn2 != 0.0) ql_reflection(alpha, xn2, beta, taun, scal);
#pragma unroll
      for (int k = 0; k < RR; k++) {
        const int row = lane + 32 * k;
        const bool in = row >= lo && row < hi;
        const double w = x[0][k] * scal;
        vn[row] = row == hi ? 1.0 : (in ? w : 0.0);
        if (row < h) s.P[pc * s.ld + row] = row == hi ? beta : (in ? w : x[0][k]);
      }
      if (lane == 0) {
        vn[32 * RR] = taun;
        s.taus[next] = taun;
      }
      __syncwarp();
      named_bar_arrive(1 + (next & 1), NTHREADS);
      // the column is done: the others move up (the last slot keeps a copy,
      // which no reflection reads)
#pragma unroll
      for (int e = 0; e + 1 < SL; e++)
#pragma unroll
        for (int k = 0; k < RR; k++) x[e][k] = x[e + 1][k];
      next += 4;
    }
    if (tau != 0.0) {
#pragma unroll
      for (int gr = 0; gr < NG; gr++) {
        if (next + 32 * gr >= nb) break;
        double u[8];
#pragma unroll
        for (int e = 0; e < 8; e++) u[e] = 0.0;
#pragma unroll
        for (int k = 0; k < RR; k++) {
          const double vk = v[32 * k];
#pragma unroll
          for (int e = 0; e < 8; e++)
            if (8 * gr + e < SL) u[e] = fma(vk, x[(8 * gr + e) % SL][k], u[e]);
        }
        const double w = tau * warp_sum8(u);
        if ((lane & 3) == 0) s.wb[8 * gr + (lane >> 2)] = w;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < RR; k++) {
          const double vk = v[32 * k];
#pragma unroll
          for (int e = 0; e < 8; e++)
            if (8 * gr + e < SL) x[(8 * gr + e) % SL][k] = fma(-vk, s.wb[8 * gr + e], x[(8 * gr + e) % SL][k]);
        }
      }
      __syncwarp();
    }
    if (!mine && i + 1 < nb) named_bar_sync(1 + ((i + 1) & 1), NTHREADS);
    vb = vn;
  }
}

// The same reflections for a panel of any height, in shared memory: the
// pivot column's norm, then its scaling, the dots (a group of threads per
// column) and the rank-1 update, with a barrier after each.
__device__ __forceinline__ void ql_factor_tall(const QlSmem& s) {
  const int tid = threadIdx.x, h = s.h, nb = s.nb, ld = s.ld;
  double* const red = s.vb;         // NTHREADS / 32 partial norms
  double* const wq = s.vb + 16;     // tau v^T c of the columns on the left
  for (int i = 0; i < nb; i++) {
    const int pc = nb - 1 - i, lr0 = s.lo[pc], lp = s.hi[pc];
    double* pv = s.P + pc * ld;
    double tau = 0.0;
    if (lp > lr0) {
      double part = 0.0;
      for (int q = lr0 + tid; q < lp; q += NTHREADS) part = fma(pv[q], pv[q], part);
#pragma unroll
      for (int m = 16; m > 0; m >>= 1) part += __shfl_xor_sync(0xffffffffu, part, m);
      if ((tid & 31) == 0) red[tid >> 5] = part;
      __syncthreads();
      const double xn2 = (red[0] + red[1]) + (red[2] + red[3]);
      if (xn2 != 0.0) {
        double beta, scal;
        ql_reflection(pv[lp], xn2, beta, tau, scal);
        __syncthreads();  // everyone has read pv[lp] and the norm
        for (int q = lr0 + tid; q < lp; q += NTHREADS) pv[q] *= scal;
        __syncthreads();
        for (int q2 = tid >> 3; q2 < pc; q2 += NTHREADS / 8) {
          const double* cq = s.P + q2 * ld;
          double a = 0.0, b = 0.0;
          int q = lr0 + (tid & 7);
          for (; q + 8 < lp; q += 16) {
            a = fma(pv[q], cq[q], a);
            b = fma(pv[q + 8], cq[q + 8], b);
          }
          if (q < lp) a = fma(pv[q], cq[q], a);
          a += b;
          // the eight threads of a column are all in this round or none is
          const unsigned mask = 0xffu << (tid & 24);
          for (int m = 4; m > 0; m >>= 1) a += __shfl_xor_sync(mask, a, m);
          if ((tid & 7) == 0) wq[q2] = tau * (a + cq[lp]);
        }
        __syncthreads();
        for (int q = lr0 + tid; q <= lp; q += NTHREADS) {
          const double vq = (q == lp) ? 1.0 : pv[q];
#pragma unroll 4
          for (int q2 = 0; q2 < pc; q2++) s.P[q2 * ld + q] = fma(-vq, wq[q2], s.P[q2 * ld + q]);
        }
        __syncthreads();
        if (tid == 0) pv[lp] = beta;
      }
    }
    if (tid == 0) s.taus[i] = tau;
    __syncthreads();
  }
}

// The T factor from the explicit reflectors (column nb - 1 - i of the panel)
// in 8 x 8 blocks: G(bi, bj) = W_bi^T W_bj by FP64 MMAs, the diagonal blocks
// by LAPACK's recurrence, then by block rows
// T(bi, :) = -T(bi, bi) G(bi, :) T(:bi, :bi).
__device__ __forceinline__ void ql_t_factor(const QlSmem& s) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  const int nblk = (s.nb + 7) >> 3, ldt = s.ldt, h4 = (s.h + 3) & ~3;
  double* const T = s.T;
  double* const Zs = s.scr;
  int at = 0;
  for (int bi = 0; bi < nblk; bi++)
    for (int bj = 0; bj <= bi; bj++, at++) {
      if (at % (NTHREADS / 32) != warp) continue;
      const int ia = 8 * bi + g, ib = 8 * bj + g;
      const double* const pa = s.P + (s.nb - 1 - min(ia, s.nb - 1)) * s.ld;
      const double* const pb = s.P + (s.nb - 1 - min(ib, s.nb - 1)) * s.ld;
      double c[2] = {0.0, 0.0};
#pragma unroll 4
      for (int k = q; k < h4; k += 4) dmma8(c, ia < s.nb ? pa[k] : 0.0, ib < s.nb ? pb[k] : 0.0);
      T[(8 * bj + 2 * q) * ldt + 8 * bi + g] = c[0];
      T[(8 * bj + 2 * q + 1) * ldt + 8 * bi + g] = c[1];
    }
  __syncthreads();
  for (int bi = warp; bi < nblk; bi += NTHREADS / 32) {
    // T(r, i) = -tau_i sum_{i < k <= r} T(r, k) w_k^T w_i, lane r the row r
    double* const D = T + 8 * bi * ldt + 8 * bi;
    const int r = lane & 7;
    double t[8];
#pragma unroll
    for (int i = 7; i >= 0; i--) {
      const double tau = 8 * bi + i < s.nb ? s.taus[8 * bi + i] : 0.0;
      double v = 0.0;
#pragma unroll
      for (int k = 7; k > i; k--) v = fma(k <= r ? t[k] : 0.0, D[i * ldt + k], v);
      t[i] = r == i ? tau : (r > i ? -tau * v : 0.0);
    }
    __syncwarp();
    if (lane < 8) {
#pragma unroll
      for (int i = 0; i < 8; i++) D[i * ldt + r] = t[i];
    }
  }
  __syncthreads();
  for (int bi = 1; bi < nblk; bi++) {
    double out[2][2];
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int bj = warp + 4 * e;
      if (bj >= bi) break;
      double c[2] = {0.0, 0.0};
      for (int k = 8 * bj; k < 8 * bi; k += 4)
        dmma8(c, T[(k + q) * ldt + 8 * bi + g], T[(8 * bj + g) * ldt + k + q]);
      __syncwarp();
      Zs[2 * q * QL_SLD + g] = c[0];
      Zs[(2 * q + 1) * QL_SLD + g] = c[1];
      __syncwarp();
      out[e][0] = out[e][1] = 0.0;
      dmma8(out[e], -T[(8 * bi + q) * ldt + 8 * bi + g], Zs[g * QL_SLD + q]);
      dmma8(out[e], -T[(8 * bi + 4 + q) * ldt + 8 * bi + g], Zs[g * QL_SLD + 4 + q]);
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int bj = warp + 4 * e;
      if (bj >= bi) break;
      T[(8 * bj + 2 * q) * ldt + 8 * bi + g] = out[e][0];
      T[(8 * bj + 2 * q + 1) * ldt + 8 * bi + g] = out[e][1];
    }
    __syncthreads();
  }
}

// Blocked Householder QL of a factored update (update_factor.c:29-47).
// For child c = aux[0] of front k, with V_k = L_k^T L_k (L_k lower, the
// parent's update block, operand a of QL_GATHER) and the child's relative
// indices r split as r[:N1] < nn <= r[N1:], the N2 columns
// C(:, j) = L_k(:, jj_j), jj_j = r[N1 + j] - nn, are reduced to [0; L22] by
// reflections applied last column first.  The reflection of column j acts on
// rows [jj_j, prow_j], prow_j = na - N2 + j, with LAPACK's dlarfg/dlarfx
// conventions: alpha = C(prow_j, j), x = C(jj_j:prow_j, j),
// beta = -sign(alpha) * hypot(alpha, ||x||), tau = (beta - alpha) / beta,
// v = [x / (alpha - beta); 1]; tau = 0 when x is empty or zero.
//
// A QL_PANEL task factors columns [c0, c1) (rows [row0, row1] =
// [jj_c0, prow_{c1-1}], the rows its reflections touch) and writes, for the
// columns to its left (updated by MROW/GEMM tasks):
//   W' (operand b): column c0 + i = reflector i, i = c1 - 1 - j (the order
//     they are applied), explicit over rows [row0, row1];
//   T  (operand c, nb x nb lower, ld c.ld): H_{c0} ... H_{c1-1} = I - W' T W'^T
//     (LAPACK dlarft 'B','C': T(i,i) = tau_i,
//      T(i+1:, i) = -tau_i T(i+1:, i+1:) W'(:, i+1:)^T w'_i).
// A panel is a serial chain of reflections: their latency bounds it.  Up to
// 512 rows it is held in registers (56 columns of 128 rows, 32 of 256, 12 of
// 512).  The build spills 40 bytes a thread with these sizes; with 80 entries
// a thread instead of 64 factored completion on 3-D 40^3 took 70 ms instead
// of 63, as a spilled register costs an L2 round trip where two panels take an
// SM's shared memory.  Taller panels stay in shared memory.  With every panel
// in shared memory and seven barriers a reflection, a reflection took 4.9k
// cycles; now 1.7k (128 rows) to 3.0k.
static __device__ void run_ql(const RunArgs& ra, const Task& t, double* smem) {
  const FrontDesc ch = ra.fronts[t.aux[0]];
  const FrontDesc f = ra.fronts[ch.parent];
  const int N = ch.na, nn = f.nn, na = f.na;
  const int32_t* __restrict__ r = ra.relidx + ch.relptr;
  int lo = 0, hi = N;
  while (lo < hi) { int mid = (lo + hi) >> 1; if (__ldg(r + mid) < nn) lo = mid + 1; else hi = mid; }
  const int N1 = lo, N2 = N - N1;
  const int c0 = t.aux[1], c1 = t.aux[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (t.aux[3] == QL_GATHER) {
    const double* __restrict__ Lk = ra.bases[t.a.base] + t.a.off;
    double* __restrict__ C = ra.bases[t.c.base] + t.c.off;
    const int ldl = t.a.ld, ldc = t.c.ld;
    for (int j = c0 + warp; j < c1; j += NTHREADS / 32) {
      const int jj = __ldg(r + N1 + j) - nn;
#pragma unroll 8
      for (int i = lane; i < na; i += 32)
        C[(int64_t)j * ldc + i] = (i >= jj) ? __ldcg(Lk + (int64_t)jj * ldl + i) : 0.0;
    }
    return;
  }
  double* __restrict__ C = ra.bases[t.a.base] + t.a.off;
  double* __restrict__ W = ra.bases[t.b.base] + t.b.off;
  double* __restrict__ Tg = ra.bases[t.c.base] + t.c.off;
  const int ldc = t.a.ld, ldw = t.b.ld, ldt = t.c.ld;
  const int nb = c1 - c0;
  const int row0 = __ldg(r + N1 + c0) - nn, row1 = na - N2 + c1 - 1;
  const int h = row1 - row0 + 1;
  if (nb <= 0 || nb > ql_max_cols(h) || h <= 0 || ql_panel_doubles(h, nb) > ra.smem_doubles) {
    if (tid == 0) atomicCAS(&ra.ctl[1], DE_NONE, DE_BAD_TASK);
    return;
  }
  QlSmem s;
  const int nb8 = nb > 1 ? (nb + 7) & ~7 : 0, tsize = ql_ld(nb8) * nb8;
  s.h = h;
  s.nb = nb;
  s.ld = nb > 1 ? ql_ld(h) : h;
  s.ldt = ql_ld(nb8);
  s.P = smem;
  s.T = s.P + s.ld * nb;
  s.scr = s.T + tsize + warp * 8 * QL_SLD;
  s.wb = s.T + tsize + (nb > 1 ? NTHREADS / 32 * 8 * QL_SLD : 0);
  s.vb = s.wb + (h <= QL_REG_ROWS ? 16 * (NTHREADS / 32) : 0);
  s.wb += 16 * warp;
  s.taus = s.vb + ql_vb_doubles(h);
  s.lo = reinterpret_cast<int*>(s.taus + ql_scalars(nb));
  s.hi = s.lo + ql_scalars(nb);
  double* const Cp = C + (int64_t)c0 * ldc + row0;
  if (tid < nb) {
    s.lo[tid] = __ldg(r + N1 + c0 + tid) - nn - row0;  // first row of x (local)
    s.hi[tid] = na - N2 + c0 + tid - row0;             // pivot row (local)
  }
  for (int pc = warp; pc < nb; pc += NTHREADS / 32)
    for (int q = lane; q < h; q += 32) cp_async8_zfill(s.P + pc * s.ld + q, Cp + (int64_t)pc * ldc + q, true);
  cp_async_commit();
  cp_async_wait_all();
  __syncthreads();
  if (h <= 128) ql_factor<14, 4>(s);
  else if (h <= 256) ql_factor<8, 8>(s);
  else if (h <= QL_REG_ROWS) ql_factor<3, 16>(s);
  else ql_factor_tall(s);
  __syncthreads();
  // the panel back to C, then W' (explicit reflectors) in its place, with
  // zeros below it up to the leading dimension
  for (int pc = warp; pc < nb; pc += NTHREADS / 32) {
    double* const col = s.P + pc * s.ld;
    double* const dst = Cp + (int64_t)pc * ldc;
    double* const w = W + (int64_t)(c0 + nb - 1 - pc) * ldw + row0;
    const int a = s.lo[pc], b = s.hi[pc];
    for (int q = lane; q < s.ld; q += 32) {
      const double x = q < h ? col[q] : 0.0, v = (q < a || q > b) ? 0.0 : (q == b ? 1.0 : x);
      if (q < h) {
        dst[q] = x;
        w[q] = v;
      }
      col[q] = v;
    }
  }
  if (nb == 1) {
    if (tid == 0) Tg[0] = s.taus[0];
    return;
  }
  __syncthreads();
  ql_t_factor(s);
  for (int b = warp; b < nb; b += NTHREADS / 32)
    for (int a = lane; a < nb; a += 32) Tg[(int64_t)b * ldt + a] = (a >= b) ? s.T[b * s.ldt + a] : 0.0;
}

// ------------------------------------------------------- solve vectors
// Extraction of a child's rows out of [x_p; u_p], or (add) their addition into
// it: elements idx < tot, row i0 + idx mod ni of u_c, column j0 + idx / ni,
// EV per thread at a time.
struct VecChild {
  const int32_t* r;  // relative indices of the child
  double *uc, *xp, *up;
  int nn, na, Nc, ldx, i0, ni, j0, tot;
};
template <int EV>
__device__ __forceinline__ void vec_child(const VecChild& a, bool add) {
  for (int base = 0; base < a.tot; base += EV * NTHREADS) {
    int row[EV], col[EV];
    double v[EV];
#pragma unroll
    for (int e = 0; e < EV; e++) {
      const int idx = base + threadIdx.x + e * NTHREADS;
      const int j = idx / max(a.ni, 1), i = a.i0 + idx - j * a.ni;
      col[e] = a.j0 + j;
      row[e] = (idx < a.tot) ? __ldg(a.r + i) : -1;
      if (add) v[e] = (idx < a.tot) ? __ldcg(a.uc + i + (int64_t)(a.j0 + j) * a.Nc) : 0.0;
    }
    auto entry = [&](int e) {
      return row[e] < a.nn ? a.xp + row[e] + (int64_t)col[e] * a.ldx : a.up + (row[e] - a.nn) + (int64_t)col[e] * a.na;
    };
    if (add) {
      // rows of one child are distinct, but other children add into the
      // same rows at the same time: atomic adds
#pragma unroll
      for (int e = 0; e < EV; e++)
        if (row[e] >= 0) atomicAdd(entry(e), v[e]);
      continue;
    }
#pragma unroll
    for (int e = 0; e < EV; e++) v[e] = row[e] < 0 ? 0.0 : __ldcg(entry(e));
#pragma unroll
    for (int e = 0; e < EV; e++) {
      const int idx = base + threadIdx.x + e * NTHREADS;
      if (row[e] >= 0) a.uc[a.i0 + idx - (col[e] - a.j0) * a.ni + (int64_t)col[e] * a.Nc] = v[e];
    }
  }
}

// Vector operations of the triangular solve sweep (T_VEC, sub-operation
// aux[0], nrhs = t.n right-hand sides).  Bp / x_k live at operand a or c
// with leading dimension n; the per-front vector updates u_k (na x nrhs,
// ld na) start at WS + b.off + vpos[k] * nrhs.
static __device__ void run_vec(const RunArgs& ra, const Task& t, double* smem) {
  const int mode = t.aux[0], nrhs = t.n;
  if (mode == VEC_GATHER || mode == VEC_SCATTER) {
    const int r0 = t.aux[1], r1 = t.aux[2];
    double* __restrict__ Bp = ra.bases[t.c.base] + t.c.off;
    const int ldp = t.c.ld;
    double* __restrict__ Bu = ra.bases[B_RHS];
    const int64_t ldb = ra.ldb;
    const int rows = r1 - r0;
    for (int base = 0; base < rows * nrhs; base += 4 * NTHREADS) {
      double v[4];
      int64_t src[4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int idx = base + threadIdx.x + e * NTHREADS;
        const int i = r0 + idx % max(rows, 1), j = idx / max(rows, 1);
        src[e] = (idx < rows * nrhs) ? __ldg(ra.perm + i) + (int64_t)j * ldb : -1;
        if (mode == VEC_GATHER) v[e] = (src[e] >= 0) ? ra.alpha * __ldcg(Bu + src[e]) : 0.0;
        else v[e] = (src[e] >= 0) ? __ldcg(Bp + i + (int64_t)j * ldp) : 0.0;
      }
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int idx = base + threadIdx.x + e * NTHREADS;
        const int i = r0 + idx % max(rows, 1), j = idx / max(rows, 1);
        if (src[e] < 0) continue;
        if (mode == VEC_GATHER) Bp[i + (int64_t)j * ldp] = v[e];
        else Bu[src[e]] = v[e];
      }
    }
    return;
  }
  double* __restrict__ WS = ra.bases[B_WS];
  const int64_t vbase = t.b.off;
  // right-hand-side columns [j0, j1) of this task (aux[3] == 0: all)
  const int j0 = t.aux[2], j1 = t.aux[3] > 0 ? t.aux[3] : nrhs, nc = j1 - j0;
  constexpr int E = 8;  // elements per thread with their loads in flight together
  if (mode == VEC_ASM) {
    const FrontDesc f = ra.fronts[t.aux[1]];
    double* __restrict__ xk = ra.bases[t.a.base] + t.a.off;
    const int ldx = t.a.ld;
    double* __restrict__ uk = ra.bases[t.c.base] + t.c.off;
    const int nj = f.nj;
    if ((int64_t)nj * nc <= ENGINE_SMEM_BASE_DOUBLES) {
      // [x_k; u_k] columns staged in shared memory (u_k part zero), the
      // children added there, the result stored once
      for (int base = 0; base < nj * nc; base += E * NTHREADS) {
        double v[E];
#pragma unroll
        for (int e = 0; e < E; e++) {
          const int idx = base + threadIdx.x + e * NTHREADS;
          const int i = idx % nj, j = j0 + idx / nj;
          v[e] = (idx < nj * nc && i < f.nn) ? __ldcg(xk + i + (int64_t)j * ldx) : 0.0;
        }
#pragma unroll
        for (int e = 0; e < E; e++) {
          const int idx = base + threadIdx.x + e * NTHREADS;
          if (idx < nj * nc) smem[idx] = v[e];
        }
      }
      __syncthreads();
      for (int l = f.chend - 1; l >= f.chbeg; l--) {
        const FrontDesc ch = ra.fronts[ra.chidx[l]];
        const int Nc = ch.na, tot = Nc * nc;
        const int32_t* __restrict__ r = ra.relidx + ch.relptr;
        const double* __restrict__ uc = WS + vbase + ch.vpos * nrhs + (int64_t)j0 * Nc;
        for (int base = 0; base < tot; base += E * NTHREADS) {
          int dst[E];
          double v[E];
#pragma unroll
          for (int e = 0; e < E; e++) {
            const int idx = base + threadIdx.x + e * NTHREADS;
            const int i = idx % max(Nc, 1), j = idx / max(Nc, 1);
            dst[e] = (idx < tot) ? __ldg(r + i) + j * nj : -1;
            v[e] = (idx < tot) ? __ldcg(uc + idx) : 0.0;
          }
          // a child's relative indices are distinct: no two elements of one
          // pass meet in shared memory
#pragma unroll
          for (int e = 0; e < E; e++)
            if (dst[e] >= 0) smem[dst[e]] += v[e];
        }
        __syncthreads();
      }
      for (int idx = threadIdx.x; idx < nj * nc; idx += NTHREADS) {
        const int i = idx % nj, j = j0 + idx / nj;
        if (i < f.nn) xk[i + (int64_t)j * ldx] = smem[idx];
        else uk[(i - f.nn) + (int64_t)j * f.na] = smem[idx];
      }
      return;
    }
    // too tall for shared memory: zero u_k's columns, add in global memory
    for (int idx = threadIdx.x; idx < f.na * nc; idx += NTHREADS)
      uk[(idx % f.na) + (int64_t)(j0 + idx / f.na) * f.na] = 0.0;
    __syncthreads();
    for (int l = f.chend - 1; l >= f.chbeg; l--) {
      const FrontDesc ch = ra.fronts[ra.chidx[l]];
      const int Nc = ch.na, tot = Nc * nc;
      const int32_t* __restrict__ r = ra.relidx + ch.relptr;
      const double* __restrict__ uc = WS + vbase + ch.vpos * nrhs + (int64_t)j0 * Nc;
      for (int base = 0; base < tot; base += E * NTHREADS) {
        double* dst[E];
        double v[E], old[E];
#pragma unroll
        for (int e = 0; e < E; e++) {
          const int idx = base + threadIdx.x + e * NTHREADS;
          const int i = idx % max(Nc, 1), j = j0 + idx / max(Nc, 1);
          dst[e] = nullptr;
          v[e] = 0.0;
          if (idx < tot) {
            const int row = __ldg(r + i);
            dst[e] = (row < f.nn) ? xk + row + (int64_t)j * ldx : uk + (row - f.nn) + (int64_t)j * f.na;
            v[e] = __ldcg(uc + idx);
          }
        }
#pragma unroll
        for (int e = 0; e < E; e++) old[e] = dst[e] ? __ldcg(dst[e]) : 0.0;
#pragma unroll
        for (int e = 0; e < E; e++)
          if (dst[e]) *dst[e] = old[e] + v[e];
      }
      __syncthreads();
    }
    return;
  }
  if (mode == VEC_ZERO) {
    double* __restrict__ z = ra.bases[t.c.base] + t.c.off;
    const int64_t cnt = (int64_t)t.m * t.n;
    for (int64_t i = threadIdx.x; i < cnt; i += NTHREADS) z[i] = 0.0;
    return;
  }
  // VEC_EXTRACT / VEC_ADD for child aux1 of the front p described by
  // operands a (x_p) and c (u_p): rows [i0, i1) of u_c, columns [j0, j1)
  const FrontDesc ch = ra.fronts[t.aux[1]];
  const FrontDesc f = ra.fronts[ch.parent];
  double* __restrict__ xp = ra.bases[t.a.base] + t.a.off;
  const int ldx = t.a.ld;
  double* __restrict__ up = ra.bases[t.c.base] + t.c.off;
  const int Nc = ch.na;
  const int i0 = t.m, i1 = t.k > 0 ? t.k : Nc, ni = max(i1 - i0, 0), tot = ni * nc;
  const int32_t* __restrict__ r = ra.relidx + ch.relptr;
  double* __restrict__ uc = WS + vbase + ch.vpos * nrhs;
  // 16 elements per thread with their loads in flight together: the planner's
  // chunks (2048 elements) take one pass, two L2 round trips in an extraction
  // and one in an addition, whose values need not wait for the indices; at
  // most 512 elements take four (twelve empty ones are a microsecond: an
  // extraction on small fronts 2.5 us instead of 1.5).
  const VecChild c{r, uc, xp, up, f.nn, f.na, Nc, ldx, i0, ni, j0, tot};
  if (tot <= 4 * NTHREADS) vec_child<4>(c, mode == VEC_ADD);
  else vec_child<16>(c, mode == VEC_ADD);
}

// ---------------------------------------------------------------- kernel
// ------------------------------------------------------------ bundles
// Small-subtree bundles.  A T_SUBTREE / T_PSUBTREE task carries up to four
// ranges of supernodes, one per warp: warp w owns [aux[w], bundle_last(t, w)]
// (aux[w] < 0: idle).  Each range is a union of complete subtrees,
// contiguous in postorder, whose fronts all have nj <= SUB_NJ, so a range
// needs nothing from outside but, for projected_inverse, its roots' V_k.
// The warp processes its fronts alone (cholesky in postorder, projected
// inverse parents first), one row of the front per lane, in its own
// shared-memory matrices (row-major, stride SUB_LD).  The update matrices
// inside a range pass through the workspace at their usual offsets and are
// written and read by the same warp (ordered by __syncwarp); the parents of
// a range's roots wait on the whole task.  Arithmetic and summation orders
// are those of the one-front tasks (T_FRONT / T_PFRONT).
__device__ __forceinline__ int bundle_last(const Task& t, int w) {
  return w == 0 ? t.m : w == 1 ? t.n : w == 2 ? t.k : t.cdiag;
}

// Global loads go SUB_E at a time into registers before they are stored (a
// load is not moved above a store to shared memory, so one by one each costs
// a round trip: a bundle of the 256 uneven grids took 72 us in cholesky and
// 67 in projected_inverse, now 60 and 63).
constexpr int SUB_E = 8;

// Columns [c0, c1) of a matrix whose column c begins at src + c * ld, rows
// >= c, into the lane's row of a front (from entry to0 on); all lanes call.
__device__ __forceinline__ void sub_load(double* row, const double* __restrict__ src, int ld, int c1, bool lower,
                                         bool active, int lane, int to0) {
  for (int c0 = 0; c0 < c1; c0 += SUB_E) {
    double v[SUB_E];
#pragma unroll
    for (int e = 0; e < SUB_E; e++) {
      const int c = c0 + e;
      v[e] = (active && c < c1 && (!lower || lane >= c)) ? __ldcg(src + (int64_t)c * ld + lane) : 0.0;
    }
#pragma unroll
    for (int e = 0; e < SUB_E; e++)
      if (active && c0 + e < c1) row[to0 + c0 + e] = v[e];
  }
}

// cholesky.c:33-72 for one front of at most SUB_NJ rows, by one warp.
static __device__ void chol_front_warp(const RunArgs& ra, int k, double* F, int lane) {
  const FrontDesc f = ra.fronts[k];
  const int nn = f.nn, na = f.na, nj = f.nj;
  double* __restrict__ X = ra.bases[B_X] + f.blk;
  double* __restrict__ W = ra.bases[B_WS];
  double* row = F + lane * SUB_LD;
  sub_load(row, X, nj, nn, true, lane < nj, lane, 0);
  if (lane < nj)
    for (int c = nn; c < nj; c++) row[c] = 0.0;
  __syncwarp();
  // extend-add, children last to first (the reference's stack order)
  for (int l = f.chend - 1; l >= f.chbeg; l--) {
    const FrontDesc ch = ra.fronts[ra.chidx[l]];
    const int Nc = ch.na;
    const double* __restrict__ Uc = W + ch.upd;
    const int r = lane < Nc ? __ldg(ra.relidx + ch.relptr + lane) : 0;
    double* dst = F + r * SUB_LD;
    for (int q0 = 0; q0 < Nc; q0 += SUB_E) {
      double v[SUB_E];
      int rq[SUB_E];
#pragma unroll
      for (int e = 0; e < SUB_E; e++) {
        const int q = q0 + e;
        rq[e] = __shfl_sync(0xffffffffu, r, q & 31);
        v[e] = (lane < Nc && q <= lane) ? __ldcg(Uc + (int64_t)q * Nc + lane) : 0.0;
      }
#pragma unroll
      for (int e = 0; e < SUB_E; e++)
        if (lane < Nc && q0 + e <= lane) dst[rq[e]] += v[e];
    }
    __syncwarp();
  }
  // partial Cholesky of the nn pivot columns; the trailing block becomes U_k
  int first_bad = -1;
  for (int j = 0; j < nn; j++) {
    const double d = F[j * SUB_LD + j];
    const bool bad = !(d > 0.0);
    if (bad && first_bad < 0) first_bad = j;
    const double lj = sqrt(bad ? 1.0 : d), rl = 1.0 / lj;
    double a = 0.0;
    if (lane > j && lane < nj) {
      a = row[j] * rl;
      row[j] = a;
    }
    __syncwarp();
    if (lane == j) row[j] = lj;
    for (int c0 = j + 1; c0 < nj; c0 += SUB_E) {
      double u[SUB_E], w[SUB_E];
#pragma unroll
      for (int e = 0; e < SUB_E; e++) {
        const int c = min(c0 + e, nj - 1);
        u[e] = F[c * SUB_LD + j];
        w[e] = row[c];
      }
#pragma unroll
      for (int e = 0; e < SUB_E; e++)
        if (c0 + e <= lane && lane < nj) row[c0 + e] = fma(-a, u[e], w[e]);
    }
    __syncwarp();
  }
  if (lane == 0 && first_bad >= 0) atomicCAS(&ra.ctl[2], 0, first_bad + 1);
  // separator rows: L21 L11^{-1}, the reference's off-diagonal layout (:72)
  if (lane >= nn && lane < nj)
    for (int j = nn - 1; j >= 0; j--) {
      double v = row[j];
      for (int l2 = j + 1; l2 < nn; l2++) v = fma(-row[l2], F[l2 * SUB_LD + j], v);
      row[j] = v / F[j * SUB_LD + j];
    }
  __syncwarp();
  for (int c = 0; c < nn; c++)
    if (lane >= c && lane < nj) X[(int64_t)c * nj + lane] = row[c];
  double* __restrict__ U = W + f.upd;
  for (int q = 0; q < na; q++)
    if (lane >= nn + q && lane < nj) U[(int64_t)q * na + (lane - nn)] = row[nn + q];
  __syncwarp();
}

// projected_inverse.c:33-73 for one front of at most SUB_NJ rows, by one
// warp: G holds L11, then M = L11^{-1}, then S21; F holds [W, V_k], then
// [Y11; S21 | V_k].
static __device__ void pinv_front_warp(const RunArgs& ra, int k, double* G, double* F, int lane) {
  const FrontDesc f = ra.fronts[k];
  const int nn = f.nn, na = f.na, nj = f.nj;
  double* __restrict__ X = ra.bases[B_X] + f.blk;
  double* __restrict__ W = ra.bases[B_WS];
  const double* __restrict__ V = W + f.upd;
  // L11 into G, with zeros above its diagonal; W and V_k into F
  sub_load((lane < nn ? G : F) + lane * SUB_LD, X, nj, nn, true, lane < nj, lane, 0);
  sub_load(F + (nn + lane) * SUB_LD, V, na, na, true, lane < na, lane, nn);
  __syncwarp();
  // M = L11^{-1} in place, columns last to first
  int first_bad = -1;
  for (int j = nn - 1; j >= 0; j--) {
    const double d = G[j * SUB_LD + j];
    if (d == 0.0 && first_bad < 0) first_bad = j;
    const double ajj = 1.0 / (d == 0.0 ? 1.0 : d);
    double ti = 0.0;
    if (lane > j && lane < nn)
      for (int l = j + 1; l <= lane; l++) ti = fma(G[lane * SUB_LD + l], G[l * SUB_LD + j], ti);
    __syncwarp();
    if (lane > j && lane < nn) G[lane * SUB_LD + j] = -ajj * ti;
    if (lane == j) G[j * SUB_LD + j] = ajj;
    __syncwarp();
  }
  if (lane == 0 && first_bad >= 0) atomicCAS(&ra.ctl[2], 0, first_bad + 1);
  // Y11 = M^T M (lower part), rows < nn of F
  if (lane < nn)
    for (int j = 0; j <= lane; j++) {
      double v = 0.0;
      for (int l = lane; l < nn; l++) v = fma(G[l * SUB_LD + lane], G[l * SUB_LD + j], v);
      F[lane * SUB_LD + j] = v;
    }
  __syncwarp();
  if (na > 0) {
    // S21 = -V_k W (V_k read as symmetric from its lower part) into G
    if (lane < na)
      for (int j = 0; j < nn; j++) {
        double v = 0.0;
        for (int l = 0; l < na; l++) {
          const double vil = (lane >= l) ? F[(nn + lane) * SUB_LD + nn + l] : F[(nn + l) * SUB_LD + nn + lane];
          v = fma(vil, F[(nn + l) * SUB_LD + j], v);
        }
        G[lane * SUB_LD + j] = -v;
      }
    __syncwarp();
    // Y11 -= S21^T W
    if (lane < nn)
      for (int j = 0; j <= lane; j++) {
        double v = 0.0;
        for (int l = 0; l < na; l++) v = fma(G[l * SUB_LD + lane], F[(nn + l) * SUB_LD + j], v);
        F[lane * SUB_LD + j] -= v;
      }
    __syncwarp();
    if (lane < na)
      for (int j = 0; j < nn; j++) F[(nn + lane) * SUB_LD + j] = G[lane * SUB_LD + j];
    __syncwarp();
  }
  // the children's updates F(r_c, r_c), lower parts
  for (int l = f.chbeg; l < f.chend; l++) {
    const FrontDesc ch = ra.fronts[ra.chidx[l]];
    const int Nc = ch.na;
    double* __restrict__ Uc = W + ch.upd;
    const int r = lane < Nc ? __ldg(ra.relidx + ch.relptr + lane) : 0;
    const double* src = F + r * SUB_LD;
    for (int q = 0; q < Nc; q++) {
      const int rq = __shfl_sync(0xffffffffu, r, q);
      if (lane < Nc && q <= lane) Uc[(int64_t)q * Nc + lane] = src[rq];
    }
  }
  for (int c = 0; c < nn; c++)
    if (lane < nj) X[(int64_t)c * nj + lane] = (lane < nn && lane < c) ? 0.0 : F[lane * SUB_LD + c];
  __syncwarp();
}

static __device__ void run_subtrees(const RunArgs& ra, const Task& t, double* smem) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lo = t.aux[warp];
  if (lo < 0) return;
  const int hi = bundle_last(t, warp);
  if (t.op == T_SUBTREE) {
    double* F = smem + warp * SUB_NJ * SUB_LD;
    for (int k = lo; k <= hi; k++) chol_front_warp(ra, k, F, lane);
  } else {
    double* G = smem + warp * 2 * SUB_NJ * SUB_LD;
    for (int k = hi; k >= lo; k--) pinv_front_warp(ra, k, G, G + SUB_NJ * SUB_LD, lane);
  }
}

static_assert(NTHREADS == 128, "a bundle has one range per warp of a 4-warp CTA");
static_assert(8 * SUB_NJ * SUB_LD <= ENGINE_SMEM_BASE_DOUBLES, "bundle fronts exceed the engine's shared memory");

// One kernel per build (engine.h: EngineBuild): code that a launch never
// reaches still costs it registers and spills.  With the tcgen05 tiles in
// it, a launch of the FP64 sweeps measured 17-60 % slower at 40^3, although
// no tcgen05 instruction ran; with the register-resident Householder panels
// in it, cholesky + projected_inverse took 12.17 ms there against 11.99
// without them; with the solve tasks, 10.37 against 10.35 (97^2 with extra
// edges 2.22 against 2.20).
template <int BUILD>
__global__ void __launch_bounds__(NTHREADS, 2) engine_kernel(RunArgs ra) {
  constexpr bool TC = BUILD == EB_TCGEN05;
  constexpr bool LATE = BUILD == EB_SOLVE;
  constexpr bool FRONTS = BUILD == EB_BASE || TC;  // small fronts and bundles (cholesky, projected_inverse)
  extern __shared__ __align__(16) double smem[];
  __shared__ int s_task;
  __shared__ int s_abort;
  __shared__ int s_next;      // dynamic: the waiter this CTA released and runs next, or -1
  __shared__ int s_succ[2];   // dynamic: waiter range of the current task
  __shared__ int s_pre[32];   // dynamic: its first 32 waiters (cp.async during the task)
  __shared__ __align__(16) Task s_t;
  static_assert(sizeof(Task) == 36 * 4, "task record is 36 words");
  SmemLayout sm{smem, smem + TILE * LDS};
  __shared__ int s_lo;        // dynamic: this CTA's copy of the finished frontier
  __shared__ uint32_t s_tmem;                 // tensor-memory base of the TF32 tiles
  __shared__ __align__(8) uint64_t s_mbar[2]; // their MMA-completion barriers
  if (threadIdx.x == 0) {
    s_next = -1;
    s_lo = 0;
  }
  TcState ts;
  ts.mbar = s_mbar;
  ts.ncommit[0] = ts.ncommit[1] = 0;
  ts.tmem = 0;
  if (TC) {
    // 64 columns of tensor memory (a 64 x 64 FP32 accumulator) for the
    // whole launch: two CTAs per SM take 128 of the 512 columns
    if (threadIdx.x < 32) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 64;" ::"r"(smem_u32(&s_tmem))
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
      mbar_init(&s_mbar[0]);
      mbar_init(&s_mbar[1]);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    ts.tmem = s_tmem;
  }
  int claim = -1;  // static: the next task (thread 32)
  if (!ra.dynamic && threadIdx.x == 32) claim = atomicAdd(&ra.ctl[0], 1);
  for (;;) {
    if (ra.dynamic) {
      // warp 0: the next task (handed over by the last one, or claimed), its
      // record and waiter range in one round of loads, its first waiters
      // prefetched asynchronously
      if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        __syncwarp();
        const unsigned long long t0 = ra.trace ? global_ns() : 0ull;
        int c = s_next;
        if (c < 0) c = claim_task(ra, &s_lo);
        if (c < ra.ntasks) {
          const uint32_t* src = reinterpret_cast<const uint32_t*>(ra.tasks + c);
          uint32_t* dst = reinterpret_cast<uint32_t*>(&s_t);
          const uint32_t v0 = __ldg(src + lane);
          const uint32_t v1 = lane < 4 ? __ldg(src + 32 + lane) : 0u;
          const int so = (lane == 4 || lane == 5) ? __ldg(ra.succ_off + c + lane - 4) : 0;
          dst[lane] = v0;
          if (lane < 4) dst[32 + lane] = v1;
          const int b = __shfl_sync(0xffffffffu, so, 4), e = __shfl_sync(0xffffffffu, so, 5);
          if (lane == 0) {
            s_succ[0] = b;
            s_succ[1] = e;
          }
          if (lane < e - b) cp_async4(&s_pre[lane], ra.succ + b + lane);
          cp_async_commit();
          if (lane == 0 && ra.trace) {
            ra.trace[4 * (int64_t)c] = t0;
            ra.trace[4 * (int64_t)c + 1] = global_ns();
          }
        }
        if (lane == 0) s_task = c;
      }
      __syncthreads();
      if (s_task >= ra.ntasks) break;
    } else {
      // warp 1: the record of the task it has claimed, then the task's waits,
      // one per lane (32 at a time), so that the wait records and the
      // counters are read in one round each.  With claim, record and waits
      // after the release, all by thread 0 and warp 0, the per-task overhead
      // was about 0.5 us more: 256 uneven 2-D grids (1.09 M tasks) 52.5 ms
      // against 50.2, projected_inverse on 2-D 1000^2 9.7 against 9.1.
      if (threadIdx.x >> 5 == 1) {
        const int lane = threadIdx.x & 31;
        const int ti = __shfl_sync(0xffffffffu, claim, 0);
        int abort = 0;
        if (ti < ra.ntasks) {
          const uint32_t* src = reinterpret_cast<const uint32_t*>(ra.tasks + ti);
          uint32_t* dst = reinterpret_cast<uint32_t*>(&s_t);
          const uint32_t v0 = __ldg(src + lane), v1 = lane < 4 ? __ldg(src + 32 + lane) : 0u;
          dst[lane] = v0;
          if (lane < 4) dst[32 + lane] = v1;
          if (lane == 0 && ra.trace) ra.trace[4 * (int64_t)ti] = global_ns();
          __syncwarp();
          int timed_out = 0;
          const int npre = ((s_t.op == T_POTRF && s_t.k > 0) || s_t.op == T_TRSV) ? (int)s_t.cdiag
                           : is_narrow<BUILD>(s_t) ? 0 : (int)s_t.nwait;
          for (int w0 = 0; w0 < npre; w0 += 32) {
            if (w0 + lane < npre) {
              const int2 wt = ra.waits[s_t.wait_off + w0 + lane];
              int64_t spins = 0;
              unsigned ns = 16;
              while (ld_acquire(ra.counters + wt.x) < wt.y) {
                if (++spins > ra.spin_limit) {
                  atomicCAS(&ra.ctl[1], 0, DE_TIMEOUT);
                  abort = timed_out = 1;
                  break;
                }
                if ((spins & 15) == 0 && ld_volatile(&ra.ctl[1]) != 0) { abort = 1; break; }
                __nanosleep(ns);
                if (ns < 128) ns <<= 1;
              }
            }
            if (__any_sync(0xffffffffu, abort)) {
              abort = 1;
              break;
            }
          }
          timed_out = __any_sync(0xffffffffu, timed_out);
          if (lane == 0) {
            if (timed_out) atomicAdd(&ra.ctl[3], 1);  // CTAs whose wait ran out
            if (!abort && ld_volatile(&ra.ctl[1]) != 0) abort = 1;
            if (ra.trace) ra.trace[4 * (int64_t)ti + 1] = global_ns();
          }
        }
        if (lane == 0) {
          s_task = ti;
          s_abort = abort;
        }
      }
      __syncthreads();
      if (s_task >= ra.ntasks || s_abort) break;
    }
    const int ti = s_task;
    const Task& t = s_t;
    claim = -1;
    switch (is_narrow<BUILD>(t) ? T_TRSV : t.op) {
      case T_GEMM:
      case T_LA: run_gemm_or_la<TC, !LATE>(ra, t, sm, ts, claim); break;
      case T_MROW: run_mrow(ra, t, sm); break;
      case T_POTRF: run_potrf(ra, t, smem, ti); break;
      case T_ASM: run_asm(ra, t, smem); break;
      case T_FRONT:
        if (FRONTS) run_front(ra, t, smem);
        else if (threadIdx.x == 0) atomicCAS(&ra.ctl[1], 0, DE_BAD_TASK);
        break;
      case T_PFRONT:
        if (FRONTS) run_pfront(ra, t, smem);
        else if (threadIdx.x == 0) atomicCAS(&ra.ctl[1], 0, DE_BAD_TASK);
        break;
      case T_SUBTREE:
      case T_PSUBTREE:
        if (FRONTS) run_subtrees(ra, t, smem);
        else if (threadIdx.x == 0) atomicCAS(&ra.ctl[1], 0, DE_BAD_TASK);
        break;
      case T_EXTRACT: run_extract(ra, t, smem); break;
      case T_COPY: run_copy(ra, t); break;
      case T_VEC:
        if (BUILD == EB_SOLVE) run_vec(ra, t, smem);
        else if (threadIdx.x == 0) atomicCAS(&ra.ctl[1], 0, DE_BAD_TASK);
        break;
      case T_TRSV:
        if (BUILD == EB_SOLVE) run_trsv(ra, t, smem, ti, claim);
        else if (threadIdx.x == 0) atomicCAS(&ra.ctl[1], 0, DE_BAD_TASK);
        break;
      case T_QL:
        if (BUILD == EB_PANELS) run_ql(ra, t, smem);
        else if (threadIdx.x == 0) atomicCAS(&ra.ctl[1], 0, DE_BAD_TASK);
        break;
      case T_NOP: break;
      case T_SUM: run_sum(ra, t); break;
      case T_SIGNAL:
        if (threadIdx.x == 0 && t.aux[0] >= 0 && t.aux[0] < ra.nio_out) raise_io_flag(ra.io_out + t.aux[0]);
        break;
      case T_ARRIVAL:
        if (threadIdx.x == 0) wait_arrival(ra, t.aux[0]);
        break;
      default:
        if (threadIdx.x == 0) atomicCAS(&ra.ctl[1], 0, DE_BAD_TASK);
        break;
    }
    const int op = t.op, group = t.group;
    // static: the next task is claimed before this one's end is published,
    // so that its record and waits are fetched (warp 1) beside the release
    // (warp 0).  Its holder still publishes first, whatever the claimed task
    // waits on.  LATE: beside the release, since in a chain of products, which
    // has idle CTAs enough, a claim before it delays the end: a product with
    // the factor of 3-D 40^3 ('N', one column) took 8.11 ms, now 7.95, with
    // a dense one of order 1500 2.51, now 2.44.
    if (!LATE && !ra.dynamic && threadIdx.x == 32 && claim < 0) claim = atomicAdd(&ra.ctl[0], 1);
    __syncthreads();
    if (LATE && !ra.dynamic && threadIdx.x == 32 && claim < 0) claim = atomicAdd(&ra.ctl[0], 1);
    if (threadIdx.x == 0 && ra.trace) {
      ra.trace[4 * (int64_t)ti + 2] = global_ns();
      ra.trace[4 * (int64_t)ti + 3] = (unsigned long long)sm_id() | ((unsigned long long)op << 32);
    }
    if (!ra.dynamic) {
      // the task's counter and its group's, by two lanes at once
      const int c = threadIdx.x == 0 ? ti : group;
      if (threadIdx.x < 2 && c >= 0) red_release_add(ra.counters + c, 1);
    } else if (threadIdx.x < 32) {
      const int nx = finish_task(ra, ti, group, s_succ[0], s_succ[1], s_pre, op == T_POTRF && t.k > 0);
      if (threadIdx.x == 0) s_next = nx;
    }
  }
  if (ra.nio_out > 0) {
    // the last CTA to leave raises every output flag (already raised after a
    // complete sweep; after an aborted one the waiting copies still proceed)
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&ra.ctl[6], 1) == (int)gridDim.x - 1)
      for (int j = 0; j < ra.nio_out; j++) raise_io_flag(ra.io_out + j);
  }
  if (TC) {
    // every tile waited for its last commit, so no MMA is in flight
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x < 32)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 64;" ::"r"(ts.tmem) : "memory");
  }
}

static_assert(2 * TILE * LDS <= ENGINE_SMEM_BASE_DOUBLES, "GEMM staging exceeds the engine's shared memory");
static_assert(GEMM_STAGES * STAGE_DOUBLES <= ENGINE_SMEM_BASE_DOUBLES, "GEMM ring exceeds the engine's shared memory");
static_assert(POTRF_SMEM_DOUBLES <= ENGINE_SMEM_BASE_DOUBLES, "POTRF exceeds the engine's shared memory");

// Launch, shared-memory attribute and occupancy of one build, for the
// translation unit that compiles it (engine.h: EngineBuild).
template <int BUILD>
cudaError_t build_launch(const RunArgs& ra, int grid, size_t smem, cudaStream_t stream) {
  engine_kernel<BUILD><<<grid, NTHREADS, smem, stream>>>(ra);
  return cudaGetLastError();
}
template <int BUILD>
cudaError_t build_set_smem(size_t smem) {
  return cudaFuncSetAttribute(engine_kernel<BUILD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}
template <int BUILD>
cudaError_t build_occupancy(int* blocks_per_sm, size_t smem) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, engine_kernel<BUILD>, NTHREADS, smem);
}

}  // namespace chb

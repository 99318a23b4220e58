// potrf_block16 (chompack_b200/csrc/block16.cuh) on the CPU, a fiber per lane:
// a lane runs on until it reaches a warp-wide operation, and only then the
// next one starts, so that a missing __syncwarp() gives wrong results.
#include <ucontext.h>

#include <cmath>
#include <vector>

#define __device__
#define __forceinline__ inline

static struct { int x; } threadIdx;
static ucontext_t sched_ctx, lane_ctx[32];
static bool done[32];
static double mma_a[32], mma_b[32];

static void __syncwarp() { swapcontext(&lane_ctx[threadIdx.x], &sched_ctx); }
static double rsqrt(double x) { return (double)(1.0L / sqrtl((long double)x)); }

static void dmma8(double (&c)[2], double a, double b) {
  const int lane = threadIdx.x, g = lane >> 2, q = lane & 3;
  mma_a[lane] = a;
  mma_b[lane] = b;
  __syncwarp();
  for (int e = 0; e < 2; e++)
    for (int k = 0; k < 4; k++) c[e] = std::fma(mma_a[4 * g + k], mma_b[4 * (2 * q + e) + k], c[e]);
  __syncwarp();
}

using std::fma;
#include "block16.cuh"

static constexpr int LD = 20;
static double *g_l, *g_m, g_t[64];
static int g_factor, g_cols, g_info;

static void lane_main() {
  const int info = potrf_block16<LD, LD>(g_l, g_m, g_t, g_factor != 0, g_cols);
  if (threadIdx.x == 0) g_info = info;
  done[threadIdx.x] = true;
  __syncwarp();
}

// l, m: 16 columns of leading dimension 20 (m may be l); the lanes take their
// turns upwards or downwards.  Returns what potrf_block16 returns.
extern "C" int block16(double* l, double* m, int factor, int cols, int downwards) {
  static std::vector<char> stacks(32 * 65536);
  g_l = l, g_m = m, g_factor = factor, g_cols = cols;
  for (int i = 0; i < 32; i++) {
    getcontext(&lane_ctx[i]);
    lane_ctx[i].uc_stack.ss_sp = stacks.data() + i * 65536;
    lane_ctx[i].uc_stack.ss_size = 65536;
    lane_ctx[i].uc_link = nullptr;
    makecontext(&lane_ctx[i], lane_main, 0);
    done[i] = false;
  }
  for (bool more = true; more;) {
    more = false;
    for (int i = 0; i < 32; i++) {
      threadIdx.x = downwards ? 31 - i : i;
      if (done[threadIdx.x]) continue;
      swapcontext(&sched_ctx, &lane_ctx[threadIdx.x]);
      more = true;
    }
  }
  return g_info;
}

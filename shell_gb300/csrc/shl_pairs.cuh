// shl_pairs.cuh -- closest points of a block's triangle pairs (internal).
//
// The fifteen tests of a pair are FP64 without contraction and GB300 issues
// two FP64 lanes per clock and SM, so a kernel that runs them all is bound by
// the FP64 pipe.  FP32 bounds (shl_prune.h) leave one test (interior against
// vertex, crossing edges), three (vertex against edge) or six (vertex against
// vertex) per pair, 3.4 on average in a folded shell and different ones from
// pair to pair, so a block lists its pairs' remaining tests in shared memory
// and deals them out densely: a warp runs 32 edge tests, or 32 vertex tests,
// whichever pairs they belong to.  Dealt out within each warp, 2.2 edge and
// 1.2 vertex tests per pair took three and two trips; over the block they take
// 2.2 and 1.2.  Each thread then takes its own pair's results in the order of
// the tests, with the strict comparison of shl_pair_compute, so the result is
// the same bit for bit.  Folded level-6 shell, 1.7 M pairs: the contact forces
// 6.26 -> 2.35 ms, the narrow phase of a list build 5.75 -> 1.56 ms (dealt out
// per warp 2.87 and 2.06); still bound by the FP64 pipe (80-83 % busy).
#ifndef SHL_PAIRS_CUH_
#define SHL_PAIRS_CUH_

#include <cstdint>

#include "shl_geom.h"
#include "shl_prune.h"

namespace shl {

constexpr int kPairBlock = 256;  // threads of a block that calls pair_compute_block

// a block's scratch: its pairs' vertices, one round's results, the test list
struct PairWork {
  double p[18][kPairBlock];
  double res[6][kPairBlock];  // d2, dc, the two parameters
  uint16_t item[9 * kPairBlock];
  uint32_t warp_sum[kPairBlock / 32];
};

// All threads of the block call it; those without a pair (active = false) only
// help.  P1, P2: the pair's vertices (shl_pair_compute's arguments).
__device__ __forceinline__ void pair_compute_block(bool active, const double* const* P1, const double* const* P2,
                                                   PairWork& w, shl_pair_geom* g) {
  const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  unsigned mask = 0;
  if (active) {
    double q[2][3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        q[0][k][c] = P1[k][c];
        q[1][k][c] = P2[k][c];
        w.p[3 * k + c][tid] = q[0][k][c];
        w.p[9 + 3 * k + c][tid] = q[1][k][c];
      }
    const double* const q1[3] = {q[0][0], q[0][1], q[0][2]};
    const double* const q2[3] = {q[1][0], q[1][1], q[1][2]};
    mask = shl_pair_mask(q1, q2);
  }
  // the best test so far: its d2 as bits.  d2 is a sum of squares, whose bits
  // compare as unsigned integers the way the doubles do, or NaN, whose bits with
  // either sign are above DBL_MAX's (a face without area gives 0/0, and the
  // device's NaN has its sign set: as a signed integer it would be the smallest)
  unsigned long long best = (unsigned long long)__double_as_longlong(SHL_DBL_MAX);
  int best_k = -1;
  double dc[3] = {0.0, 0.0, 0.0}, par[2] = {0.0, 0.0};
#pragma unroll 1
  for (int vertex = 0; vertex < 2; ++vertex) {
    unsigned m = vertex ? mask >> 9 : mask & 0x1ffu;
    const uint32_t cnt = __popc(m);
    uint32_t end = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= (unsigned)o) end += y;
    }
    if (lane == 31) w.warp_sum[warp] = end;
    __syncthreads();
    uint32_t total = 0;
#pragma unroll
    for (int k = 0; k < kPairBlock / 32; ++k) {
      const uint32_t x = w.warp_sum[k];
      if (k < (int)warp) end += x;
      total += x;
    }
    uint32_t at = end - cnt;
    for (uint32_t i = at; m; m &= m - 1) w.item[i++] = (uint16_t)((tid << 4) | (unsigned)(__ffs(m) - 1));
    __syncthreads();
#pragma unroll 1
    for (uint32_t base = 0; base < total; base += kPairBlock) {
      const uint32_t i = base + tid;
      if (i < total) {
        const unsigned it = w.item[i], src = it >> 4, k = it & 15u;
        const int a = (int)k / 3, b = (int)k - 3 * a;
        double d[3], s[2];
        if (!vertex) {
          const int a1 = a == 2 ? 0 : a + 1, b1 = b == 2 ? 0 : b + 1;
          double s0[3], s1[3], t0[3], t1[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            s0[c] = w.p[3 * a + c][src];
            s1[c] = w.p[3 * a1 + c][src];
            t0[c] = w.p[9 + 3 * b + c][src];
            t1[c] = w.p[9 + 3 * b1 + c][src];
          }
          shl_segment_segment(s0, s1, t0, t1, d, s);
        } else {
          const int pv = 9 * a + 3 * b, pf = 9 - 9 * a;
          double v[3], f0[3], f1[3], f2[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            v[c] = w.p[pv + c][src];
            f0[c] = w.p[pf + c][src];
            f1[c] = w.p[pf + 3 + c][src];
            f2[c] = w.p[pf + 6 + c][src];
          }
          shl_point_triangle(v, f0, f1, f2, d, s);
        }
        w.res[0][tid] = shl_v3_dot(d, d);
        w.res[1][tid] = d[0];
        w.res[2][tid] = d[1];
        w.res[3][tid] = d[2];
        w.res[4][tid] = s[0];
        w.res[5][tid] = s[1];
      }
      __syncthreads();
      for (; at < end && at < base + kPairBlock; ++at) {
        const uint32_t r = at - base;
        const unsigned long long d2 = (unsigned long long)__double_as_longlong(w.res[0][r]);
        if (d2 < best) {
          best = d2;
          best_k = (int)(w.item[at] & 15u) + 9 * vertex;
          dc[0] = w.res[1][r]; dc[1] = w.res[2][r]; dc[2] = w.res[3][r];
          par[0] = w.res[4][r]; par[1] = w.res[5][r];
        }
      }
      __syncthreads();
    }
  }
  shl_pair_none(g);
  const double d2 = __longlong_as_double((long long)best);
  if (best_k >= 9)
    shl_pair_take_vertex((best_k - 9) / 3, (best_k - 9) % 3, d2, dc, par, g);
  else if (best_k >= 0)
    shl_pair_take_edges(best_k / 3, best_k % 3, d2, dc, par, g);
}

}  // namespace shl

#endif  // SHL_PAIRS_CUH_

/*
 * shl_prune.h -- which of the fifteen closest-point tests of a pair of
 * triangles can hold the minimum.
 *
 * shl_pair_compute (shl_geom.h) takes the smallest of nine edge-edge and six
 * vertex-face distances, each solved in FP64 with every operation rounded on
 * its own.  All but one or two of the tests are far above the minimum, and
 * GB300 issues 64 FP32 operations per FP64 operation, so the distances are
 * first bounded in FP32: a test whose lower bound lies above the smallest upper
 * bound cannot win, and leaving it out leaves the result (the first test that
 * attains the smallest computed value) unchanged bit for bit.
 *
 * The coordinates are taken relative to the first vertex (FP64 difference) and
 * scaled to unit size, so the bounds are absolute: every vector is at most 2
 * long and eps = 2^-24.
 *  - Edge-edge.  Any (s, t) in the unit square gives a distance at or above
 *    the minimum; the FP32 parameters miss the minimising ones by what the
 *    rounding of the 2x2 system does, which raises d^2 by at most the rounding
 *    of its coefficients: for nearly parallel edges the parameter error grows,
 *    but the quadratic flattens in proportion, and the end that a clamped
 *    parameter takes follows the sign of the numerator, not of the vanishing
 *    determinant.  Largest difference from FP64 (layers, slivers, parallel,
 *    touching, needle edges): 20 eps in 6e8 edge pairs of a host build (no
 *    contraction, true division); 13 eps in the 1e7 edge pairs that the GPU test
 *    of the block search sends through the device build (contraction, fast
 *    division).  The bound allows SHL_PRUNE_E = 128 eps.
 *  - Vertex-face.  Projection clearly outside: the minimum over the face's
 *    three edges (same bound).  Otherwise the plane's distance, less its
 *    rounding (SHL_PRUNE_P eps / sin of the corner angle).  A face with a
 *    corner angle below 0.01 keeps its tests.
 * Non-finite or out-of-range input keeps every test.
 */
#ifndef SHL_PRUNE_H_
#define SHL_PRUNE_H_

#include <math.h>

#include "shl_distance.h"

#define SHL_PRUNE_EPS 5.9604645e-8f
#define SHL_PRUNE_E (128.f * SHL_PRUNE_EPS)
#define SHL_PRUNE_P 64.f
#define SHL_PRUNE_ALL 0x7fffu

#ifdef __CUDA_ARCH__
#define SHL_FDIV(a, b) __fdividef((a), (b))
#define SHL_RSQRTF(a) rsqrtf(a)
#define SHL_SATF(a) __saturatef(a)
#else
#define SHL_FDIV(a, b) ((a) / (b))
#define SHL_RSQRTF(a) (1.0f / sqrtf(a))
#define SHL_SATF(a) ((a) > 0.f ? ((a) < 1.f ? (a) : 1.f) : 0.f)
#endif

SHL_HD float shl_f3_dot(const float* a, const float* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }

/* squared distance of the segments p + s d1, q + t d2 (s, t in [0, 1]), r = p - q */
SHL_HD float shl_f_segments(const float* d1, const float* d2, const float* r, float a, float e)
{
  const float f = shl_f3_dot(d2, r), c = shl_f3_dot(d1, r), b = shl_f3_dot(d1, d2);
  const float num = b * f - c * e, den = fmaxf(a * e - b * b, 1e-30f);
  /* the clamped optimum has the sign of num also where den is all rounding */
  float s = num > 0.f ? (num < den ? SHL_FDIV(num, den) : 1.f) : 0.f;
  const float tn = b * s + f;
  float t = e > 0.f ? SHL_SATF(SHL_FDIV(tn, e)) : 0.f;
  if (!(tn >= 0.f && tn <= e) || !(e > 0.f)) s = a > 0.f ? SHL_SATF(SHL_FDIV(b * t - c, a)) : 0.f;
  float w[3];
  for (int k = 0; k < 3; ++k) w[k] = r[k] + s * d1[k] - t * d2[k];
  return shl_f3_dot(w, w);
}

/* squared distance of a point to the segment q + t d, r = point - q */
SHL_HD float shl_f_point_segment(const float* d, const float* r, float e)
{
  const float t = e > 0.f ? SHL_SATF(SHL_FDIV(shl_f3_dot(d, r), e)) : 0.f;
  float w[3];
  for (int k = 0; k < 3; ++k) w[k] = r[k] - t * d[k];
  return shl_f3_dot(w, w);
}

/* Bit 3 i + j: edge i of element 1 against edge j of element 2; bit
 * 9 + 3 i + j: vertex j of element i + 1 against the other face. */
SHL_HD unsigned shl_pair_mask(const double* const* p1, const double* const* p2)
{
  float P[2][3][3];
  float M2 = 0.f;
  for (int k = 0; k < 3; ++k) {
    for (int c = 0; c < 3; ++c) {
      P[0][k][c] = k == 0 ? 0.f : (float)SHL_SUB(p1[k][c], p1[0][c]);
      P[1][k][c] = (float)SHL_SUB(p2[k][c], p1[0][c]);
    }
    M2 = fmaxf(M2, fmaxf(shl_f3_dot(P[0][k], P[0][k]), shl_f3_dot(P[1][k], P[1][k])));
  }
  if (!(M2 > 1e-30f && M2 < 1e30f)) return SHL_PRUNE_ALL;
  const float sc = SHL_RSQRTF(M2);
  float E[2][3][3], el[2][3];
  for (int t = 0; t < 2; ++t)
    for (int k = 0; k < 3; ++k)
      for (int c = 0; c < 3; ++c) P[t][k][c] *= sc;
  for (int t = 0; t < 2; ++t)
    for (int k = 0; k < 3; ++k) {
      const int k1 = k == 2 ? 0 : k + 1;
      for (int c = 0; c < 3; ++c) E[t][k][c] = P[t][k1][c] - P[t][k][c];
      el[t][k] = shl_f3_dot(E[t][k], E[t][k]);
    }
  float lb[15];
  float ub = 3.0e38f;
  bool bad = false;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      float r[3];
      for (int c = 0; c < 3; ++c) r[c] = P[0][i][c] - P[1][j][c];
      const float d2 = shl_f_segments(E[0][i], E[1][j], r, el[0][i], el[1][j]);
      bad = bad || !(d2 < 3.0e38f);
      lb[3 * i + j] = d2 - SHL_PRUNE_E;
      ub = fminf(ub, d2 + SHL_PRUNE_E);
    }
  for (int i = 0; i < 2; ++i) {
    const float(*B)[3] = P[1 - i]; /* the face */
    const float(*Eb)[3] = E[1 - i];
    const float* lb2 = el[1 - i];
    /* ab = Eb[0], ac = -Eb[2] */
    const float n[3] = {Eb[0][2] * Eb[2][1] - Eb[0][1] * Eb[2][2], Eb[0][0] * Eb[2][2] - Eb[0][2] * Eb[2][0],
                        Eb[0][1] * Eb[2][0] - Eb[0][0] * Eb[2][1]};
    const float nn = shl_f3_dot(n, n), ll = lb2[0] * lb2[2];
    const bool ok = nn > 1e-4f * ll && nn > 1e-12f;
    const float in = ok ? SHL_RSQRTF(nn) : 0.f;
    const float len = sqrtf(lb2[0]) + sqrtf(lb2[2]);
    const float obl = sqrtf(ll) * in; /* 1 / sin of the corner angle */
    const float dp = SHL_PRUNE_P * SHL_PRUNE_EPS * (1.f + obl);
    const float tau = SHL_PRUNE_P * SHL_PRUNE_EPS * len * in * (1.f + obl);
    for (int j = 0; j < 3; ++j) {
      const float* q = P[i][j];
      float r0[3], r1[3], r2[3];
      for (int c = 0; c < 3; ++c) {
        r0[c] = q[c] - B[0][c];
        r1[c] = q[c] - B[1][c];
        r2[c] = q[c] - B[2][c];
      }
      /* barycentric coordinates of the projection, times nn: (ap x ac).n and (ab x ap).n */
      const float cv[3] = {r0[2] * Eb[2][1] - r0[1] * Eb[2][2], r0[0] * Eb[2][2] - r0[2] * Eb[2][0],
                           r0[1] * Eb[2][0] - r0[0] * Eb[2][1]};
      const float cw[3] = {Eb[0][1] * r0[2] - Eb[0][2] * r0[1], Eb[0][2] * r0[0] - Eb[0][0] * r0[2],
                           Eb[0][0] * r0[1] - Eb[0][1] * r0[0]};
      const float v = shl_f3_dot(cv, n) * in * in, w = shl_f3_dot(cw, n) * in * in, u = 1.f - v - w;
      const float h = fabsf(shl_f3_dot(r0, n)) * in;
      float low;
      if (!ok) {
        low = -1.f;
      } else if (v < -tau || w < -tau || u < -3.f * tau) {
        const float e0 = shl_f_point_segment(Eb[0], r0, lb2[0]), e1 = shl_f_point_segment(Eb[1], r1, lb2[1]),
                    e2 = shl_f_point_segment(Eb[2], r2, lb2[2]);
        low = fminf(e0, fminf(e1, e2)) - SHL_PRUNE_E;
      } else {
        const float hl = fmaxf(h - dp, 0.f), hu = h + dp;
        low = hl * hl;
        if (v > tau && w > tau && u > 3.f * tau) ub = fminf(ub, hu * hu);
      }
      lb[9 + 3 * i + j] = low;
    }
  }
  if (bad) return SHL_PRUNE_ALL;
  unsigned mask = 0;
  for (int k = 0; k < 15; ++k)
    if (!(lb[k] > ub)) mask |= 1u << k;
  return mask;
}

#endif /* SHL_PRUNE_H_ */

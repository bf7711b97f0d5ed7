// shl_split.cuh -- the FP64 path's element force, in double-float arithmetic with
// a face's three components on three lanes (internal).
//
// A face's force is a long dependent chain (about 10,000 double-float
// instructions in one thread): with a thread per face the kernel was bound by
// the latency of that chain and by fetching 180 KB of straight-line code, 34 us
// for a mesh of any size up to ten thousand faces, and at 200,000 faces two
// rounds of them on 24 % of the warp slots.  Here lane 3 f + c of a warp holds
// component c of every vector of the warp's face f (ten faces per warp): vector
// operations are one instruction instead of three, cross products and dot
// products exchange neighbours' components by shuffles, and each row of the
// stress resultants is one lane's.  The chain is a third as long and needs 96
// registers, so that twice the warps share an SM.  Cold, in us, against the thread
// per face: 1,280 faces 59 -> 30, 81,920 faces 77 -> 47, 163,840 faces 132 -> 72
// (warm, 8,820 faces 34 -> 15).  Of that, summing products in one accumulator, exact
// power-of-two weights and sums made by one lane for all three are 84 -> 72 at
// 163,840 faces.  Bound by FP32 issue at the large end (61-64 % of the slots) and by
// the chain at the small.
//
// The mechanics are those of the relative-displacement form: no step subtracts
// nearly equal quantities.
//   du_a = displacement derivatives, d_k = second derivatives (material frame)
//   alpha_11 = (A1 + du1/2).du1, alpha_22 = (A2 + du2/2).du2,
//   alpha_12 = A1.du2 + du1.(A2 + du2)                    (shear doubled)
//   Dn = a1 x a2 - A1 x A2 = A1 x du2 + du1 x (A2 + du2)
//   |a1 x a2|^2 - L0^2 = (2 L0 N0 + Dn).Dn, n - N0 = dn from them
//   beta_k = -t_k, t_k = D_k.dn + d_k.n, h_k = B_k + t_k  (shear doubled)
//   sum_k m_k p_ak (ShellSystem.C:1223-1233) = (W x a2, a1 x W) / |a1 x a2|,
//   W = M - (M.n) n, M = m0 v1 + m1 v2 + 2 m2 v3, M.n = m0 h0 + m1 h1 + 2 m2 h2
// On a regular patch the basis and its derivatives at the centroid are integers
// over 972, 324 and 108: the contractions with the patch nodes and back to them
// multiply by exact small integers, and the denominators are folded into the
// face's constants.
#ifndef SHL_SPLIT_CUH_
#define SHL_SPLIT_CUH_

#include <cstdint>

#include "shl_df.cuh"
#include "shl_internal.cuh"

namespace shl {

// basis (phi, d/dv, d/dw, d2/dv2, d2/dw2, d2/dvdw) of a regular patch's slots at
// the centroid, times 972, 162, 162, 18, 18, 18 (kSplitDen1, kSplitDen2: most of
// the derivatives are powers of two)
#define SHL_REGULAR_BASIS { \
    {276, -78, -78, -4, -4, 4}, {276, 78, 0, -4, -16, -8}, {276, 0, 78, -16, -4, -8}, \
    {42, -30, 0, 8, -4, -2},    {3, -5, -4, 4, 2, 3},      {3, -4, -5, 2, 4, 3}, \
    {42, 0, -30, -4, 8, -2},    {42, 30, 30, 8, 8, 10},    {3, 5, 1, 4, 0, 1}, \
    {3, 4, -1, 2, 0, -1},       {3, 1, 5, 0, 4, 1},        {3, -1, 4, 0, 2, -1}}

static_assert(kSplitFaces * 3 <= 32, "three lanes per face (lanes 30 and 31 repeat the last face)");

__device__ __forceinline__ df2 scale2(float s, df2 x) { return {s * x.h, s * x.l}; }  // s a power of two or 0
__device__ __forceinline__ df2 lane_of(df2 x, int src) {
  return {__shfl_sync(0xffffffffu, x.h, src), __shfl_sync(0xffffffffu, x.l, src)};
}

// a sum of products; its terms' errors go to l, normalised once at the end (a
// product and its sum cost 12 instructions, where df2's operators take 18)
struct Acc {
  float h = 0.f, l = 0.f;
  __device__ __forceinline__ void first(float w, df2 x) {
    h = __fmul_rn(w, x.h);
    l = __fmaf_rn(w, x.l, __fmaf_rn(w, x.h, -h));
  }
  __device__ __forceinline__ void two_sum(float p, float e) {
    const float s = __fadd_rn(h, p);
    const float bb = __fsub_rn(s, h);
    const float err = __fadd_rn(__fsub_rn(h, __fsub_rn(s, bb)), __fsub_rn(p, bb));
    l = __fadd_rn(l, __fadd_rn(e, err));
    h = s;
  }
  __device__ __forceinline__ void add(float w, df2 x) {
    const float p = __fmul_rn(w, x.h);
    two_sum(p, __fmaf_rn(w, x.l, __fmaf_rn(w, x.h, -p)));
  }
  __device__ __forceinline__ void add(float2 w, df2 x) {
    const float p = __fmul_rn(w.x, x.h);
    two_sum(p, __fmaf_rn(w.y, x.h, __fmaf_rn(w.x, x.l, __fmaf_rn(w.x, x.h, -p))));
  }
  // w a power of two: the product is exact
  __device__ __forceinline__ void first_exact(float w, df2 x) {
    h = __fmul_rn(w, x.h);
    l = __fmul_rn(w, x.l);
  }
  __device__ __forceinline__ void add_exact(float w, df2 x) {
    const float s = __fmaf_rn(w, x.h, h);
    const float bb = __fsub_rn(s, h);
    const float err = __fadd_rn(__fsub_rn(h, __fsub_rn(s, bb)), __fmaf_rn(w, x.h, -bb));
    l = __fadd_rn(l, __fmaf_rn(w, x.l, err));
    h = s;
  }
  // w a compile-time integer
  __device__ __forceinline__ void first_int(int w, df2 x) {
    if ((w & (w - 1)) == 0 || (-w & (-w - 1)) == 0) first_exact((float)w, x);
    else first((float)w, x);
  }
  __device__ __forceinline__ void add_int(int w, df2 x) {
    if ((w & (w - 1)) == 0 || (-w & (-w - 1)) == 0) add_exact((float)w, x);
    else add((float)w, x);
  }
  __device__ __forceinline__ void first(df2 x, df2 y) {
    h = __fmul_rn(x.h, y.h);
    l = __fmaf_rn(x.l, y.h, __fmaf_rn(x.h, y.l, __fmaf_rn(x.h, y.h, -h)));
  }
  __device__ __forceinline__ void add(df2 x, df2 y) {
    const float p = __fmul_rn(x.h, y.h);
    two_sum(p, __fmaf_rn(x.l, y.h, __fmaf_rn(x.h, y.l, __fmaf_rn(x.h, y.h, -p))));
  }
  __device__ __forceinline__ df2 value() const {
    df2 r;
    df_quick_two_sum(h, l, r.h, r.l);
    return r;
  }
};

__device__ __forceinline__ df2 dot2(df2 x0, df2 y0, df2 x1, df2 y1) {
  Acc a;
  a.first(x0, y0);
  a.add(x1, y1);
  return a.value();
}
__device__ __forceinline__ df2 dot3(df2 x0, df2 y0, df2 x1, df2 y1, df2 x2, df2 y2) {
  Acc a;
  a.first(x0, y0);
  a.add(x1, y1);
  a.add(x2, y2);
  return a.value();
}
__device__ __forceinline__ df2 dot4(df2 x0, df2 y0, df2 x1, df2 y1, df2 x2, df2 y2, df2 x3, df2 y3) {
  Acc a;
  a.first(x0, y0);
  a.add(x1, y1);
  a.add(x2, y2);
  a.add(x3, y3);
  return a.value();
}
__device__ __forceinline__ df2 pick(int c, df2 x0, df2 x1, df2 x2) { return c == 0 ? x0 : (c == 1 ? x1 : x2); }

// a warp's shared memory: its faces' constants; for irregular patches also the
// group's basis (float pairs) and the patch ids
struct SplitWarp {
  alignas(16) df2 face[kSplitFaces * kSplitStride];
  float2 basis[kMaxSlots * 6];
  int32_t id[kMaxSlots * kSplitFaces];
};
static_assert(sizeof(SplitWarp) % 16 == 0 && kSplitStride * sizeof(df2) % 16 == 0, "16-byte copies");

__device__ __forceinline__ void split_copy16(void* smem, const void* gmem) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem) : "memory");
}

// component c of u_pred at node nd
__device__ __forceinline__ df2 split_u(const DevBuf& b, int nd, int c) {
  const float2 x = __ldg(reinterpret_cast<const float2*>(b.upk) + 4 * (size_t)nd + c);
  return {x.x, x.y};
}

// One warp: faces first .. first + nf of patch group gd (nf <= kSplitFaces).
template <bool REG>
__device__ __forceinline__ void split_faces(const DevBuf& b, const StepConst& sc, const ElemGroups& eg,
                                            const GroupDesc& gd, uint32_t first, uint32_t nf, double pressure,
                                            double vol_p, SplitWarp& w) {
  const uint32_t lane = threadIdx.x & 31u;
  const int c = (int)(lane % 3u), base = (int)lane - c;
  const int cj = c == 2 ? 0 : c + 1, ck = c == 0 ? 2 : c - 1;
  const int lj = base + cj, lk = base + ck;  // the lanes of the next two components
  const uint32_t f = lane / 3u < nf ? lane / 3u : nf - 1;
  const bool valid = lane / 3u < nf && lane < 3u * kSplitFaces;
  const uint32_t i = first + f;
  const int np = REG ? 12 : gd.n_slots;
  __syncwarp();
  {
    constexpr uint32_t per_face = kSplitStride * sizeof(df2) / 16;
    const char* src = reinterpret_cast<const char*>(b.face_df) + (size_t)first * kSplitStride * sizeof(df2);
    for (uint32_t t = lane; t < nf * per_face; t += 32)
      split_copy16(reinterpret_cast<char*>(w.face) + 16 * t, src + 16 * (size_t)t);
  }
  df2 x[REG ? 12 : 1];  // the patch's displacements (this lane's component)
  if (REG) {
    int nd[12];
    const int4* id = reinterpret_cast<const int4*>(b.patch12) + 3 * (size_t)i;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int4 v = __ldg(&id[q]);
      nd[4 * q] = v.x; nd[4 * q + 1] = v.y; nd[4 * q + 2] = v.z; nd[4 * q + 3] = v.w;
    }
#pragma unroll
    for (int s = 0; s < 12; ++s) x[REG ? s : 0] = split_u(b, nd[s], c);
  } else {
    for (uint32_t t = lane; t < 6u * (uint32_t)np; t += 32) w.basis[t] = __ldg(&eg.basis_df[gd.basis_off + t]);
    for (uint32_t t = lane; t < (uint32_t)np * nf; t += 32)
      w.id[(t / nf) * kSplitFaces + t % nf] = __ldg(&b.patch[(size_t)(t / nf) * sc.F + first + t % nf]);
    __syncwarp();
  }
  const bool need_x = sc.pressure_base == SHL_CS_CYLINDRICAL || sc.pressure_base == SHL_CS_SPHERICAL;
  // G[k] = sum_s B[s][k] u_s (times the denominators on a regular patch)
  const signed short RB[12][6] = SHL_REGULAR_BASIS;  // folds into the unrolled code
  df2 G[6];
  {
    Acc a[6];
    if (REG) {
#pragma unroll
      for (int s = 0; s < 12; ++s)
#pragma unroll
        for (int k = 1; k < 6; ++k) {
          if (RB[s][k] == 0) continue;
          if (s == 0)
            a[k].first_int(RB[s][k], x[REG ? s : 0]);
          else
            a[k].add_int(RB[s][k], x[REG ? s : 0]);
        }
      if (need_x) {
#pragma unroll
        for (int s = 0; s < 12; ++s) a[0].add((float)RB[s][0], x[REG ? s : 0]);
      }
    } else {
#pragma unroll 2
      for (int s = 0; s < np; ++s) {
        const df2 us = split_u(b, w.id[s * kSplitFaces + f], c);
#pragma unroll
        for (int k = 0; k < 6; ++k) a[k].add(w.basis[6 * s + k], us);
      }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) G[k] = a[k].value();
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncwarp();
  const df2* fc = w.face + f * kSplitStride;
  const df2 R00 = fc[SF_R00], R01 = fc[SF_R01], R10 = fc[SF_R10], R11 = fc[SF_R11];
  const df2 du1 = dot2(R00, G[1], R10, G[2]), du2 = dot2(R01, G[1], R11, G[2]);
  const df2 A1 = fc[SF_A1 + c], a1 = A1 + du1, a2 = fc[SF_A2 + c] + du2;
  const df2 d1 = dot3(fc[SF_C11A], G[3], fc[SF_C11B], G[4], fc[SF_C11C], G[5]);
  const df2 d2 = dot3(fc[SF_C22A], G[3], fc[SF_C22B], G[4], fc[SF_C22C], G[5]);
  const df2 d3 = dot3(fc[SF_C12A], G[3], fc[SF_C12B], G[4], fc[SF_C12C], G[5]);
  // the sum of a value over the face's three lanes, in component order on each
  auto sum3 = [&](df2 v) { return (lane_of(v, base) + lane_of(v, base + 1)) + lane_of(v, base + 2); };
  // three such sums, one made by each lane and handed to the others
  auto sum3x3 = [&](df2 v0, df2 v1, df2 v2, df2& s0, df2& s1, df2& s2) {
    const df2 next = lane_of(pick(ck, v0, v1, v2), lj), prev = lane_of(pick(cj, v0, v1, v2), lk);
    const df2 t = (pick(c, v0, v1, v2) + next) + prev;
    s0 = lane_of(t, base); s1 = lane_of(t, base + 1); s2 = lane_of(t, base + 2);
  };
  df2 al0, al1, al2;
  sum3x3((A1 + scale2(0.5f, du1)) * du1, (fc[SF_A2 + c] + scale2(0.5f, du2)) * du2, dot2(A1, du2, du1, a2), al0, al1,
         al2);
  const df2 a2j = lane_of(a2, lj), a2k = lane_of(a2, lk);
  df2 Dn;
  {
    const df2 du1j = lane_of(du1, lj), du1k = lane_of(du1, lk), du2j = lane_of(du2, lj), du2k = lane_of(du2, lk);
    Dn = dot4(fc[SF_A1 + cj], du2k, -fc[SF_A1 + ck], du2j, du1j, a2k, -du1k, a2j);
  }
  const df2 N0 = fc[SF_N + c], L0 = fc[SF_L0];
  const df2 dL2 = sum3((scale2(2.f, L0 * N0) + Dn) * Dn);  // |a1 x a2|^2 - L0^2
  const df2 jac2 = L0 * L0 + dL2, jac = df_sqrt(jac2);
  const df2 invjac = df_recip(jac);
  const df2 s_n = -(dL2 * df_recip((L0 + jac) * jac));  // L0 / jac - 1
  const df2 dn = dot2(Dn, invjac, N0, s_n);
  const df2 a3 = N0 + dn;
  const df2 D1 = fc[SF_D1 + c], D2 = fc[SF_D2 + c], D3 = fc[SF_D3 + c];
  df2 t0, t1, t2;
  sum3x3(dot2(D1, dn, d1, a3), dot2(D2, dn, d2, a3), dot2(D3, dn, d3, a3), t0, t1, t2);
  const df2 h0 = fc[SF_B] + t0, h1 = fc[SF_B + 1] + t1, h2 = fc[SF_B + 2] + t2;
  // stress resultants times JxW: row c of H on lane c
  const df2 JxW = fc[SF_JXW];
  df2 n0, n1, n2, m0, m1, m2, energy;  // energy: on lane 1 the membrane's, on lane 2 the bending's
  {
    const int q1 = c == 0 ? 1 : c + 2, q2 = c == 0 ? 2 : c + 3;
    const df2 Hc0 = fc[SF_H + c], Hc1 = fc[SF_H + q1], Hc2 = fc[SF_H + q2];
    const float on = (float)sc.internal_scale;  // 1, or 0 for the pressure-only force
    const df2 n = (scale2(on, fc[SF_K]) * JxW) * dot3(Hc0, al0, Hc1, al1, Hc2, al2);
    const df2 m = (scale2(-on, fc[SF_D]) * JxW) * dot3(Hc0, t0, Hc1, t1, scale2(2.f, Hc2), t2);
    const df2 en = n * pick(c, al0, al1, al2), em = -(m * pick(c, t0, t1, scale2(2.f, t2)));
    const df2 en0 = lane_of(en, base), em0 = lane_of(em, base);
    const df2 other = lane_of(c == 2 ? en : em, c == 1 ? base + 2 : base + 1);
    energy = ((c == 1 ? en0 : em0) + (c == 1 ? en : em)) + other;
    n0 = lane_of(n, base); n1 = lane_of(n, base + 1); n2 = lane_of(n, base + 2);
    m0 = lane_of(m, base); m1 = lane_of(m, base + 1); m2 = lane_of(m, base + 2);
  }
  // the share positions: in flight during the rest
  uint32_t pos[REG ? 12 : 1];
  const uint32_t slot0 = gd.slot_base + (i - gd.first) * (uint32_t)np;
  if (REG) {
    const uint4* sp = reinterpret_cast<const uint4*>(b.slot_pos + slot0);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const uint4 v = __ldg(&sp[q]);
      pos[REG ? 4 * q : 0] = v.x; pos[REG ? 4 * q + 1 : 0] = v.y;
      pos[REG ? 4 * q + 2 : 0] = v.z; pos[REG ? 4 * q + 3 : 0] = v.w;
    }
  }
  if (valid) {
    // the measurements per unit area (area = jac / 2, and the metric's determinant is jac^2)
    const uint32_t e = __ldg(&b.perm[i]);
    // (two values a lane: a value's conversion is FP64, 16 cycles of the SM's pipe)
    const df2 g0 = fc[SF_G] + scale2(2.f, al0), g1 = fc[SF_G + 1] + scale2(2.f, al1), g2 = fc[SF_G + 2] + al2;
    const df2 ei = energy * invjac;
    double* to = c == 0 ? b.area : (c == 1 ? b.etens : b.ebend);
    to[e] = df_to_double(c == 0 ? scale2(0.5f, jac) : ei);
    // Gaussian curvature h0 h1 - h2 h2 on lane 1, mean (h0 g1 + h1 g0) / 2 - h2 g2 on lane 2,
    // over the determinant: by 1 / jac twice, both the root's and the reciprocal's
    // rounding would count double (mean curvature's error 2.0e-14 -> 2.3e-14)
    const df2 k = dot3(h0, c == 1 ? h1 : scale2(0.5f, g1), h1, c == 1 ? dfv(0.f) : scale2(0.5f, g0), -h2,
                       c == 1 ? h2 : g2) * df_recip(jac2);
    if (c > 0) (c == 1 ? b.kG : b.kM)[e] = df_to_double(k);
  }
  df2 Y1, Y2;
  {
    const df2 sm = dot3(m0, h0, m1, h1, scale2(2.f, m2), h2);
    const df2 W = dot4(m0, D1 + d1, m1, D2 + d2, scale2(2.f, m2), D3 + d3, -sm, a3) * invjac;
    const df2 Wj = lane_of(W, lj), Wk = lane_of(W, lk), a1j = lane_of(a1, lj), a1k = lane_of(a1, lk);
    Y1 = dot4(n0, a1, n2, a2, Wj, a2k, -Wk, a2j);
    Y2 = dot4(n1, a2, n2, a1, a1j, Wk, -a1k, Wj);
  }
  // pressure (ShellSystem.C:1509-1568), over the basis denominator on a regular patch
  constexpr double phi = REG ? 1.0 / 972.0 : 1.0;
  df2 pv = dfv(0.f);
  {
    const double pf = pressure * __ldg(&b.pscale[i]);
    df2 dir = a3;
    if (sc.pressure_base == SHL_CS_CARTESIAN) {
      dir = dfv(c == sc.pressure_dir ? 1.f : 0.f);
    } else if (need_x) {
      if (sc.pressure_base == SHL_CS_CYLINDRICAL && sc.pressure_dir == 0) {
        dir = dfv(c == 0 ? 1.f : 0.f);
      } else {
        df2 xq = fc[SF_X + c] + df_from_double(phi) * G[0];
        if (sc.pressure_base == SHL_CS_CYLINDRICAL && c == 0) xq = dfv(0.f);
        const df2 r2 = sum3(xq * xq);
        dir = r2.h > 0.f ? df_recip(df_sqrt(r2)) * xq : dfv(0.f);
      }
    }
    if (pf != 0.0) pv = dir * df_from_double(pf * phi);
    if (vol_p != 0.0) pv = pv + a3 * df_from_double(vol_p * phi);
  }
  const df2 y11 = -(m0 * a3), y22 = -(m1 * a3), y12 = -scale2(2.f, m2 * a3);
  df2 Z[6];
  Z[0] = -(JxW * pv);
  Z[1] = dot2(fc[SF_R00], Y1, fc[SF_R01], Y2);
  Z[2] = dot2(fc[SF_R10], Y1, fc[SF_R11], Y2);
  Z[3] = dot3(fc[SF_C11A], y11, fc[SF_C22A], y22, fc[SF_C12A], y12);
  Z[4] = dot3(fc[SF_C11B], y11, fc[SF_C22B], y22, fc[SF_C12B], y12);
  Z[5] = dot3(fc[SF_C11C], y11, fc[SF_C22C], y22, fc[SF_C12C], y12);
  auto put = [&](uint32_t at, df2 t) {
    reinterpret_cast<float2*>(b.qe)[3 * (size_t)at + c] = make_float2(t.h, t.l);
  };
  if (REG) {
#pragma unroll
    for (int s = 0; s < 12; ++s) {
      Acc a;
      a.first_int(RB[s][0], Z[0]);
#pragma unroll
      for (int k = 1; k < 6; ++k)
        if (RB[s][k] != 0) a.add_int(RB[s][k], Z[k]);
      if (valid) put(pos[REG ? s : 0], a.value());
    }
  } else {
#pragma unroll 1
    for (int s = 0; s < np; ++s) {
      Acc a;
#pragma unroll
      for (int k = 0; k < 6; ++k) a.add(w.basis[6 * s + k], Z[k]);
      if (valid) put(__ldg(&b.slot_pos[slot0 + s]), a.value());
    }
  }
}

// warp `chunk` of the mesh: ten faces of one patch group (eg.g[].block_start counts warps)
__device__ __forceinline__ void split_chunk(const DevBuf& b, const StepConst& sc, const ElemGroups& eg, uint32_t chunk,
                                            double pressure, double vol_p, SplitWarp& w) {
  int g = 0;
  while (g + 1 < eg.n && chunk >= eg.g[g + 1].block_start) ++g;
  const GroupDesc gd = eg.g[g];
  const uint32_t done = (chunk - gd.block_start) * kSplitFaces;
  const uint32_t nf = min((uint32_t)kSplitFaces, gd.count - done);
  if (g == 0)
    split_faces<true>(b, sc, eg, gd, gd.first + done, nf, pressure, vol_p, w);
  else
    split_faces<false>(b, sc, eg, gd, gd.first + done, nf, pressure, vol_p, w);
}

template <int BS, int MINB>
__global__ void __launch_bounds__(BS, MINB) k_elements_split(DevBuf b, StepConst sc, ElemGroups eg, uint32_t n_chunks) {
  const Ctl* ctl = b.ctl;
  if (ctl->halted != 0 || ctl->paused != 0) return;
  extern __shared__ __align__(16) unsigned char split_smem[];
  SplitWarp& w = reinterpret_cast<SplitWarp*>(split_smem)[threadIdx.x >> 5];
  const uint32_t chunk = blockIdx.x * (BS / 32) + (threadIdx.x >> 5);
  if (chunk >= n_chunks) return;
  split_chunk(b, sc, eg, chunk, ctl->pressure, ctl->volume_pressure, w);
}

}  // namespace shl

#endif  // SHL_SPLIT_CUH_

// Float32 point evaluator of the lean programs (LP_* forms) in the mixed build
// mode: one or two primitives under a stage, in plain float32, together with a
// bound of the error that the host derives per op (lean_error, px_api.cu).
//
// Coordinates are relative to the op's anchor.  Every constant is the lower end
// of its float32 interval (p32), every operation rounds to nearest.  lean_error
// repeats these expressions on (magnitude, error) pairs -- an operation's error
// is what its operands' errors make of it plus 2^-24 of its result -- so that
// |value - exact| <= err[0] - 2^-30 (the second primitive: err[1]) holds for every
// point of the op's bricks,
// where `exact` is the expression on the exact inputs and 2^-30 m covers the
// reference's own float64 rounding.  A value beyond the bound has the
// reference's sign; anything nearer is left to intervals and float64.
//
// Why this and not intervals (sdf32.cuh): a directed lower and upper bound of
// everything costs 2 to 4 instructions per operation and twice the registers; a
// point costs one, and because coordinates are those of the op, not of the world,
// the bound is some 50 to 300 roundings of the op's size: 1e-4 of a voxel for most
// shapes at 80 voxels per metre (870 voxels of the penthouse left undecided).  With
// tickets of several items (voxel_lean_kernel), lean voxel kernels of the penthouse
// at 80: 204 -> 92 us, at 128: 450 -> 202; the synthetic scene 980 -> 285 us; 256
// edits 187 -> 73 us; its classify pass 72 -> 56 us.
#pragma once
#include "px_internal.cuh"

namespace px {

// sqrt(v), v >= 0, from the hardware reciprocal square root (maximum relative
// error 2^-22.9 by the PTX manual): relative error below 2^-22.3 with the
// product's rounding, 2^-50 absolute below 2^-100.  (The bounds rely on 8 * 2^-24 for
// a length, squares and sums included: eb_len.)
__device__ __forceinline__ float root_f(float v) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fmaxf(v, 0x1p-100f)));
  return v * r;
}
__device__ __forceinline__ float len2_f(float a, float b) { return root_f(__fmaf_rn(b, b, a * a)); }
__device__ __forceinline__ float len3_f(float a, float b, float c) {
  return root_f(__fmaf_rn(c, c, __fmaf_rn(b, b, a * a)));
}
// the distance of a shape extruded by h from its section's d (shapes.ts: cylinder, prism, stadium)
__device__ __forceinline__ float extrude_f(float d, float h) {
  return fminf(fmaxf(d, h), 0.f) + len2_f(fmaxf(d, 0.f), fmaxf(h, 0.f));
}

// shapes.ts:146-161.  The crossing tests run on the polygon of the rounded vertices
// (each edge from its two vertices, the same height compared at both its ends), so
// the parity is exactly that polygon's except within a few roundings of an edge.
template <int N>
__device__ __forceinline__ void polygon_f(const float2* __restrict__ r, int n, const float (&px_)[N],
                                          const float (&py_)[N], float (&out)[N]) {
  float d[N];
  bool flip[N];
  const float x0 = __ldg(&r[0].x), y0 = __ldg(&r[1].x);
  float vjx = __ldg(&r[6 * (n - 1)].x), vjy = __ldg(&r[6 * (n - 1) + 1].x);
#pragma unroll
  for (int q = 0; q < N; q++) {
    const float ax = px_[q] - x0, ay = py_[q] - y0;
    d[q] = __fmaf_rn(ay, ay, ax * ax);
    flip[q] = false;
  }
#pragma unroll 1
  for (int i = 0; i < n; i++, r += 6) {
    const float vix = __ldg(&r[0].x), viy = __ldg(&r[1].x), ex = __ldg(&r[3].x), ey = __ldg(&r[4].x),
                inv = __ldg(&r[5].x);
    const float cx = vjx - vix, cy = vjy - viy;
#pragma unroll
    for (int q = 0; q < N; q++) {
      const float wx = px_[q] - vix, wy = py_[q] - viy;
      const float t = __saturatef(__fmaf_rn(wx, ex, wy * ey) * inv);
      const float bx = __fmaf_rn(-ex, t, wx), by = __fmaf_rn(-ey, t, wy);
      d[q] = fminf(d[q], __fmaf_rn(by, by, bx * bx));
      const bool c1 = py_[q] >= viy, c2 = py_[q] < vjy, c3 = cx * wy > cy * wx;
      flip[q] = flip[q] != (c1 == c2 && c2 == c3);
    }
    vjx = vix;
    vjy = viy;
  }
#pragma unroll
  for (int q = 0; q < N; q++) {
    const float s = root_f(d[q]);
    out[q] = flip[q] ? -s : s;
  }
}

// shapes.ts:164-173
template <int N>
__device__ __forceinline__ void polyline_f(const float2* __restrict__ r, int n, const float (&px_)[N],
                                           const float (&py_)[N], float (&out)[N]) {
  float d[N];
#pragma unroll
  for (int q = 0; q < N; q++) d[q] = INFINITY;
#pragma unroll 1
  for (int i = 0; i < n; i++, r += 5) {
    const float ax = __ldg(&r[0].x), ay = __ldg(&r[1].x), ex = __ldg(&r[2].x), ey = __ldg(&r[3].x), inv = __ldg(&r[4].x);
#pragma unroll
    for (int q = 0; q < N; q++) {
      const float wx = px_[q] - ax, wy = py_[q] - ay;
      const float t = __saturatef(__fmaf_rn(wx, ex, wy * ey) * inv);
      const float bx = __fmaf_rn(-ex, t, wx), by = __fmaf_rn(-ey, t, wy);
      d[q] = fminf(d[q], __fmaf_rn(by, by, bx * bx));
    }
  }
#pragma unroll
  for (int q = 0; q < N; q++) out[q] = root_f(d[q]);
}

// One primitive (w: opcode | count << 8, parameters p) at N points.
template <int N>
__device__ __forceinline__ void prim_f(uint32_t w, const float2* __restrict__ p, const float (&x)[N],
                                       const float (&y)[N], const float (&z)[N], float (&out)[N]) {
  auto c = [&](int k) { return __ldg(&p[k].x); };
  const int cnt = (int)(w >> 8);
  float a[N], b[N], h[N];
  switch (w & 0xffu) {
    case OP_BOX: case OP_ROUNDBOX: {
      const float c0 = c(0), c1 = c(1), c2 = c(2), h0 = c(3), h1 = c(4), h2 = c(5);
      const float r = (w & 0xffu) == OP_ROUNDBOX ? c(6) : 0.f;
#pragma unroll
      for (int q = 0; q < N; q++) {
        const float qx = fabsf(x[q] - c0) - h0, qy = fabsf(y[q] - c1) - h1, qz = fabsf(z[q] - c2) - h2;
        out[q] = (len3_f(fmaxf(qx, 0.f), fmaxf(qy, 0.f), fmaxf(qz, 0.f)) + fminf(fmaxf(fmaxf(qx, qy), qz), 0.f)) - r;
      }
      return;
    }
    case OP_SPHERE: {
      const float c0 = c(0), c1 = c(1), c2 = c(2), r = c(3);
#pragma unroll
      for (int q = 0; q < N; q++) out[q] = len3_f(x[q] - c0, y[q] - c1, z[q] - c2) - r;
      return;
    }
    case OP_ELLIPSOID: {  // parameters 1/rx, 1/ry, 1/rz
#pragma unroll
      for (int q = 0; q < N; q++)
        out[q] = (len3_f((x[q] - c(0)) * c(3), (y[q] - c(1)) * c(4), (z[q] - c(2)) * c(5)) - 1.f) * c(6);
      return;
    }
    case OP_CAPSULE: {  // a, ba, 1/bb, r
      const float c0 = c(0), c1 = c(1), c2 = c(2), ux = c(3), uy = c(4), uz = c(5), inv = c(6), r = c(7);
#pragma unroll
      for (int q = 0; q < N; q++) {
        const float px_ = x[q] - c0, py_ = y[q] - c1, pz_ = z[q] - c2;
        const float t = __saturatef(__fmaf_rn(pz_, uz, __fmaf_rn(py_, uy, px_ * ux)) * inv);
        out[q] = len3_f(__fmaf_rn(-ux, t, px_), __fmaf_rn(-uy, t, py_), __fmaf_rn(-uz, t, pz_)) - r;
      }
      return;
    }
    case OP_CYL_X: case OP_CYL_Y: case OP_CYL_Z: case OP_TORUS_X: case OP_TORUS_Y: case OP_TORUS_Z: {
      const uint32_t op = w & 0xffu;
      const uint32_t axis = op >= OP_TORUS_X ? op - OP_TORUS_X : op - OP_CYL_X;
      const float c0 = c(0), c1 = c(1), c2 = c(2), r = c(3), r2 = c(4);
#pragma unroll
      for (int q = 0; q < N; q++) {
        const float dx = x[q] - c0, dy = y[q] - c1, dz = z[q] - c2;
        a[q] = axis == 0 ? dy : dx;
        b[q] = axis == 2 ? dy : dz;
        h[q] = axis == 0 ? dx : axis == 1 ? dy : dz;
        const float dr = len2_f(a[q], b[q]) - r;
        out[q] = op >= OP_TORUS_X ? len2_f(dr, h[q]) - r2 : extrude_f(dr, fabsf(h[q]) - r2);
      }
      return;
    }
    case OP_LATHE_SOLID: case OP_LATHE_SHELL: {
      const bool shell = (w & 0xffu) == OP_LATHE_SHELL;
#pragma unroll
      for (int q = 0; q < N; q++) {
        a[q] = len2_f(x[q] - c(0), z[q] - c(2));
        b[q] = y[q] - c(1);
      }
      if (!shell) {
        polygon_f<N>(p + 3, cnt, a, b, out);
        return;
      }
      polyline_f<N>(p + 4, cnt - 1, a, b, out);
      const float t = c(3);
#pragma unroll
      for (int q = 0; q < N; q++) out[q] = out[q] - t;
      return;
    }
    case OP_PRISM: {
#pragma unroll
      for (int q = 0; q < N; q++) {
        a[q] = x[q] - c(0);
        b[q] = z[q] - c(1);
      }
      polygon_f<N>(p + 4, cnt, a, b, out);
      const float cy = c(2), hh = c(3);
#pragma unroll
      for (int q = 0; q < N; q++) out[q] = extrude_f(out[q], fabsf(y[q] - cy) - hh);
      return;
    }
    case OP_STADIUM: {
      const float c0 = c(0), c1 = c(1), hx = c(2), r = c(3), cy = c(4), hh = c(5);
#pragma unroll
      for (int q = 0; q < N; q++)
        out[q] = extrude_f(len2_f(fmaxf(fabsf(x[q] - c0) - hx, 0.f), z[q] - c1) - r, fabsf(y[q] - cy) - hh);
      return;
    }
  }
#pragma unroll
  for (int q = 0; q < N; q++) out[q] = NAN;  // not a primitive: undecided
}

// A stage (LP_* kinds) at N points (x, y, z[q]): none, one rotation about an axis
// (pivot's two coordinates, cos, sin: shapes.ts:263-320), or a run composed into
// x' = M x + t (M row by row, then t).  ROT / AFF: the kinds that occur.
template <int N, bool ROT, bool AFF>
__device__ __forceinline__ void stage_f(uint32_t kind, const float2* __restrict__ p, float x, float y, const float (&z)[N],
                                        float (&X)[N], float (&Y)[N], float (&Z)[N]) {
  auto c = [&](int k) { return __ldg(&p[k].x); };
  if constexpr (AFF) {
    if (!ROT || kind == LP_AFFINE) {
#pragma unroll
      for (int r = 0; r < 3; r++) {
        const float base = __fmaf_rn(c(3 * r + 1), y, __fmaf_rn(c(3 * r), x, c(9 + r))), m = c(3 * r + 2);
#pragma unroll
        for (int q = 0; q < N; q++) (r == 0 ? X[q] : r == 1 ? Y[q] : Z[q]) = __fmaf_rn(m, z[q], base);
      }
    }
  }
  if constexpr (ROT) {
    if (AFF && kind == LP_AFFINE) return;
    const float p0 = kind ? c(0) : 0.f, p1 = kind ? c(1) : 0.f, co = kind ? c(2) : 0.f, si = kind ? c(3) : 0.f;
#pragma unroll
    for (int q = 0; q < N; q++) {
      X[q] = x;
      Y[q] = y;
      Z[q] = z[q];
      if (!kind) continue;
      const float u = (kind == 1 ? y : x) - p0, v = (kind == 3 ? y : z[q]) - p1;
      const float nu = __fmaf_rn(co, u, __fmaf_rn(si, v, p0)), nv = __fmaf_rn(co, v, __fmaf_rn(-si, u, p1));
      if (kind == 1) Y[q] = nu;
      else X[q] = nu;
      if (kind == 3) Y[q] = nv;
      else Z[q] = nv;
    }
  }
}

// A lean program at N points of one column (x, y, z[q]): [lo, hi] around each exact
// value, from the error bounds of its primitives (a far second primitive's large
// coordinates then widen nothing but itself).  FORMS: 1 (one primitive) or 3 (any
// form); ROT / AFF: the stage kinds that occur.
template <int N, int FORMS, bool ROT, bool AFF>
__device__ __forceinline__ void lean_f(const FoldArgs& a, const OpDev* __restrict__ V, float x, float y,
                                       const float (&z)[N], float (&lo)[N], float (&hi)[N]) {
  const uint4 l0 = __ldg(reinterpret_cast<const uint4*>(V->lw));
  const float2* __restrict__ P = a.p32;
  const float E = V->err[0];
  float X[N], Y[N], Z[N], d[N];
  stage_f<N, ROT, AFF>((l0.x >> 16) & 15u, P + l0.w, x, y, z, X, Y, Z);
  prim_f<N>(l0.y, P + l0.z, X, Y, Z, d);
#pragma unroll
  for (int q = 0; q < N; q++) {
    lo[q] = __fsub_rd(d[q], E);
    hi[q] = __fadd_ru(d[q], E);
  }
  if (!(l0.x >> 24) && (FORMS == 1 || (l0.x & 0xffu) == 1u)) return;
  const uint4 l1 = __ldg(reinterpret_cast<const uint4*>(V->lw) + 1);
  if (FORMS > 1 && (l0.x & 0xffu) > 1u) {
    if ((l0.x & 0xffu) == 3u) stage_f<N, ROT, AFF>((l0.x >> 20) & 15u, P + l1.z, x, y, z, X, Y, Z);
    prim_f<N>(l1.x, P + l1.y, X, Y, Z, d);
    const uint32_t comb = (l0.x >> 8) & 0xffu;
    const float E2 = V->err[1];
#pragma unroll
    for (int q = 0; q < N; q++) {
      const float v = comb == LP_NEGMAX ? -d[q] : d[q];
      const float l = __fsub_rd(v, E2), h = __fadd_ru(v, E2);
      const bool nan = !(v == v && lo[q] == lo[q]);  // undecided, which minima and maxima would hide
      lo[q] = nan ? -INFINITY : comb == LP_MIN ? fminf(lo[q], l) : fmaxf(lo[q], l);
      hi[q] = nan ? INFINITY : comb == LP_MIN ? fminf(hi[q], h) : fmaxf(hi[q], h);
    }
  }
  if (l0.x >> 24) {  // offset (penthouse.ts:250); both ends of its interval, rounded outward
    const float2 o = __ldg(&P[l1.w]);
#pragma unroll
    for (int q = 0; q < N; q++) {
      lo[q] = __fadd_rd(lo[q], o.x);
      hi[q] = __fadd_ru(hi[q], o.y);
    }
  }
}

}  // namespace px

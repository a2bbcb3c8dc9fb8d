// pg_ttfilter.cuh -- which of the fifteen distances of a triangle pair
// (pg_tritri.cuh) can decide its contact, in FP32.
//
// The narrow phase takes the smallest of six vertex-triangle and nine
// edge-edge distances, each about 80 FP64 operations, after six edge-crossing
// tests; GB300 runs 64 FP32 operations in the time of one of FP64.  For each
// of the fifteen this finds its closest points in FP32, and from them a lower
// bound: with w the difference of the two points, the features' extents along
// w are |w| times at least the bound apart, whatever the error of the points
// themselves.  A candidate whose bound exceeds the smallest distance found
// cannot be the smallest in FP64, and a pair whose bound along the best w
// exceeds 2r is apart; one that it does not separate at all may intersect.
// Rounding: coordinates are taken relative to a vertex of the pair, `tol`
// covers the error of the float vertices (given with them), of the FP32 dot
// products (under 8 2^-24 of the largest coordinate) and of the FP64
// distances, whose points lie on their features up to rounding.  That the
// FP64 minimum does not exceed `upper` is checked on it when it is known.
// Degenerate triangles, whose FP64 tests may answer anything, are not judged.
#pragma once
#include <math.h>

#ifdef __CUDACC__
#define PG_TF __host__ __device__ __forceinline__
#else
#define PG_TF inline
#endif

namespace pgtf {

PG_TF float dot(const float *a, const float *b) { return a[0]*b[0] + a[1]*b[1] + a[2]*b[2]; }
PG_TF float mn(float a, float b) { return a < b ? a : b; }
PG_TF float mx(float a, float b) { return a > b ? a : b; }
PG_TF float clamp01(float x) { return x < 0.0f ? 0.0f : (x > 1.0f ? 1.0f : x); }
// quotient and inverse root to a few units in the last place: the points and
// directions they give serve whatever their error, the bounds have room for it
PG_TF float quot(float a, float b)
{
#ifdef __CUDA_ARCH__
  return __fdividef(a, b);
#else
  return a / b;
#endif
}
PG_TF float iroot(float x)
{
#ifdef __CUDA_ARCH__
  return rsqrtf(x);
#else
  return 1.0f / sqrtf(x);
#endif
}

// closest point of triangle (v[0], v[1], v[2]) to p, in FP32 (any point of
// the triangle serves)
PG_TF void vertex_face(const float *p, const float v[3][3], float *q)
{
  float ab[3], ac[3], ap[3];
  for (int k = 0; k < 3; k ++) { ab[k] = v[1][k] - v[0][k]; ac[k] = v[2][k] - v[0][k]; ap[k] = p[k] - v[0][k]; }
  const float g11 = dot(ab, ab), g12 = dot(ab, ac), g22 = dot(ac, ac);
  const float d1 = dot(ab, ap), d2 = dot(ac, ap);
  const float d3 = d1 - g11, d4 = d2 - g12, d5 = d1 - g12, d6 = d2 - g22;
  const float vc = d1*d4 - d3*d2, vb = d5*d2 - d1*d6, va = d3*d6 - d5*d4;
  // the region's parameters by selection, with one division (q = a + s ab + t ac)
  const float e43 = d4 - d3, e56 = d5 - d6;
  const bool r0 = d1 <= 0.0f && d2 <= 0.0f, r1 = d3 >= 0.0f && d4 <= d3, r2 = vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f,
             r3 = d6 >= 0.0f && d5 <= d6, r4 = vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f,
             r5 = va <= 0.0f && e43 >= 0.0f && e56 >= 0.0f;
  const float num = r2 ? d1 : r4 ? d2 : r5 ? e43 : 1.0f;
  const float den = r2 ? d1 - d3 : r4 ? d2 - d6 : r5 ? e43 + e56 : va + vb + vc;
  const float x = quot(num, den);
  float s = vb * x, t = vc * x;
  if (r5) { s = 1.0f - x; t = x; }
  if (r4) { s = 0.0f; t = x; }
  if (r3) { s = 0.0f; t = 1.0f; }
  if (r2) { s = x; t = 0.0f; }
  if (r1) { s = 1.0f; t = 0.0f; }
  if (r0) { s = 0.0f; t = 0.0f; }
  for (int k = 0; k < 3; k ++) q[k] = v[0][k] + s*ab[k] + t*ac[k];
}

// difference of the closest points of segments p1 + s d1 and p2 + t d2
PG_TF void edge_edge(const float *p1, const float *q1, const float *p2, const float *q2, float *w)
{
  float d1[3], d2[3], r[3];
  for (int k = 0; k < 3; k ++) { d1[k] = q1[k] - p1[k]; d2[k] = q2[k] - p2[k]; r[k] = p1[k] - p2[k]; }
  const float a = dot(d1, d1), e = dot(d2, d2), f = dot(d2, r), c = dot(d1, r), b = dot(d1, d2);
  const float den = a*e - b*b;
  float s = den > 1e-6f*a*e ? clamp01(quot(b*f - c*e, den)) : 0.0f;
  float t = quot(b*s + f, e);
  const bool low = t < 0.0f, high = t > 1.0f;
  if (low || high) s = clamp01(quot(low ? -c : b - c, a));
  t = clamp01(t);
  for (int k = 0; k < 3; k ++) w[k] = (p1[k] + s*d1[k]) - (p2[k] + t*d2[k]);
}

enum { APART = 0, NEAR = 1, FULL = 2 };

// a: triangle A's vertices, b: B's, ea and eb the bounds on their vertices'
// errors (infinite for a degenerate triangle), reach = 2r.  NEAR: the
// distances named by the mask (bits 0-2: A's vertices to B, 3-5: B's to A,
// 6 + 3 i + j: A's edge i to B's edge j) decide, the smallest is at most
// *upper, and the triangles do not intersect; APART: they are farther than
// reach; FULL: the whole narrow phase is needed.
PG_TF int judge(const float a[3][3], const float b[3][3], float ea, float eb, float reach, unsigned *mask, float *upper,
                float *size)
{
  float A[3][3], B[3][3], L = 0.0f, sum = 0.0f;
  for (int v = 0; v < 3; v ++)
    for (int k = 0; k < 3; k ++)
    {
      A[v][k] = a[v][k] - a[0][k];
      B[v][k] = b[v][k] - a[0][k];
      L = mx(L, mx(fabsf(A[v][k]), fabsf(B[v][k])));
      sum += fabsf(A[v][k]) + fabsf(B[v][k]);
    }
  *mask = 0;
  *upper = 0.0f;
  *size = L;
  // (written so that a NaN is not judged)
  if (!(sum < 1e15f) || !(L > 1e-15f) || !(ea < 1e15f) || !(eb < 1e15f)) return FULL;
  const float tol = 1.5f*(ea + eb) + 2e-6f*L;
  float lb[15], best = 3e38f, bw[3] = {0.0f, 0.0f, 0.0f};
#ifdef __CUDA_ARCH__
  #pragma unroll
#endif
  for (int i = 0; i < 15; i ++)
  {
    float w[3], lo;
    if (i < 3)
    {
      float q[3];
      vertex_face(A[i], B, q);
      for (int k = 0; k < 3; k ++) w[k] = A[i][k] - q[k];
      lo = dot(w, A[i]) - mx(mx(dot(w, B[0]), dot(w, B[1])), dot(w, B[2]));
    }
    else if (i < 6)
    {
      float q[3];
      vertex_face(B[i-3], A, q);
      for (int k = 0; k < 3; k ++) w[k] = q[k] - B[i-3][k];
      lo = mn(mn(dot(w, A[0]), dot(w, A[1])), dot(w, A[2])) - dot(w, B[i-3]);
    }
    else
    {
      const int m = (i - 6) / 3, n = (i - 6) % 3, m1 = (m + 1) % 3, n1 = (n + 1) % 3;
      edge_edge(A[m], A[m1], B[n], B[n1], w);
      lo = mn(dot(w, A[m]), dot(w, A[m1])) - mx(dot(w, B[n]), dot(w, B[n1]));
    }
    const float w2 = dot(w, w);
    lb[i] = w2 > 1e-36f ? lo * iroot(w2) : 0.0f;
    if (w2 < best) { best = w2; for (int k = 0; k < 3; k ++) bw[k] = w[k]; }
  }
  if (!(best < 3e38f)) return FULL;
  const float d = best > 1e-36f ? best * iroot(best) : 0.0f;
  const float la = mn(mn(dot(bw, A[0]), dot(bw, A[1])), dot(bw, A[2]));
  const float hb = mx(mx(dot(bw, B[0]), dot(bw, B[1])), dot(bw, B[2]));
  const float gap = best > 1e-36f ? (la - hb) * iroot(best) : 0.0f;
  if (gap - tol > reach * 1.000001f) return APART;
  if (!(gap > tol)) return FULL;
  const float up = d * 1.000001f + tol;
  unsigned m = 0;
#ifdef __CUDA_ARCH__
  #pragma unroll
#endif
  for (int i = 0; i < 15; i ++) if (!(lb[i] - tol > up)) m |= 1u << i;
  *mask = m;
  *upper = up;
  return m ? NEAR : FULL;
}

// grid cell of coordinate x along an axis of `dim` cells; beyond them, the
// nearest.  A NaN (a scene that has blown up) takes cell 0: converted to an
// integer it would name a cell outside of the table.
PG_TF int grid_cell(double x, double org, double h, int dim)
{
  const double q = (x - org) / h;
  return q >= (double)dim ? dim - 1 : q >= 1.0 ? (int)q : 0;
}

// Float copies of a triangle's vertices relative to org, and the bound on
// their error: infinite when the triangle is degenerate (a height below 1e-4
// of its longest edge, tested in FP64) or not finite
PG_TF float float_triangle(const double v[3][3], const double n[3], const double l2[3], const double *org, float f[3][3])
{
  float m = 0.0f, sum = 0.0f;
  for (int a = 0; a < 3; a ++)
    for (int k = 0; k < 3; k ++)
    {
      f[a][k] = (float)(v[a][k] - org[k]);
      m = mx(m, fabsf(f[a][k]));
      sum += fabsf(f[a][k]);
    }
  double l = l2[0] > l2[1] ? l2[0] : l2[1];
  l = l > l2[2] ? l : l2[2];
  const bool good = sum < 1e15f && l > 1e-24 && n[0]*n[0] + n[1]*n[1] + n[2]*n[2] > 1e-8*l*l;
  return good ? 1.2e-7f * m : INFINITY;
}

} // namespace pgtf

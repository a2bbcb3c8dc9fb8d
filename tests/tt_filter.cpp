// The FP32 filter of the mesh contacts (pg_ttfilter.cuh) against the whole
// FP64 narrow phase (pg_tritri.cuh), both as the device compiles them:
// triangles apart must make no contact, pairs settled by a few distances must
// take the same first smallest distance as all fifteen and must not
// intersect, and the plane test must not matter beyond 1e-9 of the size.
// Random triangles: near misses, parallel and shared faces, crossings,
// slivers, a small one against a large one, far from the origin.
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include <random>
#include "../parmec_gb300/csrc/pg_tritri.cuh"
#include "../parmec_gb300/csrc/pg_ttfilter.cuh"

static std::mt19937_64 rng(11);
static double uni() { return (rng() >> 11) * 0x1p-53; }
static double sym() { return 2.0 * uni() - 1.0; }

int main(int argc, char **argv)
{
  const long n = argc > 1 ? atol(argv[1]) : 100000;
  long bad = 0, verdicts[3] = {0, 0, 0}, redone = 0;
  double asked = 0.0;
  for (long it = 0; it < n; it ++)
  {
    const int kind = it % 8;
    const double off = kind == 7 ? 50.0 : (it & 8 ? 1.0 : 0.0), size = pow(10.0, -3.0 + 3.0 * uni());
    double a[3][3], b[3][3];
    for (int v = 0; v < 3; v ++)
      for (int k = 0; k < 3; k ++) { a[v][k] = size * sym(); b[v][k] = size * (kind == 5 ? 40.0 : 1.0) * sym(); }
    const double gap = size * (it % 3 ? 0.2 : 0.2 * (1.0 + 1e-9 * sym()));
    if (kind == 1 || kind == 2)                          // parallel faces of aligned boxes, diagonals either way
    {
      const double s = size, c[4][2] = {{0, 0}, {s, 0}, {s, s}, {0, s}};
      const int p[4][3] = {{0, 1, 2}, {0, 2, 3}, {1, 2, 3}, {0, 1, 3}};
      const int x = (int)(rng() % 4), y = (int)(rng() % 4);
      const double tilt = it & 16 ? 1e-8 : 0.0;
      for (int v = 0; v < 3; v ++)
      {
        a[v][0] = c[p[x][v]][0]; a[v][1] = c[p[x][v]][1]; a[v][2] = s * tilt * sym();
        b[v][0] = c[p[y][v]][0] + (kind == 2 ? s * (double)(rng() % 2) : 0.0); b[v][1] = c[p[y][v]][1];
        b[v][2] = gap + s * tilt * sym();
      }
    }
    if (kind == 3)                                       // a face beside the edge of a perpendicular one
      for (int v = 0; v < 3; v ++) { a[v][2] = 0.0; b[v][0] = a[v][1] + 1e-12 * sym(); b[v][1] = a[v][2]; b[v][2] += gap; }
    if (kind == 4 && it % 16 == 4)                       // slivers and points
      for (int k = 0; k < 3; k ++) b[2][k] = b[0][k] + (b[1][k] - b[0][k]) * (it % 32 == 4 ? 0.3 : 0.0) + 1e-9 * size * sym() * (it % 64 / 32);
    if (kind == 6)                                       // a shared vertex or edge, nearly
      for (int v = 0; v < 1 + (int)(it % 16 / 8); v ++)
        for (int k = 0; k < 3; k ++) b[v][k] = a[v][k] + gap * (k == 2);
    for (int v = 0; v < 3; v ++) for (int k = 0; k < 3; k ++) { a[v][k] += off; b[v][k] += off; }
    if (it % 1000 == 999) b[1][1] = it % 2000 == 999 ? NAN : INFINITY;
    const double r = size * (it % 5 ? 0.1 : 0.5 * uni());
    const double *A[3] = {a[0], a[1], a[2]}, *B[3] = {b[0], b[1], b[2]}, org[3] = {0.0, 0.0, 0.0};
    pgtt::Tri TA, TB;
    pgtt::tri_prep(A, TA);
    pgtt::tri_prep(B, TB);
    float fa[3][3], fb[3][3];
    const float ea = pgtf::float_triangle(a, TA.n, TA.l2, org, fa), eb = pgtf::float_triangle(b, TB.n, TB.l2, org, fb);
    unsigned mask;
    float upper, extent;
    const int v = pgtf::judge(fa, fb, ea, eb, (float)(r + r), &mask, &upper, &extent);
    verdicts[v] ++;
    if (v == pgtf::FULL) continue;
    double point[3], normal[3], pa[3], pb[3];
    const double depth = pgtt::contact(A, B, r, r, point, normal);
    if (v == pgtf::APART) { bad += depth > 0.0; continue; }
    double d2[15], best = 1.7976931348623157e308, few = best;
    int at = -1, few_at = -1;
    for (int i = 0; i < 15; i ++)
    {
      double q[3], c1[3], c2[3], w[3];
      if (i < 3) { pgtt::point_triangle(A[i], B[0], B[1], B[2], TB.e[0], TB.ac, q); pgtt::sub(A[i], q, w); d2[i] = pgtt::dot(w, w); }
      else if (i < 6) { pgtt::point_triangle(B[i-3], A[0], A[1], A[2], TA.e[0], TA.ac, q); pgtt::sub(q, B[i-3], w); d2[i] = pgtt::dot(w, w); }
      else { const int m = (i-6)/3, k = (i-6)%3; d2[i] = pgtt::segment_segment(A[m], TA.e[m], TA.l2[m], B[k], TB.e[k], TB.l2[k], c1, c2); }
      if (d2[i] < best) { best = d2[i]; at = i; }
      if ((mask >> i & 1) && d2[i] < few) { few = d2[i]; few_at = i; }
      asked += mask >> i & 1;
    }
    if (few_at < 0 || !(few <= (double)upper * (double)upper)) { redone ++; continue; }
    bad += at != few_at || pgtt::triangle_triangle(A, B, pa, pb) != best;
    bad += pgtt::apart(A, B, r, r) && (r + r) - sqrt(best) > 1e-9 * (double)extent;
  }
  printf("%ld %ld %ld %ld %ld %.2f\n", bad, verdicts[0], verdicts[1], verdicts[2], redone, asked / verdicts[1]);
  return 0;
}

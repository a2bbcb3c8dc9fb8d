// pg_meshcontact.cu -- mesh-mesh contact between triangles of different
// particles (an extension; off unless pg_session_mesh_contact turns it on).
//
// Every step, before the force sums, box and difference arrays of each mesh
// triangle (1); when a vertex has moved by half the skin since the last
// search, the pair list anew (2-4); then the narrow phase of the list (5) and
// the sums (6):
//   1. each triangle's edges, squared edge lengths and plane normal, a float
//      copy of its vertices for the filter, and whether a vertex moved by half
//      the skin;
//   2. each triangle's box (its vertices' bounds widened by the swept radius r
//      and the skin) and its grid cell, or the "big" range for triangles
//      larger than a cell; a stable radix sort of the triangles by cell, and
//      the cell ranges;
//   3. each triangle finds its partners among the triangles of the 27 cells
//      around its own (and among the big ones), keeps those whose boxes
//      overlap, and sorts them by index.  A pair is found by one triangle
//      only: between two small triangles (or two big ones) by the lower
//      index, between a small and a big one by the small one;
//   4. the pairs, in the order of the finding triangles and their sorted
//      partners (an exclusive scan of the counts gives each triangle's
//      offset), with the tangential state of the pairs of the last list, by
//      (finder, partner); two entries a pair, sorted by particle;
//   5. whether a pair's boxes without the skin overlap with positive measure
//      (triangles closer than 2r have such boxes), and which of its fifteen
//      feature distances can decide its contact, in FP32 with certain bounds
//      (pg_ttfilter.cuh): most pairs are apart, the others ask for 7 distances
//      on average (parallel faces tie).  Those are taken in FP64 by one thread
//      each, every warp one kind on all its lanes; then one thread per near
//      pair takes the first of the smallest, the contact it gives
//      (pg_tritri.cuh) and the granular law.  Pairs that may intersect and
//      degenerate triangles take the whole narrow phase.  Bound by the FP64
//      pipe; evaluating all fifteen distances and six crossing tests of
//      every pair that a plane test left took 3.2 ms a step on the 64x64
//      lattice (658,000 pairs), the whole stage now takes 0.8 ms;
//   6. the force of each active pair goes to its two particles (+f to the
//      finder's, -f to the partner's): the entries of active pairs, selected
//      in the list's order, are summed per particle in chunks of PG_TT_CHUNK:
//      lane L of 32 takes entries L, L+32, ... of the chunk from zero and the
//      32 lane sums are added in lane order; then the chunk sums in chunk
//      order from zero, one thread per particle and component.  A particle
//      with many contacts (a base plate under a whole lattice) spreads over
//      many blocks.  k_integrate adds these sums after gravity.
// The CPU oracle restates the same definitions with a brute-force search.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdio>
#include "pg_items.cuh"
#include "pg_launch.h"
#include "pg_meshcontact.h"
#include "pg_tritri.cuh"
#include "pg_ttfilter.cuh"

namespace {

constexpr int TPB = 128;
inline int nblk(long long n) { return (int)((n + TPB - 1) / TPB); }

__device__ __forceinline__ bool mesh_tri(const PgDev &d, int t) { return d.triobs[t] >= 0; }

__device__ __forceinline__ void tri_vertices(const PgDev &d, int t, double v[3][3])
{
  for (int a = 0; a < 3; a ++)
    for (int c = 0; c < 3; c ++) v[a][c] = d.tri[3*a + c][t];
}

// box keys: lo < hi on the keys is the FP64 comparison lo < hi
__device__ __forceinline__ unsigned long long lo_key(double x)
{
  const unsigned long long b = pgtt::bits(x);
  return pgtt::nan_b(b) ? ~0ULL : pgtt::okey(b);
}
__device__ __forceinline__ unsigned long long hi_key(double x)
{
  const unsigned long long b = pgtt::bits(x);
  return pgtt::nan_b(b) ? 0ULL : pgtt::okey(b);
}

// 1. every step: boxes, FP64 differences, float copies, and whether a vertex
// coordinate moved by half the skin since the last search (a NaN did)
__global__ void __launch_bounds__(TPB) k_tt_boxes(PgDev d, PgTT g)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  bool moved = false;
  if (t < d.trinum && mesh_tri(d, t))
  {
    double v[3][3];
    tri_vertices(d, t, v);
    const double *vp[3] = {v[0], v[1], v[2]};
    pgtt::Tri T;
    pgtt::tri_prep(vp, T);
    double *o = g.geo + (size_t)PG_TT_GEO * t;
    for (int a = 0; a < 3; a ++)
      for (int c = 0; c < 3; c ++) { o[3*a + c] = v[a][c]; o[9 + 3*a + c] = T.e[a][c]; }
    for (int a = 0; a < 3; a ++) { o[18 + a] = T.l2[a]; o[21 + a] = T.ac[a]; o[24 + a] = T.n[a]; }
    o[27] = (g.r + g.r) * sqrt(pgtt::dot(T.n, T.n));
    float f[3][3];
    const float err = pgtf::float_triangle(v, T.n, T.l2, g.org, f);
    for (int a = 0; a < 3; a ++)
      g.fv[(size_t)a * d.trinum + t] = make_float4(f[a][0], f[a][1], f[a][2], a == 0 ? err : 0.0f);
    for (int c = 0; c < 3; c ++)
    {
      const double a = v[0][c], b = v[1][c], e = v[2][c];
      double l = a < b ? a : b, h = a > b ? a : b;
      l = l < e ? l : e;
      h = h > e ? h : e;
      g.box[c][t] = lo_key(l - g.r);
      g.box[3+c][t] = hi_key(h + g.r);
    }
    const double lim = 0.4999 * g.skin;
    for (int a = 0; a < 3; a ++)
      for (int c = 0; c < 3; c ++) moved |= !(fabs(v[a][c] - g.ref[3*a + c][t]) <= lim);
  }
  if (__syncthreads_or(moved) && threadIdx.x == 0) g.moved[0] = 1;
}

// 2. a search: reference vertices, search boxes and cell keys.  The boxes are
// FP64, as the ones they stand for: single precision would widen them by the
// distance from the origin (10 mm cubes 1 mm apart had no pair near it, 8,124
// at 10 km, and too many for a triangle's list at 300 km).
__global__ void __launch_bounds__(TPB) k_tt_keys(PgDev d, PgTT g)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.trinum) return;
  unsigned key = g.none;
  PgTTBox bx;
  bx.owner = -1;
  bx.big = 0;
  for (int c = 0; c < 3; c ++) bx.lo[c] = bx.hi[c] = 0;
  if (mesh_tri(d, t))
  {
    double v[3][3], mid[3];
    tri_vertices(d, t, v);
    const double w = g.r + 0.5 * g.skin;
    for (int c = 0; c < 3; c ++)
    {
      const double a = v[0][c], b = v[1][c], e = v[2][c];
      for (int k = 0; k < 3; k ++) g.ref[3*k + c][t] = v[k][c];
      double l = a < b ? a : b, h = a > b ? a : b;
      l = l < e ? l : e;
      h = h > e ? h : e;
      mid[c] = 0.5*((l - g.r) + (h + g.r));
      bx.lo[c] = lo_key(l - w);
      bx.hi[c] = hi_key(h + w);
    }
    bx.owner = d.triobs[t];
    bx.big = g.big[t];
    if (bx.big) key = (unsigned)g.ncells;
    else
    {
      int ix[3];
      for (int c = 0; c < 3; c ++) ix[c] = pgtf::grid_cell(mid[c], g.org[c], g.h, g.dim[c]);
      key = (unsigned)((ix[2]*g.dim[1] + ix[1])*g.dim[0] + ix[0]);
    }
    g.cell[t] = (int)key;
  }
  g.sbox[t] = bx;
  g.keys[0][t] = key;
  g.vals[0][t] = t;
}

// cell ranges over the sorted keys
__global__ void __launch_bounds__(TPB) k_tt_ranges(PgTT g, int n)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const unsigned key = g.keys[0][k];
  if (key == g.none) return;
  if (k == 0 || g.keys[0][k-1] != key) g.cstart[key] = k;
  if (k == n-1 || g.keys[0][k+1] != key) g.cend[key] = k + 1;
}

// 3. partners found by triangle t, sorted by index: counted (FILL false), or
// written to the pair list with the state carried from the previous one.
// One warp per triangle: the lanes take the ranges of the 27 cells around
// its own and the big range, then test 32 candidates at a time, so that 32
// loads are in flight where one thread a triangle followed one chain of them
// (231 us a search on 3,000 triangles, all of it latency).
template <bool FILL>
__global__ void __launch_bounds__(TPB) k_tt_find(PgDev d, PgTT g)
{
  constexpr unsigned all = 0xffffffffu;
  __shared__ int lists[TPB / 32][PG_TT_KMAX];
  const int lane = threadIdx.x & 31;
  int *list = lists[threadIdx.x >> 5];
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (t >= d.trinum) return;
  const PgTTBox me = g.sbox[t];
  int cnt = 0;
  if (me.owner >= 0)
  {
    // this lane's range of sorted triangles
    int b = 0, n = 0;
    if (lane < 27 && !me.big)
    {
      const int cell = g.cell[t];
      const int x = cell % g.dim[0] + lane % 3 - 1, y = (cell / g.dim[0]) % g.dim[1] + lane / 3 % 3 - 1;
      const int z = cell / (g.dim[0] * g.dim[1]) + lane / 9 - 1;
      if (x >= 0 && y >= 0 && z >= 0 && x < g.dim[0] && y < g.dim[1] && z < g.dim[2])
      {
        const int c = (z*g.dim[1] + y)*g.dim[0] + x;
        b = g.cstart[c];
        n = g.cend[c] - b;
      }
    }
    if (lane == 27) { b = g.cstart[g.ncells]; n = g.cend[g.ncells] - b; }
    int upto = n;                                        // inclusive sums of the ranges' lengths
    for (int o = 1; o < 32; o <<= 1)
    {
      const int v = __shfl_up_sync(all, upto, o);
      if (lane >= o) upto += v;
    }
    const int total = __shfl_sync(all, upto, 31);
    for (int q0 = 0; q0 < total; q0 += 32)
    {
      const int q = q0 + lane;
      int lo = 0;                                        // the first range that ends beyond q
      for (int o = 16; o > 0; o >>= 1) if (__shfl_sync(all, upto, lo + o - 1) <= q) lo += o;
      lo = lo < 31 ? lo : 31;
      const int k = __shfl_sync(all, b, lo) + q - (__shfl_sync(all, upto, lo) - __shfl_sync(all, n, lo));
      bool hit = false;
      int u = 0;
      if (q < total)
      {
        u = g.vals[0][k];
        const PgTTBox o = g.sbox[u];
        hit = u != t && o.owner != me.owner && (me.big == o.big ? u > t : !me.big);
        for (int c = 0; c < 3; c ++) hit = hit && me.lo[c] < o.hi[c] && o.lo[c] < me.hi[c];
      }
      const unsigned m = __ballot_sync(all, hit);
      const int at = cnt + __popc(m & ((1u << lane) - 1u));
      if (hit && at < PG_TT_KMAX) list[at] = u;
      cnt += __popc(m);
    }
    if (cnt > PG_TT_KMAX)
    {
      // partners in the skin alone never end a run: the host searches without
      if (lane == 0 && g.skin > 0.0) g.moved[0] = 2;
      else if (lane == 0) pgk::set_err(d, PG_ERR_CAPACITY, 40, t, cnt);
      cnt = PG_TT_KMAX;
    }
  }
  if (!FILL)
  {
    if (lane == 0) g.cnt[t] = cnt;
    return;
  }
  __syncwarp();
  const int o = g.off[t], pb = g.poff[t], pe = g.poff[t+1];
  for (int a = lane; a < cnt; a += 32)
  {
    const int u = list[a];
    int rank = 0;
    for (int c = 0; c < cnt; c ++) rank += list[c] < u;
    const int k = o + rank;
    g.pf[k] = t;
    g.pu[k] = u;
    int lo = pb, hi = pe;
    while (lo < hi)
    {
      const int mid = (lo + hi) >> 1;
      if (g.ppu[mid] < u) lo = mid + 1;
      else hi = mid;
    }
    const bool kept = lo < pe && g.ppu[lo] == u && g.pact[lo];
    g.act[k] = kept;
    for (int c = 0; c < 3; c ++) g.st[c][k] = kept ? g.pst[c][lo] : 0.0;
  }
}

// 4. exclusive scan of the counts in one block (off[n] = total); a total
// beyond 31 bits is given as the largest int, which no list may hold
__global__ void __launch_bounds__(1024) k_tt_scan(const int *in, int *out, int n, int *total)
{
  __shared__ long long part[1024];
  const int tid = threadIdx.x;
  const int per = (n + 1023) / 1024;
  const int b = tid * per, e = b + per < n ? b + per : n;
  long long s = 0;
  for (int i = b; i < e; i ++) s += in[i];
  part[tid] = s;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1)
  {
    const long long v = tid >= o ? part[tid - o] : 0;
    __syncthreads();
    part[tid] += v;
    __syncthreads();
  }
  long long acc = tid ? part[tid - 1] : 0;
  for (int i = b; i < e; i ++) { const int v = in[i]; out[i] = (int)acc; acc += v; }
  if (tid == 1023) out[n] = *total = (int)min(part[1023], 0x7fffffffLL);
}

// the boxes of pair k overlap with positive measure this step
__device__ __forceinline__ bool boxes_overlap(const PgTT &g, int f, int u)
{
  bool in = true;
  for (int c = 0; c < 3; c ++) in = in && g.box[c][f] < g.box[3+c][u] && g.box[c][u] < g.box[3+c][f];
  return in;
}

// overlapping and active pairs of the last step
__global__ void __launch_bounds__(TPB) k_tt_counts(PgTT g, int *out2)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int a = __syncthreads_count(k < g.np && boxes_overlap(g, g.pf[k], g.pu[k]));
  const int b = __syncthreads_count(k < g.np && g.act[k]);
  if (threadIdx.x == 0) { atomicAdd(out2, a); atomicAdd(out2 + 1, b); }
}

// 5a. what each pair needs, in FP32 (pg_ttfilter.cuh): the pairs farther
// than 2r get their result (inactive), the others a place in the list of
// near pairs with the distances that can decide them, or in the list of
// pairs that need every test.  One thread per pair; list places and item
// ranges by one atomic per list and warp, counted in 64 bits: a pair asks for
// up to nine distances of a kind.
__device__ __forceinline__ long long warp_take(unsigned long long *count, int n)
{
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int s = n;
  for (int o = 1; o < 32; o <<= 1)
  {
    const int v = __shfl_up_sync(all, s, o);
    if (lane >= o) s += v;
  }
  long long base = 0;
  if (lane == 31 && s) base = (long long)atomicAdd(count, (unsigned long long)s);
  base = __shfl_sync(all, base, 31);
  return base + s - n;
}

__global__ void __launch_bounds__(TPB) k_tt_judge(PgDev d, PgTT g)
{
  // the block's pairs whose boxes overlap, on its first threads
  __shared__ int some[TPB], warps[TPB / 32];
  const int q = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  bool in = false;
  if (q < g.np)
  {
    in = boxes_overlap(g, g.pf[q], g.pu[q]);
    if (!in) g.act[q] = 0;
  }
  const unsigned m0 = __ballot_sync(0xffffffffu, in);
  if (lane == 0) warps[warp] = __popc(m0);
  __syncthreads();
  int at = __popc(m0 & ((1u << lane) - 1u)), count = 0;
  for (int w = 0; w < TPB / 32; w ++)
  {
    if (w < warp) at += warps[w];
    count += warps[w];
  }
  if (in) some[at] = q;
  __syncthreads();
  if (warp * 32 >= count) return;
  const int k = threadIdx.x < count ? some[threadIdx.x] : -1;
  int verdict = pgtf::APART;
  unsigned mask = 0;
  float upper = 0.0f, size = 0.0f;
  if (k >= 0)
  {
    const int f = g.pf[k], u = g.pu[k];
    const size_t T = d.trinum;
    float a[3][3], b[3][3], ea = 0.0f, eb = 0.0f;
    for (int v = 0; v < 3; v ++)
    {
      const float4 x = g.fv[v*T + f], y = g.fv[v*T + u];
      a[v][0] = x.x; a[v][1] = x.y; a[v][2] = x.z;
      b[v][0] = y.x; b[v][1] = y.y; b[v][2] = y.z;
      if (v == 0) { ea = x.w; eb = y.w; }
    }
    verdict = pgtf::judge(a, b, ea, eb, (float)(g.r + g.r), &mask, &upper, &size);
    if (verdict == pgtf::APART) g.act[k] = 0;
  }
  int nv = verdict == pgtf::NEAR ? __popc(mask & 63u) : 0, ne = verdict == pgtf::NEAR ? __popc(mask >> 6) : 0;
  const long long vb = warp_take(g.qn + 2, nv), eb = warp_take(g.qn + 3, ne);
  if (verdict == pgtf::NEAR && (vb + nv > g.vcap || eb + ne > g.ecap)) verdict = pgtf::FULL;   // no room for its items
  const long long np = warp_take(g.qn, verdict == pgtf::NEAR);
  if (verdict == pgtf::NEAR && np >= PG_TT_NEAR) verdict = pgtf::FULL;                         // nor for their number
  const long long z = warp_take(g.qn + 1, verdict == pgtf::FULL);
  // (items of a pair that found no room in the other list name no pair)
  if (nv + ne && verdict == pgtf::FULL)
  {
    for (long long j = vb; j < vb + nv && j < g.vcap; j ++) g.vit[j] = ~0u;
    for (long long j = eb; j < eb + ne && j < g.ecap; j ++) g.eit[j] = ~0u;
  }
  if (verdict == pgtf::FULL) g.full[z] = k;
  if (verdict != pgtf::NEAR) return;
  g.near[np] = {k, mask, (int)vb, (int)eb, upper, size};
  int j = (int)vb;
  for (unsigned m = mask & 63u; m; m &= m - 1) g.vit[j ++] = (unsigned)np << 4 | (unsigned)(__ffs(m) - 1);
  j = (int)eb;
  for (unsigned m = mask >> 6; m; m &= m - 1) g.eit[j ++] = (unsigned)np << 4 | (unsigned)(__ffs(m) - 1);
}

// 5b. the vertex-triangle and the edge-edge distances asked for, one thread
// each, so that a warp runs one kind on all its lanes: the first vb blocks
// take the one kind, the others the other
__device__ __forceinline__ void tt_vertex_face(const PgTT &g, const pg::Num<pg::f64> &N, int first, int by)
{
  const int n = (int)min(g.qn[2], (unsigned long long)g.vcap);
  for (int w = first; w < n; w += by)
  {
    const unsigned it = g.vit[w];
    if (it == ~0u) continue;
    const int k = g.near[it >> 4].pair, i = it & 15u;
    const int tp = i < 3 ? g.pf[k] : g.pu[k], tt = i < 3 ? g.pu[k] : g.pf[k], vi = i < 3 ? i : i - 3;
    const double *P = g.geo + (size_t)PG_TT_GEO * tp + 3*vi, *T = g.geo + (size_t)PG_TT_GEO * tt;
    const pg::f64 p[3] = {N(P[0]), N(P[1]), N(P[2])};
    pg::f64 v[9], ab[3], ac[3], q[3], h[3], x0, x1;
    for (int c = 0; c < 9; c ++) v[c] = N(T[c]);
    for (int c = 0; c < 3; c ++) { ab[c] = N(T[9 + c]); ac[c] = N(T[21 + c]); }
    const int region = pgtt::point_triangle_region(p, v, v + 3, v + 6, ab, ac, &x0, &x1);
    pgtt::point_triangle_at(region, x0, x1, v, v + 3, v + 6, ab, ac, q);
    if (i < 3) pgtt::sub(p, q, h);
    else pgtt::sub(q, p, h);
    double *o = g.vres + 3 * (size_t)w;
    o[0] = pgtt::dot(h, h);
    o[1] = x0;
    o[2] = x1;
    g.vit[w] = (unsigned)region;
  }
}

__device__ __forceinline__ void tt_edge_edge(const PgTT &g, const pg::Num<pg::f64> &N, int first, int by)
{
  const int n = (int)min(g.qn[3], (unsigned long long)g.ecap);
  for (int w = first; w < n; w += by)
  {
    const unsigned it = g.eit[w];
    if (it == ~0u) continue;
    const int k = g.near[it >> 4].pair, i = (it & 15u) / 3u, j = (it & 15u) % 3u;
    const double *A = g.geo + (size_t)PG_TT_GEO * g.pf[k], *B = g.geo + (size_t)PG_TT_GEO * g.pu[k];
    pg::f64 p1[3], d1[3], p2[3], d2[3], s, t, c1[3], c2[3], h[3];
    for (int c = 0; c < 3; c ++)
    {
      p1[c] = N(A[3*i + c]); d1[c] = N(A[9 + 3*i + c]);
      p2[c] = N(B[3*j + c]); d2[c] = N(B[9 + 3*j + c]);
    }
    pgtt::segment_params(p1, d1, N(A[18+i]), p2, d2, N(B[18+j]), &s, &t);
    pgtt::segment_at(p1, d1, s, c1);
    pgtt::segment_at(p2, d2, t, c2);
    pgtt::sub(c1, c2, h);
    double *o = g.eres + 3 * (size_t)w;
    o[0] = pgtt::dot(h, h);
    o[1] = s;
    o[2] = t;
  }
}

// One launch: the second kind fills the SMs as the first runs out (16x16
// lattice: 23 + 21 us in two launches, 33 in one).
__global__ void __launch_bounds__(TPB) k_tt_distances(PgTT g, int vb)
{
  const pg::Num<pg::f64> N;
  const int b = blockIdx.x;
  if (b < vb) tt_vertex_face(g, N, b * TPB + threadIdx.x, vb * TPB);
  else tt_edge_edge(g, N, (b - vb) * TPB + threadIdx.x, (gridDim.x - vb) * TPB);
}

// granular force of pair k with the contact found (depth > 0: active)
template <class R>
__device__ __forceinline__ void tt_force(const PgDev &d, const PgTT &g, const pg::Num<R> &N, int k, int f, int u,
                                         R depth, const R *point, const R *normal, double step)
{
  const bool active = depth > 0.0, was = g.act[k] != 0;
  g.act[k] = active ? 1 : 0;
  if (!active) return;
  R st[3], fr[3];
  for (int c = 0; c < 3; c ++) st[c] = N(was ? g.st[c][k] : 0.0);
  const int pa = d.triobs[f], pb = d.triobs[u];
  // contact point velocities (forces.ispc:226-246) and their difference
  R vij[3];
  const R za[3] = {point[0]-d.position[0][pa], point[1]-d.position[1][pa], point[2]-d.position[2][pa]};
  const R zb[3] = {point[0]-d.position[0][pb], point[1]-d.position[1][pb], point[2]-d.position[2][pb]};
  for (int c = 0; c < 3; c ++)
  {
    const int c1 = (c+1)%3, c2 = (c+2)%3;
    const R vi = d.angular[3+c1][pa]*za[c2] - d.angular[3+c2][pa]*za[c1] + d.linear[c][pa];
    const R vj = d.angular[3+c1][pb]*zb[c2] - d.angular[3+c2][pb]*zb[c1] + d.linear[c][pb];
    vij[c] = vj - vi;
  }
  const int ij = pgk::pairing(d, d.tricol[f], d.tricol[u]);
  if (d.ikind[ij] != 0) pgk::set_err(d, PG_ERR_UNSUPPORTED, 41, k, ij);
  const R ma = 1.0 / (N(d.invm[pa]) + d.invm[pb]);
  pgtt::granular(d.iparam[0][ij], d.iparam[1][ij], d.iparam[6][ij], d.iparam[2][ij], d.iparam[3][ij], ma,
                 normal, vij, depth, step, st, fr);
  for (int c = 0; c < 3; c ++)
  {
    g.st[c][k] = st[c];
    g.f[c][k] = fr[c];
    g.p[c][k] = point[c];
  }
}

// the whole narrow phase of a pair
__device__ __noinline__ double tt_contact(const PgDev &d, const PgTT &g, int f, int u, double *point, double *normal)
{
  double va[3][3], vb[3][3];
  tri_vertices(d, f, va);
  tri_vertices(d, u, vb);
  const double *A[3] = {va[0], va[1], va[2]}, *B[3] = {vb[0], vb[1], vb[2]};
  return pgtt::contact(A, B, g.r, g.r, point, normal);
}

// 5c. each near pair's contact from its distances: the first of the smallest,
// as the full search keeps it; then the granular force.  The plane test,
// which calls a pair apart that the distances would call touching only
// within its rounding, is taken for depths below 1e-9 of the pair's size.
// Bound by FP64 issue and by the gathers before it: 16 warps an SM hide more of
// them than 12 or 20 (a step of the 64x64 lattice 898 us against 910 and 904;
// 926 with constants as operands and 12).  In blocks of one warp the last wave
// of a small scene is spread over more SMs (a step of the 16x16 lattice 176 ->
// 173 us).
__global__ void __launch_bounds__(32, 16) k_tt_near(PgDev d, PgTT g, double step)
{
  const pg::Num<pg::f64> N;
  const int n = (int)min(g.qn[0], (unsigned long long)PG_TT_NEAR);
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < n; w += gridDim.x * blockDim.x)
  {
    const PgTTNear e = g.near[w];
    const int k = e.pair, f = g.pf[k], u = g.pu[k];
    double best = 1.7976931348623157e308;
    int at = -1, cand = 0, jv = e.vbase, je = e.ebase;
    for (unsigned m = e.mask; m; m &= m - 1)
    {
      const int i = __ffs(m) - 1;
      const int slot = i < 6 ? jv ++ : je ++;
      const double d2 = i < 6 ? g.vres[3*(size_t)slot] : g.eres[3*(size_t)slot];
      if (d2 < best) { best = d2; at = slot; cand = i; }
    }
    pg::f64 point[3], normal[3], depth;
    if (at < 0 || !(best > 0.0) || !(best <= (double)e.upper * (double)e.upper))
    {
      double po[3], no[3];
      depth = N(tt_contact(d, g, f, u, po, no));
      for (int c = 0; c < 3; c ++) { point[c] = N(po[c]); normal[c] = N(no[c]); }
    }
    else
    {
      const double *A = g.geo + (size_t)PG_TT_GEO * f, *B = g.geo + (size_t)PG_TT_GEO * u;
      pg::f64 pa[3], pb[3], v[9], x[3], y[3];
      if (cand < 6)
      {
        const double *P = (cand < 3 ? A : B) + 3 * (cand < 3 ? cand : cand - 3), *T = cand < 3 ? B : A;
        pg::f64 q[3];
        for (int c = 0; c < 9; c ++) v[c] = N(T[c]);
        for (int c = 0; c < 3; c ++) { x[c] = N(T[9 + c]); y[c] = N(T[21 + c]); }
        pgtt::point_triangle_at((int)g.vit[at], N(g.vres[3*(size_t)at+1]), N(g.vres[3*(size_t)at+2]), v, v + 3, v + 6,
                                x, y, q);
        for (int c = 0; c < 3; c ++) { pa[c] = cand < 3 ? N(P[c]) : q[c]; pb[c] = cand < 3 ? q[c] : N(P[c]); }
      }
      else
      {
        const int i = (cand - 6) / 3, j = (cand - 6) % 3;
        for (int c = 0; c < 3; c ++) { x[c] = N(A[3*i + c]); y[c] = N(A[9 + 3*i + c]); }
        pgtt::segment_at(x, y, N(g.eres[3*(size_t)at+1]), pa);
        for (int c = 0; c < 3; c ++) { x[c] = N(B[3*j + c]); y[c] = N(B[9 + 3*j + c]); }
        pgtt::segment_at(x, y, N(g.eres[3*(size_t)at+2]), pb);
      }
      depth = pgtt::contact_at(pa, pb, N(best), g.r, g.r, point, normal);
      if (depth > 0.0 && !(depth > 1e-9 * (double)e.size))
      {
        const double *Av[3] = {A, A + 3, A + 6}, *Bv[3] = {B, B + 3, B + 6};
        if (pgtt::beyond_plane_of(A, A + 24, A[27], Bv) || pgtt::beyond_plane_of(B, B + 24, B[27], Av)) depth = N(-1.0);
      }
    }
    tt_force(d, g, N, k, f, u, depth, point, normal, step);
  }
  // 5d. the pairs that need every test: triangles that may intersect,
  // degenerate ones, and those whose distances found no room
  const int nf = (int)g.qn[1];
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < nf; w += gridDim.x * blockDim.x)
  {
    const int k = g.full[w], f = g.pf[k], u = g.pu[k];
    double po[3], no[3];
    const pg::f64 depth = N(tt_contact(d, g, f, u, po, no));
    const pg::f64 point[3] = {N(po[0]), N(po[1]), N(po[2])}, normal[3] = {N(no[0]), N(no[1]), N(no[2])};
    tt_force(d, g, N, k, f, u, depth, point, normal, step);
  }
}

// resident blocks over every SM, for the loops over device-side counts
template <class K>
int resident_blocks(K k, int tpb = TPB)
{
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, tpb, 0);
  return (sms > 0 ? sms : 152) * (per > 0 ? per : 4);
}

// 6a. with the list: two entries per pair, keyed by particle
__global__ void __launch_bounds__(TPB) k_tt_entries(PgDev d, PgTT g)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= g.np) return;
  g.ekeys[0][2*k] = (unsigned)d.triobs[g.pf[k]];
  g.ekeys[0][2*k+1] = (unsigned)d.triobs[g.pu[k]];
  g.evals[0][2*k] = 2*k;
  g.evals[0][2*k+1] = 2*k + 1;
}

// particles with more than PG_TT_CHUNK entries, from their ranges of the
// sorted entries (pfirst and plast, for now)
__global__ void __launch_bounds__(TPB) k_tt_segments(PgTT g, int n)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const unsigned key = g.ekeys[0][k];
  if (k == 0 || g.ekeys[0][k-1] != key) g.pfirst[key] = k;
  if (k == n-1 || g.ekeys[0][k+1] != key) g.plast[key] = k + 1;
}

__global__ void __launch_bounds__(TPB) k_tt_big(PgDev d, PgTT g)
{
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= d.parnum) return;
  const int n = g.plast[w] - g.pfirst[w];
  if (n <= PG_TT_CHUNK) return;
  const int b = atomicAdd(g.moved + 2, 1);
  g.bigp[b] = w;
  g.bigoff[b] = atomicAdd(g.moved + 3, (n + PG_TT_CHUNK - 1) / PG_TT_CHUNK);
}

// which big particle a chunk belongs to (one block per big particle)
__global__ void __launch_bounds__(TPB) k_tt_chmap(PgTT g)
{
  const int b = blockIdx.x, w = g.bigp[b];
  const int nc = (g.plast[w] - g.pfirst[w] + PG_TT_CHUNK - 1) / PG_TT_CHUNK;
  for (int c = threadIdx.x; c < nc; c += blockDim.x) g.chmap[g.bigoff[b] + c] = b;
}

// 6b. every step: the active entries in their order: one bit per entry and
// their number per tile, the scan of the tiles, the selection
constexpr int TILE_THREADS = 256;

__global__ void __launch_bounds__(TILE_THREADS) k_tt_active(PgTT g)
{
  __shared__ int sum;
  if (threadIdx.x == 0) sum = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, n = 2 * g.np;
  for (int it = 0; it < PG_TT_TILE / TILE_THREADS; it ++)
  {
    const int e = blockIdx.x * PG_TT_TILE + it * TILE_THREADS + threadIdx.x;
    const unsigned m = __ballot_sync(0xffffffffu, e < n && g.act[g.evals[0][e] >> 1] != 0);
    if (lane == 0)
    {
      g.ebits[e >> 5] = m;
      atomicAdd(&sum, __popc(m));
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) g.etile[blockIdx.x] = sum;
}

// Each block counts the tiles before its own again instead of waiting for a
// scan in a launch of its own (tiles of 4 bytes, in L2).
__global__ void __launch_bounds__(TILE_THREADS) k_tt_select(PgTT g)
{
  __shared__ int tiles[TILE_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = 2 * g.np;
  int tile = 0;
  for (int t = threadIdx.x; t < (int)blockIdx.x; t += TILE_THREADS) tile += g.etile[t];
  tile = __reduce_add_sync(0xffffffffu, tile);
  if (lane == 0) tiles[warp] = tile;
  __syncthreads();
  tile = 0;
  for (int t = 0; t < TILE_THREADS / 32; t ++) tile += tiles[t];
  // the tile's 32 words, one a lane: active entries before each
  const unsigned word = g.ebits[blockIdx.x * (PG_TT_TILE / 32) + lane];
  int before = __popc(word);
  for (int o = 1; o < 32; o <<= 1)
  {
    const int v = __shfl_up_sync(0xffffffffu, before, o);
    if (lane >= o) before += v;
  }
  before += tile - __popc(word);
  for (int it = 0; it < PG_TT_TILE / TILE_THREADS; it ++)
  {
    const int wd = it * (TILE_THREADS / 32) + warp;
    const int e = blockIdx.x * PG_TT_TILE + wd * 32 + lane;
    const unsigned m = __shfl_sync(0xffffffffu, word, wd);
    const int rank = __shfl_sync(0xffffffffu, before, wd) + __popc(m & ((1u << lane) - 1u));
    if (e >= n) continue;
    const int on = m >> lane & 1u;
    const unsigned p = g.ekeys[0][e];
    if (on) g.elist[rank] = g.evals[0][e];
    if (e == 0 || g.ekeys[0][e-1] != p) g.pfirst[p] = rank;
    if (e == n-1 || g.ekeys[0][e+1] != p) g.plast[p] = rank + on;
  }
}

// 6c. sums of entries [b, e) of elist, e - b <= PG_TT_CHUNK: lane sums over
// entries lane, lane+32, ..., then the lane sums in lane order, one lane per
// component.  Four entries' loads are issued before the first is added.
// Returns component `lane`, force then torque.
__device__ __forceinline__ double chunk_sum(const PgTT &g, const double *x, int b, int e, double (*part)[6])
{
  const int lane = threadIdx.x & 31;
  double s[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (int q0 = b + lane; q0 < e; q0 += 128)
  {
    int v[4];
    #pragma unroll
    for (int j = 0; j < 4; j ++) v[j] = q0 + 32*j < e ? g.elist[q0 + 32*j] : -1;
    double f[4][3], p[4][3];
    #pragma unroll
    for (int j = 0; j < 4; j ++)
    {
      const int k = v[j] >= 0 ? v[j] >> 1 : 0;
      for (int c = 0; c < 3; c ++) { f[j][c] = g.f[c][k]; p[j][c] = g.p[c][k]; }
    }
    #pragma unroll
    for (int j = 0; j < 4; j ++)
    {
      if (v[j] < 0) break;
      if (v[j] & 1) { f[j][0] = -f[j][0]; f[j][1] = -f[j][1]; f[j][2] = -f[j][2]; }
      s[0] += f[j][0]; s[1] += f[j][1]; s[2] += f[j][2];
      const double a[3] = {p[j][0]-x[0], p[j][1]-x[1], p[j][2]-x[2]};
      s[3] += a[1]*f[j][2] - a[2]*f[j][1];
      s[4] += a[2]*f[j][0] - a[0]*f[j][2];
      s[5] += a[0]*f[j][1] - a[1]*f[j][0];
    }
  }
  for (int c = 0; c < 6; c ++) part[lane][c] = s[c];
  __syncwarp();
  double acc = 0.0;
  if (lane < 6) for (int L = 0; L < 32; L ++) acc += part[L][lane];
  return acc;
}

// Component q of the same sum by a block: the warps take the entries' terms
// side by side, the first adds them up.  A chain of 40 + 64 FP64 instructions
// of 64 clocks where the sum of all six by one warp has 600; for the long sums
// of few particles, where the chip waits for the chain (a full chunk 57 us by
// one warp, 13 by six blocks), not for thousands of short ones (4,097
// particles: 35 us by a warp each, 73 by blocks).
__device__ __forceinline__ double chunk_component(const PgTT &g, int w, int q, int b, int e, const PgDev &d, double (*term)[32])
{
  constexpr int EACH = PG_TT_CHUNK / TPB;                // entries a lane
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c1 = q < 3 ? q : (q + 1) % 3, c2 = (q + 2) % 3;   // torque q-3: a[c1] f[c2] - a[c2] f[c1]
  const double x1 = d.position[c1][w], x2 = d.position[c2][w];
  int v[EACH];
  #pragma unroll
  for (int j = 0; j < EACH; j ++)
  {
    const int k = b + lane + 32 * (warp * EACH + j);
    v[j] = k < e ? g.elist[k] : -1;
  }
  double f1[EACH], f2[EACH], p1[EACH], p2[EACH];
  #pragma unroll
  for (int j = 0; j < EACH; j ++)
  {
    const int k = v[j] >= 0 ? v[j] >> 1 : 0;
    f1[j] = g.f[c1][k];
    if (q >= 3) { f2[j] = g.f[c2][k]; p1[j] = g.p[c1][k]; p2[j] = g.p[c2][k]; }
  }
  #pragma unroll
  for (int j = 0; j < EACH; j ++)
  {
    if (v[j] < 0) break;
    const double s1 = v[j] & 1 ? -f1[j] : f1[j];
    if (q < 3) term[warp * EACH + j][lane] = s1;
    else
    {
      const double s2 = v[j] & 1 ? -f2[j] : f2[j];
      term[warp * EACH + j][lane] = (p1[j]-x1)*s2 - (p2[j]-x2)*s1;
    }
  }
  __syncthreads();
  if (warp != 0) return 0.0;
  double s = 0.0;
  for (int j = 0; b + lane + 32*j < e; j ++) s += term[j][lane];
  __syncwarp();
  term[0][lane] = s;
  __syncwarp();
  double acc = 0.0;
  if (lane == 0) for (int L = 0; L < 32; L ++) acc += term[0][L];
  return acc;
}

// The first 6 nchunks blocks take a component of a chunk each, of the
// particles that may have more than one chunk (k_tt_totals adds theirs up),
// the others a warp a particle of at most one.
__global__ void __launch_bounds__(TPB, 4) k_tt_sums(PgDev d, PgTT g, int nchunks)
{
  __shared__ union { double part[TPB / 32][32][6]; double term[PG_TT_CHUNK / 32][32]; } sh;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if ((int)blockIdx.x < 6 * nchunks)
  {
    const int c = blockIdx.x / 6, k = blockIdx.x % 6, q = g.chmap[c], w = g.bigp[q], n = g.plast[w] - g.pfirst[w];
    const int b = g.pfirst[w] + (c - g.bigoff[q]) * PG_TT_CHUNK, e = min(b + PG_TT_CHUNK, g.plast[w]);
    if (b >= e || n <= PG_TT_CHUNK) return;
    const double acc = chunk_component(g, w, k, b, e, d, sh.term);
    if (threadIdx.x == 0) g.csum[k][c] = acc;
    return;
  }
  const int w = (blockIdx.x - 6 * nchunks) * (TPB / 32) + warp;
  if (w >= d.parnum) return;
  const int b = g.pfirst[w], e = g.plast[w];
  if (e - b > PG_TT_CHUNK) return;
  double acc = 0.0;
  if (e > b)
  {
    const double x[3] = {d.position[0][w], d.position[1][w], d.position[2][w]};
    acc += chunk_sum(g, x, b, e, sh.part[warp]);
  }
  if (lane < 3) d.ttF[lane][w] = acc;
  else if (lane < 6) d.ttT[lane - 3][w] = acc;
}

__global__ void __launch_bounds__(TPB) k_tt_totals(PgDev d, PgTT g)
{
  const int q = (blockIdx.x * blockDim.x + threadIdx.x) / 6, k = (blockIdx.x * blockDim.x + threadIdx.x) % 6;
  if (q >= g.nbig) return;
  const int w = g.bigp[q], n = g.plast[w] - g.pfirst[w];
  if (n <= PG_TT_CHUNK) return;
  const double *s = g.csum[k] + g.bigoff[q];
  const int nc = (n + PG_TT_CHUNK - 1) / PG_TT_CHUNK;
  double acc = 0.0;
  #pragma unroll 8
  for (int c = 0; c < nc; c ++) acc += s[c];
  if (k < 3) d.ttF[k][w] = acc;
  else d.ttT[k - 3][w] = acc;
}

} // namespace

int pg_tt_key_bits(int ncells)
{
  int b = 1;
  while ((1u << b) <= (unsigned)ncells + 1u) b ++;      // ncells + 1 ranges and the sentinel above them
  return b;
}

void pg_tt_prepare(const PgDev &d, PgTT &g, cudaStream_t s)
{
  if (d.trinum <= 0) return;
  cudaMemsetAsync(g.moved, 0, 4 * sizeof(int), s);
  k_tt_boxes<<<nblk(d.trinum), TPB, 0, s>>>(d, g);
}

void pg_tt_search(const PgDev &d, PgTT &g, cudaStream_t s)
{
  const int T = d.trinum;
  if (T <= 0) return;
  k_tt_keys<<<nblk(T), TPB, 0, s>>>(d, g);
  pg_launch_radix_sort(g.keys[0], g.vals[0], g.keys[1], g.vals[1], g.hist, T, g.passes, nullptr, s);
  cudaMemsetAsync(g.cstart, 0, (size_t)(g.ncells + 1) * sizeof(int), s);
  cudaMemsetAsync(g.cend, 0, (size_t)(g.ncells + 1) * sizeof(int), s);
  k_tt_ranges<<<nblk(T), TPB, 0, s>>>(g, T);
  k_tt_find<false><<<nblk(32LL * T), TPB, 0, s>>>(d, g);
  k_tt_scan<<<1, 1024, 0, s>>>(g.cnt, g.off, T, g.moved + 1);
}

void pg_tt_list(const PgDev &d, PgTT &g, cudaStream_t s)
{
  cudaMemsetAsync(g.pfirst, 0, (size_t)d.parnum * sizeof(int), s);
  cudaMemsetAsync(g.plast, 0, (size_t)d.parnum * sizeof(int), s);
  if (g.np <= 0) return;
  k_tt_find<true><<<nblk(32LL * d.trinum), TPB, 0, s>>>(d, g);
  k_tt_entries<<<nblk(g.np), TPB, 0, s>>>(d, g);
  pg_launch_radix_sort(g.ekeys[0], g.evals[0], g.ekeys[1], g.evals[1], g.ehist, 2 * g.np, g.epasses, nullptr, s);
  k_tt_segments<<<nblk(2LL * g.np), TPB, 0, s>>>(g, 2 * g.np);
  k_tt_big<<<nblk(d.parnum), TPB, 0, s>>>(d, g);
}

void pg_tt_chunk_map(PgTT &g, cudaStream_t s)
{
  if (g.nbig > 0) k_tt_chmap<<<g.nbig, TPB, 0, s>>>(g);
}

void pg_tt_forces(const PgDev &d, const PgTT &list, cudaStream_t s, double step)
{
  PgTT g = list;
  g.vcap = std::min(g.vcap, g.vmost);
  g.ecap = std::min(g.ecap, g.emost);
  if (g.np > 0)
  {
    static const int bd = resident_blocks(k_tt_distances), bn = resident_blocks(k_tt_near, 32);
    auto upto = [](int most, long long n) { const int b = nblk(n); return b < most ? b : most; };
    const int bv = upto(bd, 6LL * g.np), be = upto(bd, 9LL * g.np);
    const int tiles = (2 * g.np + PG_TT_TILE - 1) / PG_TT_TILE;
    cudaMemsetAsync(g.qn, 0, 4 * sizeof(*g.qn), s);
    k_tt_judge<<<nblk(g.np), TPB, 0, s>>>(d, g);
    k_tt_distances<<<bv + be, TPB, 0, s>>>(g, bv);
    k_tt_near<<<std::min((g.np + 31) / 32, bn), 32, 0, s>>>(d, g, step);
    k_tt_active<<<tiles, TILE_THREADS, 0, s>>>(g);
    k_tt_select<<<tiles, TILE_THREADS, 0, s>>>(g);
  }
  const int nchunks = g.nbig > 0 ? g.nchunks : 0;
  if (d.parnum > 0) k_tt_sums<<<6 * nchunks + nblk(32LL * d.parnum), TPB, 0, s>>>(d, g, nchunks);
  if (g.nbig > 0)
  {
    k_tt_totals<<<nblk(6LL * g.nbig), TPB, 0, s>>>(d, g);
  }
}

void pg_tt_count(const PgDev &d, const PgTT &g, int *out2, cudaStream_t s)
{
  cudaMemsetAsync(out2, 0, 2 * sizeof(int), s);
  if (d.trinum > 0 && g.np > 0) k_tt_counts<<<nblk(g.np), TPB, 0, s>>>(g, out2);
}

// kernels of a search, of its list, and of one step's contacts and sums
int pg_tt_search_kernels(const PgTT &g, int trinum) { return 4 + pg_sort_kernel_count(trinum, g.passes); }

int pg_tt_list_kernels(const PgTT &g)
{
  return g.np > 0 ? 4 + pg_sort_kernel_count(2 * g.np, g.epasses) + (g.nbig > 0 ? 1 : 0) : 0;
}

int pg_tt_step_kernels(const PgTT &g) { return 2 + (g.np > 0 ? 5 : 0) + (g.nbig > 0 ? 1 : 0); }

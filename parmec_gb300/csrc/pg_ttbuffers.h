// pg_ttbuffers.h -- the arrays of the mesh-contact pair list that grow with it.
//
// `mem` hands out device memory: make(&p, n) allocates n zeroed elements into
// p, drop(&p) gives p back and nulls it, copy(to, from, n) moves elements on
// the device before anything that follows; make and copy return 0 or a status.
// Wherever a call fails, every pointer of g is null or live, g.cap (g.ccap)
// says 0 until all arrays of that size are there, and the previous list, whose
// contact state the next search takes, is whole: the call can be repeated.
#pragma once
#include <algorithm>
#include "pg_launch.h"
#include "pg_meshcontact.h"

// room for np pairs; the previous list's g.pnp pairs move with it
template <class Mem>
int pg_tt_pair_room(PgTT &g, int np, Mem &mem)
{
  const int cap = np + np / 2 + 1024;
  int rc = 0;
  auto make = [&](auto &p, size_t n) { if (rc == 0) rc = mem.make(&p, n); };
  // the work of the narrow phase and the entries hold nothing between searches
  g.cap = 0;
  auto drop = [&](auto &p) { mem.drop(&p); };
  drop(g.pf); drop(g.pu); drop(g.act); drop(g.near); drop(g.full); drop(g.vit); drop(g.eit); drop(g.vres); drop(g.eres);
  for (int k = 0; k < 2; k ++) { drop(g.ekeys[k]); drop(g.evals[k]); }
  drop(g.ehist); drop(g.ebits); drop(g.etile); drop(g.elist); drop(g.bigp); drop(g.bigoff);
  for (int c = 0; c < 3; c ++) { drop(g.st[c]); drop(g.f[c]); drop(g.p[c]); }
  // the previous list: its old arrays go once the new ones hold it
  int *ppu = nullptr;
  unsigned char *pact = nullptr;
  double *pst[3] = {};
  make(ppu, cap);
  make(pact, cap);
  for (int c = 0; c < 3; c ++) make(pst[c], cap);
  if (rc == 0 && g.pnp > 0)
  {
    rc = mem.copy(ppu, g.ppu, g.pnp);
    if (rc == 0) rc = mem.copy(pact, g.pact, g.pnp);
    for (int c = 0; c < 3 && rc == 0; c ++) rc = mem.copy(pst[c], g.pst[c], g.pnp);
  }
  if (rc == 0)
  {
    std::swap(ppu, g.ppu);
    std::swap(pact, g.pact);
    for (int c = 0; c < 3; c ++) std::swap(pst[c], g.pst[c]);
  }
  drop(ppu);
  drop(pact);
  for (int c = 0; c < 3; c ++) drop(pst[c]);
  make(g.pf, cap); make(g.pu, cap); make(g.act, cap);
  for (int c = 0; c < 3; c ++) { make(g.st[c], cap); make(g.f[c], cap); make(g.p[c], cap); }
  // room for 2 vertex-triangle and 3 edge-edge distances a pair (the spring
  // lattice, whose faces lie parallel, asks for 1.3 and 2.4); pairs beyond
  // it take the whole narrow phase
  g.vcap = (int)std::min(2LL * cap, (long long)PG_TT_DISTANCES);
  g.ecap = (int)std::min(3LL * cap, (long long)PG_TT_DISTANCES);
  make(g.near, cap); make(g.full, cap);
  make(g.vit, g.vcap); make(g.eit, g.ecap);
  make(g.vres, 3 * (size_t)g.vcap); make(g.eres, 3 * (size_t)g.ecap);
  const size_t E = 2 * (size_t)cap, tiles = (E + PG_TT_TILE - 1) / PG_TT_TILE;
  for (int k = 0; k < 2; k ++) { make(g.ekeys[k], E); make(g.evals[k], E); }
  make(g.ehist, pg_sort_hist_len((int)E));
  make(g.ebits, tiles * (PG_TT_TILE / 32));
  make(g.etile, tiles);
  make(g.elist, E);
  make(g.bigp, E / PG_TT_CHUNK + 1); make(g.bigoff, E / PG_TT_CHUNK + 1);
  if (rc == 0) g.cap = cap;
  return rc;
}

// room for the chunk sums of the big particles
template <class Mem>
int pg_tt_chunk_room(PgTT &g, int chunks, Mem &mem)
{
  const int cap = chunks + chunks / 2;
  g.ccap = 0;
  mem.drop(&g.chmap);
  for (int c = 0; c < 6; c ++) mem.drop(&g.csum[c]);
  int rc = mem.make(&g.chmap, (size_t)cap);
  for (int c = 0; c < 6 && rc == 0; c ++) rc = mem.make(&g.csum[c], (size_t)cap);
  if (rc == 0) g.ccap = cap;
  return rc;
}

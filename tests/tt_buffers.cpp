// The arrays of the mesh-contact pair list (pg_ttbuffers.h) where an
// allocation or a copy fails: every call that can fail fails once, on lists
// that grow with and without a previous list.  No pointer may be left to
// memory that was given back, no memory given back twice or lost, the room
// said to be there must be there, the previous list must be whole, and the
// same call must succeed afterwards.  Then the largest list there may be: its
// arrays must have room for what the kernels number in it, in their types.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include "../parmec_gb300/csrc/pg_ttbuffers.h"

size_t pg_sort_hist_len(int n) { return 256 * ((size_t)n / 2048 + 2); }

static long bad = 0;

struct FakeMem
{
  std::map<void *, size_t> live;
  int fail_at = -1, calls = 0;
  bool pretend = false;                                  // sizes alone
  size_t total = 0;
  bool fails() { return calls ++ == fail_at; }
  template <class T> int make(T **p, size_t n)
  {
    if (fails()) return -3;
    if (n > ((size_t)1 << 34)) bad ++;                   // a length that went below zero
    total += n * sizeof(T);
    void *q = pretend ? (void *)(live.size() * 64 + 64) : calloc(n ? n : 1, sizeof(T));
    live[q] = n * sizeof(T);
    *p = (T *)q;
    return 0;
  }
  template <class T> void drop(T **p)
  {
    if (*p)
    {
      if (!live.erase((void *)*p)) bad ++;               // given back before, or never made
      else free((void *)*p);
    }
    *p = nullptr;
  }
  template <class T> int copy(T *to, const T *from, size_t n)
  {
    if (fails()) return -3;
    const auto a = live.find((void *)to), b = live.find((void *)from);
    if (a == live.end() || b == live.end() || a->second < n * sizeof(T) || b->second < n * sizeof(T)) { bad ++; return 0; }
    memcpy(to, from, n * sizeof(T));
    return 0;
  }
};

struct Check
{
  FakeMem &mem;
  size_t seen = 0;
  template <class T> void operator()(T *p, size_t n)
  {
    if (!p) { bad += n > 0; return; }
    const auto it = mem.live.find((void *)p);
    seen ++;
    if (it == mem.live.end() || it->second < n * sizeof(T)) bad ++;
  }
};

// every array of g: live, with room for what g says (nothing says more than 0: null is fine)
static void check(const PgTT &g, FakeMem &mem)
{
  Check c{mem};
  const size_t n = g.cap, pn = g.cap > g.pnp ? (size_t)g.cap : (size_t)g.pnp, E = 2 * n, tiles = (E + PG_TT_TILE - 1) / PG_TT_TILE;
  c(g.pf, n); c(g.pu, n); c(g.act, n); c(g.ppu, pn); c(g.pact, pn); c(g.near, n); c(g.full, n);
  for (int k = 0; k < 3; k ++) { c(g.st[k], n); c(g.f[k], n); c(g.p[k], n); c(g.pst[k], pn); }
  c(g.vit, n ? g.vcap : 0); c(g.eit, n ? g.ecap : 0); c(g.vres, n ? 3 * (size_t)g.vcap : 0); c(g.eres, n ? 3 * (size_t)g.ecap : 0);
  for (int k = 0; k < 2; k ++) { c(g.ekeys[k], E); c(g.evals[k], E); }
  c(g.ehist, n ? pg_sort_hist_len((int)E) : 0); c(g.ebits, tiles * (PG_TT_TILE / 32)); c(g.etile, tiles); c(g.elist, E);
  c(g.bigp, n ? E / PG_TT_CHUNK + 1 : 0); c(g.bigoff, n ? E / PG_TT_CHUNK + 1 : 0);
  c(g.chmap, g.ccap);
  for (int k = 0; k < 6; k ++) c(g.csum[k], g.ccap);
  bad += c.seen != mem.live.size();                      // memory that nothing names
}

static void previous(PgTT &g, bool write)
{
  for (int k = 0; k < g.pnp; k ++)
    if (write) { g.ppu[k] = k; g.pact[k] = k & 1; for (int c = 0; c < 3; c ++) g.pst[c][k] = k + 0.25 * c; }
    else
    {
      bad += g.ppu[k] != k || g.pact[k] != (k & 1);
      for (int c = 0; c < 3; c ++) bad += g.pst[c][k] != k + 0.25 * c;
    }
}

int main()
{
  long tried = 0;
  for (int carried = 0; carried < 2; carried ++)
    for (int grow = 0; grow < 2; grow ++)
      for (int k = 0; ; k ++)
      {
        FakeMem mem;
        PgTT g;
        if (carried)
        {
          if (pg_tt_pair_room(g, 10, mem) || pg_tt_chunk_room(g, 3, mem)) bad ++;
          g.pnp = 700;
          previous(g, true);
        }
        check(g, mem);
        mem.calls = 0;
        mem.fail_at = k;
        const int rc = grow ? pg_tt_chunk_room(g, 5, mem) : pg_tt_pair_room(g, 2000, mem);
        const bool failed = mem.calls > k;
        bad += failed != (rc != 0);
        bad += failed && (grow ? g.ccap : g.cap) != 0;
        check(g, mem);
        previous(g, false);
        mem.fail_at = -1;
        if (grow ? pg_tt_chunk_room(g, 5, mem) : pg_tt_pair_room(g, 2000, mem)) bad ++;
        bad += grow ? g.ccap < 5 : g.cap < 2000;
        check(g, mem);
        previous(g, false);
        tried ++;
        if (!failed) break;
      }
  for (const int np : {0x10000000, 0x10000001, PG_TT_MOST})
  {
    FakeMem mem;
    mem.pretend = true;
    PgTT g;
    if (pg_tt_pair_room(g, np, mem)) bad ++;
    check(g, mem);
    const long long cap = g.cap, stride = 1 << 22;       // stride: threads of the largest grid
    bad += cap < np || 2 * cap > 0x7fffffff;             // two entries a pair, in an int
    bad += g.vcap <= 0 || g.ecap <= 0 || g.vcap + stride > 0x7fffffff || g.ecap + stride > 0x7fffffff;
    bad += ((PG_TT_NEAR - 1LL) << 4 | 15) > 0xffffffffLL; // a near pair's place and the distance, in 32 bits
  }
  printf("%ld %ld\n", bad, tried);
  return 0;
}

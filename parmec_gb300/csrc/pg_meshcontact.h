// pg_meshcontact.h -- device state of the mesh-mesh contact stage
// (pg_meshcontact.cu): triangle boxes and cell sort, the pairs of this and
// the previous step, and the per-particle entry sort.
#pragma once
#include <cuda_runtime.h>
#include "pg_state.h"

#define PG_TT_KMAX 256            // partners one triangle may find (a warp's list in the search)
#define PG_TT_SOON 4              // steps a list serves at least, or the skin grows
#define PG_TT_LATE 32             // steps a list serves at most, or a grown skin shrinks

// a pair whose contact a few distances decide: candidates (bits as in
// pgtf::judge), where their results start, a bound on the smallest
struct PgTTNear { int pair; unsigned mask; int vbase, ebase; float upper, size; };
#define PG_TT_GEO 28
// pairs a list may hold: its entries, three a pair with the room to grow, are
// numbered by 31 bits.  Distances are numbered by 31 bits with room for a
// grid's stride above, near pairs by 28 (four name the distance).
#define PG_TT_MOST 0x2a000000
#define PG_TT_DISTANCES 0x7f000000
#define PG_TT_NEAR 0x10000000

// a triangle's box at a search, widened by r and half the skin, in the keys of
// PgTT.box, its particle (-1: not of a mesh) and whether it is big
struct PgTTBox { unsigned long long lo[3], hi[3]; int owner, big; };

struct PgTT
{
  double r = 0.0;                 // swept radius of every mesh triangle
  double h = 0.0, org[3] = {0, 0, 0};
  int dim[3] = {1, 1, 1}, ncells = 1;
  unsigned none = 0;              // sentinel key (above every cell)
  int passes = 2, epasses = 2;    // radix-sort passes of the two sorts
  unsigned char *big = nullptr;   // [trinum] 1: larger than a cell
  // [trinum] this step's box widened by r, as keys whose unsigned order is
  // the IEEE order of the coordinates (-0 = +0): min xyz (NaN: above every
  // key), max xyz (NaN: 0), so that a NaN fails every overlap test
  unsigned long long *box[6] = {};
  // the pair list: every pair of triangles whose boxes, widened by half the
  // skin, overlapped at the last search, in (finder, partner) order; valid
  // while no vertex coordinate has moved by half the skin since.  The skin
  // starts at skin0 and doubles, up to skin_most, where a list served fewer than
  // PG_TT_SOON steps; a grown one halves where it served more than PG_TT_LATE.
  double skin = 0.0, skin0 = 0.0, skin_most = 0.0;
  int since = 0;                  // steps the list has served
  int valid = 0;
  int *moved = nullptr;           // [4]: a vertex moved, pairs found, big particles, their chunks
  double *ref[9] = {};            // [trinum] vertices at the last search
  PgTTBox *sbox = nullptr;        // [trinum] search boxes
  int *cell = nullptr;            // [trinum] grid cell of a small triangle's box centre
  unsigned *keys[2] = {}; int *vals[2] = {}; unsigned *hist = nullptr;
  int *cstart = nullptr, *cend = nullptr;   // [ncells + 1]: the last range holds the big triangles
  int *cnt = nullptr, *off = nullptr;       // [trinum], [trinum + 1]
  int cap = 0, np = 0;            // pair capacity and pairs
  int most = PG_TT_MOST;          // more pairs than these are refused
  int *pf = nullptr, *pu = nullptr;         // [cap] finder and partner of each pair
  // the narrow phase's work (pg_ttfilter.cuh): float copies of the triangles
  // and their FP64 differences, the pairs that may touch with what decides
  // them, the pairs that need every test, and the distances to take
  float4 *fv = nullptr;           // [3][trinum] vertices relative to org; w of the first: error bound
  double *geo = nullptr;          // [trinum][PG_TT_GEO] vertices, edges, squared edges, third minus first vertex, normal, 2r |normal|
  PgTTNear *near = nullptr;       // [cap]
  int *full = nullptr;            // [cap]
  unsigned *vit = nullptr, *eit = nullptr;  // [vcap], [ecap] near pair << 4 | candidate; vit then holds the region
  double *vres = nullptr, *eres = nullptr;  // [.cap][3] squared distance and the closest points' parameters
  int vcap = 0, ecap = 0;
  int vmost = PG_TT_DISTANCES, emost = PG_TT_DISTANCES;   // not all of the room is taken (a self-test)
  unsigned long long *qn = nullptr;   // [4] near pairs, full pairs, vertex-face and edge-edge distances
  unsigned char *act = nullptr;   // [cap] in contact
  double *st[3] = {}, *f[3] = {}, *p[3] = {};   // tangential state, force on the finder's particle, point
  // the previous list, pnp pairs (state carried by (finder, partner) at a search)
  int pnp = 0;
  int *poff = nullptr, *ppu = nullptr;
  unsigned char *pact = nullptr;
  double *pst[3] = {};
  // the pairs' two entries sorted by particle (ekeys[0]: particle, evals[0]:
  // 2 pair + side), made with the list; each step takes the active ones, in
  // that order, into elist
  unsigned *ekeys[2] = {}; int *evals[2] = {}; unsigned *ehist = nullptr;
  unsigned *ebits = nullptr;      // active entries, one bit each
  int *etile = nullptr;           // active entries before each tile of PG_TT_TILE
  int *elist = nullptr;
  int *pfirst = nullptr, *plast = nullptr;  // [parnum] each particle's range of elist
  // particles with more than PG_TT_CHUNK entries in the list: their chunks
  int nbig = 0, nchunks = 0;
  int *bigp = nullptr, *bigoff = nullptr;   // [cap / PG_TT_CHUNK + 1] particle, first chunk
  int *chmap = nullptr;           // [ccap] chunk -> big particle's place
  double *csum[6] = {};           // [ccap] chunk sums (force, torque)
  int ccap = 0;
};

#define PG_TT_CHUNK 1024          // entries of a chunk: summed by a warp, or by six blocks where a particle has several
#define PG_TT_TILE 1024           // entries of one tile of the selection of active entries

int pg_tt_key_bits(int ncells);
void pg_tt_prepare(const PgDev &d, PgTT &g, cudaStream_t s);              // boxes and geometry; sets moved[0]
void pg_tt_search(const PgDev &d, PgTT &g, cudaStream_t s);               // pairs of each triangle; total in moved[1]
void pg_tt_list(const PgDev &d, PgTT &g, cudaStream_t s);                 // the list of g.np pairs and its entry order
void pg_tt_chunk_map(PgTT &g, cudaStream_t s);                            // chunks of the big particles
void pg_tt_forces(const PgDev &d, const PgTT &g, cudaStream_t s, double step);  // contacts and per-particle sums
void pg_tt_count(const PgDev &d, const PgTT &g, int *out2, cudaStream_t s);   // overlapping and active pairs
int pg_tt_search_kernels(const PgTT &g, int trinum);
int pg_tt_list_kernels(const PgTT &g);
int pg_tt_step_kernels(const PgTT &g);

// pg_quad.cuh -- the particle update of a scene that leaves schedulers idle:
// four lanes a particle, component c of every vector in lane c of the four
// (the fourth lane repeats the first).  Included by pg_step.cu.
//
// Such a scene has a few warps a scheduler at most, and its update lasts as
// long as one warp's chain: loads that wait for one another, FP64 instructions
// at 64 clocks each whatever the number of lanes, and the instructions between
// them at 5 to 10.  A lane that sums one component of force and torque takes 7
// FP64 instructions a contact instead of 18, a product with a matrix 5 instead
// of 15 and the exponential map about 20 instead of 50; vectors are put
// together by shuffles.  What the update reads of the particle is asked for at
// the start, and the entries of its contacts PG_QUAD_WIDE at a time, those it
// is master of and those it is slave of in one list (8 at a time, or both
// lists' first entries ahead of everything, cost more instructions than they
// save of the wait).  Every component is the expression k_integrate evaluates:
// the same bits.  The update of 216 and of 4,096 falling spheres 23 -> 20 and
// 25 -> 21 us, of a 64x64 lattice's nodes 33 -> 26; a third of what is left is
// the launch and the end of the step.
#pragma once

#define PG_QUAD_WIDE 4

struct Quad
{
  unsigned mask;                // the four lanes
  int c, c1, c2;                // this lane's component, the next and the one after
  __device__ __forceinline__ Quad()
  {
    const int lane = threadIdx.x & 31, q = lane & 3;
    mask = 0xfu << (lane & 28);
    c = q == 3 ? 0 : q;
    c1 = c == 2 ? 0 : c + 1;
    c2 = c == 0 ? 2 : c - 1;
  }
  // component k of a vector
  __device__ __forceinline__ double of(double x, int k) const { return __shfl_sync(mask, x, k, 4); }
  __device__ __forceinline__ void all(double x, double *v) const { v[0] = of(x, 0); v[1] = of(x, 1); v[2] = of(x, 2); }
  // the sum of the three components in their order
  __device__ __forceinline__ double sum(double x) const { const double a = of(x, 0), b = of(x, 1), e = of(x, 2); return a + b + e; }
  __device__ __forceinline__ double dot(double a, double b) const { return sum(a*b); }
  // component c of a x b
  __device__ __forceinline__ double cross(double a, double b) const
  {
    const double a1 = of(a, c1), a2 = of(a, c2), b1 = of(b, c1), b2 = of(b, c2);
    return a1*b2 - a2*b1;
  }
  // component c of the product with a matrix whose row (or, transposed, column) c is r
  __device__ __forceinline__ double mul(const double *r, double x) const
  {
    double v[3];
    all(x, v);
    return r[0]*v[0] + r[1]*v[1] + r[2]*v[2];
  }
  __device__ __forceinline__ bool every(bool ok) const { return __all_sync(mask, ok); }
  // v0, v1, v2 by this lane's component
  __device__ __forceinline__ double own(double v0, double v1, double v2) const { return c == 0 ? v0 : c == 1 ? v1 : v2; }
};

// C = (j*I) B, as iso_nvmul
__device__ __forceinline__ double quad_iso(const Quad &q, double j, double x)
{
  double v[3];
  q.all(x, v);
  if (finite_d(v[0]) && finite_d(v[1]) && finite_d(v[2])) return zero_terms(j*x, q.own(v[1], v[2], v[0]), q.own(v[2], v[0], v[1]));
  const double m0 = q.c == 0 ? j : 0.0, m1 = q.c == 1 ? j : 0.0, m2 = q.c == 2 ? j : 0.0;
  return m0*v[0] + m1*v[1] + m2*v[2];
}

// sin(x)/x and (1 - cos(x))/x^2 as exp_terms, the first by the lanes of
// components 0 and 2, the second by those of 1: the two series side by side
// are 12 FP64 instructions instead of 24, their first terms 4 instead of 8
__device__ __forceinline__ void quad_exp_terms(const Quad &q, double angsq, double *psx, double *pcx)
{
  const bool cosine = q.c == 1;
  double x = 0.0;
  bool done = false;
  const double c0 = cosine ? 0.5 : 1.0, k1 = cosine ? -4.166666666666667E-2 : -1.666666666666667E-1,
               k2 = cosine ? 1.388888888888889E-3 : 8.333333333333333E-3;
  if (dbits(angsq) < 0x3ed0000000000000ULL)
  {
    const double p = (k1 + k2 * angsq) * angsq;
    x = c0 + p;
    done = q.every(cosine ? sum_settled<54>(p) : sum_settled<53>(p));
  }
  if (!done)
  {
    if (gt_nonneg(3.0461741978671E-02, angsq))
    {
      const double k3 = cosine ? -2.480158730158730E-5 : -1.984126984126984E-4,
                   k4 = cosine ? 2.755731922398589E-7 : 2.755731922398589E-6,
                   k5 = cosine ? -2.087675698786810E-9 : -2.505210838544172E-8,
                   k6 = cosine ? 1.147074559772972E-11 : 1.605904383682161E-10;
      x = c0 + (k1 + (k2 + (k3 + (k4 + (k5 + k6 * angsq)*angsq)*angsq)*angsq)*angsq)*angsq;
    }
    else
    {
      double sx, cx;
      exp_series(angsq, &sx, &cx);
      x = cosine ? cx : sx;
    }
  }
  *psx = q.of(x, 0);
  *pcx = q.of(x, 1);
}

// row c of the exponential map of the rotation vector w, as expmap
__device__ __forceinline__ void quad_expmap(const Quad &q, double w, double *row, bool typo)
{
  double s[3], sx, cx;
  q.all(w*w, s);
  const double angsq = s[0] + s[1] + s[2];
  quad_exp_terms(q, angsq, &sx, &cx);
  // element (c, c): 1 - cx (the other squares); (c, c+1): cx w_c w_c+1 - sx w_c+2;
  // (c, c+2): cx w_c w_c+2 + sx w_c+1.  The product of the third and the first
  // component is the reference's w_1 w_2 when asked for.
  const double w1 = q.of(w, q.c1), w2 = q.of(w, q.c2);
  const double m = cx*(typo && q.c == 2 ? w2*w : w*w1), t = sx*w;
  const double d0 = -cx*(q.own(s[2], s[2], s[1]) + q.own(s[1], s[0], s[0])) + 1.0;
  const double d1 = m - q.of(t, q.c2);
  const double d2 = q.of(m, q.c2) + q.of(t, q.c1);
  row[0] = q.own(d0, d2, d1);
  row[1] = q.own(d1, d0, d2);
  row[2] = q.own(d2, d1, d0);
}

__device__ __forceinline__ void quad_restrain(const Quad &q, double &v, double *const dir[9], int r)
{
  for (int k = 0; k < 3; k ++)
  {
    const double l = dir[3*k + q.c][r];
    const double dt = q.dot(v, l);
    v = v - dt*l;
  }
}

// the referential angular velocity of an isotropic body, as spin_iso
__device__ __forceinline__ void quad_spin_iso(const Quad &q, double &O, double &Tb, double js, double is, double step, double half,
                                              bool typo)
{
  double row[3];
  quad_expmap(q, -half*O, row, typo);
  double B = q.mul(row, quad_iso(q, js, O));
  B = B + half*Tb;
  const double A = quad_iso(q, is, B);
  B = quad_iso(q, js, A);
  Tb -= q.cross(A, B);
  Tb *= step;
  O = O + quad_iso(q, is, Tb);
}

// gyro_settled with each lane bounding its own component
__device__ __forceinline__ bool quad_settled(const Quad &q, double O, double Tb, double js, double is, double step, double half)
{
  const float tiny = 1.2e-38f, up = 1.000001f;
  if (q.every(dbits(O) == 0 && (dbits(Tb) << 1) == 0)) return finite_d(js) && finite_d(is) && finite_d(step) && finite_d(half);
  const float of = mag32(O), tf = mag32(Tb), jf = mag32(js), jinv = mag32(is), sf = mag32(step), hf = mag32(half);
  const float o1 = __shfl_sync(q.mask, of, q.c1, 4), o2 = __shfl_sync(q.mask, of, q.c2, 4);
  const float om = fmaxf(fmaxf(of, o1), o2) * up + tiny;
  const float th = hf * om * 1.75f;                       // bounds the half turn
  const float qs = jinv * sf * up, qh = jinv * hf * up;
  bool ok = of + tf < 3e17f && th < 0.1f && jf > 1e-30f && jinv > 1e-30f && fabsf(jf * jinv - 1.0f) < 1e-4f &&
            sf > 1e-30f && sf < 1e18f && qs < 1e30f && qh < 1e30f;
  const float a = (of * up + tiny) * 1.0001f + om * (th * th + 1e-6f) + qh * (tf * up + tiny);
  const float P = jf * up * __shfl_sync(q.mask, a, q.c1, 4) * __shfl_sync(q.mask, a, q.c2, 4), r = 4.6e-16f * P;
  const bool torque = tf > 1e-20f && qs * tf > 1e-37f && (dbits(Tb) & 0xfffffffffffffull) != 0 && r <= 1.1e-16f * pow2_floor(tf);
  const bool spin = qs * (tf * up + tiny) + (qs * 4.6e-16f) * P * up + 1e-36f <= 5.5e-17f * pow2_floor(of);
  return q.every(ok && (torque || spin));
}

// `last` in the adaptive force sums: the master sides are summed here, as
// k_contacts_sum would, and the step chosen, as by k_adapt_min
template <int MODE>
__global__ void __launch_bounds__(32) k_integrate_quad(PgDev d, double step, double half, double hstep, int oblocks, int last)
{
  constexpr bool ADAPT = MODE == INT_FORCES_ADAPT;
  constexpr bool FUSED = MODE == INT_FUSED || MODE == INT_DYN_FUSED;
  constexpr bool SUMS = MODE != INT_DYNAMICS && MODE != INT_DYN_FUSED;
  constexpr bool MOVES = MODE != INT_FORCES && MODE != INT_FORCES_ADAPT;
  bool need = false;
  unsigned long long chosen = 0x7fefffffffffffffull;        // DBL_MAX
  const double step0 = step;
  if (FUSED && (int)blockIdx.x < oblocks)
  {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const double st = d.hs ? 0.5*(d.hs[0] + d.hs[1]) : step;
    if (t < d.trinum) need = pgk::obstacles_front(d, t, st);
    if (d.ellnum) flag_rebuild(d, need);
    pgk::step_done(d, step0, last);
    return;
  }
  const Quad q;
  const int c = q.c;
  const bool writes = (threadIdx.x & 3) != 3;
  const int i = ((int)blockIdx.x - oblocks) * 8 + (int)(threadIdx.x >> 2);
  if (i < d.parnum)
  {
    // what the update reads of the particle, asked for before anything waits
    const int sc = d.pscene[i], e = d.pell ? d.pell[i] : -1, E = d.ellnum, row = *d.stepno;
    const int rb = SUMS && E ? d.soff[i] : 0, re = SUMS && E ? d.soff[i+1] : 0;
    const bool masters = SUMS && e >= 0 && d.cwork && (!ADAPT || last);
    const double po = d.position[c][i], ma = d.mass[i];
    double Lr[3], Lc[3], O = 0.0, o = 0.0, v = 0.0, Jr[3], Ir[3], im = 0.0, X = 0.0, C = 0.0, C0 = 0.0;
    bool iso = false, skip = false;
    if (MOVES || ADAPT) for (int k = 0; k < 3; k ++) Lr[k] = d.rotation[3*k + c][i];
    if (MOVES)
    {
      skip = d.flags[i] & PG_FLAG_SKIP;
      iso = d.piso && d.piso[i];
      O = d.angular[c][i];
      o = d.angular[3+c][i];
      v = d.linear[c][i];
      im = d.invm[i];
      for (int k = 0; k < 3; k ++)
      {
        Lc[k] = d.rotation[3*c + k][i];
        Jr[k] = d.inertia[3*k + c][i];
        Ir[k] = d.inverse[3*k + c][i];
      }
      if (FUSED && e >= 0)
      {
        X = d.position[3+c][i];
        C = d.center[3+c][e];
        C0 = d.cref[c][e];
      }
    }
    const bool runs = sc >= 0 && d.sactive[sc];
    const double grav = SUMS && sc >= 0 ? d.sgrav[3*sc + c] : 0.0;
    const double damp = MOVES ? d.t_damping[(size_t)row * d.tab_row + c] : 0.0, spin_damp = MOVES ? d.t_damping[(size_t)row * d.tab_row + 3 + c] : 0.0;
    const int own = masters ? d.ncnt[e] : 0;
    if (MODE == INT_FORCES_ADAPT || MODE == INT_DYN_FUSED)
    {
      step = d.hs[0];
      half = 0.5*step;
      hstep = 0.5*(step+d.hs[1]);
    }
    if (runs)
    {
    const double js = MOVES ? q.of(Jr[0], 0) : 0.0, is = MOVES ? q.of(Ir[0], 0) : 0.0;
    const bool typo = (d.compat & PG_COMPAT_EXPMAP) != 0;
    double F = 0.0, T = 0.0, kact = 0.0, krd = 0.0, kro = 0.0, kmax = 0.0, emax = 0.0;
    // the stiffness of an arm, component c of its diagonal and of its off-diagonal terms (krot_add)
    auto arm_stiffness = [&](double A)
    {
      const double dt = q.dot(A, A);
      double a[3];
      q.all(A, a);
      krd += dt - A*A;
      kro += -(c == 2 ? a[1] : a[0]) * (c == 0 ? a[1] : a[2]);
    };
    if (ADAPT && e >= 0 && !masters)
    {
      kact = d.akact[c][i];
      krd = d.akrot[c][i];
      kro = d.akrot[3+c][i];
      kmax = d.akmax[i];
      emax = d.aemax[i];
    }
    if (!SUMS)
    {
      F = d.force[c][i];
      T = d.torque[c][i];
    }
    else
    {
    // the contacts the particle's sphere is master of, in slot order (summed
    // before, into fm and tm, where another pass needs them), then those it is
    // slave of, in master order (forces.ispc:539-569)
    constexpr int W = PG_QUAD_WIDE;
    if (e >= 0 && !masters) { F = d.fm[c][i]; T = d.tm[c][i]; }
    const int n = own + re - rb;
    const double po1 = q.of(po, q.c1), po2 = q.of(po, q.c2);
    const double *nf = d.nfrc[c], *nf1 = d.nfrc[q.c1], *nf2 = d.nfrc[q.c2], *np1 = d.npnt[q.c1], *np2 = d.npnt[q.c2];
    for (int m0 = 0; m0 < n; m0 += W)
    {
      int ref[W];
      bool on[W];
      double f[W], f1[W], f2[W], p1[W], p2[W];
      #pragma unroll
      for (int j = 0; j < W; j ++)
      {
        const int m = m0 + j;
        ref[j] = m < own ? m * d.estride + e : m < n ? d.rref[rb + m - own] : -1;
      }
      #pragma unroll
      for (int j = 0; j < W; j ++) on[j] = ref[j] >= 0 && d.nflag[ref[j]] != 0;
      #pragma unroll
      for (int j = 0; j < W; j ++)
        if (on[j])
        {
          const int r = ref[j];
          f[j] = nf[r]; f1[j] = nf1[r]; f2[j] = nf2[r];
          p1[j] = np1[r]; p2[j] = np2[r];
        }
      #pragma unroll
      for (int j = 0; j < W; j ++)
      {
        if (!on[j]) continue;
        const bool slave = m0 + j >= own;
        const int r = ref[j];
        const double g = slave ? -f[j] : f[j], g1 = slave ? -f1[j] : f1[j], g2 = slave ? -f2[j] : f2[j];
        const double a1 = p1[j] - po1, a2 = p2[j] - po2;
        F += g;
        T += a1*g2 - a2*g1;
        if (ADAPT)
        {
          // master side (forces.ispc:505-522): the normal; slave side
          // (forces.ispc:539-567): the force direction, and the contact's own
          // stiffness and damping (the reference reads slave records whose
          // kcur/ecur nothing sets)
          const int ms = r % d.estride, code = d.ncode[r];
          double u;
          if (slave)
          {
            u = g;
            double len = sqrt(q.dot(g, g));
            if (len != 0.0)
            {
              len = 1.0/len;
              u *= len;
            }
            else u = 0.0;
          }
          else u = d.nnrm[c][r];
          kact += fabs(u);
          const int ij = pairing(d, d.ellcol[ms], code >= 0 ? d.ellcol[code] : d.tricol[-code-1]);
          const double kc = d.iparam[0][ij];
          double ec;
          if (d.nen) ec = d.nen[r];
          else
          {
            const int pj = slave ? i : code >= 0 ? d.part[code] : d.triobs[-code-1];
            ec = d.iparam[1][ij] * 2.0 * sqrt(kc*(pj >= 0 ? 1.0 / (d.invm[d.part[ms]] + d.invm[pj]) : ma));
          }
          kmax = kc > kmax ? kc : kmax;
          emax = ec > emax ? ec : emax;
          arm_stiffness(q.mul(Lr, q.of(a2, q.c1)));
        }
      }
    }
    F = add_times_zero(F, ma, grav);
    if (d.tt_on)
    {
      // mesh-mesh contacts (pg_meshcontact.cu), summed per particle beforehand
      F = F + d.ttF[c][i];
      T = T + d.ttT[c][i];
    }

    // spring force flushes, in the order a single springs_task applies them
    if (d.sprnum)
    {
      const int vb = d.sev_first[i], ve = d.sev_first[i+1];
      for (int ev = vb; ev < ve; ev ++)
      {
        const int4 w = d.sev[ev];
        const int type = w.x & 1, run = (w.x >> 1) - 1;
        const double *fr = d.spr_out[c], *tq = d.spr_out[(type == 0 ? 3 : 6) + c];
        double af = 0.0, at = 0.0;
        bool started = false;
        if (run >= 0)
        {
          // a long run, its groups summed in the same order by k_spring_run_groups
          run_total(d, run, w, c, af, at);
        }
        else
        for (int s = w.y; s < w.z; s ++)
        {
          if (type == 1 && d.sprpart[1][s] < 0) continue;
          const double x = fr[s], y = tq[s];
          if (!started && !w.w) { af = x; at = y; }
          else { af += x; at += y; }
          started = true;
        }
        if (type == 0) { F += af; T += at; }
        else { F -= af; T -= at; }
        if (ADAPT)
        {
          // the run's stiffness partials (forces.ispc:1212-1345): sums from
          // zero in spring order, maxima for stiffness and damping
          double p = 0.0, pd = 0.0, px = 0.0, km = 0.0, em = 0.0;
          if (run >= 0)
          {
            p = d.sbig_ad[11*run + c];
            pd = d.sbig_ad[11*run + 3 + c];
            px = d.sbig_ad[11*run + 6 + c];
            km = d.sbig_ad[11*run + 9];
            em = d.sbig_ad[11*run + 10];
          }
          else
          {
            const int ao = type == 0 ? 5 : 11;
            for (int s = w.y; s < w.z; s ++)
            {
              if (type == 1 && d.sprpart[1][s] < 0) continue;
              p = p + d.sad[c][s];
              pd = pd + d.sad[ao + c][s];
              px = px + d.sad[ao + 3 + c][s];
              const double xk = d.sad[3][s], xe = d.sad[4][s];
              km = xk > km ? xk : km;
              em = xe > em ? xe : em;
            }
          }
          kact += p;
          krd += pd;
          kro += px;
          kmax = km > kmax ? km : kmax;
          emax = em > emax ? em : emax;
        }
      }
    }

    // torsion spring torque flushes (trqspr_task, forces.ispc:1667-2055),
    // after every translational spring flush, in the same run rule
    if (d.trqsprnum)
    {
      for (int ev = d.tev_first[i]; ev < d.tev_first[i+1]; ev ++)
      {
        const int4 w = d.tev[ev];
        const int type = w.x & 1;
        double at = 0.0, kp = 0.0;
        bool started = false;
        for (int s = w.y; s < w.z; s ++)
        {
          if (type == 1 && d.trqsprpart[1][s] < 0) continue;
          const double y = d.tq_out[c][s];
          if (!started && !w.w) at = y;
          else at += y;
          if (ADAPT) kp = kp + d.tq_k[c][s];
          started = true;
        }
        if (type == 0) T += at;
        else T -= at;
        if (ADAPT) krd += kp;
      }
    }

    // prescribe_body_forces (parmec.cpp:2202-2224): the particle's force and
    // torque are exported, then the prescribed ones added
    if ((MODE == INT_FUSED || MODE == INT_FORCES_ADAPT) && d.pbfnum)
    {
      const int s = d.pbf_slot[i];
      if (s >= 0)
      {
        if (writes)
        {
          d.pbfin[c][s] = F;
          d.pbfin[3+c][s] = T;
        }
        F += d.pbfout[c][s];
        T += d.pbfout[3+c][s];
      }
    }
    }
    if (ADAPT && writes)
    {
      d.akact[c][i] = kact;
      d.akrot[c][i] = krd;
      d.akrot[3+c][i] = kro;
      if (c == 0)
      {
        d.akmax[i] = kmax;
        d.aemax[i] = emax;
      }
    }
    if (!MOVES)
    {
      if (writes) { d.force[c][i] = F; d.torque[c][i] = T; }
      if (ADAPT && last)
      {
        double J[9];
        for (int k = 0; k < 9; k ++) J[k] = d.inertia[k][i];
        double ka[3], kr[6], om, ra;
        q.all(kact, ka);
        q.all(krd, kr);
        q.all(kro, kr + 3);
        const double h = critical_step(ka, kmax, emax, kr, ma, J, &om, &ra);
        chosen = (unsigned long long)__double_as_longlong(h);
      }
    }
    if (MOVES)
    {
    // restrain_forces (restrain.ispc:93-133), in input order; the drop-in
    // entry points run it as its own export
    if (FUSED && d.rstnum)
      for (int rr = d.rst_first[i]; rr < d.rst_first[i+1]; rr ++)
      {
        quad_restrain(q, F, d.rstlin, d.rst_list[rr]);
        quad_restrain(q, T, d.rstang, d.rst_list[rr]);
      }

    // prescribe_acceleration (input.cpp:4247-4341); the drop-in entry points
    // leave prescribed motion to the host, as parmec.cpp does
    const bool prs = FUSED && d.prsnum;
    const int pb = prs ? d.prs_first[i] : 0, pe = prs ? d.prs_first[i+1] : 0;
    for (int pp = pb; pp < pe; pp ++)
    {
      const int s = d.prs_list[pp];
      const double lin = d.t_prs_lin[(size_t)row * d.tab_row + 3*s + c];
      const double ang = d.t_prs_ang[(size_t)row * d.tab_row + 3*s + c];
      if (d.prslin[s] && d.linkind[s] == 1) F = ma * lin;
      else if (d.prslin[s] && d.linkind[s] == 0) F = 0.0;
      if (d.prsang[s] && d.angkind[s] == 1) T = q.mul(Jr, ang);
      else if (d.prsang[s] && d.angkind[s] == 0) T = 0.0;
    }

    // dynamics_task (dynamics.ispc:30-169)
    double x = po;
    if (!skip)
    {
      if (!q.every(!nonzero_d(damp))) F -= ma * damp * v;
      if (!q.every(!nonzero_d(spin_damp)))
      {
        const double t = q.mul(Lc, spin_damp*o);
        const double b = iso ? quad_iso(q, js, t) : q.mul(Jr, t);
        T -= q.mul(Lr, b);
      }
      const bool free_spin = q.every((dbits(T) << 1) == 0 && finite_d(Lc[0]) && finite_d(Lc[1]) && finite_d(Lc[2]));
      double Tb = 0.0;
      if (!(iso && free_spin)) Tb = q.mul(Lc, T);
      if (iso && quad_settled(q, O, Tb, js, is, step, half))
      {
        // O + J^-1 (h Tb); unchanged, bit for bit, without a torque
        if (!free_spin) O = O + is*(step*Tb);
      }
      else if (iso)
      {
        if (free_spin) Tb = q.mul(Lc, T);                // the signs of its zeros
        quad_spin_iso(q, O, Tb, js, is, step, half, typo);
      }
      else
      {
        double er[3];
        quad_expmap(q, -half*O, er, typo);
        double B = q.mul(er, q.mul(Jr, O));
        B = B + half*Tb;
        const double A = q.mul(Ir, B);
        B = q.mul(Jr, A);
        Tb -= q.cross(A, B);
        Tb *= step;
        O = O + q.mul(Ir, Tb);
      }
      im *= step;
      v = v + im*F;
      double L2[3];
      bool still = finite_d(hstep) && (long long)dbits(hstep) >= 0;
      for (int k = 0; k < 3; k ++) still = still && finite_d(Lr[k]) && dbits(Lr[k]) != 0x8000000000000000ull;
      if (q.every(still && dbits(O) == 0))
      {
        // no spin: exp(0) is the identity and L stands; L O is zero, negative
        // where all three products are
        for (int k = 0; k < 3; k ++) L2[k] = Lr[k];
        o = __longlong_as_double((long long)(dbits(Lr[0]) & dbits(Lr[1]) & dbits(Lr[2]) & 0x8000000000000000ull));
      }
      else
      {
        double er[3];
        quad_expmap(q, hstep*O, er, typo);
        for (int k = 0; k < 3; k ++) L2[k] = q.mul(Lr, er[k]);
        o = q.mul(L2, O);
      }
      x += hstep*v;

      // prescribe_velocity (input.cpp:4344-4421)
      for (int pp = pb; pp < pe; pp ++)
      {
        const int s = d.prs_list[pp];
        if (d.prslin[s] && d.linkind[s] == 0) v = d.t_prs_lin[(size_t)row * d.tab_row + 3*s + c];
        if (d.prsang[s] && d.angkind[s] == 0)
        {
          o = d.t_prs_ang[(size_t)row * d.tab_row + 3*s + c];
          double col[3];
          for (int k = 0; k < 3; k ++) col[k] = q.own(q.of(L2[0], k), q.of(L2[1], k), q.of(L2[2], k));
          O = q.mul(col, o);
        }
      }

      if (writes)
      {
        for (int k = 0; k < 3; k ++) d.rotation[3*k + c][i] = L2[k];
        d.position[c][i] = x;
        d.angular[c][i] = O;
        d.angular[3+c][i] = o;
        d.linear[c][i] = v;
      }
      for (int k = 0; k < 3; k ++) Lr[k] = L2[k];
    }
    else
    {
      // skipped particle: prescribe_velocity still applies (it runs after dynamics)
      for (int pp = pb; pp < pe; pp ++)
      {
        const int s = d.prs_list[pp];
        if (d.prslin[s] && d.linkind[s] == 0 && writes) d.linear[c][i] = d.t_prs_lin[(size_t)row * d.tab_row + 3*s + c];
        if (d.prsang[s] && d.angkind[s] == 0)
        {
          const double oo = d.t_prs_ang[(size_t)row * d.tab_row + 3*s + c];
          const double Oc = q.mul(Lc, oo);
          if (writes) { d.angular[c][i] = Oc; d.angular[3+c][i] = oo; }
        }
      }
    }
    if (writes) { d.force[c][i] = F; d.torque[c][i] = T; }

    // ellipsoids_task for this particle's sphere (shapes.ispc:29-98)
    if (FUSED && e >= 0)
    {
      bool at = dbits(C) == dbits(X) && finite_d(X) && finite_d(x) && nonzero_d(x);
      for (int k = 0; k < 3; k ++) at = at && finite_d(Lr[k]);
      const double ce = q.every(at) ? x : x + q.mul(Lr, C - X);
      if (writes) d.center[c][e] = ce;
      // the displacement since the rebuild, squared in FP32: its rounding
      // (1e-6) is far inside the margin between 0.45 and 0.5 of the skin
      const float r = mag32(ce - C0), rr = r*r;
      const float r0 = __shfl_sync(q.mask, rr, 0, 4), r1 = __shfl_sync(q.mask, rr, 1, 4), r2 = __shfl_sync(q.mask, rr, 2, 4);
      need = r0 + r1 + r2 > d.half_skin_sq_f;
    }
    }
    }
  }
  if (ADAPT && last) adapt_min(d, chosen);
  if (FUSED && d.ellnum) flag_rebuild(d, need);
  if (FUSED) pgk::step_done(d, step0, last);
}

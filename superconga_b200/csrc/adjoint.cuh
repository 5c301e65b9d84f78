// Reverse-mode derivatives of one frozen-boundary evaluation of the
// self-consistency map (included at the end of engine.cu; FP64 contexts).
//
// The functional is
//   L(Delta, A, b) = w_omega * Omega + sum_r (beta_x(r) j_x(r) + beta_y(r) j_y(r)),
// with Omega the free energy of ComputeFreeEnergy (ComputeFreeEnergy.h:281-414)
// and j the current of ComputeCurrent (ComputeCurrent.h:175-222), both from
// one pass of Riccati sweeps over every angle with the incoming boundary
// values held fixed (IntegrationIteratorOzaki.h:302-404 without the boundary
// update).  b is the external field B_ext = pi Phi / area of the gauge
// (RiccatiSolver.h:137-139).
//
// L is linear in the frame sums Re I and Re g of every angle, so the
// derivative starts from seeds on the frame lattice: the transposes of the
// rotation back (insertRotatedGridAdditive) and of the frame extension
// (extendValuesAtBoundary) applied to the reference-grid weights.  The adjoint
// sweep then runs, per trajectory column, the two Riccati recursions forward,
// storing both coherence functions at every site, and integrates the two
// adjoint recursions in reverse.  Complex sensitivities are carried as
// G = dL/dRe z + i dL/dIm z: G_z = conj(f'(z)) G_w for holomorphic w = f(z),
// G_z = k conj(G_w) for w = k conj(z).  The frame-lattice sensitivities of the
// rotated order parameter and of the Doppler shift are finally scattered back
// through the transposed bilinear lookups onto the reference grid.

namespace {

struct AdjArgs {
  SweepArgs<double> S;
  int tile0, n_tiles;        // tiles of this launch
  Cx<double> *g_all;         // gamma of every site, [tile - tile0][row][energy][column of tile]
  const double2 *seed;       // [slot][n1*n1] (seed of Re I, seed of Re g)
  double2 *grad_d;           // [slot][n1*n1] dL/dDelta_frame
  double *grad_e;            // [slot][n1*n1] dL/d(Doppler shift)
};

__device__ __forceinline__ Cx<double> cadd(Cx<double> a, Cx<double> b) { return {a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ Cx<double> cconj(Cx<double> a) { return {a.re, -a.im}; }
__device__ __forceinline__ Cx<double> cscale(Cx<double> a, double s) { return {a.re * s, a.im * s}; }
__device__ __forceinline__ Cx<double> cinv(Cx<double> a) {
  const double n = 1.0 / (a.re * a.re + a.im * a.im);
  return {a.re * n, -a.im * n};
}

// Reverse mode of riccati_step<double> (same intermediates): given gw for g1,
// returns the sensitivities of g0, of the step's order parameter D and of the
// real part of the step's energy.
__device__ __forceinline__ void riccati_step_adj(double dre, double dim, double ere, double eim,
                                                 Cx<double> g0, double h, Cx<double> gw,
                                                 Cx<double> &gg0, Cx<double> &gD, double &ge) {
  typedef Cx<double> C;
  const double q = 0.25 * h;
  const C a{q * dim, q * dre};
  const C ihe{-h * eim, h * ere};
  const C ag = cmul(a, g0);
  const C b{2.0 * ag.re + ihe.re - 1.0, 2.0 * ag.im + ihe.im};
  const C t{ag.re + ihe.re + 1.0, ag.im + ihe.im};
  const C tg = cmul(t, g0);
  const C c{tg.re - h * dim, tg.im + h * dre};
  const C bb = cmul(b, b), ac = cmul(a, c);
  const C s = csqrt_dev<double>(bb.re - 4.0 * ac.re, bb.im - 4.0 * ac.im);
  const C den{s.re - b.re, s.im - b.im};
  const C rden = cinv(den);
  const C g1 = cmul(cscale(c, 2.0), rden);
  // g1 = 2 c / den
  C Gc = cmul(cconj(cscale(rden, 2.0)), gw);
  const C Gden = cmul(cconj(cscale(cmul(g1, rden), -1.0)), gw);
  // den = s - b
  C Gb = cscale(Gden, -1.0);
  // s = sqrt(disc)
  const C Gdisc = cmul(cconj(cscale(cinv(s), 0.5)), Gden);
  // disc = b^2 - 4 a c
  Gb = cadd(Gb, cmul(cconj(cscale(b, 2.0)), Gdisc));
  C Ga = cmul(cconj(cscale(c, -4.0)), Gdisc);
  Gc = cadd(Gc, cmul(cconj(cscale(a, -4.0)), Gdisc));
  // c = t g0 + i h D
  const C Gt = cmul(cconj(g0), Gc);
  gg0 = cmul(cconj(t), Gc);
  // t = a g0 + i h e + 1;  b = 2 a g0 + i h e - 1
  const C Gag = cadd(Gt, cscale(Gb, 2.0));
  const C Gihe = cadd(Gt, Gb);
  Ga = cadd(Ga, cmul(cconj(g0), Gag));
  gg0 = cadd(gg0, cmul(cconj(a), Gag));
  // i h e: G_e = -i h G
  ge = h * Gihe.im;
  // i h D: G_D = -i h G
  gD = C{h * Gc.im, -h * Gc.re};
  // a = (i h / 4) conj(D): G_D += (i h / 4) conj(G_a)
  gD = cadd(gD, C{q * Ga.im, q * Ga.re});
}

// Reverse mode of step_fast at the same site constants: given gw for g1,
// returns the sensitivity of g0 and adds those of the step's order parameter
// and of the real part of its energy to gD and ge.  With the step written as
//   u = a g0, beta = u + B1, t = beta + B1 + 2, c = t g0 + P, w = B1^2 - a P - 2 u,
//   s = sqrt(w), g1 = c / (s - beta)      (a = (i h / 4) conj(D), P = i h D,
//                                          B1 = (i h e - 1) / 2)
// the reverse is a dozen complex products on values the forward step has too;
// |w| and 1 / |w| come from one estimate.
__device__ __forceinline__ Cx<double> step_fast_adj(const SiteConst<double> &S, double s0, double sh, double d,
                                                    double h, Cx<double> g0, Cx<double> gw, Cx<double> &gD,
                                                    double &ge) {
  typedef Cx<double> C;
  const double urd = S.ar * g0.re - (S.ai * g0.im + d), uim = S.ar * g0.im + S.ai * g0.re;
  const double br = urd - 0.5, bi = uim + sh;
  const double tr = (urd - d) + 1.0, ti = bi + sh;
  const double cre = tr * g0.re - (ti * g0.im + S.hdi), cim = tr * g0.im + (ti * g0.re + S.hdr);
  const double xh = (0.5 * ((d * d + s0) - d) - urd) + 0.125, y = -(d * sh + (0.5 * sh + uim));
  const double xx = xh * xh + (y * y + 1e-300);  // |w|^2 / 4
  const double rm = rsqrt_(xx), m = xx * rm;     // 2 / |w|, |w| / 2
  const double U = m + xh, rho = rsqrt_pos(U);
  const double sr = U * rho, si = y * rho;
  const double dr = sr - br, di = si - bi;
  const double inv = rcp_pos(dr * dr + di * di);
  // conj(1 / den) = den / |den|^2
  const C Gc = cmul(C{dr * inv, di * inv}, gw);
  const C g1{(cre * dr + cim * di) * inv, (cim * dr - cre * di) * inv};
  const C Gb = cmul(C{g1.re, -g1.im}, Gc);  // of beta: minus the sensitivity of den
  // s: -Gb; w = s^2: conj(1 / (2 s)) = s / (2 |w|), 1 / (2 |w|) = rm / 4
  const double q4 = -0.25 * rm;
  const C Gw = cmul(C{sr * q4, si * q4}, Gb);
  const C Gt{g0.re * Gc.re + g0.im * Gc.im, g0.re * Gc.im - g0.im * Gc.re};  // conj(g0) Gc
  C G0{tr * Gc.re + ti * Gc.im, tr * Gc.im - ti * Gc.re};                    // conj(t) Gc
  const C Gu{Gt.re + Gb.re - 2.0 * Gw.re, Gt.im + Gb.im - 2.0 * Gw.im};
  G0.re += S.ar * Gu.re + S.ai * Gu.im;  // conj(a) Gu
  G0.im += S.ar * Gu.im - S.ai * Gu.re;
  // Re e through i h e: B1 carries half of it, t a further half.
  //   G of i h e = Gt + Gb / 2 + conj(B1) Gw, B1 = (-1/2 - d, sh); its imaginary part
  ge += h * (Gt.im + 0.5 * Gb.im - ((0.5 + d) * Gw.im + sh * Gw.re));
  // P = (-hdi, hdr): G_P = Gc - conj(a) Gw;  a: G_a = conj(g0) Gu - conj(P) Gw
  const C GP{Gc.re - (S.ar * Gw.re + S.ai * Gw.im), Gc.im - (S.ar * Gw.im - S.ai * Gw.re)};
  const C Ga{g0.re * Gu.re + g0.im * Gu.im + (S.hdi * Gw.re - S.hdr * Gw.im),
             g0.re * Gu.im - g0.im * Gu.re + (S.hdi * Gw.im + S.hdr * Gw.re)};
  // i h D: G_D = -i h G_P;  (i h / 4) conj(D): G_D += (i h / 4) conj(G_a)
  gD.re += h * GP.im + 0.25 * h * Ga.im;
  gD.im += -h * GP.re + 0.25 * h * Ga.re;
  return G0;
}

// The adjoint of one tile of trajectory columns, the half-warps as in
// sweep_tile: gammaTilde down and gamma up first, each storing every site (the
// sweep's scratch and g_all), then the adjoint of each recursion back along
// its column, both reading both functions.  A site's sensitivities are written
// by the half-warp that reaches it first and completed by the other after the
// middle.  EMAX energies per thread; LG threads per column and function.
//
// What bounds it: FP64 issue and the latency of its loads (about 90 bytes per
// site and energy stored and read).  Storing both functions instead of
// replaying 16-site segments from checkpoints (twice, in local arrays of 4 KB
// a thread) halves the Riccati steps.
template <int EMAX, int LG>
__global__ void __launch_bounds__(128, 3) k_adjoint(const AdjArgs J) {
  typedef Cx<double> C;
  const SweepArgs<double> &A = J.S;
  const int local = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (local >= J.n_tiles) return;  // whole warps
  const int tile = J.tile0 + local;
  const int lane = threadIdx.x & 31, sub = lane & 15;
  const bool down = lane >= 16;
  constexpr int G = 1 << LG, T = 16 >> LG;
  const int g = sub & (G - 1);
  const int item = tile * T + (sub >> LG);
  const unsigned gmask = ((1u << G) - 1u) << (lane & ~(G - 1));
  const int4 it = item < A.n_items ? A.items[item] : make_int4(0, 0, 0, -1);
  const int a = it.x, x = it.y, lo = it.z, n_rows = it.w - it.z + 1;
  const int n1 = A.n1, ne = A.ne;
  const size_t nn1 = (size_t)n1 * n1;
  const double h = A.ang[a].hs;
  const int e0 = g * EMAX, ecount = min(max(ne - e0, 0), EMAX);
  double hd[EMAX], rr[EMAX];  // h e_im / 2, residue
#pragma unroll
  for (int j = 0; j < EMAX; ++j) {
    hd[j] = 0.5 * h * ((j < ecount) ? A.e_im[e0 + j] : 1.0);
    rr[j] = (j < ecount) ? A.res[e0 + j] : 0.0;
  }
  const size_t ax = (size_t)a * n1 + x;
  const int in_base = (down ? A.idx_in_gt : A.idx_in_g)[ax];
  const double *dist_in = down ? A.dist_in_gt : A.dist_in_g;
  const C *bin = down ? A.bin_gt : A.bin_g;
  const int l_entry = down ? 3 : 2;

  // Records and both functions of row 0 of the column; rows are s_row apart.
  const double4 *rec = (const double4 *)A.scratch2 + rec_index(A, LG, item, 0);
  const ptrdiff_t s_row = (ptrdiff_t)ne * T;
  C *gt_all = A.scratch + scratch_index(A, LG, item, 0, e0);
  C *g_all = J.g_all + scratch_index(A, LG, item - J.tile0 * T, 0, e0);
  C *own = down ? gt_all : g_all;
  const C *other = down ? g_all : gt_all;
  const int turns = __reduce_max_sync(0xffffffffu, n_rows);

  C coh[EMAX];
#pragma unroll
  for (int j = 0; j < EMAX; ++j) coh[j] = C{0, 0};
  bool bounded = true;
  int n_in = 0, pcode = SITE_GENERAL;
  double p0 = 0, p1 = 0, p2 = 0;
  // ------------------------------------------------------------- forward --
  double4 nx{};
  if (n_rows > 0) nx = rec[(ptrdiff_t)(down ? n_rows - 1 : 0) * T];
  for (int k = 0; k < turns; ++k) {
    __syncwarp();
    if (k >= n_rows) continue;
    const int r = down ? n_rows - 1 - k : k;
    const double4 fr = nx;
    if (k + 1 < n_rows) nx = rec[(ptrdiff_t)(down ? r - 1 : r + 1) * T];
    const int code = site_code(fr.w), l = code & SITE_LABEL;
    const double dre = down ? -fr.x : fr.x, dim = fr.y, es = fr.z;
    if (code == 1 && pcode < SITE_GENERAL && bounded) {
      const SiteConst<double> S = site_const<double>((dre + p0) * 0.5, (dim + p1) * 0.5, (es + p2) * 0.5, h);
      const double s0 = 2.0 * S.s0h - S.sh * S.sh;
#pragma unroll
      for (int j = 0; j < EMAX; ++j) coh[j] = step_fast(S, s0, S.sh, hd[j], coh[j]);
    } else {
      const bool entry = l == l_entry;
      const double st = entry ? dist_in[in_base + n_in] * h : h;
      const double mre = entry ? dre : (dre + p0) * 0.5, mim = entry ? dim : (dim + p1) * 0.5,
                   mes = entry ? es : (es + p2) * 0.5;
#pragma unroll
      for (int j = 0; j < EMAX; ++j) {
        C g0 = coh[j];
        if (entry) {
          g0 = j < ecount ? bin[(size_t)(in_base + n_in) * A.ne_stride + e0 + j] : C{0, 0};
          if (!(g0.re * g0.re + g0.im * g0.im < 1.002)) bounded = false;
        }
        coh[j] = l == 0 ? C{0, 0} : riccati_step<double>(mre, mim, mes, j < ecount ? A.e_im[e0 + j] : 1.0, g0, st);
      }
      n_in += entry;
    }
#pragma unroll
    for (int j = 0; j < EMAX; ++j)
      if (j < ecount) own[(ptrdiff_t)r * s_row + j * T] = coh[j];
    pcode = code;
    p0 = dre;
    p1 = dim;
    p2 = es;
  }
  __syncwarp();

  // ------------------------------------------------------------- reverse --
  // The row visited by step k, from the column's end of this function back:
  // its order-parameter and shift sensitivities collect the step at the row
  // (half, midpoint) and the step visited before (the other half, in pend).
  const size_t site0 = (size_t)(a - A.slot_base) * nn1 + (size_t)lo * n1 + x;
  const int below = n_rows >> 1, odd = n_rows & 1;
  const int first = down ? below : n_rows - below;  // rows this half-warp reaches before the other one
  const int delay = down ? odd : 0;
  const int turns2 = __reduce_max_sync(0xffffffffu, n_rows + odd);
  C lam[EMAX];
#pragma unroll
  for (int j = 0; j < EMAX; ++j) lam[j] = C{0, 0};
  C pend{0, 0};
  double pend_e = 0.0;
  // Inputs one row ahead: the record and seed, the other function, and this
  // function's value before the row's step (the next row visited).
  C o_nx[EMAX], in_nx[EMAX], me[EMAX];
  double4 r_nx{};
  double2 sd_nx{};
  auto fetch = [&](int k) {  // inputs of step k (coh of the same row is me)
    const int r = down ? k : n_rows - 1 - k;
    const ptrdiff_t before = (ptrdiff_t)(down ? r + 1 : r - 1);  // the row stepped from
    const bool has = k + 1 < n_rows;
    sd_nx = J.seed[site0 + (size_t)r * n1];
    if (has) r_nx = rec[before * T];
#pragma unroll
    for (int j = 0; j < EMAX; ++j)
      if (j < ecount) {
        o_nx[j] = other[(ptrdiff_t)r * s_row + j * T];
        in_nx[j] = has ? own[before * s_row + j * T] : C{0, 0};
      }
  };
#pragma unroll
  for (int j = 0; j < EMAX; ++j) o_nx[j] = in_nx[j] = me[j] = C{0, 0};
  double4 fr{};
  if (n_rows > 0) {
    const int r = down ? 0 : n_rows - 1;
    fr = rec[(ptrdiff_t)r * T];
#pragma unroll
    for (int j = 0; j < EMAX; ++j)
      if (j < ecount) me[j] = own[(ptrdiff_t)r * s_row + j * T];
    fetch(0);
  }
  for (int turn = 0; turn < turns2; ++turn) {
    __syncwarp();
    const int k = turn - delay;
    if (k < 0 || k >= n_rows) continue;
    const int r = down ? k : n_rows - 1 - k;
    C ot[EMAX], gin[EMAX];
#pragma unroll
    for (int j = 0; j < EMAX; ++j) {
      ot[j] = o_nx[j];
      gin[j] = in_nx[j];
    }
    const double4 frp = r_nx;  // the record the step comes from
    const double2 sd = sd_nx;
    if (k + 1 < n_rows) fetch(k + 1);
    const int code = site_code(fr.w), l = code & SITE_LABEL, bcode = site_code(frp.w);
    const double dre = down ? -fr.x : fr.x, dim = fr.y, es = fr.z;
    C ownD{0, 0}, nextD{0, 0};
    double own_e = 0.0, next_e = 0.0;
    if (l != 0) {
#pragma unroll
      for (int j = 0; j < EMAX; ++j) {
        // Re I = -sum r [Im(conj(D) g - D gt)]: with the sign of this
        // function's order parameter, G += s r (Im D, -Re D); the direct
        // dependence on D once, by gamma: s r i (g + conj(gt)).
        const double sr = sd.x * rr[j];
        lam[j].re += sr * dim;
        lam[j].im -= sr * dre;
        if (!down) {
          ownD.re -= sr * (me[j].im - ot[j].im);
          ownD.im += sr * (me[j].re + ot[j].re);
        }
        // Re g = Im q, q = (1 - p) / (1 + p), p = g gt: G_p = conj(dq/dp) (0, s r).
        const C p = cmul(me[j], ot[j]);
        const double nr = 1.0 + p.re, inv = rcp_pos(nr * nr + p.im * p.im);
        const C ip{nr * inv, -p.im * inv}, i2 = cmul(ip, ip);
        const double s2 = -2.0 * sd.y * rr[j];
        const C Gp{s2 * i2.im, s2 * i2.re};
        lam[j].re += ot[j].re * Gp.re + ot[j].im * Gp.im;
        lam[j].im += ot[j].re * Gp.im - ot[j].im * Gp.re;
      }
      if (l == l_entry) {
        --n_in;
        const double st = dist_in[in_base + n_in] * h;
#pragma unroll
        for (int j = 0; j < EMAX; ++j)
          if (j < ecount) {
            C gg0, gD;
            double ge;
            riccati_step_adj(dre, dim, es, A.e_im[e0 + j], bin[(size_t)(in_base + n_in) * A.ne_stride + e0 + j], st,
                             lam[j], gg0, gD, ge);
            ownD = cadd(ownD, gD);
            own_e += ge;
          }
#pragma unroll
        for (int j = 0; j < EMAX; ++j) lam[j] = C{0, 0};
      } else {
        const bool has = k + 1 < n_rows;
        const double q0 = has ? (down ? -frp.x : frp.x) : 0.0, q1 = has ? frp.y : 0.0, q2 = has ? frp.z : 0.0;
        const double mre = (dre + q0) * 0.5, mim = (dim + q1) * 0.5, mes = (es + q2) * 0.5;
        C nD{0, 0};
        double nE = 0.0;
        if (code == 1 && has && bcode < SITE_GENERAL && bounded) {
          const SiteConst<double> S = site_const<double>(mre, mim, mes, h);
          const double s0 = 2.0 * S.s0h - S.sh * S.sh;
#pragma unroll
          for (int j = 0; j < EMAX; ++j) lam[j] = step_fast_adj(S, s0, S.sh, hd[j], h, gin[j], lam[j], nD, nE);
        } else {
#pragma unroll
          for (int j = 0; j < EMAX; ++j)
            if (j < ecount) {
              C gg0, gD;
              double ge;
              riccati_step_adj(mre, mim, mes, A.e_im[e0 + j], gin[j], h, lam[j], gg0, gD, ge);
              nD = cadd(nD, gD);
              nE += ge;
              lam[j] = gg0;
            }
        }
        ownD = cadd(ownD, cscale(nD, 0.5));
        own_e += 0.5 * nE;
        if (has) {
          nextD = cscale(nD, 0.5);
          next_e = 0.5 * nE;
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < EMAX; ++j) lam[j] = C{0, 0};
    }
    ownD = cadd(ownD, pend);
    own_e += pend_e;
    pend = nextD;
    pend_e = next_e;
    // gammaTilde's order parameter is -conj(Delta): G_Delta = -conj(G).
    double v[4] = {down ? -ownD.re : ownD.re, ownD.im, own_e, 0.0};
    group_sum4_scatter(v, g, LG, gmask);
    const size_t site = site0 + (size_t)r * n1;
    const bool add = A.accumulate || k >= first;  // earlier energy passes, the other half-warp
    double *gd = (double *)(J.grad_d + site), *gv = J.grad_e + site;
    if constexpr (LG == 0) {
      gd[0] = v[0] + (add ? gd[0] : 0.0);
      gd[1] = v[1] + (add ? gd[1] : 0.0);
      *gv = v[2] + (add ? *gv : 0.0);
    } else if constexpr (LG == 1) {
      if (g == 0) {
        gd[0] = v[0] + (add ? gd[0] : 0.0);
        gd[1] = v[1] + (add ? gd[1] : 0.0);
      } else {
        *gv = v[0] + (add ? *gv : 0.0);
      }
    } else {
      const int which = g >> (LG - 2);
      if ((g & ((1 << (LG - 2)) - 1)) == 0 && which < 3) {
        double *d = which == 2 ? gv : gd + which;
        *d = v[0] + (add ? *d : 0.0);
      }
    }
    fr = frp;
#pragma unroll
    for (int j = 0; j < EMAX; ++j) me[j] = gin[j];
  }
}

// The transposes of the bilinear lookups are gathers: the sites of the lattice
// `from` (side n_from) whose lookup in the lattice `to` (side n_to, rotation c,
// s) has site (x, y) among its four corners lie within sqrt(2) of (x, y)
// rotated the other way, so the 3 x 3 sites from `base` on are looked up the
// way the forward kernels do and the matching corner's weight is taken.
// Against scattering with FP64 atomics into cleared buffers (456^2 grain, 128
// angles, with the clearing): seeds 1.18 -> 1.07 ms, fields 2.41 -> 1.44 ms.
struct Transposed {
  int bx, by;  // first candidate
};
__device__ __forceinline__ Transposed transposed_lookup(int x, int y, int n_from, int n_to, double c, double s) {
  const double ct = (double)(n_to - 1) / 2.0, cf = (double)(n_from - 1) / 2.0;
  const double X = (double)x - ct, Y = (double)y - ct;
  // inverse rotation, then the smallest integer above the centre - sqrt(2)
  const double xf = X * c + Y * s + cf, yf = Y * c - X * s + cf;
  return Transposed{(int)ceil(xf - 1.4143), (int)ceil(yf - 1.4143)};
}
// The weight with which the lookup of from-site (u, v) reads to-site (x, y).
__device__ __forceinline__ double corner_weight(int u, int v, int x, int y, int n_from, int n_to, double c, double s) {
  Bilinear b;
  if (!rotated_lookup(u, v, n_from, n_to, c, s, b)) return 0.0;
  const int d = y * n_to + x - b.i00;
  const double wx = (d == 0 || d == n_to) ? 1.0 - b.xf : b.xf, wy = (d == 0 || d == 1) ? 1.0 - b.yf : b.yf;
  return (d == 0 || d == 1 || d == n_to || d == n_to + 1) ? wx * wy : 0.0;
}

// Seeds on the frame lattice of the angles from a_begin on (blockIdx.y): the
// transpose of the rotation back (k_rotate_back) applied to the reference-grid
// weights alpha (of Re I, already times the integrand factor's partner
// T h^2 w_omega) and beta (of j_x, j_y, already times the current's factor).
__global__ void __launch_bounds__(256) k_adj_seeds(int n0, int n1, int a_begin, const AngleParams *__restrict__ ang,
                                                   const double *__restrict__ alpha, const double *__restrict__ beta,
                                                   double2 *seed) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const size_t nn0 = (size_t)n0 * n0, nn1 = (size_t)n1 * n1;
  if (t >= (int)nn1) return;
  const int x = t % n1, y = t / n1;
  const AngleParams &P = ang[a_begin + blockIdx.y];
  const Transposed T = transposed_lookup(x, y, n0, n1, P.cB, P.sB);
  double si = 0.0, sg = 0.0;
  if (T.bx > -3 && T.bx < n0 && T.by > -3 && T.by < n0) {
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const int u = T.bx + k % 3, v = T.by + k / 3;
      if (u < 0 || u >= n0 || v < 0 || v >= n0) continue;
      const double w = corner_weight(u, v, x, y, n0, n1, P.cB, P.sB);
      if (w == 0.0) continue;
      const size_t i = (size_t)v * n0 + u;
      si = fma(w, alpha[i], si);
      sg = fma(w, beta[i] * P.sx + beta[nn0 + i] * P.sy, sg);
    }
  }
  seed[(size_t)blockIdx.y * nn1 + t] = make_double2(si * P.w, sg);
}

// Transpose of the frame extension (k_halo): a halo site's seed moves to its
// sources in equal parts.
__global__ void k_adj_halo_t(int n_entries, int entry0, int n1, const int *__restrict__ entry_angle,
                             int slot_base, const int *__restrict__ site, const int *__restrict__ off,
                             const int *__restrict__ src, double2 *seed) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n_entries) return;
  const int e = entry0 + k;
  double *s = (double *)(seed + (size_t)(entry_angle[e] - slot_base) * n1 * n1);
  const double2 v = ((double2 *)s)[site[e]];
  ((double2 *)s)[site[e]] = make_double2(0.0, 0.0);
  const int b = off[e], en = off[e + 1];
  const double inv = 1.0 / (double)(en - b);
  for (int i = b; i < en; ++i) {
    atomicAdd(s + 2 * (size_t)src[i], v.x * inv);
    atomicAdd(s + 2 * (size_t)src[i] + 1, v.y * inv);
  }
}

// Frame sensitivities back onto the reference grid: the transposes of the
// bilinear lookups of frame_fields (order parameter, induced vector
// potential), gathered per reference site over the angles of one part
// (blockIdx.z) and added to the gradients.  rows: first and last row of every
// frame column (the sensitivities exist there only).
__global__ void __launch_bounds__(256) k_adj_fields_t(SweepArgs<double> A, int a_begin, int a_end,
                                                      const int2 *__restrict__ rows,
                                                      const double2 *__restrict__ grad_d,
                                                      const double *__restrict__ grad_e, double *g_dext,
                                                      double *g_avec) {
  const int n1 = A.n1, n0 = A.n0;
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= n0 || y >= n0) return;
  const size_t nn1 = (size_t)n1 * n1, nn0 = (size_t)n0 * n0;
  const int n = a_end - a_begin;
  const int k0 = a_begin + (int)((long long)n * blockIdx.z / gridDim.z);
  const int k1 = a_begin + (int)((long long)n * (blockIdx.z + 1) / gridDim.z);
  double dr[MAX_COMP] = {0, 0, 0, 0}, di[MAX_COMP] = {0, 0, 0, 0}, ax = 0.0, ay = 0.0;
  for (int a = k0; a < k1; ++a) {
    const AngleParams &P = A.ang[a];
    const Transposed T = transposed_lookup(x, y, n1, n0, P.cD, P.sD);
    const size_t slot = (size_t)(a - a_begin) * nn1;
    double gr = 0.0, gi = 0.0, ge = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int u = T.bx + i;
      if (u < 0 || u >= n1) continue;
      const int2 lh = rows[(size_t)a * n1 + u];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int v = T.by + j;
        if (lh.x < 0 || v < lh.x || v > lh.y) continue;
        const size_t f = slot + (size_t)v * n1 + u;
        const double w = corner_weight(u, v, x, y, n1, n0, P.cD, P.sD);
        if (w != 0.0) {
          const double2 gd = grad_d[f];
          gr = fma(w, gd.x, gr);
          gi = fma(w, gd.y, gi);
        }
        if (A.has_vp) {
          const double wa = corner_weight(u, v, x, y, n1, n0, P.cA, P.sA);
          if (wa != 0.0) ge = fma(wa, grad_e[f], ge);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < MAX_COMP; ++c)
      if (c < A.nc) {
        dr[c] = fma(P.eta[c], gr, dr[c]);
        di[c] = fma(P.eta[c], gi, di[c]);
      }
    ax = fma(P.vx, ge, ax);
    ay = fma(P.vy, ge, ay);
  }
  const size_t i = (size_t)y * n0 + x;
#pragma unroll
  for (int c = 0; c < MAX_COMP; ++c)
    if (c < A.nc) {
      atomicAdd(g_dext + (size_t)(2 * c) * nn0 + i, dr[c]);
      atomicAdd(g_dext + (size_t)(2 * c + 1) * nn0 + i, di[c]);
    }
  if (A.has_vp) {
    atomicAdd(g_avec + i, A.q * A.lam_scale * ax);
    atomicAdd(g_avec + nn0 + i, A.q * A.lam_scale * ay);
  }
}

// dL/dB_ext: the Doppler shift's derivative with respect to the field (the
// gauge potential of unit field) times its sensitivity, over the chunk's
// trajectory columns (it does not vanish where the field is zero).
__global__ void __launch_bounds__(256) k_adj_field(SweepArgs<double> A, const double *__restrict__ grad_e,
                                                   double *g_b) {
  const int n1 = A.n1, lane = threadIdx.x & 31;
  const int item = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;  // a warp per column
  double gb = 0.0;
  if (item < A.n_items) {
    const int4 it = A.items[item];
    const AngleParams &P = A.ang[it.x];
    const double off = -0.5 * (double)(n1 - 1), xp = ((double)it.y + off) * A.h;
    const double *g = grad_e + (size_t)(it.x - A.slot_base) * n1 * n1 + it.y;
    for (int y = it.z + lane; y <= it.w; y += 32) {
      const double yp = ((double)y + off) * A.h;
      double ax1, ay1;
      gauge_potential(A.gauge, 1.0, A.area, xp * P.cE - yp * P.sE, xp * P.sE + yp * P.cE, ax1, ay1);
      gb += g[(size_t)y * n1] * A.q * (P.vx * ax1 + P.vy * ay1);
    }
  }
  double q[1] = {gb};
  __shared__ double sum;
  block_reduce(q, 0ull, &sum, 1);
  __syncthreads();
  if (threadIdx.x == 0 && sum != 0.0) atomicAdd(g_b, sum);
}

// Transpose of extend_reference: an extension site's sensitivity moves to its
// sources in equal parts.
__global__ void k_adj_rext_t(int n_fields, int nn, int n_sites, const int *__restrict__ site,
                             const int *__restrict__ off, const int *__restrict__ src, double *g) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int f = blockIdx.y;
  if (k >= n_sites || f >= n_fields) return;
  double *gf = g + (size_t)f * nn;
  const double v = gf[site[k]];
  gf[site[k]] = 0.0;
  const int b = off[k], e = off[k + 1];
  const double inv = 1.0 / (double)(e - b);
  for (int i = b; i < e; ++i) atomicAdd(gf + src[i], v * inv);
}

struct AdjCoef {
  double v[MAX_COMP];
};

// Explicit terms of the free energy: sum_c |Delta_c|^2 (ln(T/Tc_c) + T sum r/e)
// inside the grain (times h^2 w_omega), and the mask of the order parameter
// (zero outside the grain, OrderParameter.h:180-199).
__global__ void k_adj_explicit(int n0, int nc, const uint8_t *__restrict__ dom, const double *__restrict__ x,
                               AdjCoef coef, double *g) {
  const size_t nn = (size_t)n0 * n0;
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= nn) return;
  for (int c = 0; c < nc; ++c)
    for (int p = 0; p < 2; ++p) {
      const size_t k = (size_t)(2 * c + p) * nn + i;
      g[k] = dom[i] ? g[k] + 2.0 * coef.v[c] * x[k] : 0.0;
    }
}

// Magnetic term h^2 w_omega (0.5 / lambda^2) sum B^2 with B the curl of the
// stored vector potential (curl_kernel, GridFunctions_GPU.h:326-352).
__global__ void k_adj_curl_t(int n0, double h, double scale, const double *__restrict__ avec, double *g_avec) {
  const size_t nn = (size_t)n0 * n0;
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= nn) return;
  const int x = (int)(i % n0), y = (int)(i / n0);
  const int xn = min(x + 1, n0 - 1), xp = max(x - 1, 0);
  const int yn = min(y + 1, n0 - 1), yp = max(y - 1, 0);
  const double *ax = avec, *ay = avec + nn;
  const double dx = (double)(xn - xp), dy = (double)(yn - yp);
  const double bz = ((ay[(size_t)y * n0 + xn] - ay[(size_t)y * n0 + xp]) / dx -
                     (ax[(size_t)yn * n0 + x] - ax[(size_t)yp * n0 + x]) / dy) / h;
  const double gbz = 2.0 * scale * bz / h;
  atomicAdd(g_avec + nn + (size_t)y * n0 + xn, gbz / dx);
  atomicAdd(g_avec + nn + (size_t)y * n0 + xp, -gbz / dx);
  atomicAdd(g_avec + (size_t)yn * n0 + x, -gbz / dy);
  atomicAdd(g_avec + (size_t)yp * n0 + x, gbz / dy);
}

// Frozen-boundary evaluation: g(x), j and the free energy of the current
// state without an accelerator step and without the boundary update.
void evaluate_once(sc_ctx *c) {
  const HostSetup &S = c->S;
  if (!c->boundary_initialized) boundary_initial<double>(c);
  extend_reference(c);
  run_chunks<double>(c, 0);
  const size_t nn = c->nn0();
  double *delta = c->xstate.p, *avec = c->xstate.p + (size_t)2 * S.nc * nn;
  launch_finalize(c, delta, avec);
}

// Reference-grid weights of Re I (free energy) and of the current, zero
// outside the grain; beta_j null: no current term.
__global__ void k_adj_weights(size_t nn, const uint8_t *__restrict__ dom, double w_fe, double w_j,
                              const double *__restrict__ beta_j, double *alpha, double *beta) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= nn) return;
  const bool in = dom[i] != 0;
  alpha[i] = in ? w_fe : 0.0;
  beta[i] = in && beta_j ? beta_j[i] * w_j : 0.0;
  beta[nn + i] = in && beta_j ? beta_j[nn + i] * w_j : 0.0;
}

struct AdjBuffers {
  DevArray<double> g_all, grad_e, g_dext, g_avec, g_b, alpha, beta, beta_in;
  DevArray<int2> rows;  // [angle][column]: first and last row
};
void AdjDeleter::operator()(AdjBuffers *p) const { delete p; }

// One launch over the tiles [t0, t0 + n) with four energies in flight per
// thread pair: EMAX energies per thread, LG threads per column and function.
template <int EMAX>
void launch_adjoint(sc_ctx *c, const AdjArgs &J) {
  const unsigned blocks = grid1((size_t)J.n_tiles * 32, 128);
  switch (J.S.log_groups) {
    case 0: k_adjoint<EMAX, 0><<<blocks, 128, 0, c->stream>>>(J); break;
    case 1: k_adjoint<EMAX, 1><<<blocks, 128, 0, c->stream>>>(J); break;
    case 2: k_adjoint<EMAX, 2><<<blocks, 128, 0, c->stream>>>(J); break;
    case 3: k_adjoint<EMAX, 3><<<blocks, 128, 0, c->stream>>>(J); break;
    default: k_adjoint<EMAX, 4><<<blocks, 128, 0, c->stream>>>(J); break;
  }
  check_launch(c);
}

// The gradients into the buffers g_dext, g_avec and g_b; beta_j on the device
// or null.  The buffers are the context's and stay allocated.
void adjoint_run(sc_ctx *c, AdjBuffers &B, double w_omega, const double *beta_j) {
  const HostSetup &S = c->S;
  const size_t nn = c->nn0();
  const size_t nn1 = (size_t)S.n1 * S.n1;
  auto ensure = [](DevArray<double> &a, size_t n) {
    if (a.n < n) a.alloc(n);
  };
  // The adjoint's own mapping: two energies per thread, at most 16 threads per
  // column and function (energy passes above 32); a tile is its own 16 / G
  // columns.
  constexpr int ADJ_EMAX = 2;
  const int pass = std::min(c->e_pass, ADJ_EMAX * 16);
  int lg = 0;
  while ((ADJ_EMAX << lg) < pass) ++lg;
  const int T = 16 >> lg;
  size_t slots = 0, tile_bytes = 0, tiles = 0;
  for (const Chunk &ch : c->chunks) {
    const size_t ni = (size_t)(ch.item_end - ch.item_begin);
    slots = std::max(slots, (size_t)(ch.a_end - ch.a_begin));
    tile_bytes = std::max(tile_bytes, (size_t)ch.kmax * pass * T * sizeof(Cx<double>));
    tiles = std::max(tiles, (ni + T - 1) / T);
  }
  // gamma of as many tiles as fit 40% of the free memory (all of them unless
  // the sweep's own scratch already takes most of the device), at least one.
  // The buffer is kept for the next gradient; one that was made when memory
  // was short grows once all tiles, or twice as many as before, would fit.
  const size_t held = B.g_all.n * sizeof(double);
  if (held < tiles * tile_bytes) {
    size_t free_b = 0, total_b = 0;
    CUDA_TRY(cudaMemGetInfo(&free_b, &total_b));
    double budget = 0.4 * (double)(free_b + held);
    if (const char *env = std::getenv("SCB_SCRATCH_MB")) budget = std::min(budget, std::atof(env) * 1048576.0);
    const size_t fit = std::max<size_t>(1, (size_t)budget / tile_bytes);
    const size_t want = std::min(tiles, fit) * tile_bytes;
    if (!held || want == tiles * tile_bytes || want >= 2 * held) {
      try {
        B.g_all.alloc(want / sizeof(double));
      } catch (const EngineError &) {  // no piece of that size: as before
        if (!held) throw;
        B.g_all.alloc(held / sizeof(double));
      }
    }
  }
  if (B.grad_e.n < slots * nn1) B.grad_e.alloc(slots * nn1);
  ensure(B.g_dext, (size_t)2 * S.nc * nn);
  ensure(B.g_avec, 2 * nn);
  ensure(B.g_b, 1);
  ensure(B.alpha, nn);
  ensure(B.beta, 2 * nn);
  if (!B.rows.n) {
    std::vector<int2> rows((size_t)S.n_angles * S.n1);
    for (size_t k = 0; k < rows.size(); ++k) rows[k] = make_int2(S.col_lo[k], S.col_hi[k]);
    B.rows.upload(rows, c->stream);
    CUDA_TRY(cudaStreamSynchronize(c->stream));
  }
  B.g_dext.zero(c->stream);
  B.g_avec.zero(c->stream);
  B.g_b.zero(c->stream);
  const double la = S.h * S.h;
  const double jfactor = (double)(2 * S.charge_sign) * S.temperature;
  k_adj_weights<<<grid1(nn, 256), 256, 0, c->stream>>>(nn, c->dom.p, w_omega * la * S.temperature, jfactor, beta_j,
                                                      B.alpha.p, B.beta.p);
  check_launch(c);
  extend_reference(c);
  for (const Chunk &ch : c->chunks) {
    const int nslots = ch.a_end - ch.a_begin;
    SweepArgs<double> A = sweep_args<double>(c, &ch, 0);
    if (!A.n_items) continue;
    A.log_groups = lg;  // the records in the adjoint's tiles
    launch_frame_fields<double>(c, ch, A);
    // The frame-record buffer (two double2 per site and slot) holds both.
    double2 *seed = (double2 *)c->w_fr, *grad_d = seed + (size_t)nslots * nn1;
    c->frames_zeroed = false;  // the frame buffers serve as seed and gradient buffers
    {
      k_adj_seeds<<<dim3(grid1(nn1, 256), nslots), 256, 0, c->stream>>>(S.n0, S.n1, ch.a_begin, c->ang.p, B.alpha.p,
                                                                        B.beta.p, seed);
      check_launch(c);
      const int h0 = S.halo_angle_off[ch.a_begin], h1 = S.halo_angle_off[ch.a_end];
      if (h1 > h0) {
        k_adj_halo_t<<<grid1(h1 - h0, 128), 128, 0, c->stream>>>(h1 - h0, h0, S.n1, c->halo_angle.p, ch.a_begin,
                                                                  c->halo_site.p, c->halo_off.p, c->halo_src.p, seed);
        check_launch(c);
      }
    }
    AdjArgs J{};
    J.S = A;
    J.g_all = (Cx<double> *)B.g_all.p;
    J.seed = seed;
    J.grad_d = grad_d;
    J.grad_e = B.grad_e.p;
    const size_t ch_tiles = ((size_t)A.n_items + T - 1) / T;
    for (int e = 0; e < S.ne; e += pass) {
      // Energies [e, e + pass) of every column from their own boundary
      // values, adding into the gradients of the earlier passes.
      AdjArgs P = J;
      P.S.ne = std::min(pass, S.ne - e);
      P.S.accumulate = e > 0;
      P.S.e_im += e;
      P.S.res += e;
      P.S.bin_g += e;
      P.S.bin_gt += e;
      const size_t per = (size_t)ch.kmax * P.S.ne * T * sizeof(Cx<double>);
      const size_t most = std::max<size_t>(1, B.g_all.n * sizeof(double) / per);
      for (size_t t0 = 0; t0 < ch_tiles; t0 += most) {
        P.tile0 = (int)t0;
        P.n_tiles = (int)std::min(most, ch_tiles - t0);
        launch_adjoint<ADJ_EMAX>(c, P);
      }
    }
    // As in k_rotate_back: 8 x 4 patches a warp, the angles in parts.
    dim3 gridf((S.n0 + 7) / 8, (S.n0 + 31) / 32);
    gridf.z = std::max(1, std::min<int>(8, (int)((32 * c->n_sm) / (gridf.x * gridf.y)) + 1));
    k_adj_fields_t<<<gridf, dim3(8, 32), 0, c->stream>>>(A, ch.a_begin, ch.a_end, B.rows.p, grad_d, B.grad_e.p,
                                                         B.g_dext.p, B.g_avec.p);
    check_launch(c);
    k_adj_field<<<grid1((size_t)A.n_items * 32, 256), 256, 0, c->stream>>>(A, B.grad_e.p, B.g_b.p);
    check_launch(c);
  }
  // Reference extension transpose, explicit terms, mask.
  const int ns = (int)S.rext_site.size();
  if (ns) {
    dim3 grid(grid1(ns, 128), 2 * S.nc);
    k_adj_rext_t<<<grid, 128, 0, c->stream>>>(2 * S.nc, (int)nn, ns, c->rext_site.p, c->rext_off.p, c->rext_src.p,
                                               B.g_dext.p);
    check_launch(c);
  }
  double si = 0.0;
  for (int e = 0; e < S.ne; ++e) si += S.residues[e] / S.e_im[e];
  AdjCoef coef{};
  for (int k = 0; k < S.nc; ++k) coef.v[k] = w_omega * la * (std::log(S.temperature / S.tc[k]) + si * S.temperature);
  k_adj_explicit<<<grid1(nn, 256), 256, 0, c->stream>>>(S.n0, S.nc, c->dom.p, c->xstate.p, coef, B.g_dext.p);
  check_launch(c);
  if (c->has_vp() && w_omega != 0.0) {
    const double scale = w_omega * la * 0.5 / (S.lambda * S.lambda);
    k_adj_curl_t<<<grid1(nn, 256), 256, 0, c->stream>>>(S.n0, S.h, scale, c->xstate.p + (size_t)2 * S.nc * nn,
                                                          B.g_avec.p);
    check_launch(c);
  }
}

// sc_adjoint and sc_adjoint_device: beta_j and the results where `from` and
// `to` say.
int adjoint_call(sc_ctx *ctx, const char *name, double w_omega, const double *beta_j, cudaMemcpyKind from,
                 double *g_delta, double *g_a, double *g_b, cudaMemcpyKind to) {
  if (!ctx) return SC_ERR_ARG;
  ctx->drop_graph();
  if (ctx->mode != SC_MODE_FP64 || ctx->S.keldysh || ctx->batch_member) {
    ctx->err = std::string(name) + ": FP64 self-consistency contexts only";
    return SC_ERR_STATE;
  }
  if (!ctx->boundary_initialized) {
    ctx->err = std::string(name) + ": the boundary values are not set (run an iteration or sc_boundary_initial first)";
    return SC_ERR_STATE;
  }
  API_BEGIN
  if (!ctx->adj) ctx->adj.reset(new AdjBuffers());
  AdjBuffers &B = *ctx->adj;
  const size_t nn = ctx->nn0();
  if (beta_j && from == cudaMemcpyHostToDevice) {
    if (B.beta_in.n < 2 * nn) B.beta_in.alloc(2 * nn);
    CUDA_TRY(cudaMemcpyAsync(B.beta_in.p, beta_j, 2 * nn * sizeof(double), from, ctx->stream));
    beta_j = B.beta_in.p;
  }
  adjoint_run(ctx, B, w_omega, beta_j);
  if (g_delta)
    CUDA_TRY(cudaMemcpyAsync(g_delta, B.g_dext.p, (size_t)2 * ctx->S.nc * nn * sizeof(double), to, ctx->stream));
  if (g_a) CUDA_TRY(cudaMemcpyAsync(g_a, B.g_avec.p, 2 * nn * sizeof(double), to, ctx->stream));
  if (g_b) CUDA_TRY(cudaMemcpyAsync(g_b, B.g_b.p, sizeof(double), to, ctx->stream));
  CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  API_END
}

}  // namespace

extern "C" {

int sc_set_external_field(sc_ctx *ctx, double b) {
  if (!ctx || ctx->batch_member) return SC_ERR_ARG;
  ctx->drop_graph();
  ctx->S.flux_quanta = b * ctx->S.area / M_PI;
  return SC_OK;
}

int sc_get_external_field(const sc_ctx *ctx, double *b) {
  if (!ctx || !b) return SC_ERR_ARG;
  *b = M_PI * ctx->S.flux_quanta / ctx->S.area;
  return SC_OK;
}

int sc_evaluate(sc_ctx *ctx, double *free_energy) {
  if (!ctx) return SC_ERR_ARG;
  ctx->drop_graph();
  if (ctx->mode != SC_MODE_FP64 || ctx->S.keldysh || ctx->batch_member) {
    ctx->err = "sc_evaluate: FP64 self-consistency contexts only";
    return SC_ERR_STATE;
  }
  API_BEGIN
  evaluate_once(ctx);
  read_scalars(ctx);
  if (free_energy) *free_energy = ctx->host_scalars.fe;
  API_END
}

int sc_adjoint(sc_ctx *ctx, double w_omega, const double *beta_j, double *g_delta, double *g_a,
               double *g_b) {
  return adjoint_call(ctx, "sc_adjoint", w_omega, beta_j, cudaMemcpyHostToDevice, g_delta, g_a, g_b,
                      cudaMemcpyDeviceToHost);
}

int sc_adjoint_device(sc_ctx *ctx, double w_omega, const double *d_beta_j, double *d_g_delta, double *d_g_a,
                      double *d_g_b) {
  return adjoint_call(ctx, "sc_adjoint_device", w_omega, d_beta_j, cudaMemcpyDeviceToDevice, d_g_delta, d_g_a, d_g_b,
                      cudaMemcpyDeviceToDevice);
}

}  // extern "C"

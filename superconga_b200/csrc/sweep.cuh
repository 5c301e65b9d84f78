// The fused Riccati sweep (included in engine.cu's anonymous namespace).
//
// G = 2^lg threads share one trajectory column (angle, x) and one coherence
// function; thread g integrates the energies [g EMAX, g EMAX + EMAX).  Half a
// warp integrates gammaTilde down its 16 / G columns, the other half gamma up
// the same columns, at the same time (RiccatiSolverConfined.h:129-312).  Until
// the two meet in the middle of the column each stores its values
// (scratch[tile][row][energy][column]); from there on each reads what the
// other one stored at the site it has reached and forms the Green sums over
// all energies there (GreensFunctionStatic.h:92-157, ComputeFreeEnergy.h:
// 106-160).  One value per site and energy is stored and read, as in a sweep
// down and up by the same thread, but the serial chain of steps is half as
// long and twice as many threads work on a column, which is what bounds small
// grains; the order of the steps and of each sum is unchanged.
// KEL: real energies e_re + i e_im (the LDOS path, IntegrationIteratorKeldysh.h
// :219-389); instead of the energy sums, Im g of every energy is written to the
// LDOS frame buffer (GreensFunctionStatic.h:66-90, ComputeLDOS.h:123-144).

// One step of one coherence function at one site for EMAX energies
// (internal::computeStep, RiccatiSolverConfined.h:129-225): entry sites start
// from the stored boundary value with the partial step dist*h, grain sites take
// the midpoint step, exit sites also step on to the boundary and store the
// out-going value (and its conjugate on the mirrored partner angle when pout is
// set), sites outside the grain reset to zero.  eim: the imaginary parts of the
// thread's energies in memory.  Returns false when an entering value lies
// outside the unit disc, where the shortened interior step must not be used.
template <typename R, int EMAX, bool KEL>
__device__ __forceinline__ bool site_step(int l, int l_entry, int l_exit, R dre, R dim, R es, R pdre, R pdim, R pes,
                                       const R *ere, const double *e_im, Cx<R> *coh, int ecount, R h, R dist_in,
                                       const Cx<R> *bin, R dist_out, Cx<R> *bout, Cx<R> *pout) {
  const bool entry = l == l_entry;
  const R sdre = entry ? dre : (dre + pdre) * R(0.5);
  const R sdim = entry ? dim : (dim + pdim) * R(0.5);
  const R ses = entry ? es : (es + pes) * R(0.5);
  const R st = entry ? dist_in * h : h;
  bool inside = true;
#pragma unroll
  for (int j = 0; j < EMAX; ++j) {
    const bool on = j < ecount;
    const R ei = on ? (R)e_im[j] : R(1);
    Cx<R> g0 = coh[j];
    if (entry) g0 = on ? bin[j] : Cx<R>{R(0), R(0)};
    if (entry && !(g0.re * g0.re + g0.im * g0.im < R(1.002))) inside = false;
    Cx<R> v = riccati_step<R>(sdre, sdim, KEL ? ses + ere[j] : ses, ei, g0, st);
    if (l == 0) v = Cx<R>{R(0), R(0)};
    coh[j] = v;
    if (l == l_exit) {
      const Cx<R> bv = riccati_step<R>(dre, dim, KEL ? es + ere[j] : es, ei, v, dist_out * h);
      if (on) {
        bout[j] = bv;
        if (pout) pout[j] = Cx<R>{bv.re, -bv.im};
      }
    }
  }
  return inside;
}

// Sum of four values over the G threads of a group, scattered: afterwards the
// thread whose group index has bits (b1 b0) in the two highest positions holds
// the total of value 2 b1 + b0 (G >= 4), or of values {2 b0, 2 b0 + 1} in v[0],
// v[1] (G = 2).  Halving the exchanged set in each of the first two rounds
// takes 3 (G = 2: 2, G = 8: 4) shuffles instead of 4 log2(G).
__device__ __forceinline__ void group_sum4_scatter(double v[4], int g, int log_groups, unsigned mask) {
  if (log_groups == 0) return;
  int o = 1 << (log_groups - 1);
  {  // keep two of four
    const bool up = (g & o) != 0;
    const double s0 = up ? v[0] : v[2], s1 = up ? v[1] : v[3];
    const double r0 = __shfl_xor_sync(mask, s0, o), r1 = __shfl_xor_sync(mask, s1, o);
    v[0] = (up ? v[2] : v[0]) + r0;
    v[1] = (up ? v[3] : v[1]) + r1;
  }
  o >>= 1;
  if (!o) return;
  {  // keep one of two
    const bool up = (g & o) != 0;
    const double sv = up ? v[0] : v[1];
    const double r = __shfl_xor_sync(mask, sv, o);
    v[0] = (up ? v[1] : v[0]) + r;
  }
  for (o >>= 1; o > 0; o >>= 1) v[0] += __shfl_xor_sync(mask, v[0], o);
}

// Asynchronous global-to-shared copies of 16 bytes (cp.async.cg, through L2);
// with pred false nothing is read (the source must still be a valid address)
// and the 16 bytes are zero-filled.  Each thread waits only for its own
// copies (cp.async.wait_group), so no barrier is involved.
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, bool pred) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(pred ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// The sweep's staging ring: every thread keeps the inputs of the next NS - 1
// sites of its column in flight (the site's frame-field record and, past the
// middle, the other function's stored values), copied asynchronously into
// shared memory ring[stage][16-byte unit][thread], so that the latency of these
// loads spans several sites' Riccati steps instead of one.
template <typename R, int EMAX, int MINB, bool PK>
struct SweepRing {
  static constexpr bool on = PK || sizeof(R) == 8;
  static constexpr int NV_REC = sizeof(R) == 8 ? 2 : 1;
  static constexpr int NV_GT = PK ? EMAX / 2 : EMAX;  // stored values: one energy pair, one FP64 energy per unit
  static constexpr int NV = NV_REC + NV_GT;
  static constexpr int STAGE = NV * 128 * 16;
  // Shared memory of a block: all blocks of an SM together 150 KB (FP64; the
  // rest of the 228 KB is L1 for the frame stores and the neighbouring
  // kernels: C2 sweep 15.7 ms, 16.7 with 200 KB), 50 KB a block in FP32.
  static constexpr int NS_FIT = (sizeof(R) == 8 ? 150 / MINB : 50) * 1024 / STAGE;
  static constexpr int NS = on ? (NS_FIT < 2 ? 2 : (NS_FIT > 8 ? 8 : NS_FIT)) : 1;
  static constexpr int BYTES = on ? NS * STAGE : 0;  // dynamic shared memory of a block
};

// One lane's part of one tile of trajectory columns (all lanes of the warp
// call it).  s_res2: twice the residues of the energies.  LG < 0: the group
// size is taken from A at run time.
template <typename R, int EMAX, int MINB, bool KEL, int LG, bool PK>
__device__ __forceinline__ void sweep_tile(const SweepArgs<R> &A, const double *s_res2, int tile) {
  static_assert(!PK || (std::is_same<R, float>::value && EMAX % 2 == 0), "packed sweep: FP32 pairs");
  const int lgc = LG >= 0 ? LG : A.log_groups;
  const int lane = threadIdx.x & 31, sub = lane & 15;
  const bool down = lane >= 16;  // this half-warp's function: gammaTilde (down) or gamma (up)
  const int g = sub & ((1 << lgc) - 1);
  const int item = (tile << (4 - lgc)) + (sub >> lgc);
  const unsigned gmask = ((1u << (1 << lgc)) - 1u) << (lane & ~((1 << lgc) - 1));
  const int4 it = item < A.n_items ? A.items[item] : make_int4(0, 0, 0, -1);  // lanes past the end: no rows
  const int a = it.x, x = it.y, lo = it.z, n_rows = it.w - it.z + 1;
  const int n1 = A.n1, ne = A.ne;
  const size_t nn1 = (size_t)n1 * n1;
  const int T = 16 >> lgc;
  const R h = (R)A.ang[a].hs;  // h / |v_F| of this angle
  const bool burn_in = A.burn_in != 0;
  const int e0 = g * EMAX;
  const int ecount = min(max(ne - e0, 0), EMAX);

  // Interior constants of the energies: d = h e_im / 2 (rounded from FP64) and
  // what step_fast2 takes of it.
  constexpr int NP = PK ? EMAX / 2 : 1;
  R ec[PK ? 1 : EMAX], ere[KEL ? EMAX : 1];
  EnergyConst2 ec2[NP];
#pragma unroll
  for (int j = 0; j < EMAX; ++j) {
    const double d = 0.5 * A.ang[a].hs * ((j < ecount) ? A.e_im[e0 + j] : 1.0);
    if constexpr (KEL) ere[j] = (j < ecount) ? (R)A.e_re[e0 + j] : R(0);
    if constexpr (!PK) ec[j] = R(d);
    if constexpr (PK) {
      const float c[4] = {(float)(0.5 + d), (float)(1.0 + d), (float)(0.5 * (d + d * d)), (float)(3.0 * d)};
      EnergyConst2 &E = ec2[j / 2];
      if (j & 1) E.nbh.y = c[0], E.c1.y = c[1], E.d2h.y = c[2], E.d3.y = c[3];
      else E.nbh.x = c[0], E.c1.x = c[1], E.d2h.x = c[2], E.d3.x = c[3];
    }
  }
  // This function at the last site: one value per energy, or in energy pairs.
  Cx<R> coh[PK ? 1 : EMAX];
  Cx2 coh2[NP];
#pragma unroll
  for (int j = 0; j < (PK ? 1 : EMAX); ++j) coh[j] = Cx<R>{R(0), R(0)};
#pragma unroll
  for (int p = 0; p < NP; ++p) coh2[p] = Cx2{bc2(0.0f), bc2(0.0f)};

  // This function's boundary entries.  With paired angles the out-going values
  // are also the mirrored partner column's (angle + pi, x -> n1 - 1 - x): gamma
  // there is conj(gammaTilde) here and the other way round.
  const size_t ax = (size_t)a * n1 + x;
  const int l_entry = down ? 3 : 2, l_exit = down ? 2 : 3;
  int in_base = (down ? A.idx_in_gt : A.idx_in_g)[ax], out_base = (down ? A.idx_out_gt : A.idx_out_g)[ax];

  // Step k visits row k (gamma) or n_rows - 1 - k (gammaTilde).  The first
  // `first` steps store, the others read what the other function stored: rows
  // below n_rows / 2 hold gamma, the others gammaTilde.  With an odd number of
  // rows gamma starts one loop turn later, so that both functions are done
  // storing after the same turn; the warp synchronises at every turn.
  // LATE (FP32): the Green functions of a site are formed one turn later,
  // beside the step to the next site; the two are independent, and the step's
  // chain of dependent operations hides behind them.  The FP64 sweep has no
  // registers for that (C2: 17.5 -> 24.7 ms) and forms them after the step.
  constexpr bool LATE = sizeof(R) == 4;
  const int below = n_rows >> 1, odd = n_rows & 1;
  const int first = burn_in ? n_rows + 1 : (down ? n_rows - below : below);
  const int delay = down ? 0 : odd;
  const int turns = __reduce_max_sync(0xffffffffu, n_rows + odd) + (LATE ? 1 : 0);
  typedef typename Rec4<R>::type V4;
  const ptrdiff_t dir = down ? -1 : 1;
  const int row0 = down ? n_rows - 1 : 0;
  const ptrdiff_t s_row = (ptrdiff_t)(PK ? (ne + 1) >> 1 : ne) * T;
  using SV = typename std::conditional<PK, float4, Cx<R>>::type;  // stored unit
  const ptrdiff_t f_step = dir * T, s_step = dir * s_row;
  // Record and stored values of the step whose inputs are fetched next, and
  // the place where this step's values are stored.
  const V4 *fp = (const V4 *)A.scratch2 + rec_index(A, lgc, item, row0);
  SV *sp = (SV *)A.scratch + (PK ? scratch_pair_index(A, lgc, item, 0, e0 >> 1) : scratch_index(A, lgc, item, 0, e0)) +
           (ptrdiff_t)row0 * s_row;
  using RG = SweepRing<R, EMAX, MINB, PK>;
  constexpr int NS = RG::NS;
  extern __shared__ float4 ring[];  // [stage][unit][thread]
  constexpr int STAGE = RG::NV * 128;  // float4s of a stage
  float4 *const ring_me = ring + threadIdx.x;
  auto unit = [&](int at, int v) -> float4 * { return ring_me + at + v * 128; };  // at: a stage's first float4
  // Copies of the next step's inputs (its record, and the stored values when
  // with_gt) into its stage; one commit group per call.
  const SV *sq = sp;  // fetched stored values
  int kq = 0, slot_in = 0;  // next step fetched, and its stage (slot_in, slot: offsets of stages)
  auto ring_issue = [&](bool with_gt) {
    if constexpr (RG::on) {
      if (kq < n_rows) {
#pragma unroll
        for (int v = 0; v < RG::NV_REC; ++v) cp_async16(unit(slot_in, v), (const float4 *)fp + v, true);
        if (with_gt) {
#pragma unroll
          for (int jp = 0; jp < RG::NV_GT; ++jp) {
            const bool ok = (PK ? 2 * jp : jp) < ecount;
            cp_async16(unit(slot_in, RG::NV_REC + jp), ok ? (const void *)(sq + jp * T) : (const void *)fp, ok);
          }
        }
        fp += f_step;
        sq += s_step;
      }
      ++kq;
      slot_in = slot_in == (NS - 1) * STAGE ? 0 : slot_in + STAGE;
      cp_async_commit();
    }
  };
  V4 fr_nx;
  Cx2 gt2[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) gt2[p] = Cx2{bc2(0.0f), bc2(0.0f)};
  Cx<R> gt[PK ? 1 : EMAX], gt_nx[RG::on ? 1 : EMAX];  // the other function at the Green functions' site, at the next one
  auto load_gt = [&]() {
    if constexpr (!RG::on) {
#pragma unroll
      for (int j = 0; j < EMAX; ++j)
        if (j < ecount) gt_nx[j] = sq[j * T];
      sq += s_step;
    }
  };
#pragma unroll
  for (int j = 0; j < (PK ? 1 : EMAX); ++j) gt[j] = Cx<R>{R(0), R(0)};
  if constexpr (RG::on) {
    for (int k = 0; k < NS - 1; ++k) ring_issue(false);
  } else {
    if (n_rows > 0) fr_nx = fp[0];
#pragma unroll
    for (int j = 0; j < EMAX; ++j) gt_nx[j] = Cx<R>{R(0), R(0)};
  }

  using Fr = typename FrameOf<R>::type;
  // Record of the site whose Green functions are formed next.
  const ptrdiff_t o_step = dir * (ptrdiff_t)n1;
  const size_t site0 = (size_t)(a - A.slot_base) * nn1 + (size_t)(lo + (down ? n_rows - 1 - first : first)) * n1 + x;
  Fr *rec = A.fr + 2 * site0;
  typename LdosOf<R>::type *ldo = A.ldf + site0 * A.ne_stride + e0;
  // One store of four energies (16 or 32 bytes): the frame's base (an energy
  // pass's slice starts anywhere) and its sites must be aligned; e0 is a
  // multiple of four.  In FP64 four stores of 8 bytes write every 32-byte sector
  // of the frame four times (64 angles, 32 energies: sweep of a 286^2 disc 2.20
  // -> 1.93 ms, of a 487^2 square 8.34 -> 7.37 ms).
  const bool ldos_vec = KEL && EMAX == 4 && (A.ne_stride & 3) == 0 && ((size_t)A.ldf & (4 * sizeof(*ldo) - 1)) == 0;
  bool bounded = true;  // every entering value inside the unit disc
  int pcode = SITE_GENERAL, slot = 0;
  R pdre = 0, pdim = 0, pes = 0;

  auto fast_steps = [&](R dre, R dim, R es) {
    const SiteConst<R> S = site_const<R>((dre + pdre) * R(0.5), (dim + pdim) * R(0.5), (es + pes) * R(0.5), h);
    if constexpr (PK) {
      const SiteConst2 S2{bc2(S.ai), bc2(-S.ar), bc2(-S.ai), bc2(S.hdi), bc2(-S.hdr)};
      const float2 s0h_site = bc2(S.s0h - 0.5f * S.sh * S.sh), nsh_site = bc2(-S.sh), n3sh_site = bc2(-3.0f * S.sh);
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        float2 nsh = nsh_site, n3sh = n3sh_site, s0h = s0h_site;
        if constexpr (KEL) {
          const R hh = R(-0.5) * h;
          nsh = make_float2(hh * ere[2 * p] - S.sh, hh * ere[2 * p + 1] - S.sh);
          n3sh = mul2(nsh, bc2(3.0f));
          s0h = fma2(mul2(nsh, bc2(-0.5f)), nsh, bc2(S.s0h));
        }
        coh2[p] = step_fast2(S2, s0h, nsh, n3sh, ec2[p], coh2[p]);
      }
    } else {
      // FP64: s0; FP32: half of it.
      constexpr R c2 = sizeof(R) == 8 ? 2 : 1, c1 = sizeof(R) == 8 ? 1 : 0.5;
      const R s0_site = c2 * S.s0h - c1 * S.sh * S.sh;
#pragma unroll
      for (int j = 0; j < EMAX; ++j) {
        R sh = S.sh, s0 = s0_site;
        if constexpr (KEL) {
          sh += R(0.5) * h * ere[j];
          s0 = c2 * S.s0h - c1 * sh * sh;
        }
        if constexpr (sizeof(R) == 8) coh[j] = step_fast(S, s0, sh, ec[j], coh[j]);
        else coh[j] = step_fast_f32(S, s0, sh, ec[j], coh[j]);
      }
    }
  };
  auto general_steps = [&](int l, R dre, R dim, R es) {
    const bool entry = l == l_entry, exit = l == l_exit;
    Cx<R> *pout = nullptr;
    if (A.pair && exit) {
      const size_t pax = (size_t)(a + A.pair) * n1 + (n1 - 1 - x);
      const int po = (down ? A.idx_out_g : A.idx_out_gt)[pax] + out_base - (down ? A.idx_out_gt : A.idx_out_g)[ax];
      pout = (down ? A.bout_g : A.bout_gt) + (size_t)po * A.ne_stride + e0;
    }
    Cx<R> c1[EMAX];
#pragma unroll
    for (int j = 0; j < EMAX; ++j) {
      if constexpr (PK) c1[j] = (j & 1) ? Cx<R>{(R)coh2[j / 2].re.y, (R)coh2[j / 2].im.y}
                                        : Cx<R>{(R)coh2[j / 2].re.x, (R)coh2[j / 2].im.x};
      else c1[j] = coh[j];
    }
    if (!site_step<R, EMAX, KEL>(l, l_entry, l_exit, dre, dim, es, pdre, pdim, pes, ere, A.e_im + e0, c1, ecount, h,
                                 entry ? (R)(down ? A.dist_in_gt : A.dist_in_g)[in_base] : R(0),
                                 (down ? A.bin_gt : A.bin_g) + (size_t)in_base * A.ne_stride + e0,
                                 exit ? (R)(down ? A.dist_out_gt : A.dist_out_g)[out_base] : R(0),
                                 (down ? A.bout_gt : A.bout_g) + (size_t)out_base * A.ne_stride + e0, pout))
      bounded = false;
#pragma unroll
    for (int j = 0; j < EMAX; ++j) {
      if constexpr (PK) {
        if (j % 2 == 0) coh2[j / 2] = Cx2{make_float2(c1[j].re, c1[j + 1].re), make_float2(c1[j].im, c1[j + 1].im)};
      } else {
        coh[j] = c1[j];
      }
    }
    in_base += entry;
    out_base += exit;
  };
  auto store = [&]() {
    if constexpr (PK) {
#pragma unroll
      for (int p = 0; p < NP; ++p)
        if (2 * p < ecount) sp[p * T] = make_float4(coh2[p].re.x, coh2[p].re.y, coh2[p].im.x, coh2[p].im.y);
    } else {
#pragma unroll
      for (int j = 0; j < EMAX; ++j)
        if (j < ecount) sp[j * T] = coh[j];
    }
    sp += s_step;
  };
  // The residue's double, zero past the last energy (k_sweep pads its copy).
  auto res2_at = [&](int j) { return (LG >= 0 || j < ecount) ? s_res2[e0 + j] : 0.0; };
  // Green functions at a site (fields gdre, gdim; in: inside the grain) from
  // this function (coh) and the other one (gt).
  auto greens = [&](R gdre, R gdim, bool in) {
    if constexpr (!LATE) {
#pragma unroll
      for (int j = 0; j < EMAX; ++j) {
        const double2 v = *(const double2 *)unit(slot, RG::NV_REC + j);
        gt[j] = Cx<R>{(R)v.x, (R)v.y};
      }
    }
    if constexpr (KEL) {
      if (in) {
        R im[EMAX];
        if constexpr (PK) {
#pragma unroll
          for (int j = 0; j < EMAX; j += 2) {
            const float2 v = greens_g_im2(coh2[j / 2], gt2[j / 2]);
            im[j] = v.x;
            im[j + 1] = v.y;
          }
        } else {
#pragma unroll
          for (int j = 0; j < EMAX; ++j) im[j] = greens_g_im<R>(coh[j], gt[j]);
        }
        bool done = false;
        if constexpr (EMAX == 4) {
          if (ldos_vec && ecount == 4) {
            if constexpr (PK) *(float4 *)ldo = make_float4(im[0], im[1], im[2], im[3]);
            else st_d4((double *)ldo, im[0], im[1], im[2], im[3]);
            done = true;
          }
        }
        if (!done) {
#pragma unroll
          for (int j = 0; j < EMAX; ++j)
            if (j < ecount) ldo[j] = im[j];
        }
      }
      ldo += o_step * A.ne_stride;
    } else {
      // Sums over this thread's energies of r (f + f~*), r Re g and
      // r Im(conj(D) g - D gt): with p = g gt,
      // i 2 / (1 + p) = (fre, fim), and d = (other - own), v = (own + other),
      //   f + f~* = (+-(fre d.re - fim d.im), -(fre v.im + fim v.re)),
      //   Re g = -fre,   Im I = -(D_own.re d.im + D.im v.re),
      // the upper sign for gamma; D_own.re carries the sign of gammaTilde.
      double sfr = 0.0, sfi = 0.0, sg = 0.0, si = 0.0;
      if constexpr (PK) {
        const float2 hre = bc2(0.5f * gdre), him = bc2(0.5f * gdim), m1 = bc2(-1.0f);
#pragma unroll
        for (int j = 0; j < EMAX; j += 2) {
          const Cx2 u = coh2[j / 2], w = gt2[j / 2];
          const float2 nui = mul2(u.im, m1);
          const float2 pre = fma2(u.re, w.re, mul2(nui, w.im)), pim = fma2(u.re, w.im, mul2(u.im, w.re));
          const float2 den = add2(bc2(1.0f), pre);
          const float2 s = fma2(den, den, mul2(pim, pim));
          const float2 inv = make_float2(rcp_pos(s.x), rcp_pos(s.y));
          const float2 fre = mul2(pim, inv), fim = mul2(den, inv);
          const float2 dr = fma2(u.re, m1, w.re), di = add2(w.im, nui);
          const float2 vr = add2(u.re, w.re), vi = add2(u.im, w.im);
          const float2 Fre = fma2(fre, dr, mul2(mul2(fim, m1), di)), nfim = fma2(fre, vi, mul2(fim, vr));
          const float2 nii = fma2(hre, di, mul2(him, vr));
          const double r0 = res2_at(j), r1 = res2_at(j + 1);
          sfr += r0 * (double)Fre.x + r1 * (double)Fre.y;
          sfi -= r0 * (double)nfim.x + r1 * (double)nfim.y;
          sg -= r0 * (double)fre.x + r1 * (double)fre.y;
          si += r0 * (double)nii.x + r1 * (double)nii.y;
        }
      } else {
        double sd = 0.0, sv = 0.0;
#pragma unroll
        for (int j = 0; j < EMAX; ++j) {
          const Cx<R> u = coh[j], w = gt[j];
          const R pim = u.re * w.im + u.im * w.re, den = R(1) + (u.re * w.re - u.im * w.im);
          const R inv = rcp_pos(den * den + pim * pim);
          const double rr = res2_at(j);
          const R dr = w.re - u.re, di = w.im - u.im, vr = u.re + w.re, vi = u.im + w.im;
          if constexpr (sizeof(R) == 8) {
            const R wr = inv * rr, fre = pim * wr, fim = den * wr;
            sfr += fre * dr - fim * di;
            sfi -= fre * vi + fim * vr;
            sg -= fre;
          } else {
            const R fre = pim * inv, fim = den * inv;
            sfr += rr * (double)(fre * dr - fim * di);
            sfi -= rr * (double)(fre * vi + fim * vr);
            sg -= rr * (double)fre;
          }
          sd += rr * (double)di;
          sv += rr * (double)vr;
        }
        si = 0.5 * ((double)gdre * sd + (double)gdim * sv);
      }
      // The mirrored partner angle is not stored: k_rotate_back reads it
      // from this frame at the mirrored site.
      double v[4] = {in ? (down ? -sfr : sfr) : 0.0, in ? sfi : 0.0, in ? sg : 0.0, in ? si : 0.0};
      group_sum4_scatter(v, g, lgc, gmask);
      if (lgc == 0) {
        if (A.accumulate) {
          const double2 of = as_d2(rec[0]), og = as_d2(rec[1]);
          v[0] += of.x;
          v[1] += of.y;
          v[2] += og.x;
          v[3] += og.y;
        }
        rec[0] = frame_pair<Fr>(v[0], v[1]);
        rec[1] = frame_pair<Fr>(v[2], v[3]);
      } else if (lgc == 1) {
        Fr *dst = rec + g;
        if (A.accumulate) {
          const double2 o = as_d2(*dst);
          v[0] += o.x;
          v[1] += o.y;
        }
        *dst = frame_pair<Fr>(v[0], v[1]);
      } else {
        const int sh = lgc > 2 ? lgc - 2 : 0;  // low bits below the two value bits
        if ((g & ((1 << sh) - 1)) == 0) {
          auto *dst = &rec->x + (g >> sh);
          if (A.accumulate) v[0] += (double)*dst;
          *dst = (decltype(Fr::x))v[0];
        }
      }
      rec += 2 * o_step;
    }
  };

  for (int turn = 0; turn < turns; ++turn) {
    __syncwarp();
    const int k = turn - delay;
    const bool step = k >= 0 && k < n_rows;
    const bool green = LATE ? k > first && k <= n_rows : k >= first && k < n_rows;  // of the last, of this site
    const bool want_gt = k >= first;
    // Inputs of step k; the other function's values at its site are used one
    // turn later.
    V4 fr{};
    if (k == first && step) {  // the other function's stores of the rows ahead are done
      if constexpr (RG::on) {
        cp_async_wait<0>();
        kq = k;
        slot_in = slot;
        fp += f_step * (k - min(k + NS - 1, n_rows));
        sq = sp;
        for (int i = 0; i < NS - 1; ++i) ring_issue(true);
      } else {
        sq = sp;
        load_gt();
      }
    }
    if (step) {
      if constexpr (RG::on) {
        ring_issue(want_gt);
        cp_async_wait<NS - 1>();
        if constexpr (sizeof(R) == 4) {
          const float4 v = *unit(slot, 0);
          fr = V4{(R)v.x, (R)v.y, (R)v.z, (R)v.w};
        } else {
          const double2 u = *(const double2 *)unit(slot, 0), w = *(const double2 *)unit(slot, 1);
          fr = V4{(R)u.x, (R)u.y, (R)w.x, (R)w.y};
        }
      } else {
        fr = fr_nx;
        fp += f_step;
        if (k + 1 < n_rows) fr_nx = fp[0];
      }
    }
    const int code = site_code(fr.w);
    // gammaTilde uses -conj(Delta) (RiccatiSolverConfined.h:74-79).
    const R dre = down ? -fr.x : fr.x, dim = fr.y, es = fr.z;
    // Whole warps in the interior take the shortened step with no divergence,
    // storing (first half) or beside the Green functions (second half).
    const bool fast = step && code == 1 && pcode < SITE_GENERAL && bounded;
    if (__all_sync(0xffffffffu, fast && !want_gt)) {
      fast_steps(dre, dim, es);
      if (!burn_in) store();
    } else if (__all_sync(0xffffffffu, fast && green && (!LATE || (pcode & SITE_LABEL) != 0))) {
      if constexpr (LATE) greens(pdre, pdim, true);
      fast_steps(dre, dim, es);
      if constexpr (!LATE) greens(dre, dim, true);
    } else {
      if constexpr (LATE)
        if (green) greens(pdre, pdim, (pcode & SITE_LABEL) != 0);
      if (step) {
        if (fast) fast_steps(dre, dim, es);
        else general_steps(code & SITE_LABEL, dre, dim, es);
        if (!want_gt && !burn_in) store();
      }
      if constexpr (!LATE)
        if (green) greens(dre, dim, (code & SITE_LABEL) != 0);
    }
    if (step) {
      pcode = code;
      pdre = dre;
      pdim = dim;
      pes = es;
      if (want_gt) {
        if constexpr (PK) {
#pragma unroll
          for (int jp = 0; jp < RG::NV_GT; ++jp) {
            const float4 v = *unit(slot, RG::NV_REC + jp);
            gt2[jp] = Cx2{make_float2(v.x, v.y), make_float2(v.z, v.w)};
          }
        } else if constexpr (!RG::on) {
#pragma unroll
          for (int j = 0; j < EMAX; ++j) gt[j] = gt_nx[j];
          if (k + 1 < n_rows) load_gt();
        }
      }
      if constexpr (RG::on) slot = slot == (NS - 1) * STAGE ? 0 : slot + STAGE;
    }
  }
  if constexpr (RG::on) cp_async_wait<0>();
}

template <typename R, int EMAX, int MINB, bool KEL, int LG, bool PK>
__global__ void __launch_bounds__(128, MINB) k_sweep(const SweepArgs<R> A) {
  __shared__ double s_res2[128];  // twice the residues of this pass's energies, zero past the last
  for (int e = threadIdx.x; e < 128; e += blockDim.x) s_res2[e] = e < A.ne ? A.res2[e] : 0.0;
  __syncthreads();
  sweep_tile<R, EMAX, MINB, KEL, LG, PK>(A, s_res2, (blockIdx.x * blockDim.x + threadIdx.x) >> 5);
}

// The sweep of many grains in one persistent launch.  A work unit is one tile
// of trajectory columns (16 / G of them) of one grain; warps take units from a
// global counter, longest columns first (the unit list is sorted by the host),
// so ragged grains share the GPU without a tail per grain.  Each grain has its
// own G = 2^log_groups threads per column and function (the warp's unit belongs
// to one grain, so the mapping is uniform within a warp).
template <typename R, int EMAX, int MINB, bool PK>
__global__ void __launch_bounds__(128, MINB) k_sweep_batch(const SweepArgs<R> *__restrict__ args,
                                                           const int2 *__restrict__ units, int n_units,
                                                           int *counter) {
  const int lane = threadIdx.x & 31;
  for (;;) {
    int u = 0;
    if (lane == 0) u = atomicAdd(counter, 1);
    u = __shfl_sync(0xffffffffu, u, 0);
    if (u >= n_units) break;
    const int2 wu = units[u];
    const SweepArgs<R> &A = args[wu.x];
    sweep_tile<R, EMAX, MINB, false, -1, PK>(A, A.res2, wu.y);
    __syncwarp();
  }
}

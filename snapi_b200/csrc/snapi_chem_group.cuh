// snapi_chem_group.cuh -- the chemistry of the hydrostatic march solved by a group of eight lanes, its
// state in shared memory.  Included by snapi_eos.cu after Chem, whose results it reproduces bit for
// bit: every number is formed by the same operations in the same order, only on another lane.
//
// What bounds it: a march is one serial chain (ionisation sweep -> molecules -> Newton system -> update,
// 1 to 3 passes, inside the hydrostatic iterations of a depth, inside the walk over depths), FP64
// latency all along (8 cycles per dependent FMA, 137 per division, 171 per exp), and with one thread per
// march a batch of 61 pixels takes as long as one of a thousand.  Here the independent pieces of a pass
// go to the lanes of a group: the atoms of the ionisation sweep (host-made lists of equal cost), the
// exponentials of the temperature tables, the molecules, the columns of the reduced Newton system
// (electrons, hydrogen, the atoms in molecules and two right-hand sides: up to 8), the sums' chains.
// Four groups share a warp, in warp-uniform loops: a loop runs until no group of the warp needs it,
// finished groups masked.
//
// Measured (B200, one thread per march -> groups): spectra and gradient from node vectors of 61 pixels
// 25.4 -> 8.0 ms, of 4096 79.4 -> 75.6 (every march slot is taken either way); 1500 spectra from 85-node
// vectors 37.5 -> 13.3; a fit of 1000 pixels, 4 iterations, 200.8 -> 130.9, of 77 with differences 108.7 -> 40.3.
#pragma once

namespace snapi {
namespace {

constexpr int kGL = 8;           // lanes per group
constexpr int kGroupNR = kGL - 2;  // unknowns of the reduced Newton system at most (two right-hand sides)
constexpr unsigned kFull = 0xffffffffu;
constexpr size_t kGroupShared = 224 * 1024;  // shared memory of a CTA at most

// offsets (in doubles) of a group's arrays in its shared block, for one table set
struct GroupLayout {
  int sl;    // [nst] {Ut, cz}: see ChemT::SLoc
  int w2;    // [nt] the terms' weights
  int ik;    // [nmol] 1 / (K kT)
  int mcb;   // [nbf_m] edge factors of the march's opacity
  int mlf;   // [nlev_m] level factors of the march's opacity
  int N;     // [natom + 1] densities: electrons, free atoms
  int dn;    // [natom + 1] dN / dNt of the last solve
  int lx;    // [2][natom + 1] log(N / Nt) at the two latest temperatures
  // from here a new temperature overwrites what the last solve left (set_T's exponentials)
  int ex;    // [nc] the level sums' exponentials
  int ea;    // [natom + 1] {sum_z z f_z, its n_e derivative}
  int iN;    // [natom + 1] 1 / N
  int fr;    // [nref] {kept fraction, its n_e derivative}
  int dlf;   // [nref] d ln f / d n_e
  int mol;   // [nmol] {n, dn / dn_e} of the molecules
  int dd;    // [natom + 1] defects
  int xs;    // [2][NR] solutions: the Newton update, dN / dNt
  int lm;    // [nlev_m] level populations
  int total;
  int th[kGL + 1];  // the sweep's atoms by lane: [th[g], th[g + 1]) of at
  unsigned char at[kEA];
};

// NR: unknowns of the reduced Newton system (5 or 6; fewer are padded)
template <int NR>
struct GChem {
  const EosDev &E;
  const GroupLayout &L;
  double *S;  // the group's block
  int g;      // lane in the group
  // uniform over the group
  double T, kT, x5040, mstim, mhm, Nt_prev, lu_T, T1, T2;
  int have, lu_ok, nhist, capped;
  double last_gr;  // gr (ChemT) of this lane's unknown in the last Newton pass

  __device__ __forceinline__ GChem(const EosDev &e, const GroupLayout &l, double *s)
      : E(e), L(l), S(s), g(threadIdx.x & (kGL - 1)), T(-1.0), kT(0.0), x5040(0.0), mstim(0.0), mhm(0.0),
        Nt_prev(0.0), lu_T(0.0), T1(0.0), T2(0.0), have(0), lu_ok(0), nhist(0), capped(0), last_gr(0.0) {}

  __device__ __forceinline__ double2 *pair(int at) const { return reinterpret_cast<double2 *>(S + at); }
  __device__ __forceinline__ bool any(bool b) const {  // over the group
    return __ballot_sync(kFull, b) & 0xffu << (threadIdx.x & 31 & ~(kGL - 1));
  }

  // ---- what depends on T alone (ChemT::set_T and set_march) -----------------------------------------
  __device__ __forceinline__ void set_T(double Tin, bool act) {
    if (act) {
      T = Tin;
      kT = cK * T;
      const double x = 5040.0 / T;
      x5040 = x;
      for (int c = g; c < E.ncoef; c += kGL) S[L.ex + c] = exp(-2.302585 * E.cG[c] * x);
      for (int t = g; t < E.nterm; t += kGL) S[L.w2 + t] = E.g2[t] * exp(-2.302585 * E.tee[t] * x);
    }
    __syncwarp();
    if (act) {
      const double fct = 2.0 * pow((2.0 * cPI * cME * cK * T) / (cH * cH), 1.5);
      for (int s = g; s < E.nst; s += kGL) {
        const int ty = E.pft[s];
        double u = E.pfv[s];
        if (ty == SNAPI_PF_TRAV) {
          for (int t = E.t0[s]; t < E.t1[s]; ++t)
            for (int c = E.c0[t]; c < E.c1[t]; ++c) u += E.cA[c] * S[L.ex + c];
        } else if (ty == SNAPI_PF_IRWIN) {
          const double lnT = log(T);
          double sum = 0.0;
          for (int c = E.t0[s]; c < E.t1[s]; ++c) sum += E.cA[c] * pow(lnT, (double)(c - E.t0[s]));
          u = exp(sum);
        }
        pair(L.sl)[s] = make_double2(u, fct * exp(-E.eion[s] / kT));
      }
      for (int m = g; m < E.nmol; m += kGL) {
        double k = 0.0;
        if (E.meqc[m] == SNAPI_EQC_POLY) {
          const int n = E.mncoef[m];
          double sum = E.mcoef[m][n - 1];
          for (int i = n - 2; i >= 0; --i) sum = E.mcoef[m][i] + x5040 * sum;
          k = exp(2.302585093 * sum);
        } else if (E.meqc[m] == SNAPI_EQC_HMIN) {
          k = exp(2.302585093 * (0.1249 + (2.5 * log(T) / 2.302585) - 0.747 * x5040));
        } else if (E.meqc[m] == SNAPI_EQC_CONST) {
          k = E.mcoef[m][0];
        }
        S[L.ik + m] = 1.0 / (k * kT);
      }
      const double lambda = E.lambda_he;
      mstim = exp(-cH * cC / lambda / cK / T);
      for (int k = g; k < E.nbf_m; k += kGL) S[L.mcb + k] = march_edge(E, k, T);
      for (int k = g; k < E.nlev_m; k += kGL) S[L.mlf + k] = march_level(E, k, T);
      mhm = march_hminus(E, T, mstim);
    }
    __syncwarp();
  }

  // ---- ionisation sweep (ChemT::sweep_atom) -----------------------------------------------------------
  template <bool kDeriv>
  __device__ __forceinline__ void sweep_atom(int a, double ine, double pne, double ipne, double &Ea, double &Da) {
    const int s0 = E.s0[a], ns = E.ns[a], zk = E.zkeep[a];
    double2 *fr = pair(L.fr);
    int zend = ns;
    double h = 1.0, fsum = 0.0, S1 = 0.0, dfsum = 0.0, S2 = 0.0, dl0 = 0.0;
    for (int z = 0; z < ns; ++z) {
      const StageTab Q = E.stab[s0 + z];
      const double2 uc = pair(L.sl)[s0 + z];
      double U, dU;
      trav_u<kDeriv>(E, Q, uc.x, S + L.w2, x5040, ine, pne, ipne, U, dU);
      const double f = U * h;
      fsum += f;
      S1 += (double)z * f;
      double df = 0.0;
      if (kDeriv) {
        if (z == 0) dl0 = dU / U;
        else df = h * dU - f * (dl0 + (double)z * ine);
        dfsum += df;
        S2 += (double)z * df;
        if (Q.ref >= 0) fr[Q.ref] = make_double2(f, df);
      }
      h *= uc.y * ine;
      if (z + 1 >= zk && h < 1e-30 * fsum) {  // see ChemT::sweep_atom
        zend = z + 1;
        break;
      }
    }
    const double inv = 1.0 / fsum;
    Ea = S1 * inv;
    if (kDeriv) {
      Da = (S2 - dfsum * S1 * inv) * inv;
      for (int z = 0; z < zend; ++z) {
        const int r = E.stab[s0 + z].ref;
        if (r >= 0) {
          double2 v = fr[r];
          v.y = (v.y - dfsum * v.x * inv) * inv;
          v.x *= inv;
          fr[r] = v;
          if (E.stab[s0 + z].inmol) S[L.dlf + r] = v.y / v.x;
        }
      }
    }
  }

  // this lane's atoms at n_e = n into ea (and kDeriv: fr, dlf, iN)
  template <bool kDeriv>
  __device__ __forceinline__ void sweep(double n, bool act) {
    if (act) {
      const double ine = 1.0 / n, pne = cbrt(sqrt(n)), ipne = 1.0 / pne;
      for (int k = L.th[g]; k < L.th[g + 1]; ++k) {
        const int a = L.at[k];
        double2 v;
        sweep_atom<kDeriv>(a, ine, pne, ipne, v.x, v.y);
        pair(L.ea)[a + 1] = v;
        if (kDeriv && E.rmap[a + 1] >= 0) S[L.iN + a + 1] = 1.0 / S[L.N + a + 1];
      }
      if (kDeriv && g == 0) S[L.iN] = ine;
    }
    __syncwarp();
  }

  // ---- the reference's starting values (ChemT::cold_start) --------------------------------------------
  __device__ __forceinline__ void cold_start(double Nt, bool act) {
    const int na = E.natom;
    double *N = S + L.N;
    double F1 = 0.0, S1 = 0.0, n = 1.0, esum = 0.0;
    for (int a = 0; a < na; ++a) S1 += E.abund[a];
    const double S3 = S1;
    bool run = act;
    for (int pass = -2; __any_sync(kFull, run); ++pass) {
      sweep<false>(n, run);
      if (pass >= 0 && run)
        for (int a = 1 + g; a <= na; a += kGL) N[a] = (Nt - n) * E.abund[a - 1] / S3;
      __syncwarp();
      if (run) {
        if (pass < 0) {
          double F = 0.0;
          for (int a = 0; a < na; ++a) F += E.abund[a] * S[L.ea + 2 * (a + 1)];
          if (pass == -2) {
            F1 = F;
            n = Nt;
          } else {
            const double aa = F / (S3 * Nt);
            double bb = F1 / S1 - aa;
            const double cc = -bb * Nt;
            bb += 1.0 - aa * Nt;
            n = fmax((-bb + sqrt(bb * bb - 4.0 * aa * cc)) / (2.0 * aa), 1.0);
          }
        } else {
          esum = 0.0;
          for (int a = 1; a <= na; ++a) esum += S[L.ea + 2 * a] * N[a];
          n = 0.5 * (n + esum);
          if (pass + 1 >= kPolishCap) {
            capped = 1;
            run = false;
          } else if (!((1E-2 * (n + esum)) < fabs(n - esum))) {
            run = false;
          }
        }
      }
      __syncwarp();
    }
    if (act && g == 0) N[0] = n;
    __syncwarp();
  }

  // ---- Newton passes (ChemT::newton); groups without act are left alone --------------------------------
  __device__ __forceinline__ int newton(double Nt, int maxpass, bool bail, bool act) {
    const int na = E.natom, nr = E.nr, nm = E.nmol;
    int res = 0, iter = 0;
    double *N = S + L.N;
    const double2 *ea = pair(L.ea), *mol = pair(L.mol);
    const double abH = E.abund[0], iabH = 1.0 / abH;
    while (__any_sync(kFull, act)) {
      sweep<true>(act ? N[0] : 1.0, act);
      if (act) {
        for (int m = g; m < nm; m += kGL) {
          double nmv = S[L.ik + m], dm0 = 0.0;
          const int nc = E.mnc[m];
          for (int i = 0; i < nc; ++i) {
            const int a = E.matom[m][i];
            if (a == 0) {
              nmv *= N[0] * kT;
              dm0 += S[L.iN];
            } else {
              const int r = E.mref[m][i];
              nmv *= S[L.fr + 2 * r] * N[a] * kT;
              dm0 += S[L.dlf + r];
            }
          }
          dm0 *= nmv;
          pair(L.mol)[m] = make_double2(nmv, dm0);
        }
      }
      __syncwarp();
      // lane k: column k of the system (0 electrons, 1 hydrogen, ..); lane NR the defects, NR + 1 e_1
      // (dN / dNt); padding and groups without act: identity columns
      const int k = g;
      const bool colk = act && k < nr, rhs = act && g == NR;
      double col[NR], grk = 0.0, Nr = 0.0;
#pragma unroll
      for (int r = 0; r < NR; ++r) col[r] = r == g ? 1.0 : 0.0;
      if (colk || rhs) {
        // rows 0 / 1 from the atoms, then the molecules in their order
        double s0, s1;
        if (rhs) {
          s0 = -N[0];
          s1 = N[0] - Nt;
          for (int a = 1; a <= na; ++a) {
            s0 += N[a] * ea[a].x;
            s1 += N[a];
          }
          Nr = N[1];
        } else if (k == 0) {
          s0 = -1.0;
          s1 = 1.0;
          for (int a = 1; a <= na; ++a) s0 += N[a] * ea[a].y;
        } else {
          s0 = ea[E.rfull[k]].x;
          s1 = 1.0;
        }
#pragma unroll
        for (int r = 2; r < NR; ++r) col[r] = r >= nr ? 0.0 : (rhs ? N[E.rfull[r]] : (r == k ? -abH : 0.0));
        const int own = k > 0 && k < nr ? k : 0;
        const double ink = own ? S[L.iN + E.rfull[own]] : 0.0;
#pragma unroll 2
        for (int m = 0; m < nm; ++m) {
          const double2 n = mol[m];
          const double *mu = E.mrow[m];  // charge, counts of the reduced unknowns 1 ..
          const double q = mu[0], hm = mu[1];
          if (rhs) {
            s0 += q * n.x;
            s1 += n.x;
            Nr += n.x * hm;
#pragma unroll
            for (int r = 2; r < NR; ++r) col[r] += n.x * mu[r];
          } else {
            const double d = own ? n.x * mu[own] * ink : n.y;
            s0 += q * d;
            s1 += d;
            grk += hm * d;
#pragma unroll
            for (int r = 2; r < NR; ++r) col[r] -= abH * mu[r] * d;
          }
        }
        col[0] = s0;
        col[1] = s1;
      }
      Nr = __shfl_sync(kFull, Nr, NR, kGL);
      // the defects of the rows >= 2, the eliminated atoms' sums
      double c0 = 0.0, c1 = 0.0, e0 = 0.0, e1 = 0.0;
      if (rhs) {
        S[L.dd] = col[0];
        S[L.dd + 1] = col[1];
#pragma unroll
        for (int r = 2; r < NR; ++r)
          if (r < nr) {
            const double nc = col[r];
            col[r] = E.abund[E.rfull[r] - 1] * Nr - abH * nc;
            S[L.dd + E.rfull[r]] = col[r];
          }
      }
      if (act) {
        for (int q = 0; q < E.nsimple; ++q) {
          const int sa = E.simple[q];
          const double as = E.abund[sa - 1] * iabH, nc = N[sa], Es = ea[sa].x;
          const double d = E.abund[sa - 1] * Nr - abH * nc;
          c0 += Es * as;
          c1 += as;
          e0 += Es * d * iabH;
          e1 += d * iabH;
          if (g == 0) S[L.dd + sa] = d;
        }
      }
      if (rhs) {
        col[0] += e0;
        col[1] += e1;
      } else if (colk) {
#pragma unroll
        for (int r = 2; r < NR; ++r)
          if (r < nr) {
            const double ab = E.abund[E.rfull[r] - 1];
            col[r] += ab * grk;
            if (k == 1) col[r] += ab;
          }
        col[0] += c0 * grk;
        col[1] += c1 * grk;
        if (k == 1) {
          col[0] += c0;
          col[1] += c1;
        }
      } else if (act && g == NR + 1) {
#pragma unroll
        for (int r = 0; r < NR; ++r) col[r] = r == 1 ? 1.0 : 0.0;
      }
      // Gaussian elimination with partial pivoting, columns in the lanes: the owner of column c picks
      // the pivot, the others follow its swap and multipliers
      double piv = 1.0;  // this column's pivot
#pragma unroll
      for (int c = 0; c < NR; ++c) {
        int p = c;
        double best = fabs(col[c]);
#pragma unroll
        for (int r = c + 1; r < NR; ++r) {
          const double t = fabs(col[r]);
          if (t > best) { best = t; p = r; }
        }
        p = __shfl_sync(kFull, p, c, kGL);
#pragma unroll
        for (int r = c + 1; r < NR; ++r)
          if (p == r) { const double t = col[c]; col[c] = col[r]; col[r] = t; }
        const double pc = __shfl_sync(kFull, col[c], c, kGL), ipv = 1.0 / pc;
        if (g == c) piv = pc;
#pragma unroll
        for (int r = c + 1; r < NR; ++r) {
          const double f = __shfl_sync(kFull, col[r], c, kGL) * ipv;
          if (g > c) col[r] -= f * col[c];
        }
      }
      // back substitution of both right-hand sides at once (lanes NR, NR + 1)
#pragma unroll
      for (int r = NR - 1; r >= 0; --r) {
        double sum = col[r];
#pragma unroll
        for (int j = r + 1; j < NR; ++j) sum -= __shfl_sync(kFull, col[r], j, kGL) * col[j];
        const double x = sum / __shfl_sync(kFull, piv, r, kGL);
        if (g >= NR) col[r] = x;
      }
      if (act && g >= NR && g < NR + 2) {
#pragma unroll
        for (int r = 0; r < NR; ++r) S[L.xs + (g - NR) * NR + r] = col[r];
      }
      __syncwarp();
      // u = w_1 + gr . w in the unknowns' order, then every density's update
      const double *xs = S + L.xs;
      double u = act ? xs[1] : 0.0;
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const double gr = __shfl_sync(kFull, grk, r, kGL);
        if (act && r < nr) u += gr * xs[r];
      }
      bool bad = false, inf = false;
      if (act) {
        for (int a = g; a <= na; a += kGL) {
          const int r = E.rmap[a];
          const double d = S[L.dd + a];
          const double v = r >= 0 ? xs[r] : __dmul_rn(E.abund[a - 1] * u - d, iabH);
          double n = N[a] - v;
          if (n < 1E-2) n = 1E-2;
          N[a] = n;
          inf |= !isfinite(n);
          bad |= fabs(d / n) > 1E-4;
        }
      }
      const bool anybad = any(bad), anyinf = any(inf);
      if (act) {
        iter += 2;  // the reference counts two per pass (atmos_chm.cc:294, 300)
        if (bail && anyinf) { res = -1; act = false; }
        else if (iter > 2 * maxpass) { res = 0; act = false; }
        else if (!anybad) { res = 1; act = false; }
        if (!act) last_gr = grk;
      }
      __syncwarp();
    }
    return res;
  }

  // ---- the continued start (ChemT::predict, finish) ----------------------------------------------------
  // a new temperature: log(N / Nt) of the last solution joins the history (act: groups that had one)
  __device__ __forceinline__ void history(bool act) {
    if (act) {
      const int na = E.natom;
      double *l1 = S + L.lx, *l2 = l1 + na + 1;
      for (int a = g; a <= na; a += kGL) {
        l2[a] = l1[a];
        l1[a] = log(S[L.N + a] / Nt_prev);
      }
      T2 = T1;
      T1 = lu_T;
      if (nhist < 2) ++nhist;
    }
  }

  // after a solve: dN / dNt from the e_1 column
  __device__ __forceinline__ void finish(double Nt, bool act) {
    const int nr = E.nr;
    const double *xp = S + L.xs + NR;
    double u = act ? xp[1] : 0.0;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const double gr = __shfl_sync(kFull, last_gr, r, kGL);
      if (act && r < nr) u += gr * xp[r];
    }
    if (act) {
      have = 1;
      Nt_prev = Nt;
      lu_ok = 1;
      lu_T = T;
      const double iabH = 1.0 / E.abund[0];
      for (int a = g; a <= E.natom; a += kGL) {
        const int r = E.rmap[a];
        S[L.dn + a] = r >= 0 ? xp[r] : E.abund[a - 1] * u * iabH;
      }
    }
    __syncwarp();
  }

  __device__ __forceinline__ void predict(double Nt, bool act) {
    const int na = E.natom;
    const bool same = lu_ok && T == lu_T, extra = !same && nhist == 2;
    double r = T1 != T2 ? (T - T1) / (T1 - T2) : 1.0;
    r = fmin(fmax(r, 0.0), 2.0);
    const double dNt = Nt - Nt_prev, sc = Nt / Nt_prev;
    const double *l1 = S + L.lx, *l2 = l1 + na + 1;
    constexpr int kOwn = (kEA + kGL) / kGL;
    double x[kOwn];
    bool bad = false;
#pragma unroll
    for (int q = 0; q < kOwn; ++q) {
      const int a = g + q * kGL;
      x[q] = 1.0;
      if (act && a <= na) {
        const double n = S[L.N + a];
        x[q] = same ? n + S[L.dn + a] * dNt : (extra ? Nt * exp(l1[a] + (l1[a] - l2[a]) * r) : n * sc);
        bad |= !(x[q] >= 1E-2) || !isfinite(x[q]);
      }
    }
    const bool scale = any(bad) && (same || extra);
    if (act) {
#pragma unroll
      for (int q = 0; q < kOwn; ++q) {
        const int a = g + q * kGL;
        if (a <= na) S[L.N + a] = scale ? S[L.N + a] * sc : x[q];
      }
    }
    __syncwarp();
  }

  __device__ __forceinline__ void solve(double Nt, bool warm, bool act) {
    if (act) capped = 0;
    bool need = act;
#pragma unroll 1
    for (int start = warm ? 0 : 1; start < 2; ++start) {  // 0: the predicted iterate, 1: the cold start
      const bool a = need && (start || have);
      if (!__any_sync(kFull, a)) continue;
      if (start) cold_start(Nt, a);
      else predict(Nt, a);
      const int r = newton(Nt, start ? 50 : Chem::kWarmPasses, !start, a);
      if (a) {
        if (r == 1) need = false;
        else if (start) capped = 1;
      }
    }
    if (warm) finish(Nt, act);
  }

  __device__ __forceinline__ double stage_total(int s) const {
    return S[L.N + E.satom[s] + 1] * S[L.fr + 2 * E.ref[s]];
  }

  // chemistry and opacity at lambda_he (chem_point's compact path)
  __device__ __forceinline__ double march_point(double Tin, double Nt, bool warm, bool act) {
    const bool newT = act && Tin != T;
    if (__any_sync(kFull, newT)) {
      if (warm) history(newT && have && Tin != lu_T);
      set_T(Tin, newT);
    }
    solve(Nt, warm, act);
    const double ne = act ? S[L.N] : 1.0;
    double *lm = S + L.lm;
    if (act) {
      const double pne = cbrt(sqrt(ne)), ine = 1.0 / ne, ipne = 1.0 / pne;
      for (int k = g; k < E.nlev_m; k += kGL) {
        const int l = E.lev_m[k], st = E.lst[l];
        double U, dU;
        trav_u<false>(E, E.stab[st], pair(L.sl)[st].x, S + L.w2, x5040, ine, pne, ipne, U, dU);
        const double tot = stage_total(st);
        lm[k] = E.lg[l] != 0.0 ? tot * (S[L.mlf + k] / U) : tot;
      }
    }
    __syncwarp();
    if (!act) return 0.0;
    const double nH0 = stage_total(E.s0[0]);
    double op = 6.65E-25 * ne;
    for (int k = 0; k < E.nbf_m; ++k)
      op += E.sig_he[E.bf_m[k]] * (lm[E.bfl_m[k]] - lm[E.bfn_m[k]] * ne * S[L.mcb + k] * mstim);
    return op + mhm * ne * nH0;
  }

  // the march's state between depth segments: the predictors (kWords(natom) words per march)
  static __host__ __device__ __forceinline__ int words(int natom) { return 4 * (natom + 1) + 5; }
  __device__ __forceinline__ void save(double *s) const {
    const int n = E.natom + 1;
    for (int a = g; a < n; a += kGL) {
      s[a] = S[L.N + a];
      s[n + a] = S[L.dn + a];
      s[2 * n + a] = S[L.lx + a];
      s[3 * n + a] = S[L.lx + n + a];
    }
    if (g == 0) {
      double *q = s + 4 * n;
      q[0] = Nt_prev;
      q[1] = lu_T;
      q[2] = T1;
      q[3] = T2;
      q[4] = (double)(have | lu_ok << 1 | nhist << 2);
    }
  }
  __device__ __forceinline__ void load(const double *s) {
    const int n = E.natom + 1;
    for (int a = g; a < n; a += kGL) {
      S[L.N + a] = s[a];
      S[L.dn + a] = s[n + a];
      S[L.lx + a] = s[2 * n + a];
      S[L.lx + n + a] = s[3 * n + a];
    }
    const double *q = s + 4 * n;
    Nt_prev = q[0];
    lu_T = q[1];
    T1 = q[2];
    T2 = q[3];
    const int f = (int)q[4];
    have = f & 1;
    lu_ok = f >> 1 & 1;
    nhist = f >> 2;
  }
};

}  // namespace
}  // namespace snapi

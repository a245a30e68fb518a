// snapi_ali.cu -- NLTE level populations by accelerated lambda iteration for many 1-D columns
// (atmosphere::nltepops, atmos/atmos_pop.cc:67-240), one NLTE atom.
//
// The profiles do not depend on the populations, so they are formed once per call; an iteration reads
// them back.  Per batch of columns, once:
//   k_ali_tables  CTA = (column, ray, depth), thread = wavelength: the W4 profile of every bound-bound
//                 transition (FP32), and per (depth, wavelength) the bound-free factors of the temperature.
//   k_ali_turn    the background's arrays turned wavelength-fastest.
// Per iteration:
//   k_ali_formal  CTA = (column, ray, 128 wavelengths), thread = wavelength: background + active
//                 opacity / emissivity at every depth (bound-bound from the stored profiles, bound-free
//                 with the LTE-ratio correction), scalar formal solution along the ray with the diagonal
//                 operator (atmos_ppbez_rts.cc:21-219); writes I, Lambda* and 1 / total opacity.  Opacity
//                 sums, optical depths and the recursion in FP64: the NLTE grid's background spans
//                 1e-13 .. 1e32 cm^-1 (1e45 after normalisation by kappa_500, beyond FP32) and the rates
//                 use J - Lambda* S, which cancels in optically thick line cores.
//   k_ali_sums    thread = (column, depth, two transitions, wavelength slice): the profile-weighted mean
//                 intensities and operators of the transitions (atom::add, atom.cc:1865-1927) in FP64.
//   k_ali_solve   CTA = column, thread = depth: the rate equations (atom::newpops, atom_pop.cc:27-145)
//                 in FP64 with the most populated level replaced by conservation, an LU solve, the
//                 relative change; negative populations anywhere in the column -> the same step without
//                 the operator; the column stops when the maximum relative change falls below tol.
//
// The iteration multiplies a rounding difference by 30 to 300 a step until it meets the FP32 factors of the
// lines (last bits after two steps, 1e-5 after three), so every kernel keeps the order of additions of one
// sequential pass per (depth, slice): the split into kernels, batches and threads moves no bit.
//
// Bounds and measurements (B200, Ca II, 10 lines, 444 wavelengths).  With the profiles evaluated twice an
// iteration and the sums in one CTA per column, 40 running sums a thread, an iteration of 512 columns x 2 rays
// x 80 depths took 2.4 ms (formal) + 2.9 (rates), of 40 columns x 10 rays x 100 depths 1.7 + 6.4 (40 CTAs on
// 148 SMs); now 1.16 + 0.69 + 0.08 and 0.58 + 0.42 + 0.06, after 1.2 and 0.55 ms once per call.  To
// convergence 97.4 -> 33.5 ms and 410 -> 51.2 ms, the set-up included.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "snapi_internal.cuh"

using namespace snapi;

namespace {

constexpr int kAliChunk = 128;
constexpr size_t kAliWork = (size_t)24 << 30;  // work buffers of a batch of columns [bytes]
constexpr int kAliMaxLev = 16, kAliMaxLine = 32, kAliMaxBf = 16;
constexpr double kHc = kH * kC;
constexpr double kPi4 = 4.0 * kPi;
constexpr double kInvPi4 = 1.0 / kPi4, kInvHc = 1.0 / kHc;

struct AliDev {
  int ncol, nd, nl, nray, nlev, nline, nbf, nchunk;
  // a depth's sums run in nsl slices of wavelengths (l % nsl: a power of two <= 4) that meet by shuffles; the
  // work arrays hold the wavelengths by slot (slot_of), nls of them, the last ones perhaps empty
  int nsl, nls;
  double tol;
  int max_iter;
  // problem
  const double *lambda, *lw, *p5;               // [nls], by slot (empty ones 1, 0, 0); p5 = 1 / lambda^5
  const double *ray_ct, *ray_w;                 // [nray]
  const double *geo;                            // [nray][nd][3]: the interval entered from depth z, a third, opd weight
  const double *lam0, *Aul, *Blu, *Bul, *Eline; // [nline]
  const int *line_lo, *line_up;                 // [nline]
  const int *bf_lo, *bf_up;                     // [nbf]
  const float *sigma;                           // [nbf][nls], by slot
  const double *sgf;                            // sigma x fudge
  const double *A, *B;                          // [nlev][nlev]
  const int *stage, *cont_of, *tmap, *bf_of;    // [nlev], [nlev], [nlev][nlev], [nlev]
  // columns
  const double *T, *ne, *na, *kap, *vray, *dld, *adamp, *bfratio, *coll;
  const double *bgop, *bgem;
  double *pops;                                 // [ncol][nd][nlev]
  // once per call: profiles [ncol][nray][nd][nline][nls]; exp(-hc / lambda k T) and the Planck function of the
  // formal solution's FP32 temperatures, exp(-hc / lambda k T) of the rates', [ncol][nd][nls]
  float *phi;
  double *eb, *pl, *ex;
  double *ik;                                   // 1 / normalising opacity (rounded to FP32), [ncol][nd]
  double2 *fac;                                 // of the current populations (factor), [ncol][nd][nline + nbf]
  double *bo, *be;                              // the background wavelength-fastest, [ncol][nray][nd][nls]
  double *I, *L, *iop;                          // [ncol][nray][nd][nls]: I, Lambda*, 1 / total opacity
  double *sums;                                 // [ncol][3 nline + 2 nbf][nd]: norm, J, Lambda* by line; up, down by bf
  int *state, *iters;                           // [ncol]: state 0 running, 1 converged, 2 max_iter, -1 negative
  double *rel;                                  // [ncol]
};

// Slot of wavelength l: the slices' wavelengths four and four together, so that one thread of k_ali_sums reads
// four consecutive ones of its slice by one or two 16-byte loads; l back from the slot.
__host__ __device__ inline int slot_of(int l, int nsl) { return l / (4 * nsl) * (4 * nsl) + l % nsl * 4 + l / nsl % 4; }
__host__ __device__ inline int lambda_of(int s, int nsl) { return s / (4 * nsl) * (4 * nsl) + s % 4 * nsl + s / 4 % nsl; }

// The factor of transition k of a depth in the opacity and emissivity, from its populations n: {opacity,
// emissivity} of a line, rounded to FP32 as the profiles are; {lower population, upper x LTE ratio} of a
// bound-free transition (k from nline on).
__device__ __forceinline__ double2 factor(const AliDev &D, int col, int z, int k, const double *n) {
  if (k < D.nline)
    return make_double2((double)(float)(n[D.line_lo[k]] * D.Blu[k] - n[D.line_up[k]] * D.Bul[k]),
                        (double)(float)(n[D.line_up[k]] * D.Aul[k]));
  const int b = k - D.nline;
  return make_double2(n[D.bf_lo[b]], n[D.bf_up[b]] * D.bfratio[((size_t)col * D.nbf + b) * D.nd + z]);
}

// the profiles and temperature factors, once per call
constexpr int kTabThreads = 128;
__global__ void __launch_bounds__(kTabThreads) k_ali_tables(AliDev D) {
  __shared__ float iv[kAliMaxLine], ad[kAliMaxLine];
  const int z = blockIdx.x % D.nd, ray = (blockIdx.x / D.nd) % D.nray, col = blockIdx.x / (D.nd * D.nray);
  const int nd = D.nd, nl = D.nls;
  if ((int)threadIdx.x < D.nline) {
    const size_t at = ((size_t)col * D.nline + threadIdx.x) * nd + z;
    iv[threadIdx.x] = (float)(1.0 / D.dld[at]);
    ad[threadIdx.x] = (float)D.adamp[at];
  }
  __syncthreads();
  const float vr = (float)(D.vray[((size_t)col * D.nray + ray) * nd + z] / kC);
  const double T = D.T[(size_t)col * nd + z], Tf = (double)(float)T, hckT = kHc / (kK * T);
  if (ray == 0) {
    const size_t row = (size_t)col * nd + z;
    if (threadIdx.x == 0) D.ik[row] = 1.0 / (double)(float)D.kap[row];
    if ((int)threadIdx.x < D.nline + D.nbf)
      D.fac[row * (D.nline + D.nbf) + threadIdx.x] = factor(D, col, z, threadIdx.x, D.pops + row * D.nlev);
  }
  float *ph = D.phi + (size_t)blockIdx.x * D.nline * nl;
  for (int l = threadIdx.x; l < nl; l += kTabThreads) {
    if (lambda_of(l, D.nsl) >= D.nl) {  // an empty slot adds zeros to the sums
      for (int k = 0; k < D.nline; ++k) ph[(size_t)k * nl + l] = 0.f;
      D.I[(size_t)blockIdx.x * nl + l] = D.L[(size_t)blockIdx.x * nl + l] = D.iop[(size_t)blockIdx.x * nl + l] = 0.0;
      if (ray == 0 && D.nbf) D.ex[((size_t)col * nd + z) * nl + l] = 0.0;
      continue;
    }
    const double lam = D.lambda[l];
    const float lamf = (float)lam;
    for (int k = 0; k < D.nline; ++k) {
      float H, F;
      voigt(((float)(D.lam0[k] - lam) - lamf * vr) * iv[k], ad[k], H, F);
      ph[(size_t)k * nl + l] = H * iv[k];
    }
    if (ray == 0 && D.nbf) {
      const size_t at = ((size_t)col * nd + z) * nl + l;
      const double xpl = kHc / (lam * kK), pl5 = 2.0 * kHc * kC / (lam * lam * lam * lam * lam);
      const double x = xpl / Tf, il = 1.0 / lam;
      D.eb[at] = exp(-x);
      D.pl[at] = pl5 / (exp(x) - 1.0);
      D.ex[at] = exp(-hckT * il);
    }
  }
}

// the background's layout turned wavelength-fastest, once per call: CTA = (column, ray, 32 wavelengths, 32
// depths), a tile through shared memory
__global__ void __launch_bounds__(256) k_ali_turn(AliDev D) {
  __shared__ double to[32][33], te[32][33];
  const int nd = D.nd, nl = D.nl, nzt = (nd + 31) / 32, nlt = (nl + 31) / 32;
  const int zt = blockIdx.x % nzt, lt = (blockIdx.x / nzt) % nlt;
  const size_t cr = blockIdx.x / (nzt * nlt);
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int q = ty; q < 32; q += 8) {
    const int l = lt * 32 + q, z = zt * 32 + tx;
    if (l < nl && z < nd) {
      to[q][tx] = D.bgop[(cr * nl + l) * nd + z];
      te[q][tx] = D.bgem[(cr * nl + l) * nd + z];
    }
  }
  __syncthreads();
  for (int q = ty; q < 32; q += 8) {
    const int s = lt * 32 + tx, l = lambda_of(s, D.nsl), z = zt * 32 + q;  // a tile holds whole groups of slots
    if (l < nl && z < nd) {
      D.bo[(cr * nd + z) * D.nls + s] = to[l - lt * 32][q];
      D.be[(cr * nd + z) * D.nls + s] = te[l - lt * 32][q];
    }
  }
}

// Bound by the latency of its loads (59 % of the stalls; 29 % of DRAM's rate, FP64 pipe 21 %): 96 bytes a
// (wavelength, depth), 0.54 ms at the copy rate for the 1.16 it takes.  The lines' loop is unrolled by ten so that
// a cell's loads leave together (ten rays: 0.73 -> 0.58 ms against five), and six CTAs of 128 an SM leave the
// registers for it; 64 threads doubled the factors' copies (+10 to 25 %), prefetches to L2 only cost issue
// slots (+4 to 15 %), factors read through L1 instead of shared memory +47 %.
__global__ void __launch_bounds__(kAliChunk, 6) k_ali_formal(AliDev D) {
  extern __shared__ __align__(16) double2 s_fac[];  // [nd][nline + nbf] factors, [nd] 1 / normalising opacity
  const int chunk = blockIdx.x % D.nchunk;
  const int ray = (blockIdx.x / D.nchunk) % D.nray;
  const int col = blockIdx.x / (D.nchunk * D.nray);
  if (D.state[col] != 0) return;  // CTA-uniform
  const int nd = D.nd, nl = D.nls, nline = D.nline, nbf = D.nbf;
  const int nt = nline + nbf;
  double *ik = reinterpret_cast<double *>(s_fac + nd * nt);
  {
    const double2 *fac = D.fac + (size_t)col * nd * nt;
#pragma unroll 4
    for (int i = threadIdx.x; i < nd * nt; i += kAliChunk) s_fac[i] = fac[i];
    for (int z = threadIdx.x; z < nd; z += kAliChunk) ik[z] = D.ik[(size_t)col * nd + z];
  }
  __syncthreads();
  const int l = chunk * kAliChunk + threadIdx.x;  // slot
  if (l >= nl || lambda_of(l, D.nsl) >= D.nl) return;  // no barrier below
  const double lam = D.lambda[l];
  const double hc4pl = kHc / (kPi4 * lam);
  const size_t cr = (size_t)col * D.nray + ray;
  const double *bo = D.bo + cr * nd * nl + l, *be = D.be + cr * nd * nl + l;
  const float *ph = D.phi + cr * nd * nline * nl + l;
  const double *ebp = D.eb + (size_t)col * nd * nl + l, *plp = D.pl + (size_t)col * nd * nl + l;
  const double *sg = D.sgf + l, *geo = D.geo + (size_t)ray * nd * 3;
  auto cell = [&](int z, double &oo, double &ee, double &op) {
    double o = bo[(size_t)z * nl], e = be[(size_t)z * nl];
    const float *p = ph + (size_t)z * nline * nl;
    const double2 *fz = s_fac + z * nt;
#pragma unroll 10
    for (int k = 0; k < nline; ++k) {
      const double phi = (double)p[(size_t)k * nl] * hc4pl;
      const double2 q = fz[k];
      o += phi * q.x;
      e += phi * q.y;
    }
    if (nbf) {
      const double eb = ebp[(size_t)z * nl], pl = plp[(size_t)z * nl];
#pragma unroll 10
      for (int b = 0; b < nbf; ++b) {
        const double2 q = fz[nline + b];
        const double sb = sg[(size_t)b * nl];
        o += sb * (q.x - q.y * eb);
        e += sb * q.y * (1.0 - eb) * pl;
      }
    }
    op = o;
    oo = o * ik[z];
    ee = e * ik[z];
  };
  double *Io = D.I + cr * nd * nl + l, *Lo = D.L + cr * nd * nl + l, *Oo = D.iop + cr * nd * nl + l;
  auto put = [&](int z, double I, double La, double op) {
    const size_t at = (size_t)z * nl;
    Io[at] = I;
    Lo[at] = La;
    Oo[at] = 1.0 / op;
  };
  const double ct = D.ray_ct[ray];
  const int dz = ct > 0.0 ? 1 : -1, zl = ct > 0.0 ? 0 : nd - 1, zh = ct > 0.0 ? nd - 1 : 0;
  // window: p (z - dz), c (z), n (z + dz); each cell's source function and each interval's slope once
  double oop, eep, opp_, ooc, eec, opc, oon = 0.0, een = 0.0, opn = 0.0;
  cell(zl, oop, eep, opp_);
  cell(zl + dz, ooc, eec, opc);
  double sp = eep / oop, sc = eec / ooc, sn = 0.0;
  double hz = geo[3 * zl], h3 = geo[3 * zl + 1], d1 = (ooc - oop) / hz, d2 = 0.0;
  double dprev = d1;
  double I = ct > 0.0 ? 0.0 : sp;
  put(zl, I, ct > 0.0 ? 0.0 : 1.0, opp_);
  for (int z = zl + dz;; z += dz) {
    double dcur;
    if (z == zh) {
      dcur = d1;
    } else {
      cell(z + dz, oon, een, opn);
      sn = een / oon;
      // opd_interior of the three cells, its lengths' quotients from the table
      d2 = (oon - ooc) / geo[3 * z];
      const double alpha = geo[3 * z + 2];
      dcur = d1 * d2 > 0 ? d1 * d2 / (alpha * d1 + (1.0 - alpha) * d2) : 0.0;
    }
    // bezier_dtau(oop, ooc, dprev, dcur, hz)
    const double C0 = ooc - hz / 2.0 * dcur, C1 = oop + hz / 2.0 * dprev, C = 0.5 * (C0 + C1);
    const double tb = h3 * (oop + ooc + C);
    // linear weights with the Taylor branch below 1e-2 (atmos_ppbez_rts.cc:1070-1096 scalar form)
    double w0, w1, etb;
    if (tb < 1e-2) {
      etb = 1.0 - tb + tb * tb * 0.5 - tb * tb * tb / 6.0;
      w0 = tb * (0.5 - tb * (1.0 / 3.0 - tb / 8.0));
      w1 = 0.5 * tb * (1.0 - tb / 3.0 * (1.0 - tb / 4.0));
    } else {
      etb = exp(-tb);
      const double itb = 1.0 / tb;
      w0 = itb - etb * (1.0 + itb);
      w1 = 1.0 - itb + etb * itb;
    }
    I = I * etb + w0 * sp + w1 * sc;
    put(z, I, w1, opc);
    if (z == zh) break;
    oop = ooc; opp_ = opc; sp = sc;
    ooc = oon; opc = opn; sc = sn;
    hz = geo[3 * z]; h3 = geo[3 * z + 1];
    d1 = d2;
    dprev = dcur;
  }
}

// The slices of a (depth, transition pair) are adjacent lanes; a lane takes its slice's wavelengths in order,
// four by 16-byte loads (slot_of), and the slices meet by shuffles.  Slices: four where depths are few, two above
// 256, one above 512 (each column has depths to keep the chip busy then).  One wavelength a load instead took
// 1.46 ms (26 L1 tags a warp step) against 0.69; two lines a thread share I, Lambda* and the opacity.  L1
// throughput 72 %, DRAM 45 %: the profiles, 40 of 64 bytes a (wavelength, depth), are read once.
// kNorm: and the profiles' norms, which no iteration changes.
constexpr int kSumThreads = 64;
__device__ __forceinline__ void four(const double *p, double *v) {
  const double2 a = *reinterpret_cast<const double2 *>(p), b = *reinterpret_cast<const double2 *>(p + 2);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void four(const float *p, float *v) {
  const float4 a = *reinterpret_cast<const float4 *>(p);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
template <bool kNorm>
__global__ void __launch_bounds__(kSumThreads, 16) k_ali_sums(AliDev D, int nblk_line, int nblk) {
  const int col = blockIdx.x / nblk, blk = blockIdx.x % nblk;
  if (D.state[col] != 0) return;  // CTA-uniform
  const int nd = D.nd, nl = D.nls, nline = D.nline, nbf = D.nbf, nsl = D.nsl, sl = threadIdx.x % nsl;
  double *out = D.sums + (size_t)col * (3 * nline + 2 * nbf) * nd;
  const bool line = blk < nblk_line;
  const int nt = line ? nline : nbf, nq = (nt + 1) / 2;
  const int item = ((line ? blk : blk - nblk_line) * kSumThreads + (int)threadIdx.x) / nsl;
  const bool valid = item < nd * nq;  // of all the lanes of a depth at once; no lane leaves before the shuffles
  const int z = valid ? item / nq : 0, q = valid ? item % nq : 0;
  const size_t cell0 = (size_t)col * D.nray * nd + z;
  // a, b: J and Lambda* of a line (up and down of a bound-free transition), c its norm; the two transitions
  // of a thread share the reads of I, Lambda* and the opacity
  double a0 = 0.0, b0 = 0.0, c0 = 0.0, a1 = 0.0, b1 = 0.0, c1 = 0.0;
  const int k0 = 2 * q, k1 = min(k0 + 1, nt - 1);
  if (line && valid) {
    const double *n = D.pops + ((size_t)col * nd + z) * D.nlev;
    auto fac = [&](int k) { return (n[D.line_lo[k]] * D.Blu[k] - n[D.line_up[k]] * D.Bul[k]) * D.Eline[k] / kPi4; };
    const double lf0 = fac(k0), lf1 = fac(k1);
    for (int r = 0; r < D.nray; ++r) {
      const size_t cell = cell0 + (size_t)r * nd;
      const float *p0 = D.phi + (cell * nline + k0) * nl, *p1 = D.phi + (cell * nline + k1) * nl;
      const double *pI = D.I + cell * nl, *pL = D.L + cell * nl, *pO = D.iop + cell * nl;
      const double wr = D.ray_w[r];
      for (int l = 4 * sl; l < nl; l += 4 * nsl) {
        double I4[4], L4[4], O4[4], w4[4];
        float f0[4], f1[4];
        four(pI + l, I4); four(pL + l, L4); four(pO + l, O4); four(D.lw + l, w4);
        four(p0 + l, f0); four(p1 + l, f1);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double I = I4[j], Ls = L4[j], iop = O4[j], w = w4[j] * wr, wq = w * kInvPi4;
          {
            const double phi = (double)f0[j], wp = wq * phi, lf = lf0 * phi * iop;
            if (kNorm) c0 += wp;
            a0 += wp * I * lf;
            b0 += wp * Ls * lf;
          }
          {
            const double phi = (double)f1[j], wp = wq * phi, lf = lf1 * phi * iop;
            if (kNorm) c1 += wp;
            a1 += wp * I * lf;
            b1 += wp * Ls * lf;
          }
        }
      }
    }
  } else if (valid) {
    const float *s0 = D.sigma + (size_t)k0 * nl, *s1 = D.sigma + (size_t)k1 * nl;
    const double *ex = D.ex + ((size_t)col * nd + z) * nl;
    for (int r = 0; r < D.nray; ++r) {
      const double *pI = D.I + (cell0 + (size_t)r * nd) * nl;
      const double wr = D.ray_w[r];
      for (int l = 4 * sl; l < nl; l += 4 * nsl) {
        double I4[4], e4[4], w4[4], lam4[4], p4[4];
        float f0[4], f1[4];
        four(pI + l, I4); four(ex + l, e4); four(D.lw + l, w4); four(D.lambda + l, lam4); four(D.p5 + l, p4);
        four(s0 + l, f0); four(s1 + l, f1);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double I = I4[j], e = e4[j], w = w4[j] * wr, wl = w * lam4[j] * kInvHc, Ip = fma(2.0 * kHc * kC, p4[j], I);
          const double sa = wl * (double)f0[j], sb = wl * (double)f1[j];
          a0 += sa * I;
          b0 += sa * Ip * e;
          a1 += sb * I;
          b1 += sb * Ip * e;
        }
      }
    }
  }
  for (int off = 1; off < nsl; off <<= 1) {
    a0 += __shfl_xor_sync(0xffffffffu, a0, off);
    b0 += __shfl_xor_sync(0xffffffffu, b0, off);
    a1 += __shfl_xor_sync(0xffffffffu, a1, off);
    b1 += __shfl_xor_sync(0xffffffffu, b1, off);
    if (kNorm && line) {  // CTA-uniform
      c0 += __shfl_xor_sync(0xffffffffu, c0, off);
      c1 += __shfl_xor_sync(0xffffffffu, c1, off);
    }
  }
  if (sl || !valid) return;
  auto put = [&](int k, double a, double b, double c) {
    if (line) {
      if (kNorm) out[(size_t)k * nd + z] = c;
      out[(size_t)(nline + k) * nd + z] = a;
      out[(size_t)(2 * nline + k) * nd + z] = b;
    } else {
      out[(size_t)(3 * nline + k) * nd + z] = a;
      out[(size_t)(3 * nline + nbf + k) * nd + z] = b;
    }
  };
  put(k0, a0, b0, c0);
  if (k1 > k0) put(k1, a1, b1, c1);
}

// radiative rate from level `from` to `to` of one stage (atom_rad.cc:1732-1756 / 1726-1729)
__device__ double rad_rate(const AliDev &D, int from, int to, double JJ, double LL, double nf, double nt, bool alo) {
  const double a = D.A[from * D.nlev + to], b = D.B[from * D.nlev + to];
  if (!alo) return a + b * JJ;
  if (to == from) return 0.0;
  int u, lo;
  double nu, nl;
  if (to > from) { u = to; lo = from; nu = nt; nl = nf; }
  else { u = from; lo = to; nu = nf; nl = nt; }
  const double sl = nu * D.A[u * D.nlev + lo] / (nl * D.B[lo * D.nlev + u] - nu * D.B[u * D.nlev + lo]);
  return a * (1.0 - LL) + b * (JJ - LL * sl);
}

// rate equations of one depth and their solution (atom_pop.cc:27-145); returns false if singular
// (out of line: k_ali_solve calls it twice, and with both inlined nvcc 12.9 gave other populations)
__device__ __noinline__ bool solve_rates(const AliDev &D, const double *n, const double *coll, double Tz, double nez, double naz,
                            const double *Jl, const double *Ll, const double *nrm, const double *Jbu,
                            const double *Jbd, const double *bfr, bool alo, double *out) {
  const int m = D.nlev;
  double M[kAliMaxLev * kAliMaxLev], b[kAliMaxLev];
  for (int i = 0; i < m * m; ++i) M[i] = 0.0;
  for (int i = 0; i < m; ++i) b[i] = 0.0;
  for (int i = 0; i < m - 1; ++i) {
    for (int j = 0; j < m; ++j) {
      if (D.stage[j] != D.stage[i]) continue;
      const int k = D.tmap[i * m + j];
      const double JJ = k >= 0 ? Jl[k] / nrm[k] : -1.0;
      const double LL = k >= 0 ? Ll[k] / nrm[k] : 0.0;
      M[i * m + i] -= rad_rate(D, i, j, JJ, LL, n[i], n[j], alo) + coll[i * m + j];
      M[i * m + j] += rad_rate(D, j, i, JJ, LL, n[j], n[i], alo) + coll[j * m + i];
    }
    const int c = D.cont_of[i];
    if (c >= 0) {
      const int bb = D.bf_of[i];
      const double up = Jbu[bb] + coll[i * m + c];
      M[i * m + i] -= up;
      M[c * m + i] += up;
      const double down = Jbd[bb] * bfr[bb] + coll[c * m + i];  // every continuum has a bf transition
      M[i * m + c] += down;
      M[c * m + c] -= down;
    }
  }
  int rep = m - 1;
  double maxpop = n[rep];
  for (int i = 0; i < m - 1; ++i)
    if (n[i] > maxpop) { maxpop = n[i]; rep = i; }
  for (int j = 0; j < m; ++j) M[rep * m + j] = 1.0;
  b[rep] = naz;
  // LU without pivoting (Crout) and the two triangular solves
  for (int p = 0; p < m; ++p) {
    for (int i = p; i < m; ++i) {
      double s = M[i * m + p];
      for (int q = 0; q < p; ++q) s -= M[i * m + q] * M[q * m + p];
      M[i * m + p] = s;
    }
    if (M[p * m + p] == 0.0) return false;
    for (int j = p + 1; j < m; ++j) {
      double s = M[p * m + j];
      for (int q = 0; q < p; ++q) s -= M[p * m + q] * M[q * m + j];
      M[p * m + j] = s / M[p * m + p];
    }
  }
  for (int i = 0; i < m; ++i) {
    double s = b[i];
    for (int q = 0; q < i; ++q) s -= M[i * m + q] * out[q];
    out[i] = s / M[i * m + i];
  }
  for (int i = m - 1; i >= 0; --i) {
    double s = out[i];
    for (int q = i + 1; q < m; ++q) s -= M[i * m + q] * out[q];
    out[i] = s;
  }
  (void)Tz; (void)nez;
  return true;
}

// A thread per depth, up to the 1024 that snapi_ali_create accepts: 64 registers (72 without the bound, which
// refused the launch from 29 warps on).
__global__ void __launch_bounds__(1024) k_ali_solve(AliDev D) {
  __shared__ int s_neg;
  __shared__ double s_max;
  const int col = blockIdx.x, z = threadIdx.x, nd = D.nd, m = D.nlev;
  if (D.state[col] != 0) return;  // CTA-uniform
  if (threadIdx.x == 0) { s_neg = 0; s_max = 0.0; }
  __syncthreads();
  const bool valid = z < nd;
  const int zz = valid ? z : nd - 1;
  double n[kAliMaxLev], nn[kAliMaxLev];
  double *pz = D.pops + ((size_t)col * nd + zz) * m;
  for (int i = 0; i < m; ++i) n[i] = pz[i];
  const double Tz = D.T[(size_t)col * nd + zz], nez = D.ne[(size_t)col * nd + zz], naz = D.na[(size_t)col * nd + zz];
  double Jl[kAliMaxLine], Ll[kAliMaxLine], nrm[kAliMaxLine], Jbu[kAliMaxBf], Jbd[kAliMaxBf], bfr[kAliMaxBf];
  const double *su = D.sums + (size_t)col * (3 * D.nline + 2 * D.nbf) * nd + zz;
  for (int k = 0; k < D.nline; ++k) {
    nrm[k] = su[(size_t)k * nd];
    Jl[k] = su[(size_t)(D.nline + k) * nd];
    Ll[k] = su[(size_t)(2 * D.nline + k) * nd];
  }
  for (int b = 0; b < D.nbf; ++b) {
    Jbu[b] = su[(size_t)(3 * D.nline + b) * nd];
    Jbd[b] = su[(size_t)(3 * D.nline + D.nbf + b) * nd];
    bfr[b] = D.bfratio[((size_t)col * D.nbf + b) * nd + zz];
  }
  const double *cz = D.coll + ((size_t)col * nd + zz) * m * m;
  // step with the local operator; negative populations anywhere -> without it (atmos_pop.cc:185-205)
  double rmax = 0.0;
  int neg = 0;
  bool ok = solve_rates(D, n, cz, Tz, nez, naz, Jl, Ll, nrm, Jbu, Jbd, bfr, true, nn);
  for (int i = 0; i < m; ++i) {
    const double rc = nn[i] / n[i] - 1.0;
    if (!(rc >= -1.0)) neg = 1;
    rmax = fmax(rmax, fabs(rc));
  }
  if (!ok) neg = 1;
  if (valid && neg) atomicOr(&s_neg, 1);
  __syncthreads();
  int negative = s_neg;
  __syncthreads();
  if (negative) {
    if (threadIdx.x == 0) s_neg = 0;
    __syncthreads();
    ok = solve_rates(D, n, cz, Tz, nez, naz, Jl, Ll, nrm, Jbu, Jbd, bfr, false, nn);
    neg = ok ? 0 : 1;
    rmax = 0.0;
    for (int i = 0; i < m; ++i) {
      const double rc = nn[i] / n[i] - 1.0;
      if (!(rc >= -1.0)) neg = 1;
      rmax = fmax(rmax, fabs(rc));
    }
    if (valid && neg) atomicOr(&s_neg, 1);
    __syncthreads();
    negative = s_neg;
  }
  if (negative) {  // stays negative: the column stops without updating (outcome -1)
    if (threadIdx.x == 0) { D.state[col] = -1; D.iters[col] += 1; }
    return;
  }
  if (valid) {
    for (int i = 0; i < m; ++i) pz[i] = nn[i];
    const int nt = D.nline + D.nbf;
    for (int k = 0; k < nt; ++k) D.fac[((size_t)col * nd + z) * nt + k] = factor(D, col, z, k, nn);
    // max of non-negative doubles through their bit patterns
    atomicMax(reinterpret_cast<unsigned long long *>(&s_max), __double_as_longlong(rmax));
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double r = s_max;
    D.rel[col] = r;
    D.iters[col] += 1;
    if (r < D.tol) D.state[col] = 1;
    else if (D.iters[col] >= D.max_iter) D.state[col] = 2;
  }
}

}  // namespace

struct snapi_ali_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  int nd = 0, nl = 0, nray = 0, nlev = 0, ntr = 0, nline = 0, nbf = 0, nls = 0, nchunk = 0;
  std::vector<void *> bufs;  // problem constants
  AliDev D;
  int cap = 0, cap_host = 0;  // columns of the work buffers, and of the staged copies of inputs
  double *d_T = nullptr, *d_ne = nullptr, *d_na = nullptr, *d_kap = nullptr, *d_vray = nullptr, *d_dld = nullptr,
         *d_adamp = nullptr, *d_bfr = nullptr, *d_coll = nullptr, *d_pops = nullptr, *d_rel = nullptr;
  double *d_bgop = nullptr, *d_bgem = nullptr, *d_I = nullptr, *d_L = nullptr, *d_iop = nullptr, *d_sums = nullptr;
  float *d_phi = nullptr;
  double2 *d_fac = nullptr;
  double *d_eb = nullptr, *d_pl = nullptr, *d_ex = nullptr, *d_ik = nullptr, *d_bo = nullptr, *d_be = nullptr;
  int *d_state = nullptr, *d_iters = nullptr;
  double last_ms = 0.0;
  std::string err;
};

namespace {

int ali_err(snapi_ali_ctx *c, int code, const char *msg) {
  if (c) c->err = msg;
  return code;
}

template <class T>
T *upload(snapi_ali_ctx *c, const T *h, size_t n) {
  T *d = nullptr;
  if (cudaMalloc(&d, sizeof(T) * (n ? n : 1)) != cudaSuccess) return nullptr;
  c->bufs.push_back(d);
  if (n && cudaMemcpy(d, h, sizeof(T) * n, cudaMemcpyHostToDevice) != cudaSuccess) return nullptr;
  return d;
}

// Column buffers: the work buffers and the staged copies of inputs, each with its own capacity, so that a
// call that only lacks the one does not free and allocate the other again.
template <class F>
void each_work(snapi_ali_ctx *c, F f) {
  const size_t nd = c->nd, nr = c->nray, m = c->nlev, ln = c->nline, bf = c->nbf, ns = c->nls, rays = nr * ns * nd;
  f(c->d_pops, nd * m);
  f(c->d_rel, 1);
  f(c->d_state, 1);
  f(c->d_iters, 1);
  f(c->d_I, rays);
  f(c->d_L, rays);
  f(c->d_iop, rays);
  f(c->d_phi, rays * ln);
  f(c->d_eb, bf ? ns * nd : 0);
  f(c->d_pl, bf ? ns * nd : 0);
  f(c->d_ex, bf ? ns * nd : 0);
  f(c->d_bo, rays);
  f(c->d_be, rays);
  f(c->d_ik, nd);
  f(c->d_fac, nd * (ln + bf));
  f(c->d_sums, nd * (3 * ln + 2 * bf));
}
template <class F>
void each_stage(snapi_ali_ctx *c, F f) {
  const size_t nd = c->nd, nl = c->nl, nr = c->nray, m = c->nlev, ln = c->nline, bf = c->nbf;
  f(c->d_T, nd);
  f(c->d_ne, nd);
  f(c->d_na, nd);
  f(c->d_kap, nd);
  f(c->d_vray, nr * nd);
  f(c->d_dld, ln * nd);
  f(c->d_adamp, ln * nd);
  f(c->d_bfr, bf * nd);
  f(c->d_coll, nd * m * m);
  f(c->d_bgop, nr * nl * nd);
  f(c->d_bgem, nr * nl * nd);
}

void free_work(snapi_ali_ctx *c) {
  each_work(c, [](auto *&p, size_t) { cudaFree(p); p = nullptr; });
  c->cap = 0;
}
void free_stage(snapi_ali_ctx *c) {
  each_stage(c, [](auto *&p, size_t) { cudaFree(p); p = nullptr; });
  c->cap_host = 0;
}

// bytes of one column
size_t work_bytes(snapi_ali_ctx *c) {
  size_t n = 0;
  each_work(c, [&](auto *&p, size_t k) { n += k * sizeof(*p); });
  return n;
}
size_t stage_bytes(snapi_ali_ctx *c) {
  size_t n = 0;
  each_stage(c, [&](auto *&p, size_t k) { n += k * sizeof(*p); });
  return n;
}

// the buffers of C columns (stage: and the staged inputs) where they are smaller, or the first error
cudaError_t ensure_cols(snapi_ali_ctx *c, size_t C, bool stage) {
  cudaError_t e = cudaSuccess;
  auto get = [&](auto *&p, size_t n) {
    if (e == cudaSuccess) e = cudaMalloc(&p, sizeof(*p) * (n ? C * n : 1));
  };
  if (c->cap < (int)C) {
    free_work(c);
    each_work(c, get);
    if (e == cudaSuccess) c->cap = (int)C;
  }
  if (e == cudaSuccess && stage && c->cap_host < (int)C) {
    free_stage(c);
    each_stage(c, get);
    if (e == cudaSuccess) c->cap_host = (int)C;
  }
  return e;
}

// Where the kernels may read an input of a device call: 1 in place (memory of the context's GPU, managed memory, any
// where the GPU reads pageable memory), 0 copied first (another GPU's, pinned host memory), -1 not at all.
int input_place(const snapi_ali_ctx *c, const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return -1; }
  if (a.type == cudaMemoryTypeManaged) return 1;
  if (a.type == cudaMemoryTypeDevice) return a.device == c->device;
  if (a.type == cudaMemoryTypeHost) return 0;
  int pageable = 0;
  return cudaDeviceGetAttribute(&pageable, cudaDevAttrPageableMemoryAccess, c->device) == cudaSuccess && pageable ? 1 : -1;
}

size_t formal_smem(const snapi_ali_ctx *c) { return c->nd * (sizeof(double2) * (c->nline + c->nbf) + sizeof(double)); }

}  // namespace

extern "C" {

snapi_ali_ctx *snapi_ali_create(const snapi_ali_problem *p, int device, int *status) {
  auto fail = [&](snapi_ali_ctx *c, int code) -> snapi_ali_ctx * {
    if (status) *status = code;
    if (c) { fprintf(stderr, "snapi_ali_create: %s\n", c->err.c_str()); snapi_ali_destroy(c); }
    return nullptr;
  };
  if (!p) return fail(nullptr, SNAPI_EINVAL);
  snapi_ali_ctx *c = new snapi_ali_ctx();
  c->device = device;
  if (p->nd < 3 || p->nlambda < 1 || p->nray < 1 || p->nlevel < 2 || p->nlevel > kAliMaxLev || p->ntrans < 1 ||
      !p->grid || !p->lambda || !p->lambda_w || !p->fudge || !p->ray_theta || !p->ray_w || !p->trans || !p->line_c ||
      !p->line_e || !p->A || !p->B || !p->stage || !p->cont_of || !p->sigma) {
    ali_err(c, SNAPI_EINVAL, "invalid ALI problem");
    return fail(c, SNAPI_EINVAL);
  }
  const int m = p->nlevel;
  std::vector<int> llo, lup, blo, bup, tmap(m * m, -1), bfof(m, -1), lineof(p->ntrans, -1), bfidx(p->ntrans, -1);
  std::vector<double> lam0, aul, blu, bul, eline;
  for (int t = 0; t < p->ntrans; ++t) {
    const int lo = p->trans[2 * t], up = p->trans[2 * t + 1];
    if (lo < 0 || lo >= m || up < 0 || up >= m || lo == up) {
      ali_err(c, SNAPI_EINVAL, "transition levels out of range");
      return fail(c, SNAPI_EINVAL);
    }
    if (p->cont_of[lo] == up) {
      bfof[lo] = (int)blo.size();
      bfidx[t] = (int)blo.size();
      blo.push_back(lo); bup.push_back(up);
    } else {
      const int k = (int)llo.size();
      tmap[lo * m + up] = tmap[up * m + lo] = k;
      lineof[t] = k;
      llo.push_back(lo); lup.push_back(up);
      lam0.push_back(p->line_c[4 * t]); aul.push_back(p->line_c[4 * t + 1]);
      blu.push_back(p->line_c[4 * t + 2]); bul.push_back(p->line_c[4 * t + 3]);
      eline.push_back(p->line_e[t]);
    }
  }
  for (int i = 0; i < m; ++i)
    if (p->cont_of[i] >= m || (p->cont_of[i] >= 0 && bfof[i] < 0)) {
      ali_err(c, SNAPI_EINVAL, "every level with a continuum needs its bound-free transition");
      return fail(c, SNAPI_EINVAL);
    }
  if ((int)llo.size() > kAliMaxLine || (int)blo.size() > kAliMaxBf) {
    ali_err(c, SNAPI_EINVAL, "too many transitions (lines <= 32, bound-free <= 16)");
    return fail(c, SNAPI_EINVAL);
  }
  c->nd = p->nd; c->nl = p->nlambda; c->nray = p->nray; c->nlev = m; c->ntr = p->ntrans;
  c->nline = (int)llo.size(); c->nbf = (int)blo.size();
  int maxsm = 0;
  const int nsl = c->nd <= 256 ? 4 : (c->nd <= 512 ? 2 : 1), nls = (p->nlambda + 4 * nsl - 1) / (4 * nsl) * (4 * nsl);
  c->nls = nls;
  c->nchunk = (nls + kAliChunk - 1) / kAliChunk;
  if (12 * (size_t)c->nd + 16 * (size_t)(c->nline + c->nbf) * c->nd > 200 * 1024) {
    ali_err(c, SNAPI_EINVAL, "too many depths x transitions for one CTA's shared memory");
    return fail(c, SNAPI_EINVAL);
  }
  if (p->nd > 1024) { ali_err(c, SNAPI_EINVAL, "nd > 1024"); return fail(c, SNAPI_EINVAL); }
  if (cudaSetDevice(device) != cudaSuccess) { ali_err(c, SNAPI_ECUDA, "cudaSetDevice failed"); return fail(c, SNAPI_ECUDA); }
  std::vector<double> ct(p->nray), geo((size_t)p->nray * p->nd * 3, 0.0), lam(nls, 1.0), lw(nls, 0.0), p5(nls, 0.0);
  for (int r = 0; r < p->nray; ++r) {
    ct[r] = cos(p->ray_theta[r]);
    const int dz = ct[r] > 0.0 ? 1 : -1, zl = dz > 0 ? 0 : p->nd - 1, zh = p->nd - 1 - zl;
    double hp = 0.0;
    for (int z = zl; z != zh; z += dz) {
      double *g = &geo[((size_t)r * p->nd + z) * 3];
      const double h = (p->grid[z + dz] - p->grid[z]) / -ct[r];
      g[0] = h;
      g[1] = h / 3.0;
      if (z != zl) g[2] = (1.0 + hp / (hp + h)) / 3.0;
      hp = h;
    }
  }
  std::vector<float> sig((size_t)c->nbf * nls, 0.f);
  std::vector<double> sgf((size_t)c->nbf * nls, 0.0);
  for (int l = 0; l < p->nlambda; ++l) {
    const int s = slot_of(l, nsl);
    const double il = 1.0 / p->lambda[l], il2 = il * il;
    lam[s] = p->lambda[l];
    lw[s] = p->lambda_w[l];
    p5[s] = il2 * il2 * il;
    for (int t = 0; t < p->ntrans; ++t)
      if (bfidx[t] >= 0) {
        const size_t at = (size_t)bfidx[t] * nls + s;
        sig[at] = (float)p->sigma[(size_t)t * p->nlambda + l];
        sgf[at] = (double)sig[at] * (double)(float)p->fudge[l];
      }
  }
  AliDev &D = c->D;
  memset(&D, 0, sizeof D);
  D.nd = c->nd; D.nl = c->nl; D.nray = c->nray; D.nlev = m; D.nline = c->nline; D.nbf = c->nbf; D.nchunk = c->nchunk;
  D.nsl = nsl; D.nls = nls;
  bool ok = (D.geo = upload(c, geo.data(), geo.size())) && (D.lambda = upload(c, lam.data(), lam.size())) &&
            (D.lw = upload(c, lw.data(), lw.size())) && (D.p5 = upload(c, p5.data(), p5.size())) &&
            (D.ray_ct = upload(c, ct.data(), ct.size())) && (D.ray_w = upload(c, p->ray_w, p->nray)) &&
            (D.sgf = upload(c, sgf.data(), sgf.size())) &&
            (D.lam0 = upload(c, lam0.data(), lam0.size())) && (D.Aul = upload(c, aul.data(), aul.size())) &&
            (D.Blu = upload(c, blu.data(), blu.size())) && (D.Bul = upload(c, bul.data(), bul.size())) &&
            (D.Eline = upload(c, eline.data(), eline.size())) && (D.line_lo = upload(c, llo.data(), llo.size())) &&
            (D.line_up = upload(c, lup.data(), lup.size())) && (D.bf_lo = upload(c, blo.data(), blo.size())) &&
            (D.bf_up = upload(c, bup.data(), bup.size())) && (D.sigma = upload(c, sig.data(), sig.size())) &&
            (D.A = upload(c, p->A, (size_t)m * m)) && (D.B = upload(c, p->B, (size_t)m * m)) &&
            (D.stage = upload(c, p->stage, m)) && (D.cont_of = upload(c, p->cont_of, m)) &&
            (D.tmap = upload(c, tmap.data(), tmap.size())) && (D.bf_of = upload(c, bfof.data(), bfof.size()));
  if (!ok) { ali_err(c, SNAPI_ENOMEM, "device allocation failed"); return fail(c, SNAPI_ENOMEM); }
  if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreate(&c->ev0) != cudaSuccess || cudaEventCreate(&c->ev1) != cudaSuccess ||
      // the limit is per device and shared by every ALI context: the opt-in maximum, not this
      // problem's size, so a smaller context never lowers it under a larger one
      cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess ||
      cudaFuncSetAttribute(k_ali_formal, cudaFuncAttributeMaxDynamicSharedMemorySize, maxsm) != cudaSuccess) {
    ali_err(c, SNAPI_ECUDA, "stream / event / attribute set-up failed");
    return fail(c, SNAPI_ECUDA);
  }
  if (status) *status = SNAPI_OK;
  return c;
}

void snapi_ali_destroy(snapi_ali_ctx *c) {
  if (!c) return;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  free_work(c);
  free_stage(c);
  for (void *b : c->bufs) cudaFree(b);
  if (c->ev0) cudaEventDestroy(c->ev0);
  if (c->ev1) cudaEventDestroy(c->ev1);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
}

const char *snapi_ali_last_error(const snapi_ali_ctx *c) { return c ? c->err.c_str() : "null context"; }
double snapi_ali_last_kernel_ms(const snapi_ali_ctx *c) { return c ? c->last_ms : 0.0; }

int snapi_ali_iter(snapi_ali_ctx *c, int ncol, const snapi_ali_columns *in, double *pops, int max_iter, double tol,
                   double *rel_change, int *iters, int *status, int mem) {
  if (!c) return SNAPI_EINVAL;
  if (ncol < 1 || !in || !pops || max_iter < 1 || !(tol > 0.0) || (mem != SNAPI_MEM_HOST && mem != SNAPI_MEM_DEVICE) ||
      !in->T || !in->ne || !in->na || !in->kappa || !in->vray || (c->nline && (!in->dld || !in->adamp)) ||
      (c->nbf && !in->bfratio) || !in->coll || !in->bg_op || !in->bg_em)
    return ali_err(c, SNAPI_EINVAL, "snapi_ali_iter: invalid arguments");
#define ACK(call)                                                                         \
  do {                                                                                    \
    cudaError_t e_ = (call);                                                              \
    if (e_ != cudaSuccess) return ali_err(c, SNAPI_ECUDA, cudaGetErrorString(e_));         \
  } while (0)
  ACK(cudaSetDevice(c->device));
  const size_t nd = c->nd, nl = c->nl, nr = c->nray, m = c->nlev, ln = c->nline, bf = c->nbf;
  const bool host = mem == SNAPI_MEM_HOST;
  cudaStream_t s = c->stream;
  bool stage = host;  // the inputs are copied into buffers of the context
  if (!host) {
    const double *in_dev[] = {in->T, in->ne, in->na, in->kappa, in->vray, c->nline ? in->dld : in->T, c->nline ? in->adamp : in->T,
                              c->nbf ? in->bfratio : in->T, in->coll, in->bg_op, in->bg_em};
    for (const double *p : in_dev) {
      const int at = input_place(c, p);
      if (at < 0) return ali_err(c, SNAPI_EINVAL, "snapi_ali_iter: an input is not a device array");
      stage = stage || at == 0;
    }
  }
  // Batches of columns whose buffers stay within kAliWork and within half of what the GPU has free beside them.
  // Buffers that hold less than that are only replaced where more fit: the next call of a size that did not fit
  // runs in the batches that did.
  const size_t wb = work_bytes(c), hb = stage_bytes(c), per = wb + (stage ? hb : 0);
  int B = (int)std::min<size_t>(ncol, std::max<size_t>(1, kAliWork / per));
  if (c->cap < B || (stage && c->cap_host < B)) {
    size_t room = 0, total = 0;
    ACK(cudaMemGetInfo(&room, &total));
    room += c->cap * wb + c->cap_host * hb;
    B = (int)std::min<size_t>(B, std::max<size_t>(1, room / 2 / per));
    cudaError_t e;
    while ((e = ensure_cols(c, B, stage)) != cudaSuccess) {
      cudaGetLastError();
      free_work(c);
      free_stage(c);
      if (e != cudaErrorMemoryAllocation || B == 1) return ali_err(c, SNAPI_ECUDA, cudaGetErrorString(e));
      B = (B + 1) / 2;
    }
  }
  const int nthr = (int)((nd + 31) / 32 * 32);
  auto sum_blocks = [&](size_t nq) { return (int)((nd * nq * c->D.nsl + kSumThreads - 1) / kSumThreads); };
  const int nblk_line = sum_blocks((ln + 1) / 2), nblk = nblk_line + sum_blocks((bf + 1) / 2);
  std::vector<int> st(ncol);
  c->last_ms = 0.0;
  for (int c0 = 0; c0 < ncol; c0 += B) {
    const size_t C = std::min(B, ncol - c0);
    AliDev D = c->D;
    D.ncol = (int)C; D.tol = tol; D.max_iter = max_iter;
    auto input = [&](const double *&dst, const double *src, double *buf, size_t n) -> cudaError_t {
      if (!src) return cudaSuccess;
      dst = src + (size_t)c0 * n;
      if (!stage) return cudaSuccess;
      const cudaError_t e = cudaMemcpyAsync(buf, dst, sizeof(double) * C * n, host ? cudaMemcpyHostToDevice : cudaMemcpyDefault, s);
      dst = buf;
      return e;
    };
    ACK(input(D.T, in->T, c->d_T, nd));
    ACK(input(D.ne, in->ne, c->d_ne, nd));
    ACK(input(D.na, in->na, c->d_na, nd));
    ACK(input(D.kap, in->kappa, c->d_kap, nd));
    ACK(input(D.vray, in->vray, c->d_vray, nr * nd));
    if (ln) {
      ACK(input(D.dld, in->dld, c->d_dld, ln * nd));
      ACK(input(D.adamp, in->adamp, c->d_adamp, ln * nd));
    }
    if (bf) ACK(input(D.bfratio, in->bfratio, c->d_bfr, bf * nd));
    ACK(input(D.coll, in->coll, c->d_coll, nd * m * m));
    ACK(input(D.bgop, in->bg_op, c->d_bgop, nr * nl * nd));
    ACK(input(D.bgem, in->bg_em, c->d_bgem, nr * nl * nd));
    double *pb = pops + (size_t)c0 * nd * m;
    ACK(cudaMemcpyAsync(c->d_pops, pb, sizeof(double) * C * nd * m, host ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, s));
    ACK(cudaMemsetAsync(c->d_state, 0, sizeof(int) * C, s));
    ACK(cudaMemsetAsync(c->d_iters, 0, sizeof(int) * C, s));
    ACK(cudaMemsetAsync(c->d_rel, 0, sizeof(double) * C, s));
    D.pops = c->d_pops; D.I = c->d_I; D.L = c->d_L; D.iop = c->d_iop; D.phi = c->d_phi; D.eb = c->d_eb; D.pl = c->d_pl;
    D.ex = c->d_ex; D.ik = c->d_ik; D.fac = c->d_fac; D.bo = c->d_bo; D.be = c->d_be; D.sums = c->d_sums; D.state = c->d_state; D.iters = c->d_iters; D.rel = c->d_rel;
    for (int it = 0; it < max_iter; ++it) {
      ACK(cudaEventRecord(c->ev0, s));
      if (it == 0) {
        k_ali_tables<<<(unsigned)(C * nr * nd), kTabThreads, 0, s>>>(D);
        ACK(cudaGetLastError());
        k_ali_turn<<<(unsigned)(C * nr * ((nl + 31) / 32) * ((nd + 31) / 32)), 256, 0, s>>>(D);
        ACK(cudaGetLastError());
      }
      k_ali_formal<<<(unsigned)(C * nr * c->nchunk), kAliChunk, formal_smem(c), s>>>(D);
      ACK(cudaGetLastError());
      if (it == 0) k_ali_sums<true><<<(unsigned)(C * nblk), kSumThreads, 0, s>>>(D, nblk_line, nblk);
      else k_ali_sums<false><<<(unsigned)(C * nblk), kSumThreads, 0, s>>>(D, nblk_line, nblk);
      ACK(cudaGetLastError());
      k_ali_solve<<<(unsigned)C, nthr, 0, s>>>(D);
      ACK(cudaGetLastError());
      ACK(cudaEventRecord(c->ev1, s));
      ACK(cudaMemcpyAsync(st.data() + c0, c->d_state, sizeof(int) * C, cudaMemcpyDeviceToHost, s));
      ACK(cudaStreamSynchronize(s));
      float ms = 0.f;
      ACK(cudaEventElapsedTime(&ms, c->ev0, c->ev1));
      c->last_ms += ms;
      bool any = false;
      for (size_t i = 0; i < C; ++i) any = any || st[c0 + i] == 0;
      if (!any) break;
    }
    const cudaMemcpyKind o = host ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
    ACK(cudaMemcpyAsync(pb, c->d_pops, sizeof(double) * C * nd * m, o, s));
    if (rel_change) ACK(cudaMemcpyAsync(rel_change + c0, c->d_rel, sizeof(double) * C, o, s));
    if (iters) ACK(cudaMemcpyAsync(iters + c0, c->d_iters, sizeof(int) * C, o, s));
    ACK(cudaStreamSynchronize(s));
  }
  if (status) {
    std::vector<int> out(ncol);
    for (int i = 0; i < ncol; ++i) out[i] = st[i] < 0 ? -1 : 0;
    ACK(cudaMemcpy(status, out.data(), sizeof(int) * ncol, host ? cudaMemcpyHostToHost : cudaMemcpyHostToDevice));
  }
#undef ACK
  return SNAPI_OK;
}

}  // extern "C"

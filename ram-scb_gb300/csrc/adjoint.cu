// adjoint.cu -- frozen-limiter adjoint of the RAM kinetic step.
//
// With the limiter branch of every face and the clip state of every cell
// frozen (recorded by the forward sweeps, four bits per face: 0 upwind
// only, 1 beta*D, 2 X, 3 D, 4 beta*X, plus kClipBit; a call's forward and
// reverse sweeps of one direction share a byte, the forward one in the high
// nibble, read here with the shift rsh), each sweep of
// src/ModRamDrift.f90 is a linear map of its line
//   Fnew(i) = G(i) + w(i) (Phi(i-1) - Phi(i)),  Phi(f) = C(f) FBND(f),
//   FBND(f) = FUP(f) + a(f) LX(f),  LX in {beta D, X, D, beta X},
// so its adjoint is the transposed map, applied here line by line with the
// coefficients recomputed, from the forward pass's tables or, in DRIFTE, from
// EDOT and EB (the forward sweep's factored form agrees to rounding).  The
// tail of ram_run (periodic copy, magnetopause mask, ANISCH's F2(:,:,:,:,1)
// side effect), the CEX/ATMOL factors and the log-flux observation operator
// are transposed too.  dJ/dFGEOS collects the ghost cells of DRIFTR,
// including the stale ghosts an outflow line inherits from an earlier
// inflow line.
#include <math.h>

#include <type_traits>

#include "face.cuh"
#include "kernels.cuh"

namespace ramgpu {

// Transposed sweeps.  With the record frozen, one face f contributes
//   FBb(f) = dJ/dFBND(f) = C(f) * (w(f+1) le(f+1) - w(f) le(f))
// (le = lambda of an updated, unclipped cell, w the update weight: 1 for R
// and P, 1/WE, 1/WMU for E and MU) and scatters it to the cells of
// FBND(f) = FUP + a LX:  the upwind cell, and for LX = beta D | X | D |
// beta X the two cells of D (f-1,f for s=+1; f+1,f+2 for s=-1) or of X
// (f,f+1).  Every face touches cells f-1..f+2 only, so each line is
// streamed once with a rolling window of four cell accumulators in
// registers: after face f, cell f-1 is final and is written out.

// FBND(f) = FUP + a LX depends on adjacent cells only: with C >= 0 (FUP =
// F(f)) on (f-1, f) for LX = D, (f, f+1) for LX = X; with C < 0 (FUP =
// F(f+1)) on (f, f+1) for LX = X, (f+1, f+2) for LX = D.  The pair and its
// two weights, which add up to 1, are picked by integer selects, so a face
// costs two fma on the FP64 pipe whatever its case.
//
// The transposes are bound by the FP64 unit, so the two FP64 operations that
// form the weights move to integer instructions (as in face.cuh).  Backward
// ms a call on 20x25x35x72, one species and four: 0.270 -> 0.262, 0.532 ->
// 0.502.  The 46 FP64 operations a cell and call that the eight transposes
// execute (five to eight each) take 0.44 of the 0.50 ms of four species; forming the
// product FBb = C*DL on the integer pipe as well was slower or even in every
// sweep.

// v 2^-64 as a double, rounded.
__device__ __forceinline__ double fix64_to_double(uint64_t v) {
  const int lz = __clzll((long long)(v | 1ULL));
  const uint64_t r = ((uint64_t)(1021 - lz) << 52) + ((((v << lz) >> 10) + 1) >> 1);
  return bitsd(v ? r : 0ULL);
}
// Scatter of one face of coefficient C into the window (cm1, c0, c1, c2) =
// cells f-1..f+2, from q, C as the forward sweeps prepare it.  The pair's
// weights are (1-w, w) where it starts at the upwind cell, (w, 1-w) where it
// ends there, with w = ak for LX = X, -ak for LX = D, ak = k/2 (1 - U) (k =
// beta in cases 1 and 4), 0 with upwind only.  Both are formed in fixed
// point with 2^64 as 1 and rounded once; Courant numbers of 1 and more, inf
// and NaN take the FP64 form (y: U = |C| y).
__device__ __forceinline__ void face_acc_q(double FBb, double C, double y, const FaceCoef& q, int cs, uint64_t betaf,
                                           double betalim, double& cm1, double& c0, double& c1, double& c2) {
  const bool neg = is_neg(C);
  const bool dt = (cs & 1) != 0;  // LX = D (f-1, f) or (f+1, f+2)
  const bool kb = (cs == 1) | (cs == 4);
  const bool ends = dt != neg;  // (upwind only: either side, w = 0)
  double w, m;
  if (q.bad >= 0) {
    uint64_t A = kb ? beta_times<false>(q.a63, betaf) : q.a63;
    if (cs == 0) A = 0ULL;
    w = bitsd(dbits(fix64_to_double(A)) ^ (dt ? kSignMask : 0ULL));
    const uint64_t up = 0x3FF0000000000000ULL + (((A >> 11) + 1) >> 1);  // 1 + ak
    m = (dt | (A == 0ULL)) ? bitsd(up) : fix64_to_double(0ULL - A);
  } else {
    const double k = kb ? 0.5 * betalim : 0.5;
    const double ak = fma(fabs(C), -k * y, k);
    w = cs == 0 ? 0.0 : (dt ? -ak : ak);
    m = 1.0 - w;
  }
  const double b0 = ends ? w : m, b1 = ends ? m : w;
  // first cell of the pair in the window: 0 = f-1, 1 = f, 2 = f+1
  const int p = (int)neg + (int)!ends;
  const double p0 = p == 0 ? cm1 : (p == 1 ? c0 : c1);
  const double p1 = p == 0 ? c0 : (p == 1 ? c1 : c2);
  const double t0 = fma(b0, FBb, p0);
  const double t1 = fma(b1, FBb, p1);
  cm1 = p == 0 ? t0 : cm1;
  c0 = p == 0 ? t1 : (p == 1 ? t0 : c0);
  c1 = p == 1 ? t1 : (p == 2 ? t0 : c1);
  c2 = p == 2 ? t1 : c2;
}

// ak = LIMITER weight times the CORR factor a = -0.5*(C - s) of a face of
// DRIFTP: fma(C, -0.5*k, 0.5*k*s) with k = beta for cases 1, 4 and 1
// otherwise (the two faces that wrap around; hb = 0.5*beta).
__device__ __forceinline__ double face_ak(double C, bool neg, int cs, double hb) {
  const double hk = (cs == 1) | (cs == 4) ? hb : 0.5;
  return fma(C, -hk, neg ? -hk : hk);
}

// lambda of cell c of a line (stride st) masked by the clip bit.  Both
// loads are issued unconditionally (the record through the read-only path)
// so that the next cells' loads can run ahead of the window's arithmetic.
__device__ __forceinline__ double masked(const double* __restrict__ lam, const unsigned char* __restrict__ rl,
                                         long long off, int rsh) {
  const double v = lam[off];
  return ((__ldg(rl + off) >> rsh) & kClipBit) ? 0.0 : v;
}

#define WORK_LOOP(NLINES) for (Unit u((NLINES + blockDim.x - 1) / blockDim.x); u.ok(d); u.next(d))

// The loops below are peeled so that no floating-point operation in the
// main loop depends on the position along the line (the FP64 pipe is the
// bottleneck and predicated-off branches would still cost issue slots).

// ------------------------------------------------------------------ DRIFTR^T
// Cells 1..NR, ghosts NR+1, NR+2.  new(1) = F(1); faces 2..NR-1 (and NR on
// inflow lines); FBND(1) = F(2) on inflow lines, FBND(NR) = F(NR) on outflow
// lines (both 0 when closed).  The ghosts' adjoints go to dJ/dFGEOS, for an
// outflow line to the FGEOS cell its stale ghost came from.
// A CTA takes blockDim.x consecutive lines of one item.  They are contiguous
// in memory (blockDim.x*NR doubles of lambda and as many record bytes), so
// the CTA loads them into shared memory with coalesced loads, each thread
// transposes its line there, and the CTA stores the tile back coalesced.
// Read in place, the lanes' lines lie 8*NR bytes apart: every warp load
// touches 32 sectors and leans on L1, and at seven CTAs per SM L1 no longer
// held them (four times slower).  Rows of the lambda tile are NR|1 doubles
// apart, so the 8-byte accesses of a half-warp fall in distinct banks.
#ifdef RAMGPU_BOUNDS_CHECK
constexpr bool kBoundsChecked = true;
#else
constexpr bool kBoundsChecked = false;
#endif
size_t adj_r_smem(const Dev& d, int threads) {
  return (size_t)threads * (size_t)(d.nr | 1) * sizeof(double) + (size_t)threads * (size_t)d.nr;
}
template <int rsh>
__global__ void __launch_bounds__(128) k_adj_r(Dev d, const unsigned char* __restrict__ rec) {
  extern __shared__ double tile[];
  const int nr = d.nr, nt = d.nt, ne = d.ne;
  const int ts = nr | 1;
  unsigned char* rtile = (unsigned char*)(tile + (size_t)blockDim.x * ts);
  const int nlines = nt * ne * d.npa;
  for (Unit u((nlines + blockDim.x - 1) / blockDim.x); u.ok(d); u.next(d)) {  // uniform across the CTA
    const int2 item = d.items[u.it];
    const int m = item.x, s = item.y, slot = m * d.ns + s;
    const int lfirst = u.b * blockDim.x;
    const int nl = min((int)blockDim.x, nlines - lfirst);
    // bounds-checked builds: the tile's cells (the whole CTA skips it)
    if (kBoundsChecked) {
      const bool ok = rg_item(d, item) && rg_span((long long)lfirst * nr, (long long)nl * nr, 1, d.ncell);
      if (threadIdx.x == 0) rg_ok(d, ok, kRgAdjR, lfirst);
      if (!ok) continue;
    }
    double* __restrict__ gl = d.lam + (long long)slot * d.ncell + (long long)lfirst * nr;
    const unsigned char* __restrict__ gr = rec + u.it * d.ncell + (long long)lfirst * nr;
    for (int e = threadIdx.x; e < nl * nr; e += blockDim.x) {
      const int ln = e / nr;
      tile[ln * ts + (e - ln * nr)] = gl[e];
      rtile[e] = __ldg(gr + e);
    }
    __syncthreads();
    const int line = lfirst + threadIdx.x;
    const int j = line % nt, k = (line / nt) % ne, l = line / (nt * ne);
    // bounds-checked builds: the line's GRT and CR rows
    const bool lok = threadIdx.x < nl &&
        (!kBoundsChecked ||
         rg_ok(d, rg_span(((long long)l * nt + j) * nr, nr, 1, (long long)nr * nt * d.npa) &&
                      rg_span(((long long)m * nt + j) * nr, nr, 1, (long long)d.nm * nr * nt),
               kRgAdjR, line));
    if (lok) {
      double* lam = tile + threadIdx.x * ts;
      const unsigned char* rl = rtile + threadIdx.x * nr;
      const double* __restrict__ grt = d.grt + ((long long)l * nt + j) * nr;
      const double* __restrict__ cr = d.cr + ((long long)m * nt + j) * nr;
      const double p4 = d.p4[s * ne + k];
      const uint64_t betaf = beta_fix(dbits(d.betalim));
      const bool closed = d.flags & 1u;
      const int n = nr;  // >= 4
      auto mk = [&](int c) { return ((rl[c] >> rsh) & kClipBit) ? 0.0 : lam[c]; };  // masked lambda
      const double cN = fma(grt[n - 1], p4, cr[n - 1]);
      const bool inflow = is_neg(cN);
      // le(i) = lambda of updated, unclipped cell i (i = 2..NR); window = cells f-1..f+2
      double le0 = mk(1), le1 = mk(2), le2 = mk(3);
      double cm1 = lam[0], c0 = le0, c1 = le1, c2 = le2;
      if (inflow && !closed) c0 += fma(grt[0], p4, cr[0]) * le0;  // FBND(1) = F(2)
      auto face = [&](int f, double C) {
        const int cs = (rl[f - 1] >> rsh) & 7;
        face_acc_q(C * (le1 - le0), C, 1.0, face_coef(dbits(C)), cs, betaf, d.betalim, cm1, c0, c1, c2);
      };
      auto advance = [&](int f, double le3) {  // cell f-1 is final; cell f+3 enters
        lam[f - 2] = cm1;
        cm1 = c0; c0 = c1; c1 = c2; c2 = le3;
        le0 = le1; le1 = le2; le2 = le3;
      };
      int f = 2;
      for (; f <= n - 3; ++f) {
        face(f, fma(grt[f - 1], p4, cr[f - 1]));
        advance(f, mk(f + 2));
      }
      for (; f <= n - 1; ++f) {
        face(f, fma(grt[f - 1], p4, cr[f - 1]));
        advance(f, 0.0);
      }
      // face NR: transposed on inflow lines, FBND(NR) = F(NR) on outflow lines
      if (!closed) {
        if (inflow) face(n, cN);
        else c0 -= cN * le0;
      }
      lam[n - 2] = cm1;
      lam[n - 1] = c0;
      const double gN1 = c1, gN2 = c2;  // ghosts F(NR+1), F(NR+2)
      const long long nfg = (long long)nt * ne * d.npa;
      if (inflow) {
        if (d.outside[(long long)j * nr + n - 1] != 1) {
          const double fh = d.fnhs[((long long)l * nt + j) * d.nf + n - 1];
          atomicAdd(&d.gfg[slot * nfg + line], d.conf1 * fh * gN1 + d.conf2 * fh * gN2);
        }
      } else if (gN1 != 0.0) {
        const int src = stale_ghost_src(d, m, slot, j, k, l, p4);
        if (src >= 0) {
          const int jj = src % nt, ll = src / (nt * ne);
          if (d.outside[(long long)jj * nr + n - 1] != 1) {
            const double fh = d.fnhs[((long long)ll * nt + jj) * d.nf + n - 1];
            atomicAdd(&d.gfg[slot * nfg + src], d.conf1 * fh * gN1);
          }
        }
      }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nl * nr; e += blockDim.x) {
      const int ln = e / nr;
      gl[e] = tile[ln * ts + (e - ln * nr)];
    }
    __syncthreads();  // the next unit reuses the tile
  }
}

// ------------------------------------------------------------------ DRIFTP^T
// Cells 1..NT with J = 1 == J = NT: new(1) is overwritten by new(NT), faces
// J = 2..NT with FBND(1) = FBND(NT).  Faces NT-1 and NT wrap onto cells
// 1..3; they are transposed first, their contributions held in registers
// and added when the window reaches those cells (NT >= 7).
template <int rsh>
__global__ void __launch_bounds__(128) k_adj_p(Dev d, const unsigned char* __restrict__ rec) {
  const int nr = d.nr, nt = d.nt, ne = d.ne;
  const int nlines = (nr - 1) * ne * d.npa;
  WORK_LOOP(nlines) {
    const int2 item = d.items[u.it];
    const int m = item.x, s = item.y, slot = m * d.ns + s;
    const int line = u.b * blockDim.x + threadIdx.x;
    if (line >= nlines) continue;
    const int i = 1 + line % (nr - 1);
    const int kl = line / (nr - 1);
    const int k = kl % ne, l = kl / ne;
    const long long st = nr;
    const long long base = ((long long)kl * nt) * nr + i;
    // bounds-checked builds: the line's cells, its GPT and CA columns
    if (!rg_ok(d, rg_item(d, item) && rg_span(base, nt, nr, d.ncell) &&
                      rg_span((long long)l * nt * nr + i, nt, nr, (long long)nr * nt * d.npa) &&
                      rg_span((long long)m * nt * nr + i, nt, nr, (long long)d.nm * nr * nt),
               kRgAdjP, line))
      continue;
    double* __restrict__ lam = d.lam + (long long)slot * d.ncell + base;
    const unsigned char* __restrict__ rl = rec + u.it * d.ncell + base;
    const double* __restrict__ gpt = d.gpt + ((long long)l * nt) * nr + i;
    const double* __restrict__ ca = d.ca + ((long long)m * nt) * nr + i;
    const double p2 = d.p2[((long long)s * ne + k) * nr + i];
    const double hb = 0.5 * d.betalim;
    const uint64_t betaf = beta_fix(dbits(d.betalim));
    const int n = nt;
#define PC(J) fma(gpt[(long long)((J)-1) * nr], p2, ca[(long long)((J)-1) * nr])
#define PLE(J) masked(lam, rl, (long long)((J)-1) * st, rsh)
    // le(NT) takes lambda of cell 1 too (F2(1) = F2new(NT))
    const double leN = ((rl[(long long)(n - 1) * st] >> rsh) & kClipBit) ? 0.0 : lam[(long long)(n - 1) * st] + lam[0];
    const double leNm = PLE(n - 1), le2 = PLE(2);
    // w1..w3: contributions to cells 1..3, tNm2..tN: to cells NT-2..NT
    double w1 = 0.0, w2 = 0.0, w3 = 0.0, tNm2 = 0.0, tNm1 = 0.0, tN = 0.0;
    {  // face NT-1: X = F(NT)-F(NT-1); D = F(NT-1)-F(NT-2) (s=+1) or F(2)-F(1) (s=-1)
      const double C = PC(n - 1);
      const bool neg = is_neg(C);
      const int cs = (rl[(long long)(n - 2) * st] >> rsh) & 7;
      const double FBb = C * (leN - leNm);
      const double V = face_ak(C, neg, cs, hb) * FBb;
      if (neg) tN += FBb; else tNm1 += FBb;
      if (cs == 2 || cs == 4) { tN += V; tNm1 -= V; }
      else if (cs && !neg) { tNm1 += V; tNm2 -= V; }
      else if (cs) { w2 += V; w1 -= V; }
    }
    {  // face NT: X = F(2)-F(NT); D = F(NT)-F(NT-1) (s=+1) or F(3)-F(2) (s=-1)
      const double C = PC(n);
      const bool neg = is_neg(C);
      const int cs = (rl[(long long)(n - 1) * st] >> rsh) & 7;
      const double FBb = C * (le2 - leN);  // Pb(NT) = -le(NT) + Pb(1), Pb(1) = le(2)
      const double V = face_ak(C, neg, cs, hb) * FBb;
      if (neg) w2 += FBb; else tN += FBb;
      if (cs == 2 || cs == 4) { w2 += V; tN -= V; }
      else if (cs && !neg) { tN += V; tNm1 -= V; }
      else if (cs) { w3 += V; w2 -= V; }
    }
    // faces 2..NT-2 streamed; window cells 1..4 (cell 1 has no own term)
    double le0 = le2, le1 = PLE(3), lnext = PLE(4);
    double cm1 = w1, c0 = le2 + w2, c1 = le1 + w3, c2 = lnext;
    auto step = [&](int J, double add, double lec) {  // face J, then cell J+3 enters
      const double C = PC(J);
      const int cs = (rl[(long long)(J - 1) * st] >> rsh) & 7;
      face_acc_q(C * (le1 - le0), C, 1.0, face_coef(dbits(C)), cs, betaf, d.betalim, cm1, c0, c1, c2);
      lam[(long long)(J - 2) * st] = cm1;
      cm1 = c0; c0 = c1; c1 = c2; c2 = add;
      le0 = le1; le1 = lnext; lnext = lec;
    };
    for (int J = 2; J <= n - 6; ++J) {
      const double lec = PLE(J + 3);
      step(J, lec, lec);
    }
    { const double lec = PLE(n - 2); step(n - 5, lec + tNm2, lec); }
    step(n - 4, leNm + tNm1, leNm);
    step(n - 3, leN + tN, leN);
    step(n - 2, 0.0, 0.0);
    lam[(long long)(n - 3) * st] = cm1;
    lam[(long long)(n - 2) * st] = c0;
    lam[(long long)(n - 1) * st] = c1;
#undef PC
#undef PLE
  }
}

// ------------------------------------------------------------------ DRIFTE^T
// Cells 0..NE+2: G(1) = kap1 F(2) and G(0) = kap0 G(1) are extrapolated,
// G(NE+1) = G(NE+2) = 0; faces 1..NE (not 1 and NE when closed); cell 1
// is never updated (NE >= 6).
// kCo: 0 compute the face coefficients C, 1 compute and keep them in the
// DRIFTE coefficient store, 2 read them from it.  A call's two DRIFTE
// transposes (of the reverse and the forward half) share C (same DTs and
// potential), so the first keeps it for the second; the stored value is the
// recomputed one, so the results do not change.
// A warp's instructions issue in order: the cell entering the window was
// masked, and so waited for, where it was loaded, an L2 round trip per face.
// Loading a face ahead, backward ms a call with and without (one species,
// four species on 20x25x35x72): 0.291 -> 0.277, 0.560 -> 0.546, with DRIFTMU^T
// alike 0.270, 0.532.
template <int kCo, int rsh>
__global__ void __launch_bounds__(128) k_adj_e(Dev d, const unsigned char* __restrict__ rec) {
  const int nr = d.nr, nt = d.nt, ne = d.ne;
  const int nlines = (nr - 1) * nt * d.npa;
  WORK_LOOP(nlines) {
    const int2 item = d.items[u.it];
    const int m = item.x, s = item.y, slot = m * d.ns + s;
    const int line = u.b * blockDim.x + threadIdx.x;
    if (line >= nlines) continue;
    const int i = 1 + line % (nr - 1);
    const int jl = line / (nr - 1);
    const int j = jl % nt, l = jl / nt;
    const long long st = (long long)nt * nr;
    const long long base = ((long long)l * ne * nt + j) * nr + i;
    // bounds-checked builds: the line's cells, its (I,J,L) entry and UE, its
    // EDOT column, the coefficient store's item
    if (!rg_ok(d, rg_item(d, item) && rg_span(base, ne, st, d.ncell) &&
                      rg_span((long long)m * nr * nt * d.npa + ((long long)l * nt + j) * nr + i, 1, 1,
                              (long long)d.nm * nr * nt * d.npa) &&
                      rg_span((long long)s * ne * nr + i, ne, nr, (long long)d.ns * ne * nr) &&
                      (!kCo || d.item0 + u.it < d.coef_items),
               kRgAdjE, line))
      continue;
    double* __restrict__ lam = d.lam + (long long)slot * d.ncell + base;
    const unsigned char* __restrict__ rl = rec + u.it * d.ncell + base;
    double* __restrict__ cst = kCo ? coef_ptr(d, u.it) + base : nullptr;
    const long long fij = ((long long)l * nt + j) * nr + i;
    const double wet = d.wet[fij];
    const double ue = d.ue[(long long)m * nr * nt * d.npa + fij];
    const double* __restrict__ edot = d.edot + (long long)s * ne * nr + i;
    const double* __restrict__ eb = d.eb + s * ne;
    const uint64_t betaf = beta_fix(dbits(d.betalim));
    const bool closed = d.flags & 1u;
    const int n = ne;
    const double out1 = lam[0];
    // what face K needs is loaded while face K-1 is worked on: its EDOT (or
    // the stored coefficient), the lambda and the record byte of the cell
    // entering, K+3; the record bytes of faces K..K+2 wait in recs
    auto rb = [&](int c) { return (unsigned)__ldg(rl + (long long)(c - 1) * st); };
    unsigned recs = rb(1) | rb(2) << 8 | rb(3) << 16;
    // wl(K) = le(K)/WE(K) for K = 2..NE, 0 elsewhere; window = cells K-1..K+2
    const double le2 = masked(lam, rl, st, rsh), le3 = masked(lam, rl, 2 * st, rsh);
    double nc, nlam;
    unsigned nrec;
    auto ahead = [&](int K) {
      const long long o = (long long)(min(K, n) - 1) * st;
      nc = (kCo == 2) ? cst[o] : edot[(long long)(min(K, n) - 1) * nr];
      const int c = min(K + 3, n);
      nlam = lam[(long long)(c - 1) * st];
      nrec = rb(c);
    };
    ahead(1);
    double wl0 = 0.0, wl1 = le2 * d.iwe[1], wl2 = le3 * d.iwe[2];
    double cm1 = 0.0, c0 = 0.0, c1 = le2, c2 = le3;
    double vin;  // the masked lambda of cell K+3 as face(K) leaves it
    auto face = [&](int K) {
      const double C = (kCo == 2) ? nc : nc * fma(eb[K - 1], wet, ue);
      if (kCo == 1) cst[(long long)(K - 1) * st] = C;
      recs |= nrec << 24;
      vin = ((nrec >> rsh) & kClipBit) ? 0.0 : nlam;
      ahead(K + 1);
      const int cs = (recs >> rsh) & 7;
      recs >>= 8;
      const double y = d.ide[K - 1];
      FaceMu fm;
      fm.sy = sig_62(dbits(y));
      fm.sh = 2045 - (int)(dbits(y) >> 52);
      face_acc_q(C * (wl1 - wl0), C, y, face_coef_mu(dbits(C), fm), cs, betaf, d.betalim, cm1,
                 c0, c1, c2);
    };
    auto shift = [&](double lec, double wl) {
      cm1 = c0; c0 = c1; c1 = c2; c2 = lec;
      wl0 = wl1; wl1 = wl2; wl2 = wl;
    };
    if (!closed) {
      face(1);
    } else {
      recs = recs >> 8 | nrec << 16;
      vin = ((nrec >> rsh) & kClipBit) ? 0.0 : nlam;
      ahead(2);
    }
    const double g0 = cm1;  // cell 0
    { const double lec = vin; shift(lec, lec * d.iwe[3]); }
    face(2);
    const double g1 = fma(d.kap[2 * s + 0], g0, cm1);  // cell 1 (+ kap0 * cell 0)
    { const double lec = vin; shift(lec, lec * d.iwe[4]); }
    face(3);
    lam[st] = fma(d.kap[2 * s + 1], g1, cm1);  // cell 2 (+ kap1 * cell 1)
    { const double lec = vin; shift(lec, lec * d.iwe[5]); }
    int K = 4;
    for (; K <= n - 3; ++K) {
      face(K);
      lam[(long long)(K - 2) * st] = cm1;
      const double lec = vin;
      shift(lec, lec * d.iwe[K + 2]);
    }
    for (; K <= n - 1; ++K) {
      face(K);
      lam[(long long)(K - 2) * st] = cm1;
      shift(0.0, 0.0);
    }
    if (!closed) face(n);
    lam[(long long)(n - 2) * st] = cm1;
    lam[(long long)(n - 1) * st] = c0;
    lam[0] = out1;
  }
}

// ----------------------------------------------------------------- DRIFTMU^T
// Cells 1..NPA: G(1) = F(2); faces 2..NPA-2; FBND(NPA-1) = F(NPA) (0 when
// closed); cells 2..NPA-1 updated; then F2(NPA) = F2new(NPA-1)*rho
// (NPA >= 9).
// loss (may be null): the CEX/ATMOL factor table the forward sweep applied
// to its result (cells L >= 2 of its lines; the table is 1 elsewhere), so
// lambda is scaled by it as it is read, the transposed loss fused in.
// kSplit adjacent lanes share a line (few lines, long serial chains, as in the
// forward sweep): lane r writes the cells b+1..lim of its segment (b = r*S,
// lim = (r+1)*S, S = NPA/kSplit; the first from cell 2, the last to NPA).
// Cell i collects from faces i-2..i+1, so a lane runs the faces b-1..lim+1,
// three more than its cells.  Every old value a lane needs from its
// neighbours' cells is loaded before a __syncwarp, no lane writes before it.
template <bool kLoss, int rsh, int kSplit>
__global__ void __launch_bounds__(128) k_adj_mu(Dev d, const unsigned char* __restrict__ rec,
                                                const double* __restrict__ loss) {
  const int nr = d.nr, nt = d.nt, ne = d.ne, npa = d.npa;
  const int nlines = (nr - 1) * nt * ne;
  const int lpb = blockDim.x / kSplit;
  const int r = kSplit > 1 ? (int)threadIdx.x % kSplit : 0, seg = npa / kSplit;
  const bool last = r == kSplit - 1;
  for (Unit u((nlines + lpb - 1) / lpb); u.ok(d); u.next(d)) {
    const int2 item = d.items[u.it];
    const int m = item.x, s = item.y, slot = m * d.ns + s;
    const int line = u.b * lpb + (int)threadIdx.x / kSplit;
    const int lc = line < nlines ? line : 0;
    const int i = 1 + lc % (nr - 1);
    const int jk = lc / (nr - 1);
    const int j = jk % nt;
    const long long st = (long long)ne * nt * nr;
    const long long off = (long long)jk * nr + i;
    // bounds-checked builds: the line's cells, its WM and UM columns (the
    // lanes sharing a line test the same)
    const bool active = line < nlines &&
        rg_ok(d, rg_item(d, item) && rg_span(off, npa, st, d.ncell) &&
                      rg_span((long long)j * nr + i, npa, (long long)nt * nr, (long long)nr * nt * npa) &&
                      rg_span((long long)m * nt * nr * npa + (long long)j * nr + i, npa, (long long)nt * nr,
                              (long long)d.nm * nr * nt * npa),
               kRgAdjMu, line);
    double* __restrict__ lam = d.lam + (long long)slot * d.ncell + off;
    const unsigned char* __restrict__ rl = rec + u.it * d.ncell + off;
    const long long sij = (long long)nt * nr;
    const long long fij = (long long)j * nr + i;
    const double* __restrict__ wm = d.wm + fij;
    const double* __restrict__ um = d.um + (long long)m * nt * nr * npa + fij;
    const double ekv = d.ek[s * ne + jk / nt];
    const uint64_t betaf = beta_fix(dbits(d.betalim));
    const bool closed = d.flags & 1u;
    const int n = npa;
    const double* __restrict__ iwmu = d.iwmu;
#define MC(L) fma(ekv, wm[(long long)((L)-1) * sij], um[(long long)((L)-1) * sij])
    const double* __restrict__ ls = kLoss ? loss + (long long)s * d.ncell + off : nullptr;
    auto lv = [&](int L) {  // lambda of cell L (>= 2), scaled by the loss factor
      const double v = lam[(long long)(L - 1) * st];
      return kLoss ? v * ls[(long long)(L - 1) * st] : v;
    };
    auto mle = [&](int L) {  // masked as in masked(): both loads issued unconditionally
      const double v = lv(L);
      return ((__ldg(rl + (long long)(L - 1) * st) >> rsh) & kClipBit) ? 0.0 : v;
    };
    // the lane's cells b+1..lim, its faces f0..fe; loads end at cell le1, the
    // two cells after it are eA, eB: the next lane's first ones, or for the
    // last lane NPA-1, which takes rho * lambda(NPA) (F2(NPA) = F2new(NPA-1)*rho),
    // and NPA, which has no term of its own
    const int b = r ? r * seg : 1, lim = last ? n : (r + 1) * seg;
    const int f0 = r ? b - 1 : 2, fe = last ? n - 2 : lim + 1, le1 = last ? n - 2 : lim;
    double eA = 0.0, eB = 0.0, v0 = 0.0, v1 = 0.0, v2 = 0.0;
    if (active) {
      if (last) {
        eA = ((rl[(long long)(n - 2) * st] >> rsh) & kClipBit) ? 0.0 : fma(d.rho[fij], lv(n), lv(n - 1));
      } else {
        eA = mle(lim + 1);
        eB = mle(lim + 2);
      }
      v0 = mle(f0);      // cells f0, f0+1, f0+2
      v1 = mle(f0 + 1);
      v2 = mle(f0 + 2);
    }
    if (kSplit > 1) __syncwarp();
    if (active) {
      double wl0 = v0 * iwmu[f0 - 1], wl1 = v1 * iwmu[f0], wl2 = v2 * iwmu[f0 + 1];
      // window: cells f-1..f+2 (a cell before b+1 is another lane's)
      double cm1 = 0.0, c0 = r ? 0.0 : v0, c1 = r ? 0.0 : v1, c2 = v2;
      double first = 0.0;  // cell 1 -> cell 2 (G(1) = F(2))
      // what face f needs is loaded while face f-1 is worked on: its WM and
      // UM, the cell entering (its lambda, factor and record byte, for the
      // clip; cells past le1 are read at le1 and not used); the record bytes
      // of faces f..f+2 wait in recs
      auto rb = [&](int c) { return (unsigned)__ldg(rl + (long long)(c - 1) * st); };
      unsigned recs = rb(f0) | rb(f0 + 1) << 8 | rb(f0 + 2) << 16;
      double nwm, num, nlam, nls = 1.0;
      unsigned nrec;
      auto ahead = [&](int f) {
        const int fc = min(f, fe), c = min(f + 3, le1);
        const long long o = (long long)(c - 1) * st;
        nwm = wm[(long long)(fc - 1) * sij];
        num = um[(long long)(fc - 1) * sij];
        nlam = lam[o];
        if (kLoss) nls = ls[o];
        nrec = rb(min(f + 3, n));
      };
      ahead(f0);
      for (int f = f0; f <= fe; ++f) {
        const double C = fma(ekv, nwm, num);
        const double vin = nlam, lin = nls;
        recs |= nrec << 24;
        ahead(f + 1);
        const int cs = (recs >> rsh) & 7;
        // the cell entering next
        double lec = eA;
        if (f + 3 <= le1) {
          lec = ((recs >> (24 + rsh)) & kClipBit) ? 0.0 : (kLoss ? vin * lin : vin);
        } else {
          eA = eB;
          eB = 0.0;
        }
        recs >>= 8;
        face_acc_q(C * (wl1 - wl0), C, d.idmu[f - 1], face_coef_mu(dbits(C), d.mubin[f - 1]), cs, betaf,
                   d.betalim, cm1, c0, c1, c2);
        if (r == 0 && f == 2) first = cm1;
        if (f - 1 > b) lam[(long long)(f - 2) * st] = (r == 0 && f == 3) ? cm1 + first : cm1;
        cm1 = c0; c0 = c1; c1 = c2; c2 = lec;
        wl0 = wl1; wl1 = wl2; wl2 = lec * iwmu[min(f + 3, n) - 1];
      }
      if (last) {
        // window: cells NPA-2, NPA-1, NPA; FBND(NPA-1) = F(NPA): Pb(NPA-1) = -le(NPA-1)/WMU
        if (!closed) c1 -= MC(n - 1) * wl0;
        lam[(long long)(n - 3) * st] = cm1;
        lam[(long long)(n - 2) * st] = c0;
        lam[(long long)(n - 1) * st] = c1;
      }
    }
#undef MC
  }
}

// Lanes per transposed pitch-angle line, by the number of lines.  Measured
// backward ms a call (GB300, 20x25x35x72) with 1, 2, 4 lanes: one species
// (3.4 warps an SM with one lane) 0.374, 0.315, 0.291; four (14) 0.608, 0.560,
// 0.588; four members of four (55) 2.05, 2.10, 2.28.
static int adj_mu_lanes(const Dev& d) {
  const long long warps = (long long)(d.nr - 1) * d.nt * d.ne * d.nlist / 32;
  if (d.npa < 24) return 1;  // segments of at least six cells
  return warps < 8LL * d.nsm ? 4 : (warps < 24LL * d.nsm ? 2 : 1);
}

void launch_adj_sweep(const Dev& d, int w, const unsigned char* rec, int rsh, cudaStream_t st, int co,
                      const double* loss) {
  const int blk = 128;
  int nl;
  switch (w) {
    case 0: nl = d.nt * d.ne * d.npa; break;
    case 1: nl = (d.nr - 1) * d.ne * d.npa; break;
    case 2: nl = (d.nr - 1) * d.nt * d.npa; break;
    default: nl = (d.nr - 1) * d.nt * d.ne; break;
  }
  dim3 g((nl + blk - 1) / blk, d.nitems, 1);
  // the record nibble is a template parameter: 0 low (reverse half), 4 high
  auto go = [&](auto sh) {
    constexpr int R = decltype(sh)::value;
    switch (w) {
      case 0: k_adj_r<R><<<g, blk, adj_r_smem(d, blk), st>>>(d, rec); break;
      case 1: k_adj_p<R><<<g, blk, 0, st>>>(d, rec); break;
      case 2:
        if (co == 1) k_adj_e<1, R><<<g, blk, 0, st>>>(d, rec);
        else if (co == 2) k_adj_e<2, R><<<g, blk, 0, st>>>(d, rec);
        else k_adj_e<0, R><<<g, blk, 0, st>>>(d, rec);
        break;
      default: {
        const int lanes = adj_mu_lanes(d);
        const dim3 gm((nl * lanes + blk - 1) / blk, d.nitems, 1);
        if (lanes == 4) {
          if (loss) k_adj_mu<true, R, 4><<<gm, blk, 0, st>>>(d, rec, loss);
          else k_adj_mu<false, R, 4><<<gm, blk, 0, st>>>(d, rec, nullptr);
        } else if (lanes == 2) {
          if (loss) k_adj_mu<true, R, 2><<<gm, blk, 0, st>>>(d, rec, loss);
          else k_adj_mu<false, R, 2><<<gm, blk, 0, st>>>(d, rec, nullptr);
        } else {
          if (loss) k_adj_mu<true, R, 1><<<gm, blk, 0, st>>>(d, rec, loss);
          else k_adj_mu<false, R, 1><<<gm, blk, 0, st>>>(d, rec, nullptr);
        }
        break;
      }
    }
  };
  if (rsh) go(std::integral_constant<int, 4>());
  else go(std::integral_constant<int, 0>());
}

// ---------------------------------------------------------- ram_run tail^T
// Forward order: F2(:,:,NT,:,:) = F2(:,:,1,:,:); mask; ANISCH's
// F2(I,J,K,1) = F2(I,J,K,2) (I, K >= 2).  Adjoint in reverse.
__global__ void k_adj_anisch(Dev d) {
  const long long n = (long long)(d.nr - 1) * d.nt * (d.ne - 1);
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int2 item = d.items[blockIdx.y];
  const int slot = item.x * d.ns + item.y;
  const int i = 1 + (int)(t % (d.nr - 1));
  const int j = (int)((t / (d.nr - 1)) % d.nt);
  const int k = 1 + (int)(t / ((long long)(d.nr - 1) * d.nt));
  double* lam = d.lam + (long long)slot * d.ncell + ((long long)k * d.nt + j) * d.nr + i;
  const long long st = (long long)d.ne * d.nt * d.nr;
  lam[st] += lam[0];
  lam[0] = 0.0;
}

__global__ void k_adj_copy_mask(Dev d, int any_outside) {
  const long long n = (long long)d.nr * d.ne * d.npa;
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int2 item = d.items[blockIdx.y];
  const int slot = item.x * d.ns + item.y;
  const int i = (int)(t % d.nr);
  const long long kl = t / d.nr;
  double* lam = d.lam + (long long)slot * d.ncell + kl * d.nt * d.nr + i;
  if (any_outside)
    for (int j = 0; j < d.nt; ++j)
      if (d.outside[(long long)j * d.nr + i] == 1) lam[(long long)j * d.nr] = 0.0;
  lam[0] += lam[(long long)(d.nt - 1) * d.nr];
  lam[(long long)(d.nt - 1) * d.nr] = 0.0;
}

void launch_adj_tail(const Dev& d, cudaStream_t st) {
  long long n1 = (long long)(d.nr - 1) * d.nt * (d.ne - 1);
  k_adj_anisch<<<dim3((unsigned)((n1 + 255) / 256), d.nitems), 256, 0, st>>>(d);
  long long n2 = (long long)d.nr * d.ne * d.npa;
  k_adj_copy_mask<<<dim3((unsigned)((n2 + 255) / 256), d.nitems), 256, 0, st>>>(d, (d.flags >> 31) & 1u);
}

// ------------------------------------------------------------- observations
// flux = F2/FFACTOR/FNHS (src/ModRamRun.f90:214) at bin (K, L), bilinear in
// (L-shell, MLT) over the four cells (i0|i0+1, j0|j1).
__device__ __forceinline__ double obs_cell_factor(const Dev& d, int s, int i, int j, int k, int l) {
  const double ff = d.ffactor[(long long)s * d.nr * d.ne * d.npa + ((long long)l * d.ne + k) * d.nr + i];
  const double fh = d.fnhs[((long long)l * d.nt + j) * d.nf + i];
  return ff * fh;
}

__global__ void k_obs_fwd(Dev d, const ObsDev* __restrict__ obs, int nobs, int call, double* fm,
                          double* J) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nobs) return;
  const ObsDev o = obs[t];
  if (o.call != call) return;
  const int s = o.slot % d.ns;
  const double* f2 = d.f2 + (long long)o.slot * d.ncell;
  double v = 0.0;
  for (int a = 0; a < 2; ++a)
    for (int b = 0; b < 2; ++b) {
      const int i = o.i0 + a, j = b ? o.j1 : o.j0;
      const double w = (a ? o.wi : 1.0 - o.wi) * (b ? o.wj : 1.0 - o.wj);
      const long long c = (((long long)o.l * d.ne + o.k) * d.nt + j) * d.nr + i;
      const double ff = d.ffactor[(long long)s * d.nr * d.ne * d.npa + ((long long)o.l * d.ne + o.k) * d.nr + i];
      const double fh = d.fnhs[((long long)o.l * d.nt + j) * d.nf + i];
      v += w * (f2[c] / ff / fh);
    }
  fm[t] = v;
  const double r = log(v) - o.log_obs;
  atomicAdd(&J[o.member], r * r);
}

__global__ void k_obs_adj(Dev d, const ObsDev* __restrict__ obs, int nobs, int call,
                          const double* __restrict__ fm) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nobs) return;
  const ObsDev o = obs[t];
  if (o.call != call || o.item < d.item0 || o.item >= d.item0 + d.nitems) return;  // call c, this group
  const int s = o.slot % d.ns;
  const double v = fm[t];
  const double g = 2.0 * (log(v) - o.log_obs) / v;
  for (int a = 0; a < 2; ++a)
    for (int b = 0; b < 2; ++b) {
      const int i = o.i0 + a, j = b ? o.j1 : o.j0;
      const double w = (a ? o.wi : 1.0 - o.wi) * (b ? o.wj : 1.0 - o.wj);
      const long long c = (((long long)o.l * d.ne + o.k) * d.nt + j) * d.nr + i;
      atomicAdd(&d.lam[(long long)o.slot * d.ncell + c], g * w / obs_cell_factor(d, s, i, j, o.k, o.l));
    }
}

void launch_obs_fwd(const Dev& d, const ObsDev* obs, int nobs, int call, double* fm, double* J,
                    cudaStream_t st) {
  if (nobs > 0) k_obs_fwd<<<(nobs + 127) / 128, 128, 0, st>>>(d, obs, nobs, call, fm, J);
}
void launch_obs_adj(const Dev& d, const ObsDev* obs, int nobs, int call, const double* fm,
                    cudaStream_t st) {
  if (nobs > 0) k_obs_adj<<<(nobs + 127) / 128, 128, 0, st>>>(d, obs, nobs, call, fm);
}

// Order-independent digest of a branch record: two sums (mod 2^32) of
// position-mixed 32-bit hashes of its 32-bit words, read 16 bytes at a time
// (a ragged tail byte by byte).  Equal digests of two runs mean an
// unchanged pattern with overwhelming probability.  One atomic a block: with
// one a warp, 8192 to the same address, 12.6 us a call (20 MB of record),
// so 9.4.
__device__ __forceinline__ unsigned mix32(unsigned w, unsigned long long i, unsigned c1, unsigned c2) {
  unsigned h = (w + (unsigned)i * 0x9E3779B9u + (unsigned)(i >> 32)) * c1;
  h ^= h >> 15;
  h *= c2;
  return h ^ (h >> 13);
}

__global__ void __launch_bounds__(256) k_digest(const unsigned char* __restrict__ rec, long long n, unsigned long long* out) {
  unsigned lo = 0u, hi = 0u;
  const bool al = ((unsigned long long)rec & 15ULL) == 0ULL;
  const long long n16 = al ? n / 16 : 0;
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long nth = (long long)gridDim.x * blockDim.x;
  const uint4* r4 = reinterpret_cast<const uint4*>(rec);
  for (long long c = tid; c < n16; c += nth) {
    const uint4 v = r4[c];
    const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const unsigned long long i = 4ULL * c + q;
      lo += mix32(w[q], i, 0x85EBCA6Bu, 0xC2B2AE35u);
      hi += mix32(w[q], i, 0x27D4EB2Fu, 0x165667B1u);
    }
  }
  for (long long b = 16 * n16 + tid; b < n; b += nth) {
    const unsigned long long i = 0x100000000ULL + (unsigned long long)b;
    lo += mix32(rec[b], i, 0x85EBCA6Bu, 0xC2B2AE35u);
    hi += mix32(rec[b], i, 0x27D4EB2Fu, 0x165667B1u);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo += __shfl_xor_sync(0xffffffffu, lo, o);
    hi += __shfl_xor_sync(0xffffffffu, hi, o);
  }
  __shared__ unsigned long long sh[8];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = ((unsigned long long)hi << 32) + lo;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0ULL;
    for (int w = 0; w < 8; ++w) t += sh[w];
    atomicAdd(out, t);
  }
}

void launch_digest(const unsigned char* rec, long long n, unsigned long long* out, cudaStream_t st) {
  k_digest<<<1024, 256, 0, st>>>(rec, n, out);
}

}  // namespace ramgpu

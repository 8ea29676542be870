// sweeps.cu -- the four operator-split flux-limited upwind sweeps of RAM.
//
// Each kernel advances whole lines in place: thread (blockIdx.x*blockDim.x +
// threadIdx.x) owns one line of the swept axis, blockIdx.y indexes the
// (member, species) work item.  The line is streamed once through a rolling
// window G(f-1..f+2) kept in registers, so every F2 value is read once and
// written once per sweep.  The face arithmetic follows the reference:
//   DRIFTR  src/ModRamDrift.f90:95-198
//   DRIFTP  src/ModRamDrift.f90:204-279
//   DRIFTE  src/ModRamDrift.f90:285-376
//   DRIFTMU src/ModRamDrift.f90:382-473
// with the face coefficients taken from separable tables built in tables.cu
// (C = A(I,J) + G(I,J,L)*k(K) etc.).  The FP64 unit was the limit: sign, abs
// and limiter tests run on bit patterns and the whole face flux is formed in
// 64-bit fixed point (face.cuh), which leaves three FP64 operations a face:
// the coefficient and the two of the update (DRIFTMU's forward half
// multiplies the loss factor too).
#include <string.h>

#include <type_traits>

#include "ramgpu_internal.cuh"
#include "face.cuh"
#include "kernels.cuh"

namespace ramgpu {

// Branch records hold two sweeps per byte, four bits each (three case bits
// and the clip bit): a call's forward-half sweep in the high nibble
// (rsh = 4), written first, and the reverse-half sweep of the same
// direction in the low one, which ORs its code into that byte.  (The
// reverse half is transposed first; its nibble is the cheaper one to read.)
__device__ __forceinline__ unsigned rget(const unsigned char* p, int rsh) { return (unsigned)*p >> rsh; }
// The forward half writes the high nibble (rsh 4), the reverse half adds the
// low one to `old`, the byte as rold read it before the face's arithmetic (at
// the store, every face waited for the read).
__device__ __forceinline__ unsigned rold(const unsigned char* p, int rsh) { return rsh ? 0u : (unsigned)*p; }
__device__ __forceinline__ void rput(unsigned char* p, int rsh, unsigned old, unsigned v) {
  *p = (unsigned char)(rsh ? (v << 4) : (old | v));
}

// phi of a face by the FP64 unit, for what face_flux leaves out.  Out of
// line, so that its FP64 instructions are not issued predicated off.
// x, dd: the reference's X and D, u and d: the cells upwind and downwind by
// C's sign bit.  That differs from C < 0 for -0 alone, whose flux comes from
// F(f), here d, as for +0: it carries nothing but a NaN.  kRec 2: with the
// branch rcs.
struct PhiCase {
  double phi;
  int cs;
};
template <int kRec>
static __device__ __noinline__ PhiCase face_phi_fp64(double x, double dd, double u, double d, double c, double mh,
                                                     double beta, int rcs) {
  const BetaBits b(beta);
  const bool neg = is_neg(c);
  const double a = fma(c, mh, neg ? -0.5 : 0.5);
  PhiCase r;
  r.cs = rcs;
  double fb = kRec == 2 ? face_value_frozen(x, dd, u, a, b, rcs)
                        : face_value_case(x, babs_bits(b, x), dd, babs_bits(b, dd), u, a, r.cs);
  if (dbits(c) == kSignMask) fb = d;
  r.phi = __dmul_rn(c, fb);
  return r;
}

// Flux of a limited face (face.cuh) with the prepared coefficient q of C.
// v: C or a factor of it that vanishes with it; cf(): C, and mh(): -1/2 (R, P)
// or -1/2 over the bin width, formed only for the FP64 form.  kRec 1: cs is
// the branch taken; 2: the recorded branch cs is applied (the same bits as the
// recording sweep's where that is the branch the values select).  over():
// called where U >= 1 or C is not finite.
struct NoOver {
  __device__ __forceinline__ void operator()() const {}
};
template <int kRec, bool kB32, class C, class M, class O = NoOver>
__device__ __forceinline__ double face_phi(double uu, double u, double d, double v, const FaceCoef& q, double beta,
                                           uint64_t betaf, int& cs, C&& cf, M&& mh, O&& over = O()) {
  bool special;
  int taken = 0;
  double phi = bitsd(
      kRec == 2 ? face_flux_frozen<kB32>(dbits(uu), dbits(u), dbits(d), q, betaf, cs, special)
                : face_flux<kRec == 1, kB32>(dbits(uu), dbits(u), dbits(d), q, betaf, special, taken));
  if (kRec == 1) cs = taken;
  if (special) {
    if (q.bad < 0) over();
    if ((kRec != 2 || cs == 0) && face_plain(dbits(uu), dbits(u), dbits(d), dbits(v))) {
      if (kRec == 1) cs = 0;
      if (q.bad < 0 || (dbits(u) != 0ULL && (dbits(v) << 1) != 0ULL)) return __dmul_rn(cf(), u);
      return bitsd((bits64)q.sign << 32);
    }
    const bool neg = q.sign != 0;
    const PhiCase r = face_phi_fp64<kRec>(neg ? u - d : d - u, neg ? uu - u : u - uu, u, d, cf(), mh(), beta, cs);
    phi = r.phi;
    if (kRec == 1) cs = r.cs;
  }
  return phi;
}

// The line's largest Courant number, as the face with the smallest 1 - U:
// its quotient is formed once, after the line, in FP64 (a few operations a
// line; every face's took 16 integer instructions and cut the quotient).
// 1 - U has units of 2^-63, so another face's quotient may be larger than the
// one formed, by less than 2^-62/U of it: below a rounding from U = 2^-9 on.
// A limit just below its cap of 1e4 s has U = FracCFL*DTs/1e4, so up to 5e-16
// at DTs = 5 s and 3e-14 at 0.1 s (the parity bar is 1e-12), while one below
// 40 s, as sets the next step, is within a rounding at either.  Telling such
// faces apart cost more than it gives, four species on 20x25x35x72 and
// 40x49x70x144, ms a call: 0.3625, 4.634 as it is; 0.368, 4.668 with the line's
// quotients all formed where two faces tie; 0.378, 4.717 where the largest U
// is below 2^-10 and the slot's limit is not above it yet; 0.376, 4.913 with
// the quotient of a face that ties formed at once.
struct Largest {
  uint64_t a63 = 1ULL << 63;
  int at = 0;
  __device__ __forceinline__ void see(const FaceCoef& q, int f) {
    const bool less = q.a63 < a63;
    a63 = less ? q.a63 : a63;
    at = less ? f : at;
  }
};

// p[i * st], i >= 0, as one multiply-add of 32-bit factors, where a 64-bit
// index takes five instructions: the stride in cells (below 2^32: a line of
// larger ones does not fit the memory) or, where it is below 2^29, in bytes.
template <class T>
__device__ __forceinline__ T& strided(T* p, int i, unsigned st) {
  return *(T*)((uintptr_t)p + (uint64_t)((unsigned)i * (unsigned)sizeof(T)) * st);
}
template <class T>
__device__ __forceinline__ T& strided_b(T* p, int i, unsigned bytes) {
  return *(T*)((uintptr_t)p + (uint64_t)(unsigned)i * bytes);
}

// V consecutive doubles, 8*V-byte aligned.
template <int V>
struct Vec {
  double x[V];
  __device__ __forceinline__ void load(const double* p) {
    if (V == 4)
      asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                   : "=d"(x[0]), "=d"(x[1]), "=d"(x[V > 2 ? 2 : 0]), "=d"(x[V > 2 ? 3 : 0]) : "l"(p) : "memory");
    else
      asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(x[0]), "=d"(x[1]) : "l"(p) : "memory");
  }
  __device__ __forceinline__ void store(double* p) const {
    if (V == 4)
      asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(x[0]), "d"(x[1]), "d"(x[V > 2 ? 2 : 0]),
                   "d"(x[V > 2 ? 3 : 0]) : "memory");
    else
      asm volatile("st.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(x[0]), "d"(x[1]) : "memory");
  }
};

// ----------------------------------------------------------------- DRIFTR
// Line (J,K,L) along I = 1..NR.  Faces 2..NR-1 (and NR on inflow lines).
// kCfl (R, P): 1 the largest |C| of the line, 2 of its cells inside the
// magnetopause, where some lie outside.
// A thread's line is contiguous, the lanes' lines 8*NR bytes apart, so a load
// or store of one cell a lane touches 32 sectors: with V = 4 or 2 (NR a
// multiple of it: the lines are aligned) cells, GRT and CR move V at a time,
// whole sectors for V = 4, through a few slots of shared memory per thread
// that the face loop reads and writes one at a time (a loop over V unrolled
// faces does not fit the instruction cache as well).  Cells are loaded two
// groups ahead.  No barrier: a thread touches its own slots only.
template <int kCfl, int kRec, bool kB32, int V>
__global__ void __launch_bounds__(256, 4) k_sweep_r(Dev d, double dts, unsigned char* __restrict__ rec, int rsh) {
  chain_enter();
  extern __shared__ double slots[];
  const int nr = d.nr, nt = d.nt, ne = d.ne;
  // the lines of the L window [lw0, lw1) (all of them unless a pipeline
  // runs the step plane chunk by plane chunk): L is the slowest index
  const int line0 = d.lw0 * nt * ne;
  const int nlines = nt * ne * (d.lw1 - d.lw0);
  for (Unit u((nlines + blockDim.x - 1) / blockDim.x); u.ok(d); u.next(d)) {
    const int2 item = d.items[u.it];
    const int m = item.x, s = item.y, slot = m * d.ns + s;
    const int line = line0 + u.b * blockDim.x + threadIdx.x;
    unsigned long long q = kBits1em10;  // CFL quotient bits: |C| at least 1e-10
    unsigned nclip = 0;  // clip events (kRec == kRecCount)
    // bounds-checked builds: the line's cells, its GRT and CR rows
    const bool lok = line >= line0 + nlines ||
        rg_ok(d, rg_item(d, item) && rg_span((long long)line * nr, nr, 1, d.ncell) &&
                     rg_span(((long long)(line / (nt * ne)) * nt + line % nt) * nr, nr, 1, (long long)nr * nt * d.npa) &&
                     rg_span(((long long)item.x * nt + line % nt) * nr, nr, 1, (long long)d.nm * nr * nt),
              kRgSweepR, line);
    if (line < line0 + nlines && lok) {
      const int j = line % nt;
      const int l = line / (nt * ne);
      double* __restrict__ fl = d.f2 + (long long)slot * d.ncell + (long long)line * nr;
      // branch record of the frozen-limiter adjoint: one byte per face/cell
      unsigned char* __restrict__ rl = (kRec == 1 || kRec == 2) ? rec + u.it * d.ncell + (long long)line * nr : nullptr;
      const double* __restrict__ grt = d.grt + ((long long)l * nt + j) * nr;
      const double* __restrict__ cr = d.cr + ((long long)m * nt + j) * nr;
      const int* __restrict__ outside = d.outside + (long long)j * nr;
      const double p4 = d.p4[s * ne + (line / nt) % ne];
      const double beta = d.betalim;
      const uint64_t betaf = beta_fix(dbits(beta));
      auto mh = [] { return -0.5; };
      auto limit = [&](int f, double c) {
        if (kCfl == 1 || (kCfl == 2 && outside[f - 1] == 0)) q = cfl_bits(c, q);
      };
      const bool closed = d.flags & 1u;

      const int k = (line / nt) % ne;
      const double cN = fma(grt[nr - 1], p4, cr[nr - 1]);
      const double cNm = fma(grt[nr - 2], p4, cr[nr - 2]);
      const bool inflow = is_neg(cN);
      // F(NR+1), F(NR+2): boundary ghosts on inflow lines.  On an outflow line
      // F(NR+1) is read only by face NR-1 when it is upwinded from the right,
      // and then it is the stale value of the most recent inflow line in the
      // reference's K->L->J loop order (F persists across lines in DRIFTR).
      double g1 = 0.0, g2 = 0.0;
      if (inflow) {  // line index = (L*NE+K)*NT+J, the layout of FGEOS(J,K,L)
        g1 = ghost_value(d, slot, j, k, l, d.conf1);
        g2 = ghost_value(d, slot, j, k, l, d.conf2);
      } else if (is_neg(cNm)) {
        g1 = stale_ghost(d, m, slot, j, k, l, p4);
      }
      double gm, g0, gp, phi_prev;
      // face 1: FBND(1) = 0 (outflow) or F(2) (inflow)
      auto begin = [&](double c) {
        limit(1, c);
        phi_prev = c * ((inflow && !closed) ? g0 : 0.0);
      };
      // face f, 2 <= f <= NR-1: the new cell f
      auto step = [&](int f, double c, double gpp) {
        limit(f, c);
        const unsigned old = kRec == 1 ? rold(rl + (f - 1), rsh) : 0u;
        const bool neg = hi32(dbits(c)) < 0;  // (-0: face_phi_fp64)
        int cs = kRec == 2 ? (int)(rget(rl + (f - 1), rsh) & 7) : 0;
        const double phi = face_phi<kRec, kB32>(neg ? gpp : gm, neg ? gp : g0, neg ? g0 : gp, c, face_coef(dbits(c)), beta,
                                                betaf, cs, [&] { return c; }, mh);
        const double raw = (g0 - phi) + phi_prev;
        const double v = (kRec == 2) ? clip_frozen(raw, rget(rl + (f - 1), rsh)) : clip(raw);
        if (kRec == kRecCount) nclip += is_neg(raw);
        if (kRec == 1) rput(rl + (f - 1), rsh, old, cs | (is_neg(raw) ? kClipBit : 0));
        phi_prev = phi;
        gm = g0; g0 = gp; gp = gpp;
        return v;
      };
      double* slot0 = slots + threadIdx.x;
      const int bd = blockDim.x, ng = nr / V;
      if (V == 1) {
        gm = fl[0]; g0 = fl[1]; gp = fl[2];
        begin(fma(grt[0], p4, cr[0]));
        for (int f = 2; f <= nr - 1; ++f) {
          const double gpp = (f + 2 <= nr) ? fl[f + 1] : g1;
          fl[f - 1] = step(f, (f == nr - 1) ? cNm : fma(grt[f - 1], p4, cr[f - 1]), gpp);
        }
      } else {
        // slots 0..2V-1: cells, cell n at (n-1) mod 2V; 2V..3V-1: the group's
        // coefficients, replaced by its new cells
        constexpr int W = V > 1 ? V : 2;
        Vec<W> x;
        auto fill = [&](int g) {  // group g into its half (the ghosts after the last)
          if (g < ng)
            for (int t = 0; t < W; ++t) slot0[((g & 1) * W + t) * bd] = x.x[t];
          else if (g == ng) {
            slot0[(g & 1) * W * bd] = g1;
            slot0[((g & 1) * W + 1) * bd] = g2;
          }
        };
        x.load(fl);
        gm = x.x[0]; g0 = x.x[1];
        fill(0);
        if (ng > 1) x.load(fl + W);
        fill(1);
        gp = slot0[2 * bd];
        if (ng > 2) x.load(fl + 2 * W);
        for (int g = 0; g < ng; ++g) {
          Vec<W> a, b;
          a.load(grt + g * W);
          b.load(cr + g * W);
          for (int t = 0; t < W; ++t) slot0[(2 * W + t) * bd] = fma(a.x[t], p4, b.x[t]);
          int t = 0;
          if (g == 0) {
            begin(slot0[2 * W * bd]);
            slot0[2 * W * bd] = gm;  // cell 1 keeps its value
            t = 1;
          }
          const int te = g == ng - 1 ? W - 1 : W;
#pragma unroll 1
          for (; t < te; ++t) {
            double* cell = slot0 + (2 * W + t) * bd;
            const int f = g * W + t + 1;
            *cell = step(f, *cell, slot0[((f + 1) & (2 * W - 1)) * bd]);
          }
          if (g < ng - 1) {
            for (int t2 = 0; t2 < W; ++t2) a.x[t2] = slot0[(2 * W + t2) * bd];
            a.store(fl + g * W);
            fill(g + 2);
            if (g + 3 < ng) x.load(fl + (g + 3) * W);
          }
        }
      }
      // face NR (g0 = F(NR), gp = F(NR+1)): limited on inflow lines, F(NR)
      // on outflow lines
      limit(nr, cN);
      int csn = kRec == 2 ? (int)(rget(rl + (nr - 1), rsh) & 7) : 0;
      double phin = 0.0;
      if (!closed)
        phin = inflow ? face_phi<kRec, kB32>(g2, g1, g0, cN, face_coef(dbits(cN)), beta, betaf, csn, [&] { return cN; }, mh)
                      : mul_rn_int(cN, g0);
      const double rawn = (g0 - phin) + phi_prev;
      const double vn = (kRec == 2) ? clip_frozen(rawn, rget(rl + (nr - 1), rsh)) : clip(rawn);
      if (V == 1) {
        fl[nr - 1] = vn;
      } else {
        constexpr int W = V > 1 ? V : 2;
        Vec<W> a;
        for (int t = 0; t < W - 1; ++t) a.x[t] = slot0[(2 * W + t) * bd];
        a.x[W - 1] = vn;
        a.store(fl + nr - W);
      }
      if (kRec == kRecCount) nclip += is_neg(rawn);
      if (kRec == 1) rput(rl + (nr - 1), rsh, rold(rl + (nr - 1), rsh), csn | (is_neg(rawn) ? kClipBit : 0));
    }
    if (kRec == kRecCount) warp_atomic_add(&d.clipq[slot], nclip);
    if (kCfl) warp_atomic_max(&d.cflq[slot * 4 + 0], q);
  }
}

// ----------------------------------------------------------------- DRIFTP
// Line (I,K,L), I = 2..NR, along J = 1..NT, periodic with J=1 == J=NT.
// Held to 64 registers (32 warps an SM): on 40x49x70x144 553 us a launch
// against 608 with 78; running the next face's coefficient one iteration
// ahead, or unrolling by 2 or 4, took 594 to 703.
template <int kCfl, int kRec, bool kB32>
__global__ void __launch_bounds__(256, 4) k_sweep_p(Dev d, double dts, unsigned char* __restrict__ rec, int rsh) {
  chain_enter();
  const int nr = d.nr, nt = d.nt, ne = d.ne;
  const int line0 = d.lw0 * (nr - 1) * ne;  // the L window, as in DRIFTR
  const int nlines = (nr - 1) * ne * (d.lw1 - d.lw0);
  for (Unit u((nlines + blockDim.x - 1) / blockDim.x); u.ok(d); u.next(d)) {
    const int2 item = d.items[u.it];
    const int m = item.x, s = item.y, slot = m * d.ns + s;
    const int line = line0 + u.b * blockDim.x + threadIdx.x;
    unsigned long long q = kBits1em10;  // CFL quotient bits: |C| at least 1e-10
    unsigned nclip = 0;  // clip events (kRec == kRecCount)
    // bounds-checked builds: the line's cells, its GPT and CA columns
    const bool lok = line >= line0 + nlines ||
        rg_ok(d, rg_item(d, item) &&
                     rg_span((long long)(line / (nr - 1)) * nt * nr + 1 + line % (nr - 1), nt, nr, d.ncell) &&
                     rg_span((long long)(line / (nr - 1) / ne) * nt * nr + 1 + line % (nr - 1), nt, nr,
                             (long long)nr * nt * d.npa) &&
                     rg_span((long long)item.x * nt * nr + 1 + line % (nr - 1), nt, nr, (long long)d.nm * nr * nt),
              kRgSweepP, line);
    if (line < line0 + nlines && lok) {
      const int i = 1 + line % (nr - 1);
      const int kl = line / (nr - 1);
      const int k = kl % ne, l = kl / ne;
      const long long st = nr;  // stride between consecutive J
      const unsigned st8 = (unsigned)nr * 8u;
      double* __restrict__ fl = d.f2 + (long long)slot * d.ncell + ((long long)kl * nt) * nr + i;
      unsigned char* __restrict__ rl =
          (kRec == 1 || kRec == 2) ? rec + u.it * d.ncell + ((long long)kl * nt) * nr + i : nullptr;
      const double* __restrict__ gpt = d.gpt + ((long long)l * nt) * nr + i;
      const double* __restrict__ ca = d.ca + ((long long)m * nt) * nr + i;
      const int* __restrict__ outside = d.outside + i;
      const double p2 = d.p2[((long long)s * ne + k) * nr + i];
      const double beta = d.betalim;
      const uint64_t betaf = beta_fix(dbits(beta));
      auto mh = [] { return -0.5; };
  #define GJ(J) fl[(long long)((J)-1) * st]
  #define CJ(J) fma(gpt[(long long)((J)-1) * nr], p2, ca[(long long)((J)-1) * nr])
      const double G1 = GJ(1), G2 = GJ(2), G3 = GJ(3), GNm = GJ(nt - 1), GN = GJ(nt);
      // face NT first: its flux enters cell 2 through FBND(1)=FBND(NT)
      const double cN = CJ(nt);
      auto limit = [&](int J, double c) {
        if (kCfl == 1 || (kCfl == 2 && outside[(long long)(J - 1) * nr] == 0)) q = cfl_bits(c, q);
      };
      limit(nt, cN);
      int csN = kRec == 2 ? (int)(rget(rl + (long long)(nt - 1) * st, rsh) & 7) : 0;
      const bool negN = hi32(dbits(cN)) < 0;  // (-0: face_phi_fp64)
      const double phiN = face_phi<kRec, kB32>(negN ? G3 : GNm, negN ? G2 : GN, negN ? GN : G2, cN, face_coef(dbits(cN)),
                                               beta, betaf, csN, [&] { return cN; }, mh);
      double phi_prev = phiN;
      double gm = G1, g0 = G2, gp = G3;
      auto step = [&](int J, double c, double gpp, auto wrap) {
        limit(J, c);
        const unsigned old = kRec == 1 ? rold(rl + (long long)(J - 1) * st, rsh) : 0u;
        const bool neg = hi32(dbits(c)) < 0;  // (-0: face_phi_fp64)
        const unsigned char* rj = (kRec == 1 || kRec == 2) ? rl + (long long)(J - 1) * st : nullptr;
        int cs = kRec == 2 ? (int)(rget(rj, rsh) & 7) : 0;
        double phi = face_phi<kRec, kB32>(neg ? gpp : gm, neg ? gp : g0, neg ? g0 : gp, c, face_coef(dbits(c)), beta,
                                          betaf, cs, [&] { return c; }, mh);
        // The reference's D of face NT-1 against the flow is F(2)-F(1), with
        // F(1) in the place of F(NT); the two differ only in states that are
        // not periodic.
        if (decltype(wrap)::value && is_neg(c) && dbits(G1) != dbits(GN)) {
          const PhiCase r = face_phi_fp64<kRec>(gp - g0, G2 - G1, gp, g0, c, -0.5, beta,
                                                kRec == 2 ? (int)(rget(rj, rsh) & 7) : 0);
          phi = r.phi;
          cs = r.cs;
        }
        const double raw = (g0 - phi) + phi_prev;
        GJ(J) = (kRec == 2) ? clip_frozen(raw, rget(rj, rsh)) : clip(raw);
        if (kRec == kRecCount) nclip += is_neg(raw);
        if (kRec == 1) rput(rl + (long long)(J - 1) * st, rsh, old, cs | (is_neg(raw) ? kClipBit : 0));
        phi_prev = phi;
        gm = g0; g0 = gp; gp = gpp;
      };
      // The cell two faces ahead is loaded one iteration early, before this
      // face's store: the compiler cannot move a load past a store to the
      // line at a run-time stride.
      double nxt = GJ(4);
      for (int J = 2; J <= nt - 2; ++J) {
        const double nn = GJ(min(J + 3, nt));
        step(J, CJ(J), nxt, std::false_type());
        nxt = nn;
      }
      step(nt - 1, CJ(nt - 1), G2, std::true_type());
      const double rawN = (GN - phiN) + phi_prev;
      const double vN = (kRec == 2) ? clip_frozen(rawN, rget(rl + (long long)(nt - 1) * st, rsh)) : clip(rawN);
      if (kRec == kRecCount) nclip += is_neg(rawN);
      GJ(nt) = vN;
      GJ(1) = vN;
      if (kRec == 1) rput(rl + (long long)(nt - 1) * st, rsh, rold(rl + (long long)(nt - 1) * st, rsh), csN | (is_neg(rawN) ? kClipBit : 0));
  #undef GJ
  #undef CJ
    }
    if (kRec == kRecCount) warp_atomic_add(&d.clipq[slot], nclip);
    if (kCfl) warp_atomic_max(&d.cflq[slot * 4 + 1], q);
  }
}

// ----------------------------------------------------------------- DRIFTE
// Line (I,J,L), I = 2..NR, along K = 1..NE with extrapolated F(0), F(1)
// and F(NE+1) = F(NE+2) = 0.  Cell K = 1 is never written.
// kSplit adjacent lanes share a line: lane r updates the cells b+1..lim of
// its segment (b = r*S, lim = (r+1)*S with S = NE/kSplit; the first from
// cell 2, the last to NE) and first forms face b anew, whose flux enters its
// cells (face 1 for the first lane).  Every old value a lane needs from its
// neighbours' cells is loaded before a __syncwarp, and no lane writes before
// it; the flux of a face is the same bits in either lane.  S >= 4, so no
// lane but the first sees the extrapolated cells.
// Four lanes are for short lists, where 24 warps an SM are plenty: their
// instance may hold 85 registers (with 8 lanes in DRIFTMU alike; a call on
// 6x9x35x72 0.1033 -> 0.1023 ms from the graph, 0.1233 -> 0.1213 direct).
template <bool kCfl, int kRec, bool kB32, int kSplit>
__global__ void __launch_bounds__(256, kSplit > 2 ? 3 : 4) k_sweep_e(Dev d, double dts, unsigned char* __restrict__ rec, int rsh) {
  chain_enter();
  const int nr = d.nr, nt = d.nt, ne = d.ne;
  const int line0 = d.lw0 * (nr - 1) * nt;  // the L window, as in DRIFTR
  const int nlines = (nr - 1) * nt * (d.lw1 - d.lw0);
  const int lpb = blockDim.x / kSplit;  // lines per CTA
  const int r = kSplit > 1 ? (int)threadIdx.x % kSplit : 0, seg = ne / kSplit;
  const bool last = r == kSplit - 1;
  const int b = r ? r * seg : 1, lim = last ? ne : (r + 1) * seg;
  for (Unit u((nlines + lpb - 1) / lpb); u.ok(d); u.next(d)) {
    const int2 item = d.items[u.it];
    const int m = item.x, s = item.y, slot = m * d.ns + s;
    const int line = line0 + u.b * lpb + (int)threadIdx.x / kSplit;
    unsigned long long q = 0ULL;  // CFL quotient bits
    unsigned nclip = 0;  // clip events (kRec == kRecCount)
    // bounds-checked builds: the line's cells, its (I,J,L) table entry and
    // UE, its line factors (the lanes sharing a line test the same)
    const bool active = line < line0 + nlines &&
        rg_ok(d, rg_item(d, item) &&
                     rg_span(((long long)(line / (nr - 1) / nt) * ne * nt + (line / (nr - 1)) % nt) * nr + 1 +
                                 line % (nr - 1), ne, (long long)nt * nr, d.ncell) &&
                     rg_span((long long)item.x * nr * nt * d.npa + (long long)(line / (nr - 1)) * nr + 1 +
                                 line % (nr - 1), 1, 1, (long long)d.nm * nr * nt * d.npa) &&
                     rg_span((long long)item.y * nr + 1 + line % (nr - 1), 1, 1, (long long)d.ns * nr),
              kRgSweepE, line);
    const int lc = active ? line : line0;
    const int i = 1 + lc % (nr - 1);
    const int jl = lc / (nr - 1);
    const int j = jl % nt, l = jl / nt;
    const unsigned st = (unsigned)nt * nr;  // stride between consecutive K
    const long long off = ((long long)l * ne * nt + j) * nr + i;
    double* __restrict__ fl = d.f2 + (long long)slot * d.ncell + off;
    unsigned char* __restrict__ rl = (kRec == 1 || kRec == 2) ? rec + u.it * d.ncell + off : nullptr;
    const FaceBin* __restrict__ bins = d.ebin + s * ne;
  #define GK(K) strided_b(fl, (K)-1, st * 8u)
    // the window G(b-1..b+2), the next cell, and the two cells past lim
    double w0 = 0.0, w1 = 0.0, w2 = 0.0, w3 = 0.0, nxt = 0.0, hA = 0.0, hB = 0.0;
    if (active) {
      w2 = GK(b + 1);
      w3 = GK(b + 2);
      if (kSplit > 1 && r) {
        w0 = GK(b - 1);
        w1 = GK(b);
      } else {
        w1 = d.kap[2 * s + 1] * w2;
        w0 = d.kap[2 * s + 0] * w1;
      }
      nxt = GK(b + 3);
      if (kSplit > 1 && !last) {
        hA = GK(lim + 1);
        hB = GK(lim + 2);
      }
    }
    if (kSplit > 1) __syncwarp();
    if (active) {
      const long long fij = ((long long)l * nt + j) * nr + i;
      // C(K) = k(K)*v, v = UE*DTs/RLZ + k*(WET*1e3/QS*DTs/RLZ): k = EBND*(GRBND+1)/
      // (2 GRBND) comes from the bin's table, so a face's C costs one fma
      const double wet = d.wet[fij] * d.erq[s * nr + i];
      const double ue = d.ue[(long long)m * nr * nt * d.npa + fij] * d.er[i];
      const bool inside = d.outside[(long long)j * nr + i] == 0;
      const double beta = d.betalim;
      const uint64_t betaf = beta_fix(dbits(beta));
      const bool closed = d.flags & 1u;
      // Face K: its flux.  At face NE against the flow FUP = F(NE+1) = 0: that
      // flux is zero whatever the other cells (end).
      Largest big;
      auto quotient = [&](int K, double c) { q = umax64(q, dbits(c * d.ide[K - 1]) & kAbsMask); };
      auto face = [&](int K, const FaceBin& bin, double v, double gm, double g0, double gp, double gpp, int& cs,
                      auto end) {
        const FaceCoef fc = face_coef_bin(dbits(v), bin);
        if (kCfl) big.see(fc, K);
        const bool none = decltype(end)::value && fc.sign && abs_lt_inf(v), neg = fc.sign && !none;
        const double phi = face_phi<kRec, kB32>(
            neg ? gpp : gm, neg ? gp : g0, neg ? g0 : gp, v, fc, beta, betaf, cs, [&] { return bin.k * v; },
            [&] { return d.mhde[K - 1]; },
            [&] { if (kCfl && inside) quotient(K, bin.k * v); });
        if (none) cs = 0;
        return none ? 0.0 : phi;
      };
      double phi_prev;
      {
        unsigned char* rb = (kRec == 1 || kRec == 2) ? rl + (uint64_t)(b - 1) * st : nullptr;
        int cs = kRec == 2 ? (int)(rget(rb, rsh) & 7) : 0;
        phi_prev = face(b, bins[b - 1], fma(bins[b - 1].k, wet, ue), w0, w1, w2, w3, cs, std::false_type());
        if (closed && r == 0) phi_prev = 0.0;
        if (kRec == 1 && r == 0) rput(rb, rsh, rold(rb, rsh), cs);
      }
      double gm = w1, g0 = w2, gp = w3;
      auto step = [&](int K, double v, double gpp, auto end) {
        const FaceBin bin = bins[K - 1];
        const unsigned old = kRec == 1 ? rold(rl + (uint64_t)(K - 1) * st, rsh) : 0u;
        const unsigned char* rk = (kRec == 1 || kRec == 2) ? rl + (uint64_t)(K - 1) * st : nullptr;
        int cs = kRec == 2 ? (int)(rget(rk, rsh) & 7) : 0;
        double phi = face(K, bin, v, gm, g0, gp, gpp, cs, end);
        if (decltype(end)::value && closed) phi = 0.0;
        const double raw = fma(phi_prev - phi, bin.iw, g0);
        GK(K) = (kRec == 2) ? clip_frozen(raw, rget(rk, rsh)) : clip(raw);
        if (kRec == kRecCount) nclip += is_neg(raw);
        if (kRec == 1) rput(rl + (uint64_t)(K - 1) * st, rsh, old, cs | (is_neg(raw) ? kClipBit : 0));
        phi_prev = phi;
        gm = g0; g0 = gp; gp = gpp;
      };
      // the cell two faces ahead one iteration early, as in DRIFTP
      for (int K = b + 1; K <= (last ? ne - 1 : lim); ++K) {
        double nn = hA;
        if (K + 3 <= lim) nn = GK(K + 3);
        else hA = hB;
        step(K, fma(bins[K - 1].k, wet, ue), nxt, std::false_type());
        nxt = nn;
      }
      if (last) step(ne, fma(bins[ne - 1].k, wet, ue), 0.0, std::true_type());
      if (kCfl && inside) {  // |C|/DE, |C| at least 1e-10
        q = umax64(q, mul_pos_bits(kBits1em10, d.ide[ne]));
        if (big.at) {
          const double k = bins[big.at - 1].k;
          quotient(big.at, k * fma(k, wet, ue));
        }
      }
    }
  #undef GK
    if (kRec == kRecCount) warp_atomic_add(&d.clipq[slot], nclip);
    if (kCfl) warp_atomic_max(&d.cflq[slot * 4 + 2], q);
  }
}

// ---------------------------------------------------------------- DRIFTMU
// Line (I,J,K), I = 2..NR, along L = 1..NPA with F(1) = F(2); limiter on
// faces 2..NPA-2, FBND(NPA-1) = F(NPA), then the F2(NPA) extrapolation.
// kLoss: 0 none, 1 multiply the result by table lossA (loss after the sweep),
//        2 multiply the input by lossA (loss before the sweep).
// kSplit: there are few pitch-angle lines (NR-1)*NT*NE, so kSplit adjacent
// lanes share one, as in DRIFTE: lane r updates the cells b+1..lim of segment
// r (b = r*S, lim = (r+1)*S with S = NPA/kSplit; the first from cell 2, the
// last to NPA) and forms face b anew (the first lane's face 1 carries
// nothing).  S >= 4, so no lane but the first sees the F(1) = F(2) rule.
template <bool kCfl, int kLoss, int kRec, bool kB32, int kSplit>
__global__ void __launch_bounds__(256, kSplit > 4 ? 3 : 4) k_sweep_mu(Dev d, double dts, const double* __restrict__ lossA,
                                                     unsigned char* __restrict__ rec, int rsh) {
  chain_enter();
  const int nr = d.nr, nt = d.nt, ne = d.ne, npa = d.npa;
  const int nlines = (nr - 1) * nt * ne;
  const int lpb = blockDim.x / kSplit;  // lines per CTA
  const int r = kSplit > 1 ? (int)threadIdx.x % kSplit : 0, seg = npa / kSplit;
  const bool last = r == kSplit - 1;
  const int b = r ? r * seg : 1, lim = last ? npa : (r + 1) * seg;
  for (Unit u((nlines + lpb - 1) / lpb); u.ok(d); u.next(d)) {
    const int2 item = d.items[u.it];
    const int m = item.x, s = item.y, slot = m * d.ns + s;
    const int line = u.b * lpb + (int)threadIdx.x / kSplit;
    // bounds-checked builds: the line's cells, its WM and UM columns (the
    // lanes sharing a line test the same)
    const bool active = line < nlines &&
        rg_ok(d, rg_item(d, item) &&
                     rg_span((long long)(line / (nr - 1)) * nr + 1 + line % (nr - 1), npa, (long long)ne * nt * nr,
                             d.ncell) &&
                     rg_span((long long)((line / (nr - 1)) % nt) * nr + 1 + line % (nr - 1), npa, (long long)nt * nr,
                             (long long)nr * nt * npa) &&
                     rg_span((long long)item.x * nt * nr * npa + ((line / (nr - 1)) % nt) * nr + 1 + line % (nr - 1),
                             npa, (long long)nt * nr, (long long)d.nm * nr * nt * npa),
              kRgSweepMu, line);
    unsigned long long q = 0ULL;  // CFL quotient bits
    unsigned nclip = 0;  // clip events (kRec == kRecCount)
    const int lc = active ? line : 0;
    const int i = 1 + lc % (nr - 1);
    const int jk = lc / (nr - 1);
    const int j = jk % nt;
    const unsigned st = (unsigned)ne * nt * nr;  // stride between consecutive L
    const long long off = (long long)jk * nr + i;  // (K*NT + J)*NR + I
    double* __restrict__ fl = d.f2 + (long long)slot * d.ncell + off;
    unsigned char* __restrict__ rl = (kRec == 1 || kRec == 2) ? rec + u.it * d.ncell + off : nullptr;
    const double* __restrict__ la = lossA ? lossA + (long long)s * d.ncell + off : nullptr;
  #define GL(L) strided(fl, (L)-1, st)
  #define LA(L) strided(la, (L)-1, st)
  #define GLS(L) (kLoss == 2 ? GL(L) * LA(L) : GL(L))
    // the window G(b-1..b+2) (the first lane's F(1) is F(2)), the next cell,
    // and the two cells past lim
    double w0 = 0.0, w1 = 0.0, w2 = 0.0, w3 = 0.0, nxt = 0.0, hA = 0.0, hB = 0.0;
    if (active) {
      w2 = GLS(b + 1);
      w3 = GLS(b + 2);
      w0 = w1 = w2;
      if (kSplit > 1 && r) {
        w0 = GLS(b - 1);
        w1 = GLS(b);
      }
      nxt = GLS(b + 3);
      if (kSplit > 1 && !last) {
        hA = GLS(lim + 1);
        hB = GLS(lim + 2);
      }
    }
    if (kSplit > 1) __syncwarp();
    if (active) {
      const unsigned sij = (unsigned)nt * nr * 8u;  // bytes between consecutive L of (I,J,L) tables
      const long long fij = (long long)j * nr + i;
      const double* __restrict__ wm = d.wm + fij;
      const double* __restrict__ um = d.um + (long long)m * nt * nr * npa + fij;
      const FaceMu* __restrict__ bins = d.mubin;
      const double ekv = d.ek[s * ne + jk / nt];
      const bool inside = d.outside[fij] == 0;
      const double beta = d.betalim;
      const uint64_t betaf = beta_fix(dbits(beta));
      const bool closed = d.flags & 1u;
  #define CL(L) fma(ekv, strided_b(wm, (L)-1, sij), strided_b(um, (L)-1, sij))
      // face L's flux; the CFL quotient |C|/DMU is the Courant number, which
      // counts from L = 2 on (lanes that share a line form face 1 as well)
      Largest big;
      auto quotient = [&](int L, double c) { q = umax64(q, dbits(c * d.idmu[L - 1]) & kAbsMask); };
      auto face = [&](int L, const FaceMu& bin, double c, double gm, double g0, double gp, double gpp, int& cs) {
        const FaceCoef fc = face_coef_mu(dbits(c), bin);
        if (kCfl) big.see(fc, L);
        const bool neg = fc.sign;  // (-0: face_phi_fp64)
        return face_phi<kRec, kB32>(neg ? gpp : gm, neg ? gp : g0, neg ? g0 : gp, c, fc, beta, betaf, cs,
                                    [&] { return c; }, [&] { return d.mhdmu[L - 1]; },
                                    [&] { if (kCfl && inside && L > 1) quotient(L, c); });
      };
      double phi_prev = 0.0;
      if (kSplit > 1) {
        int cs = kRec == 2 ? (int)(rget(rl + (uint64_t)(b - 1) * st, rsh) & 7) : 0;
        const double phi = face(b, bins[b - 1], CL(b), w0, w1, w2, w3, cs);
        if (r) phi_prev = phi;
        else big = Largest();  // face 1 does not count
      }
      double gm = w1, g0 = w2, gp = w3;
      // cell L from its raw value, with its record
      auto put = [&](int L, double raw, int cs, unsigned old) {
        if (kRec == 1) rput(rl + (uint64_t)(L - 1) * st, rsh, old, cs | (is_neg(raw) ? kClipBit : 0));
        if (kRec == kRecCount) nclip += is_neg(raw);
        return (kRec == 2) ? clip_frozen(raw, rget(rl + (uint64_t)(L - 1) * st, rsh)) : clip(raw);
      };
      for (int L = b + 1; L <= (last ? npa - 2 : lim); ++L) {
        double nn = hA;
        if (L + 3 <= lim) nn = GLS(L + 3);
        else hA = hB;
        // read before the face's arithmetic, not at the store (four species on
        // 40x49x70x144, the two launches' mean: 633 -> 591 us; 20x25x35x72: 58.1 -> 56.3)
        const double loss = kLoss == 1 ? LA(L) : 1.0;
        const FaceMu bin = bins[L - 1];
        const unsigned old = kRec == 1 ? rold(rl + (uint64_t)(L - 1) * st, rsh) : 0u;
        int cs = kRec == 2 ? (int)(rget(rl + (uint64_t)(L - 1) * st, rsh) & 7) : 0;
        const double phi = face(L, bin, CL(L), gm, g0, gp, nxt, cs);
        double v = put(L, fma(phi_prev - phi, bin.iw, g0), cs, old);
        if (kLoss == 1) v *= loss;
        GL(L) = v;
        phi_prev = phi;
        gm = g0; g0 = gp; gp = nxt;
        nxt = nn;
      }
      // face NPA-1: FBND = F(NPA); cell NPA-1; then the F2(NPA) ghost
      if (last) {
        const int L = npa - 1;
        const FaceMu bin = bins[L - 1];
        const double c = CL(L);
        if (kCfl && inside) quotient(L, c);
        const double phi = c * (closed ? 0.0 : gp);
        const double v = put(L, fma(phi_prev - phi, bin.iw, g0), 0, kRec == 1 ? rold(rl + (uint64_t)(L - 1) * st, rsh) : 0u);
        const double vN = v * d.rho[fij];
        if (kLoss == 1) {
          GL(L) = v * LA(L);
          GL(npa) = vN * LA(npa);
        } else {
          GL(L) = v;
          GL(npa) = vN;
        }
      }
      if (kCfl && inside) {  // |C|/DMU, |C| at least 1e-32
        q = umax64(q, mul_pos_bits(kBits1em32, d.idmu[npa]));
        if (big.at) quotient(big.at, CL(big.at));
      }
    }
  #undef GL
  #undef LA
  #undef GLS
  #undef CL
    if (kRec == kRecCount) warp_atomic_add(&d.clipq[slot], nclip);
    if (kCfl) warp_atomic_max(&d.cflq[slot * 4 + 3], q);
  }
}

// ---------------------------------------------------------------- launchers
// Grid: (blocks per item, items), or a persistent grid of d.pers[w] CTAs.
static inline dim3 grid_for(const Dev& d, int w, int nlines) {
  const int blk = d.blk[w];
  if (d.pers[w] > 0) return dim3(d.pers[w], 1, 1);
  return dim3((nlines + blk - 1) / blk, d.nitems, 1);
}
// Lines of sweep w: R, P and E within the L window [lw0, lw1); every
// pitch-angle line spans all L, so DRIFTMU always takes them all.
static inline int nlines_of(const Dev& d, int w) {
  switch (w) {
    case 0: return d.nt * d.ne * (d.lw1 - d.lw0);
    case 1: return (d.nr - 1) * d.ne * (d.lw1 - d.lw0);
    case 2: return (d.nr - 1) * d.nt * (d.lw1 - d.lw0);
    default: return (d.nr - 1) * d.nt * d.ne;
  }
}

// The limiter's beta has a short fraction (face.cuh beta_times).
static inline bool beta_b32(const Dev& d) {
  uint64_t u;
  memcpy(&u, &d.betalim, sizeof(u));
  return (uint32_t)beta_fix(u) == 0u;
}
#define SWEEP_LAUNCHER(NAME, KERNEL, W)                                                                       \
  template <bool kB>                                                                                          \
  static void NAME##_b(const Dev& d, double dts, bool cfl, cudaStream_t st, unsigned char* rec, bool replay,  \
                       int rsh) {                                                                             \
    const dim3 g = grid_for(d, W, nlines_of(d, W));                                                           \
    const int b = d.blk[W];                                                                                   \
    const bool n = d.count_clips;                                                                             \
    if (rec && replay) launch_k(d.chained, KERNEL<0, 2, kB>, g, b, 0, st, d, dts, rec, rsh);                               \
    else if (rec) launch_k(d.chained, KERNEL<0, 1, kB>, g, b, 0, st, d, dts, rec, rsh);                                    \
    else if (cfl && (d.flags >> 31))                                                                          \
      launch_k(d.chained, n ? KERNEL<2, 3, kB> : KERNEL<2, 0, kB>, g, b, 0, st, d, dts, nullptr, 0);                         \
    else if (cfl) launch_k(d.chained, n ? KERNEL<1, 3, kB> : KERNEL<1, 0, kB>, g, b, 0, st, d, dts, nullptr, 0);             \
    else launch_k(d.chained, n ? KERNEL<0, 3, kB> : KERNEL<0, 0, kB>, g, b, 0, st, d, dts, nullptr, 0);                      \
  }                                                                                                           \
  void NAME(const Dev& d, double dts, bool cfl, cudaStream_t st, unsigned char* rec, bool replay, int rsh) {  \
    if (beta_b32(d)) NAME##_b<true>(d, dts, cfl, st, rec, replay, rsh);                                       \
    else NAME##_b<false>(d, dts, cfl, st, rec, replay, rsh);                                                  \
  }
SWEEP_LAUNCHER(launch_sweep_p, k_sweep_p, 1)
#undef SWEEP_LAUNCHER

template <bool kB, int V>
static void r_launch(const Dev& d, double dts, bool cfl, cudaStream_t st, unsigned char* rec, bool replay, int rsh) {
  const dim3 g = grid_for(d, 0, nlines_of(d, 0));
  const int b = d.blk[0];
  const size_t sm = V > 1 ? 3 * V * b * sizeof(double) : 0;
  const bool n = d.count_clips;
  if (rec && replay) launch_k(d.chained, k_sweep_r<0, 2, kB, V>, g, b, sm, st, d, dts, rec, rsh);
  else if (rec) launch_k(d.chained, k_sweep_r<0, 1, kB, V>, g, b, sm, st, d, dts, rec, rsh);
  else if (cfl && (d.flags >> 31)) launch_k(d.chained, n ? k_sweep_r<2, 3, kB, V> : k_sweep_r<2, 0, kB, V>, g, b, sm, st, d, dts, nullptr, 0);
  else if (cfl) launch_k(d.chained, n ? k_sweep_r<1, 3, kB, V> : k_sweep_r<1, 0, kB, V>, g, b, sm, st, d, dts, nullptr, 0);
  else launch_k(d.chained, n ? k_sweep_r<0, 3, kB, V> : k_sweep_r<0, 0, kB, V>, g, b, sm, st, d, dts, nullptr, 0);
}
// Cells per access.  While an SM's lines (32 warps of 8*NR bytes a lane) stay
// in L1 (NR up to 24), cells move one at a time: the wide accesses bring
// nothing (NR = 20, us a launch over four species: 52.1 with one, 56.7 with
// two, 51.6 with four; the call 0.386, 0.397, 0.389 ms).  Longer lines fall
// out of L1 between a lane's cells, and the widest access that divides NR
// (then every line, GRT and CR row starts on its boundary) reads and writes
// whole sectors once (NR = 40: 863, 733, 610; L2 traffic down to 0.4).  How
// much that gains depends on how the lanes' lines fall into L1's sets: on
// NR x 25x35x72, one cell against four, 72.9 and 67.5 at NR = 28, 148.8 and
// 79.8 at 32, 89.9 and 83.0 at 36, 133.1 and 90.3 at 40.  Odd NR spread over
// all sets and lose nothing one cell at a time (63.1 at 25, 65.6 at 27).  Two
// cells against one: 69.4 and 66.0, 77.9 and 73.7, 88.3 and 82.2 at NR = 26, 30
// and 34, but 444 and 440, 506 and 512, 569 and 585 on NR x 49x70x144.
static int r_width(const Dev& d) { return d.nr <= 24 || d.nr % 2 ? 1 : (d.nr % 4 ? 2 : 4); }
void launch_sweep_r(const Dev& d, double dts, bool cfl, cudaStream_t st, unsigned char* rec, bool replay, int rsh) {
  const bool kb = beta_b32(d);
  const int v = r_width(d);
  if (v == 4) (kb ? r_launch<true, 4> : r_launch<false, 4>)(d, dts, cfl, st, rec, replay, rsh);
  else if (v == 2) (kb ? r_launch<true, 2> : r_launch<false, 2>)(d, dts, cfl, st, rec, replay, rsh);
  else (kb ? r_launch<true, 1> : r_launch<false, 1>)(d, dts, cfl, st, rec, replay, rsh);
}

// Lanes per DRIFTE line.  A line is a serial chain of NE faces; with few
// lines an SM has too few warps to hide it, and splitting lines gives more,
// for one extra face and the halo loads per lane.  Measured (GB300, us a
// launch with 1, 2, 4 lanes): 34.2 k lines (one species, 20x25x35x72) 26.6,
// 25.2, 25.0, the whole call 0.231, 0.226, 0.225 ms; 136.8 k lines 54, 58,
// 68; 1.1 M lines (40x49x70x144) 580, 665, 748.  The count is that of the
// whole work list and every plane: item groups and chunks run side by side.
static int e_lanes(const Dev& d) {
  const long long warps = (long long)(d.nr - 1) * d.nt * d.npa * d.nlist / 32;
  if (d.ne < 16) return 1;  // segments of at least four cells
  return warps < 4LL * d.nsm ? 4 : (warps < 12LL * d.nsm ? 2 : 1);
}
template <bool kB, int kS>
static void e_launch(const Dev& d, double dts, bool cfl, cudaStream_t st, unsigned char* rec, bool replay, int rsh) {
  const dim3 g = grid_for(d, 2, kS * nlines_of(d, 2));
  const int b = d.blk[2];
  const bool n = d.count_clips;
  if (rec && replay) launch_k(d.chained, k_sweep_e<false, 2, kB, kS>, g, b, 0, st, d, dts, rec, rsh);
  else if (rec) launch_k(d.chained, k_sweep_e<false, 1, kB, kS>, g, b, 0, st, d, dts, rec, rsh);
  else if (cfl) launch_k(d.chained, n ? k_sweep_e<true, 3, kB, kS> : k_sweep_e<true, 0, kB, kS>, g, b, 0, st, d, dts, nullptr, 0);
  else launch_k(d.chained, n ? k_sweep_e<false, 3, kB, kS> : k_sweep_e<false, 0, kB, kS>, g, b, 0, st, d, dts, nullptr, 0);
}
void launch_sweep_e(const Dev& d, double dts, bool cfl, cudaStream_t st, unsigned char* rec, bool replay, int rsh) {
  const int lanes = e_lanes(d);
  const bool kb = beta_b32(d);
  if (lanes == 4) (kb ? e_launch<true, 4> : e_launch<false, 4>)(d, dts, cfl, st, rec, replay, rsh);
  else if (lanes == 2) (kb ? e_launch<true, 2> : e_launch<false, 2>)(d, dts, cfl, st, rec, replay, rsh);
  else (kb ? e_launch<true, 1> : e_launch<false, 1>)(d, dts, cfl, st, rec, replay, rsh);
}

// Lanes per DRIFTMU line: as set, or (0) by the number of lines, as for
// DRIFTE.  Measured whole calls (GB300, ms with 1, 2, 4 lanes), at 20x25x35x72
// unless said: one species (3.4 warps an SM with one lane) 0.264, 0.224,
// 0.203; four (14) 0.422, 0.390, 0.387; two members of four (27) 0.675,
// 0.679, 0.698; eight (109) 2.52, 2.64, 2.71; 6x9x35x72, four species (1.3)
// 0.193, 0.153, 0.134, and 0.122 with 8.  Segments keep at least six cells.
int mu_lanes(const Dev& d) {
  int want = d.mu_lanes;
  if (!want) {
    const long long warps = (long long)(d.nr - 1) * d.nt * d.ne * d.nlist / 32;
    want = warps < 2LL * d.nsm ? 8 : (warps < 16LL * d.nsm ? 4 : (warps < 24LL * d.nsm ? 2 : 1));
  }
  while (want > 1 && d.npa < 6 * want) want /= 2;
  return want;
}
template <int kLoss, bool kB, int kS>
static void mu_launch(const Dev& d, double dts, const double* loss, cudaStream_t st, unsigned char* rec, bool replay,
                      bool cfl, int rsh) {
  const dim3 g = grid_for(d, 3, kS * nlines_of(d, 3));
  const int b = d.blk[3];
  const bool n = d.count_clips;
  if (rec && replay) launch_k(d.chained, k_sweep_mu<false, kLoss, 2, kB, kS>, g, b, 0, st, d, dts, loss, rec, rsh);
  else if (rec) launch_k(d.chained, k_sweep_mu<false, kLoss, 1, kB, kS>, g, b, 0, st, d, dts, loss, rec, rsh);
  else if (cfl)
    launch_k(d.chained, n ? k_sweep_mu<true, kLoss, 3, kB, kS> : k_sweep_mu<true, kLoss, 0, kB, kS>, g, b, 0, st, d, dts, loss, nullptr, 0);
  else
    launch_k(d.chained, n ? k_sweep_mu<false, kLoss, 3, kB, kS> : k_sweep_mu<false, kLoss, 0, kB, kS>, g, b, 0, st, d, dts, loss, nullptr, 0);
}
template <int kLoss, bool kB>
static void mu_lanes_launch(const Dev& d, double dts, const double* loss, cudaStream_t st, unsigned char* rec,
                            bool replay, bool cfl, int rsh) {
  const int lanes = mu_lanes(d);
  if (lanes == 8) mu_launch<kLoss, kB, 8>(d, dts, loss, st, rec, replay, cfl, rsh);
  else if (lanes == 4) mu_launch<kLoss, kB, 4>(d, dts, loss, st, rec, replay, cfl, rsh);
  else if (lanes == 2) mu_launch<kLoss, kB, 2>(d, dts, loss, st, rec, replay, cfl, rsh);
  else mu_launch<kLoss, kB, 1>(d, dts, loss, st, rec, replay, cfl, rsh);
}
void launch_sweep_mu(const Dev& d, double dts, bool cfl, int loss_mode, const double* loss,
                     cudaStream_t st, unsigned char* rec, bool replay, int rsh) {
  const bool kb = beta_b32(d);
  if (loss_mode == 1)
    (kb ? mu_lanes_launch<1, true> : mu_lanes_launch<1, false>)(d, dts, loss, st, rec, replay, cfl, rsh);
  else if (loss_mode == 2)
    (kb ? mu_lanes_launch<2, true> : mu_lanes_launch<2, false>)(d, dts, loss, st, rec, replay, cfl, rsh);
  else
    (kb ? mu_lanes_launch<0, true> : mu_lanes_launch<0, false>)(d, dts, nullptr, st, rec, replay, cfl, rsh);
}

// Resident CTAs per SM of sweep w at block size blk (for persistent grids).
int sweep_max_blocks_per_sm(int w, int blk) {
  int n = 0;
  cudaError_t e = cudaSuccess;
  switch (w) {
    case 0: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_sweep_r<0, 0, true, 4>, blk, 3 * 4 * blk * sizeof(double)); break;
    case 1: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_sweep_p<0, 0, true>, blk, 0); break;
    case 2: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_sweep_e<false, 0, true, 1>, blk, 0); break;
    default: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_sweep_mu<false, 0, 0, true, 2>, blk, 0); break;
  }
  return e == cudaSuccess ? n : 0;
}

}  // namespace ramgpu

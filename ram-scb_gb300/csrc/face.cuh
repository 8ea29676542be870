// face.cuh -- the flux of one limited face in 64-bit fixed point.
//
// A face carries phi = C * FBND, FBND = FUP + a * LIMITER(R) * X
// (src/ModRamDrift.f90:169-183).  In terms of the upwind cell u, the cell
// downwind of it d and the one upwind of it uu (u, d, uu = F(f), F(f+1),
// F(f-1) for C >= 0 and F(f+1), F(f), F(f+2) for C < 0) both directions read
//   phi = C * (u + 1/2 (1 - U) * sgn(d-u) * lim),   U the Courant number,
//   lim = min(beta*lo, hi), lo/hi the smaller/larger of |d-u|, |u-uu|
// where u-uu and d-u have the same sign and |d-u| > 1e-27, else phi = C*u.
// (max(min(beta|D|,|X|), min(|D|,beta|X|)) is that lim for beta >= 1.)
//
// The FP64 unit issues one warp instruction per 64 cycles per scheduler
// while the integer pipes are mostly free, so the whole face runs on them:
// the three cells are aligned to u's exponent in 64-bit fixed point with
// u in [2^59, 2^60).  d and uu keep every bit down to 2^-59 of u (seven
// below u's own last place); cells of 8u and more saturate at 4u or above,
// where lim no longer depends on them (lo <= u when both differences have
// one sign).  1 - U, lim and their product stay in fixed point, so nothing
// is normalised or rounded until phi itself, which is rounded once: its
// error is below that of the FP64 sequence (a rounded X, a, FBND and phi).
// Negative, infinite, NaN and zero upwind cells, Courant numbers of 1 and
// more, a zero C and the extremes of the exponent range report `special`;
// the caller takes the FP64 form there.
//
// Bound and figures (GB300, one launch over four species on 20x25x35x72): the
// FP64 sequence held the FP64 pipe, five operations a face in DRIFTR and
// DRIFTP and up to seven in DRIFTE and DRIFTMU (phi, beta|X| and the Courant
// products were integer products already).  Here three remain (the coefficient's fma
// and the update); instruction issue (50-61 %, 170-210 instructions a face),
// the integer ALU (51-59 %) and the FP64 pipe (52-67 %) are about even.  With the
// sweeps as they are now, DRIFTR 64.5 -> 52.8 us, DRIFTP 61.8 -> 46.8, DRIFTE
// 66.8 -> 54.7, DRIFTMU 68.6 -> 56.1; on 40x49x70x144 DRIFTR 944 -> 610, DRIFTP
// 783 -> 538, DRIFTE 875 -> 572, DRIFTMU 946 -> 593.  Normalising the factor and the
// differences, as the FP64 form's integer products did, took more
// instructions than aligning the cells once.  The rare forms must stay rare:
// before face_plain and the exact threshold below, eight warps of meridian
// lines with C = 0 made the whole DRIFTE launch 71 us.
//
// Compiles for the host too (the arithmetic is tested on the CPU).
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define RG_HD __host__ __device__ __forceinline__
#else
#define RG_HD static inline
#endif

namespace ramgpu {

// v >> s with 0 for s >= 64 (also for s < 0 read as unsigned)
RG_HD uint64_t shr_clamp(uint64_t v, int s) {
#ifdef __CUDA_ARCH__
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
  return r;
#else
  return (unsigned)s > 63u ? 0ULL : v >> s;
#endif
}
// position of the top set bit (-1 for 0)
RG_HD int top_bit(uint32_t v) {
#ifdef __CUDA_ARCH__
  int r;
  asm("bfind.u32 %0, %1;" : "=r"(r) : "r"(v));
  return r;
#else
  return v ? 31 - __builtin_clz(v) : -1;
#endif
}
RG_HD uint32_t max3u(uint32_t a, uint32_t b, uint32_t c) {
#ifdef __CUDA_ARCH__
  return __vimax3_u32(a, b, c);
#else
  return a > b ? (a > c ? a : c) : (b > c ? b : c);
#endif
}
// smaller and larger of a and b, and whether a is the smaller (or equal):
// one comparison (from min/max expressions the compiler makes two)
RG_HD bool sort2(uint64_t a, uint64_t b, uint64_t& lo, uint64_t& hi) {
#ifdef __CUDA_ARCH__
  int le;
  asm("{ .reg .pred p; setp.le.u64 p, %3, %4; selp.b64 %0, %3, %4, p; selp.b64 %1, %4, %3, p; selp.s32 %2, 1, 0, p; }"
      : "=&l"(lo), "=&l"(hi), "=r"(le) : "l"(a), "l"(b));
  return le != 0;
#else
  lo = a <= b ? a : b;
  hi = a <= b ? b : a;
  return a <= b;
#endif
}
// floor(x*y / 2^64) up to one unit low (the low halves' product is left
// out), for x, y whose cross products sum below 2^64
RG_HD uint64_t mulhi_cross(uint64_t x, uint64_t y) {
  const uint32_t xh = (uint32_t)(x >> 32), xl = (uint32_t)x, yh = (uint32_t)(y >> 32), yl = (uint32_t)y;
  const uint64_t t = (uint64_t)xh * yl + (uint64_t)xl * yh;
#ifdef __CUDA_ARCH__
  uint32_t rl, rh;
  asm("mad.lo.cc.u32 %0, %2, %3, %4; madc.hi.u32 %1, %2, %3, 0;"
      : "=r"(rl), "=r"(rh) : "r"(xh), "r"(yh), "r"((uint32_t)(t >> 32)));
  return ((uint64_t)rh << 32) | rl;
#else
  return (uint64_t)xh * yh + (uint32_t)(t >> 32);
#endif
}
// significand of a normal double with its top bit at 2^63 (sign and
// exponent shift out), or at 2^62
RG_HD uint64_t sig_top(uint64_t x) { return (x << 11) | 0x8000000000000000ULL; }
RG_HD uint64_t sig_62(uint64_t x) { return ((x << 10) & 0x7FFFFFFFFFFFFFFFULL) | 0x4000000000000000ULL; }
RG_HD int hi32(uint64_t x) { return (int)(x >> 32); }

// (beta - 1) * 2^64 of the limiter's beta (1 <= beta <= 2; 2 gives 2^64 - 1).
// kB32: its low word is zero (beta a multiple of 2^-32, e.g. 1.5), which
// saves a product; the launchers choose the form.
RG_HD uint64_t beta_fix(uint64_t beta_bits) {
  return (beta_bits >> 52) >= 1024 ? ~0ULL : (beta_bits << 12);
}
// beta * v for v < 2^63
template <bool kB32>
RG_HD uint64_t beta_times(uint64_t v, uint64_t betaf) {
  const uint32_t vh = (uint32_t)(v >> 32), vl = (uint32_t)v, bh = (uint32_t)(betaf >> 32), bl = (uint32_t)betaf;
  uint64_t f = (uint64_t)vh * bh + (uint32_t)(((uint64_t)vl * bh) >> 32);
  if (!kB32) f += ((uint64_t)vh * bl) >> 32;
  return v + f;
}

// The face coefficient prepared for face_flux: C = +-m 2^-62 2^(e-1023), its
// sign bit and (1 - U) * 2^63; `bad` is negative where the fixed point does
// not hold (U >= 1, C infinite or NaN).
struct FaceCoef {
  uint64_t m;      // [2^61, 2^63)
  uint64_t a63;    // (1 - U) * 2^63
  int e;           // exponent
  uint32_t sign;   // sign bit of C
  int bad;
};
// From C with U = |C| (the R and P sweeps).
RG_HD FaceCoef face_coef(uint64_t c) {
  FaceCoef q;
  const uint32_t h = (uint32_t)(c >> 32);
  q.sign = h & 0x80000000u;
  q.e = (int)((h >> 20) & 0x7FFu);
  q.m = sig_62(c);
  q.bad = 1022 - q.e;
  q.a63 = 0x7FFFFFFFFFFFFFFFULL - shr_clamp(q.m, q.bad);
  return q;
}
// DRIFTE's coefficient is C = k*v with k > 0 from the energy bin and v from
// the line, U = |v|*(k/DE): both products are formed here from v.
struct alignas(16) FaceBin {
  double k, iw;         // k and 1/WE of the bin
  uint64_t sk, sy;      // sig_62 of k and of k/DE
  int e, sh;            // exponent of k less 1022; 2045 less that of k/DE
  double pad;
};
RG_HD FaceCoef face_coef_bin(uint64_t v, const FaceBin& b) {
  FaceCoef q;
  const uint32_t h = (uint32_t)(v >> 32);
  const int ev = (int)((h >> 20) & 0x7FFu);
  const uint64_t sv = sig_62(v);
  q.sign = h & 0x80000000u;
  q.e = ev + b.e;
  q.m = mulhi_cross(sv, b.sk) << 1;
  const uint64_t prod = mulhi_cross(sv, b.sy) << 2;  // of U, 2^62 <= prod < 2^64
  const int sh = b.sh - ev;
  q.a63 = 0x7FFFFFFFFFFFFFFFULL - shr_clamp(prod, sh);
  q.bad = sh | hi32(q.a63) | (2046 - ev);
  return q;
}
// DRIFTMU's coefficient C comes whole; U = C/DMU.
struct alignas(16) FaceMu {
  double iw;            // 1/WMU of the bin
  uint64_t sy;          // sig_62 of 1/DMU
  int sh, pad0;         // 2045 less the exponent of 1/DMU
  double pad1;
};
RG_HD FaceCoef face_coef_mu(uint64_t c, const FaceMu& b) {
  FaceCoef q;
  const uint32_t h = (uint32_t)(c >> 32);
  q.sign = h & 0x80000000u;
  q.e = (int)((h >> 20) & 0x7FFu);
  q.m = sig_62(c);
  const uint64_t prod = mulhi_cross(q.m, b.sy) << 2;
  const int sh = b.sh - q.e;
  q.a63 = 0x7FFFFFFFFFFFFFFFULL - shr_clamp(prod, sh);
  q.bad = sh | hi32(q.a63) | (2046 - q.e);
  return q;
}
// Cells of 2^100 and more, and products phi below about 2^-919, are special
// too: with those limits one sign test of the exponent of phi covers every
// zero and subnormal operand.
constexpr uint32_t kFaceTop = (1023u + 100u) << 20;
constexpr int kFaceLow = 104;
// Special faces that carry phi = C*u all the same, for cells of [0, 2^100):
// C = 0 (c: C or a factor of it that vanishes with it), u = 0 (the
// difference to uu cannot have the sign of that to d), or d and u up to
// 1e-27 (|d-u| is too).  Loss cones decay to such cells within minutes, whole
// lines of them, and a dipole's C vanishes along whole meridians.
RG_HD bool face_plain(uint64_t uu, uint64_t u, uint64_t d, uint64_t c) {
  const uint32_t hu = (uint32_t)(u >> 32), hd = (uint32_t)(d >> 32), huu = (uint32_t)(uu >> 32);
  return max3u(hu, hd, huu) < kFaceTop && (u == 0 || (c << 1) == 0 || (hu < 0x3A53CE9Au && hd < 0x3A53CE9Au));
}

// phi = C * FBND rounded, from FBND as fb (2^59 <= u < 2^60 there) and u's
// exponent eu; top: the largest high word of the cells.
RG_HD uint64_t face_round(uint64_t fb, int eu, uint32_t top, const FaceCoef& q, bool& special) {
  const uint64_t p = mulhi_cross(fb, q.m);  // < 2^60
  const int tb = top_bit((uint32_t)(p >> 32));
  const int E = eu + q.e + tb - (1049 + kFaceLow);  // exponent field less one, less kFaceLow
  const uint64_t t = p >> ((tb - 21) & 63);
  special = top >= kFaceTop || (q.bad | E | hi32(fb) | (tb - 21)) < 0;
  const uint32_t field = ((uint32_t)E << 20) + (q.sign + ((uint32_t)kFaceLow << 20));
  return ((uint64_t)field << 32) + (t >> 1) + (t & 1ULL);
}

// phi as bits, from the bits of the cells.  kCase: cs is the limiter's
// branch (0 upwind only, 1 beta*D, 2 X, 3 D, 4 beta*X).
template <bool kCase, bool kB32>
RG_HD uint64_t face_flux(uint64_t uu, uint64_t u, uint64_t d, const FaceCoef& q, uint64_t betaf, bool& special,
                         int& cs) {
  const uint32_t hu = (uint32_t)(u >> 32), hd = (uint32_t)(d >> 32), huu = (uint32_t)(uu >> 32);
  const int eu = (int)(hu >> 20);
  const uint64_t mu = ((u << 7) & 0x07FFFFFFFFFFFFFFULL) | 0x0800000000000000ULL;
  const int sd = eu + 4 - (int)(hd >> 20), suu = eu + 4 - (int)(huu >> 20);
  const uint64_t ad = shr_clamp(sig_top(d), sd > 1 ? sd : 1);
  const uint64_t auu = shr_clamp(sig_top(uu), suu > 1 ? suu : 1);
  const uint64_t X = ad - mu, D = mu - auu;
  const int32_t s = hi32(X) >> 31;  // 0 or -1
  const uint64_t sm = ((uint64_t)(uint32_t)s << 32) | (uint32_t)s;
  // |X|, |D| where both have the sign s, one unit low when it is negative
  const uint64_t ax = X ^ sm, adx = D ^ sm;
  bool act = hi32(adx) >= 0;
  if (eu < 993) {
    // |X| > 1e-27.  From eu = 993 (u >= 2^-30) on, a difference below the
    // threshold is at most one unit here, whose correction is zero.  Below
    // eu = 932 (u < 4.1e-28) only an increase can pass it: d against u + 1e-27
    // in units of 2^-151.
    constexpr uint64_t t27 = 0x9E74D1B791E08000ULL;  // sig_top of 1e-27, exponent 933
    if (eu >= 932) {
      act = act && ax > shr_clamp(t27, eu - 929);
    } else {
      const int ed = (int)(hd >> 20);
      act = act && s == 0 &&
            (ed > 935 || shr_clamp(sig_top(d), 936 - ed) > shr_clamp(sig_top(u), 936 - eu) + (t27 >> 3));
    }
  }
  uint64_t lo, hi;
  const bool dlo = sort2(adx, ax, lo, hi);
  const uint64_t bl = beta_times<kB32>(lo, betaf);
  const uint64_t lim = bl < hi ? bl : hi;
  if (kCase) {
    const int c = dlo ? (bl <= hi ? 1 : 2) : (hi <= bl ? 3 : (betaf ? 4 : 2));
    cs = (act && X != 0 && D != 0) ? c : 0;
  }
  const uint64_t corr = act ? mulhi_cross(lim, q.a63) : 0ULL;
  const uint64_t fb = mu + (corr ^ sm) + (uint32_t)(-s);
  return face_round(fb, eu, max3u(hu, hd, huu), q, special);
}

// phi as bits with the limiter's branch cs given, as a record has it: the
// correction is 1/2 (1 - U) times beta*D, X, D or beta*X (cs 1..4) with its
// sign, whatever branch the cells select; the same bits as face_flux where
// they select cs.  (With the free form, and the FP64 form wherever its branch
// was another, replaying six calls of four species on 20x25x35x72 took 2.6 ms
// from the recorded state and 4.9 from one 1 % off it; 2.2 and 2.2 with this.)
// A difference of 2^61 units and more (2u to 4u) is special
// too: face_flux never takes one, and its cell may be saturated.
template <bool kB32>
RG_HD uint64_t face_flux_frozen(uint64_t uu, uint64_t u, uint64_t d, const FaceCoef& q, uint64_t betaf, int cs,
                                bool& special) {
  const uint32_t hu = (uint32_t)(u >> 32), hd = (uint32_t)(d >> 32), huu = (uint32_t)(uu >> 32);
  const int eu = (int)(hu >> 20);
  const uint64_t mu = ((u << 7) & 0x07FFFFFFFFFFFFFFULL) | 0x0800000000000000ULL;
  const bool ofd = (cs & 1) != 0;  // D, the difference to uu
  const int so = eu + 4 - (int)((ofd ? huu : hd) >> 20);
  const uint64_t ao = shr_clamp(sig_top(ofd ? uu : d), so > 1 ? so : 1);
  const uint64_t Z = ofd ? mu - ao : ao - mu;
  const int32_t s = hi32(Z) >> 31;  // 0 or -1
  const uint64_t sm = ((uint64_t)(uint32_t)s << 32) | (uint32_t)s;
  const uint64_t az = Z ^ sm;
  const bool kb = (cs == 1) | (cs == 4);
  const uint64_t lim = cs ? (kb ? beta_times<kB32>(az, betaf) : az) : 0ULL;
  const uint64_t fb = mu + (mulhi_cross(lim, q.a63) ^ sm) + (uint32_t)(-s);
  const uint64_t phi = face_round(fb, eu, max3u(hu, hd, huu), q, special);
  special = special || (cs && (uint32_t)(az >> 32) >= 0x20000000u);
  return phi;
}

}  // namespace ramgpu

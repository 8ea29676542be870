"""The fixed-point face flux (csrc/face.cuh) in the forms of the four sweeps:
the coefficient of DRIFTR and DRIFTP (U = |C|), of DRIFTE (C = k*v, U from the
bin) and of DRIFTMU (U = |C|/DMU), each with the general and the short beta,
on the CPU against exact rationals."""
import ctypes
import pathlib
import subprocess
from fractions import Fraction as Fr

import numpy as np
import pytest

from test_face import _cells

CSRC = pathlib.Path(__file__).resolve().parent.parent / "ram-scb_gb300" / "csrc"
HARNESS = r"""
#include "face.cuh"
#include <cstring>
using namespace ramgpu;
static uint64_t bits(double x) { uint64_t u; memcpy(&u, &x, 8); return u; }
// form 0: C = v (R, P); 1: C = k*v, U = |v|*ky (E); 2: C = v, U = |v|*ky (MU)
static FaceCoef coef(int form, double v, double k, double ky) {
  if (form == 0) return face_coef(bits(v));
  if (form == 1) {
    FaceBin b;
    b.k = k; b.sk = sig_62(bits(k)); b.sy = sig_62(bits(ky));
    b.e = (int)(bits(k) >> 52) - 1022; b.sh = 2045 - (int)(bits(ky) >> 52);
    return face_coef_bin(bits(v), b);
  }
  FaceMu m;
  m.sy = sig_62(bits(ky)); m.sh = 2045 - (int)(bits(ky) >> 52);
  return face_coef_mu(bits(v), m);
}
template <bool kB32>
static void go(long n, int form, const double* uu, const double* u, const double* d, const double* v, const double* k,
               const double* ky, double beta, double* phi, int* cs, int* special) {
  for (long i = 0; i < n; ++i) {
    bool s; int c = 0;
    const uint64_t p = face_flux<true, kB32>(bits(uu[i]), bits(u[i]), bits(d[i]), coef(form, v[i], k[i], ky[i]),
                                             beta_fix(bits(beta)), s, c);
    memcpy(&phi[i], &p, 8);
    cs[i] = c;
    special[i] = s;
  }
}
extern "C" int flux(long n, int form, int b32, const double* uu, const double* u, const double* d, const double* v,
                    const double* k, const double* ky, double beta, double* phi, int* cs, int* special) {
  if (b32) go<true>(n, form, uu, u, d, v, k, ky, beta, phi, cs, special);
  else go<false>(n, form, uu, u, d, v, k, ky, beta, phi, cs, special);
  return (uint32_t)beta_fix(bits(beta)) == 0u;
}
"""


@pytest.fixture(scope="module")
def flux(tmp_path_factory):
    t = tmp_path_factory.mktemp("forms")
    (t / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC), str(t / "h.cpp"), "-o",
                    str(t / "h.so")], check=True)
    lib = ctypes.CDLL(str(t / "h.so"))

    def call(form, b32, uu, u, d, v, k, ky, beta):
        n = len(u)
        phi, cs, sp = np.zeros(n), np.zeros(n, np.int32), np.zeros(n, np.int32)
        f8 = [np.ascontiguousarray(a, dtype=np.float64) for a in (uu, u, d, v, k, ky)]
        short = lib.flux(ctypes.c_long(n), form, b32, *[a.ctypes.data_as(ctypes.c_void_p) for a in f8],
                         ctypes.c_double(beta), *[a.ctypes.data_as(ctypes.c_void_p) for a in (phi, cs, sp)])
        assert short or not b32  # the short form is for such betas alone
        return phi, cs, sp
    return call


def _exact(uu, u, d, c, cu, beta):
    """C*FBND and the limiter's branch in rationals, Courant number cu (src/ModRamDrift.f90:169-183)."""
    uu, u, d, b = Fr(uu), Fr(u), Fr(d), Fr(beta)
    s = -1 if c < 0 else 1
    x, dd = s * (d - u), s * (u - uu)
    fb, cs = u, 0
    if abs(x) > Fr(1e-27) and x * dd > 0:
        m1, m2 = min(b * abs(dd), abs(x)), min(abs(dd), b * abs(x))
        m = max(m1, m2)
        cs = (1 if m1 == b * abs(dd) else 2) if m == m1 else (3 if m2 == abs(dd) else 4)
        fb += Fr(s) / 2 * (1 - cu) * m * (1 if x > 0 else -1)
    return c * fb, cs


def _coefs(form, rng, n):
    """v, k, ky of n faces with Courant numbers below 1 over the bins of real grids."""
    cu = np.where(rng.random(n) < 0.5, rng.random(n), np.exp(-25 * rng.random(n)))
    sg = rng.choice([-1.0, 1.0], n)
    if form == 0:
        return cu * sg, np.ones(n), np.ones(n)
    y = 1.0 / np.exp(rng.uniform(np.log(1e-4), np.log(100.0), n))  # 1/DE of 0.0001..100 keV, 1/DMU
    k = np.exp(rng.uniform(np.log(1e-2), np.log(1e3), n)) if form == 1 else np.ones(n)
    ky = k * y
    return cu * sg / ky, k, ky


@pytest.mark.parametrize("beta,b32", [(1.0, 1), (1.5, 1), (1.0, 0), (1.5, 0), (1.3, 0), (2.0, 0)])
@pytest.mark.parametrize("kind", ["smooth", "steep", "ulps", "binades", "threshold", "zeros"])
@pytest.mark.parametrize("form", [0, 1, 2])
def test_face_forms_arithmetic(flux, form, kind, beta, b32):
    """phi is within 2^-53 of C*FBND plus 2^-52 of |C|*u, the bar of the R and P
    form: the last rounding, and some ten truncations of 2^-59 of u, of which
    the product k*v adds two."""
    rng = np.random.default_rng(11 + form)
    n = 1500
    uu, u, d = _cells(kind, rng, n)
    v, k, ky = _coefs(form, rng, n)
    phi, cs, sp = flux(form, b32, uu, u, d, v, k, ky, beta)
    if kind in ("smooth", "ulps", "zeros", "binades") and beta < 2.0:
        assert sp.mean() <= 0.002  # a Courant number that rounds to 1
    assert (sp == 0).mean() > 0.6
    ties = 0
    for i in np.flatnonzero(sp == 0):
        c = Fr(v[i]) * Fr(k[i])
        e, case = _exact(uu[i], u[i], d[i], c, abs(Fr(v[i])) * Fr(ky[i]), beta)
        assert abs(Fr(phi[i]) - e) <= Fr(2.0 ** -53) * abs(e) + Fr(2.0 ** -52) * abs(c) * Fr(u[i]), (i, phi[i], float(e))
        ties += case != cs[i]
    assert ties <= 0.01 * n or kind in ("binades", "ulps")  # exact ties of beta*lo and hi may name either branch


@pytest.mark.parametrize("b32", [0, 1])
@pytest.mark.parametrize("form", [0, 1, 2])
def test_face_forms_leave_out(flux, form, b32):
    """Courant numbers of 1 and more, vanishing and non-finite coefficients and
    the cells that the fixed point does not hold are reported."""
    k, ky = (1.0, 1.0) if form == 0 else ((37.5, 3.7) if form == 1 else (1.0, 141.0))
    ok = lambda u, v: flux(form, b32, [1.0], [u], [1.3], [v], [k], [ky], 1.5)[2][0] == 0  # noqa: E731
    for cu in (1e-6, 0.1, 0.999999):
        for s in (-1.0, 1.0):
            assert ok(1.1, s * cu / ky), cu
    for cu in (1.0 + 1e-15, 1.5, 2.0, 3.9, 1e3, 1e18, 1e200):
        for s in (-1.0, 1.0):
            assert not ok(1.1, s * cu / ky), cu
    for v in (0.0, -0.0, 5e-324, np.inf, -np.inf, np.nan):
        assert not ok(1.1, v), v
    for u in (np.inf, np.nan, -1.0, -0.0, 0.0, 5e-324, 1e31):
        assert not ok(u, 0.1 / ky), u

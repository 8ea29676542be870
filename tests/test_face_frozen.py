"""The fixed-point face flux with the limiter's branch given (csrc/face.cuh), as
the adjoint's frozen replay takes it: on the CPU against exact rationals and
against the free form, and on the GPU the replay of windows far from the
recorded one."""
import ctypes
import pathlib
import subprocess
import time
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
template <bool kB32>
static void go(long n, const double* uu, const double* u, const double* d, const double* c, double beta, int* cs,
               double* phi, int* special) {
  for (long i = 0; i < n; ++i) {
    const FaceCoef q = face_coef(bits(c[i]));
    const uint64_t b = beta_fix(bits(beta));
    bool s; int k = 0;
    uint64_t p;
    if (cs[i] < 0) {  // the free form, and the branch it takes
      p = face_flux<true, kB32>(bits(uu[i]), bits(u[i]), bits(d[i]), q, b, s, k);
      cs[i] = k;
    } else {
      p = face_flux_frozen<kB32>(bits(uu[i]), bits(u[i]), bits(d[i]), q, b, cs[i], s);
    }
    memcpy(&phi[i], &p, 8);
    special[i] = s;
  }
}
extern "C" void flux(long n, int b32, const double* uu, const double* u, const double* d, const double* c, double beta,
                     int* cs, double* phi, int* special) {
  if (b32) go<true>(n, uu, u, d, c, beta, cs, phi, special);
  else go<false>(n, uu, u, d, c, beta, cs, phi, special);
}
"""


@pytest.fixture(scope="module")
def flux(tmp_path_factory):
    t = tmp_path_factory.mktemp("frozen")
    (t / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC), str(t / "h.cpp"), "-o",
                    str(t / "h.so")], check=True)
    lib = ctypes.CDLL(str(t / "h.so"))

    def call(b32, uu, u, d, c, beta, cs):
        n = len(u)
        cs, phi, sp = np.array(cs, np.int32), np.zeros(n), np.zeros(n, np.int32)
        f8 = [np.ascontiguousarray(a, dtype=np.float64) for a in (uu, u, d, c)]
        lib.flux(ctypes.c_long(n), b32, *[a.ctypes.data_as(ctypes.c_void_p) for a in f8], ctypes.c_double(beta),
                 *[a.ctypes.data_as(ctypes.c_void_p) for a in (cs, phi, sp)])
        return phi, cs, sp
    return call


@pytest.mark.parametrize("beta,b32", [(1.0, 1), (1.5, 1), (1.3, 0), (2.0, 0)])
@pytest.mark.parametrize("kind", ["smooth", "steep", "ulps", "binades", "threshold", "zeros"])
def test_frozen_face_arithmetic(flux, kind, beta, b32):
    """Every branch given, whatever the cells: phi is within the free form's bar
    (2^-53 of C*FBND plus 2^-52 of |C|*u); the branch that the cells select
    gives the free form's bits, and is never left to the FP64 form by the
    size of its difference."""
    rng = np.random.default_rng(23)
    n = 1000
    uu, u, d = _cells(kind, rng, n)
    c = np.where(rng.random(n) < 0.5, rng.random(n), np.exp(-25 * rng.random(n))) * rng.choice([-1.0, 1.0], n)
    free, taken, fsp = flux(b32, uu, u, d, c, beta, [-1] * n)
    again, _, sp = flux(b32, uu, u, d, c, beta, taken)
    ok = fsp == 0
    assert np.array_equal(free[ok], again[ok]) and not sp[ok].any()
    for cs in range(5):
        phi, _, sp = flux(b32, uu, u, d, c, beta, [cs] * n)
        assert (sp == 0).mean() > (0.3 if kind == "steep" else 0.6)
        for i in np.flatnonzero(sp == 0):
            a, b, e = Fr(uu[i]), Fr(u[i]), Fr(d[i])
            lx = [0, Fr(beta) * (b - a), e - b, b - a, Fr(beta) * (e - b)][cs]
            ex = Fr(c[i]) * (b + (1 - abs(Fr(c[i]))) / 2 * lx)
            assert abs(Fr(phi[i]) - ex) <= Fr(2.0 ** -53) * abs(ex) + Fr(2.0 ** -52) * abs(Fr(c[i])) * b, (cs, i)


def _window(gpu, wl, f2, calls, kp, obs, forward):
    for s in range(len(wl.grid.species)):
        gpu.upload_f2(0, s, np.asfortranarray(f2[s]))
        gpu.set_boundary(0, s, wl.fgeos[s])
    t = time.perf_counter()
    gpu.adj_forward(calls, wl.dts, kp, calls, obs) if forward else gpu.adj_replay()
    return time.perf_counter() - t


def _obs(calls):
    return [dict(member=0, s=0, call=c, k=12, l=1, lshell=4.5, mlt=3.0, log_obs=10.0) for c in range(calls)]


@pytest.mark.gpu
def test_replay_is_affine():
    """The frozen scheme is affine in F2: replays from f(1+e), f and f(1-e) with
    e up to 0.9 lie on a line, to 1e-12 of the largest cell (the step's bar)."""
    from ramgpu import abi, workload as W
    wl = W.make_workload("tiny_pert8")
    ns, kp = len(wl.grid.species), np.array([[3.0], [4.0]])
    gpu = abi.RamGpu(wl.grid, wl.fields)
    try:
        _window(gpu, wl, wl.f2, 2, kp, _obs(2), True)
        base = [gpu.download_f2(0, s) for s in range(ns)]
        rng = np.random.default_rng(3)
        e = [np.clip(0.3 * rng.normal(size=a.shape), -0.9, 0.9) for a in wl.f2]
        ends = []
        for sign in (0.0, 1.0, -1.0):
            _window(gpu, wl, [a * (1 + sign * q) for a, q in zip(wl.f2, e)], 2, kp, _obs(2), False)
            ends.append([gpu.download_f2(0, s) for s in range(ns)])
        for s in range(ns):
            assert np.array_equal(ends[0][s], base[s])
            assert np.abs(ends[1][s] + ends[2][s] - 2 * base[s]).max() <= 1e-12 * np.abs(base[s]).max(), s
            assert np.abs(ends[1][s] - base[s]).max() > 1e-2 * np.abs(base[s]).max()
    finally:
        gpu.close()


@pytest.mark.gpu
@pytest.mark.parametrize("spread", [0.0, 0.01, 0.3])
def test_replay_costs_no_more_than_recording(spread):
    """A replay does a recording pass's sweeps and writes no record: from the
    recorded state or one far from it, it takes no longer than the recording,
    with a margin of a quarter (best of six)."""
    from ramgpu import abi, workload as W
    wl = W.make_workload("four_sp")
    calls, kp = 3, np.array([[3.0], [4.0], [5.0]])
    rng = np.random.default_rng(4)
    f2 = [a * np.exp(spread * rng.normal(size=a.shape)) for a in wl.f2]
    gpu = abi.RamGpu(wl.grid, wl.fields)
    try:
        gpu.set_graph(True)
        rec = min(_window(gpu, wl, wl.f2, calls, kp, _obs(calls), True) for _ in range(6))
        rep = min(_window(gpu, wl, f2, calls, kp, _obs(calls), False) for _ in range(6))
        assert rep <= 1.25 * rec, (rep, rec)
    finally:
        gpu.close()

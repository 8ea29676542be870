"""The fixed-point face flux (csrc/face.cuh): its arithmetic on the CPU
against exact rationals, and the sweeps that use it on the GPU against the
oracle on states that reach its limits."""
import ctypes
import pathlib
import subprocess
from fractions import Fraction as Fr

import numpy as np
import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "ram-scb_gb300" / "csrc"
HARNESS = r"""
#include "face.cuh"
#include <cstring>
using namespace ramgpu;
static uint64_t bits(double x) { uint64_t u; memcpy(&u, &x, 8); return u; }
extern "C" void flux(long n, const double* uu, const double* u, const double* d, const double* c, const double* y,
                     double beta, double* phi, int* cs, int* special) {
  for (long i = 0; i < n; ++i) {
    bool s, s2; int k = 0, k2 = 0;
    const FaceCoef q = face_coef(bits(c[i]));
    const uint64_t a = face_flux<true, false>(bits(uu[i]), bits(u[i]), bits(d[i]), q, beta_fix(bits(beta)), s, k);
    const uint64_t b = face_flux<false, false>(bits(uu[i]), bits(u[i]), bits(d[i]), q, beta_fix(bits(beta)), s2, k2);
    memcpy(&phi[i], &a, 8);
    cs[i] = k;
    special[i] = s | (a != b && !s) << 1 | (s != s2) << 2;  // plain and recording forms: the same bits
  }
}
"""


@pytest.fixture(scope="module")
def flux(tmp_path_factory):
    d = tmp_path_factory.mktemp("face")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC), str(d / "h.cpp"), "-o", str(d / "h.so")],
                   check=True)
    lib = ctypes.CDLL(str(d / "h.so"))
    p = np.ctypeslib.ndpointer

    def call(uu, u, d_, c, y, beta):
        n = len(u)
        phi, cs, sp = np.zeros(n), np.zeros(n, np.int32), np.zeros(n, np.int32)
        f8, i4 = p(np.float64), p(np.int32)
        lib.flux.argtypes = [ctypes.c_long, f8, f8, f8, f8, f8, ctypes.c_double, f8, i4, i4]
        lib.flux(n, *[np.ascontiguousarray(a, dtype=np.float64) for a in (uu, u, d_, c, y)], beta, phi, cs, sp)
        return phi, cs, sp
    return call


def _exact(uu, u, d, c, beta, y=1.0):
    """C*FBND and the limiter's branch in rationals (src/ModRamDrift.f90:169-183)."""
    neg = c < 0
    x, dd = (Fr(u) - Fr(d), Fr(uu) - Fr(u)) if neg else (Fr(d) - Fr(u), Fr(u) - Fr(uu))
    fb, cs = Fr(u), 0
    if abs(x) > Fr(1e-27) and x * dd > 0:
        b, ax, ad = Fr(beta), abs(x), abs(dd)
        m1, m2 = min(b * ad, ax), min(ad, b * ax)
        m = max(m1, m2)
        cs = (1 if m1 == b * ad else 2) if m == m1 else (3 if m2 == ad else 4)
        a = Fr(-1 if neg else 1) / 2 * (1 - abs(Fr(c)) * Fr(y))
        fb += a * m * (1 if x > 0 else -1)
    return Fr(c) * fb, cs


def _cells(kind, rng, n):
    u = np.exp(rng.uniform(-8, 12, n))
    if kind == "smooth":
        f = lambda: np.exp(rng.uniform(-0.01, 0.01, n))  # noqa: E731
    elif kind == "steep":
        f = lambda: np.exp(rng.uniform(-30, 30, n))  # noqa: E731
    elif kind == "ulps":
        f = lambda: 1.0 + rng.integers(-6, 7, n) * 2.0 ** -52  # noqa: E731
    elif kind == "binades":
        u = 2.0 ** rng.integers(-3, 3, n)
        f = lambda: 2.0 ** rng.integers(-5, 6, n) * (1 + rng.integers(-1, 2, n) * 2.0 ** -52)  # noqa: E731
    elif kind == "threshold":
        u = u * 1e-27 * np.exp(rng.uniform(-12, 12, n))
        f = lambda: np.exp(rng.uniform(-2, 2, n) * rng.integers(0, 2, n))  # noqa: E731
    else:  # zeros beside the upwind cell
        f = lambda: rng.integers(0, 2, n) * np.exp(rng.uniform(-1, 1, n))  # noqa: E731
    return u * f(), u, u * f()


@pytest.mark.parametrize("beta", [1.0, 1.5, 1.3, 2.0])
@pytest.mark.parametrize("kind", ["smooth", "steep", "ulps", "binades", "threshold", "zeros"])
def test_face_flux_arithmetic(flux, kind, beta):
    """phi is within 2^-53 of C*FBND plus 2^-52 of the upwind flux |C|*u: one
    final rounding, and the fixed point's own 2^-59 units (u's last place is
    2^-52), against two roundings of that size and more in FP64."""
    rng = np.random.default_rng(7)
    n = 4000
    uu, u, d = _cells(kind, rng, n)
    c = np.where(rng.random(n) < 0.5, rng.random(n), np.exp(-25 * rng.random(n))) * rng.choice([-1.0, 1.0], n)
    phi, cs, sp = flux(uu, u, d, c, np.ones(n), beta)
    assert not (sp & 6).any()
    if kind in ("smooth", "ulps", "zeros", "binades") and beta < 2.0:
        assert not sp.any()
    assert (sp == 0).mean() > 0.6
    ties = 0
    for i in np.flatnonzero(sp == 0):
        e, k = _exact(uu[i], u[i], d[i], c[i], beta)
        assert abs(Fr(phi[i]) - e) <= Fr(2.0 ** -53) * abs(e) + Fr(2.0 ** -52) * Fr(abs(c[i])) * Fr(u[i]), (i, phi[i], float(e))
        ties += k != cs[i]
    assert ties <= 0.01 * n or kind in ("binades", "ulps")  # exact ties of beta*lo and hi may name either branch


def test_face_flux_leaves_out(flux):
    """Forms the fixed point does not hold are reported, whatever the other operands."""
    good = [1.0, 1.1, 1.3, 0.1]
    for bad in (np.inf, np.nan, -1.0, -0.0, -1e-300, 1e31):
        for at in range(3):
            v = list(good)
            v[at] = bad
            for c in (0.1, -0.1):
                v[3] = c
                assert flux(*[[x] for x in v], [1.0], 1.5)[2][0] & 1, v
    for u in (0.0, 5e-324, 1e-310):
        assert flux([1.0], [u], [2.0], [0.1], [1.0], 1.5)[2][0] & 1
    for c in (0.0, -0.0, 1.0, -1.5, np.inf, np.nan, 5e-324):
        assert flux([1.0], [1.1], [1.2], [c], [1.0], 1.5)[2][0] & 1, c


def _states(g, fields, kind, seed):
    from ramgpu import workload as W
    rng = np.random.default_rng(seed)
    out = []
    for s in range(len(g.species)):
        a = np.asfortranarray(W.initial_f2(g, fields, s, seed + s))
        if kind == "edge":
            a = W.edge_state([a], seed=seed)[0]
        elif kind == "nonperiodic":  # F(1) and F(NT) differ
            a[:, -1] *= rng.uniform(0.5, 2.0, a[:, -1].shape)
        elif kind == "tiny":  # magnitudes on both sides of 1e-27
            a *= np.exp(rng.uniform(-8, 8, a.shape)) * 1e-27 / np.median(a)
        elif kind == "negative":  # values the clip meets
            a *= rng.choice([1.0, 1.0, 1.0, -1.0], a.shape)
        elif kind == "huge":
            a *= 1e60
        out.append(np.asfortranarray(a))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["edge", "nonperiodic", "tiny", "negative", "huge"])
@pytest.mark.parametrize("beta", [1.5, 2.0, 1.3])
def test_sweeps_at_the_limits(kind, beta):
    """Each sweep alone against the oracle, cell by cell: within 64 roundings
    of the largest of the cell's neighbours along the swept axis (a cell is
    the sum of three terms of that size at Courant numbers near one, over a
    bin width ratio below 4)."""
    from ramgpu import abi, workload as W
    import pyoracle
    wl = W.make_workload("tiny_pert8")
    g = wl.grid
    gpu = abi.RamGpu(g, wl.fields, betalim=beta)
    o = pyoracle.Oracle(g, wl.fields, betalim=beta)
    vt = o.vt_vols(5.0)
    gpu.set_kp(0, 5.0)
    for axis, (op, which) in enumerate(((abi.OP_DRIFTR, "R"), (abi.OP_DRIFTP, "P"), (abi.OP_DRIFTE, "E"),
                                        (abi.OP_DRIFTMU, "MU"))):
        f2 = _states(g, wl.fields, kind, 31)
        for s in range(len(g.species)):
            gpu.upload_f2(0, s, f2[s])
            gpu.set_boundary(0, s, wl.fgeos[s])
        gpu.apply_op(wl.dts, op)
        for s in range(len(g.species)):
            ref = f2[s].copy(order="F")
            if which == "R" and s:
                continue  # the oracle's R sweep starts its stale ghosts afresh for one species as for all
            o.sweep(which, s, ref, vt, wl.dts, fgeos=wl.fgeos[s])
            got = gpu.download_f2(0, s)
            m = np.abs(f2[s])
            if which == "R":  # the boundary ghosts belong to the last cells' neighbourhood
                m[-2:] = np.maximum(m[-2:], 4 * np.abs(wl.fgeos[s]).max())
            n = m.shape[axis]
            wrap = np.take(m, np.arange(-3, n + 3) % n if which == "P" else np.clip(np.arange(-3, n + 3), 0, n - 1), axis)
            scale = np.max([np.take(wrap, np.arange(q, q + n), axis) for q in range(7)], axis=0)
            bad = np.abs(got - ref) > 64 * 2.0 ** -53 * scale
            assert not bad.any(), (which, s, int(bad.sum()), np.argwhere(bad)[:3].tolist())
    gpu.close()


@pytest.mark.gpu
@pytest.mark.parametrize("field", ["dipole", "perturbed"])
@pytest.mark.parametrize("nr", [4, 6, 23, 25, 26, 28, 30, 32])
def test_radial_widths(nr, field):
    """Grids of every DRIFTR access width (one, two or four cells), at the
    smallest and at both sides of each rule: two calls against the oracle,
    1e-12 of the largest cell (the step's parity bar)."""
    from ramgpu import abi, workload as W
    import pyoracle
    g = W.arrays(nr, 9, 35, 72, species=(W.HYDROGEN,), mu_grid_nr=20)
    f = W.perturbed_fields(g, seed=nr) if field == "perturbed" else W.dipole_fields(g, seed=nr)
    f2, fg = np.asfortranarray(W.initial_f2(g, f, 0, nr)), W.boundary_fgeos(g, 0)
    gpu, o = abi.RamGpu(g, f), pyoracle.Oracle(g, f)
    gpu.upload_f2(0, 0, f2)
    gpu.set_boundary(0, 0, fg)
    ref = [f2.copy(order="F")]
    for c in range(2):
        gpu.set_kp(0, 3.0 + c)
        gpu.ram_run(3.0)
        out = o.ram_run(ref, [fg], 3.0, kp=3.0 + c)
        got = gpu.download_f2(0, 0)
        assert np.abs(got - ref[0]).max() <= 1e-12 * np.abs(ref[0]).max()
        assert abs(gpu.cfl(0, 0)[4] - out["dts_next"]) <= 1e-12 * out["dts_next"]
    gpu.close()


@pytest.mark.gpu
def test_lane_counts_agree():
    """DRIFTE and DRIFTMU share a line among 4 and 8 lanes for one member of
    the reduced grid and among fewer as members join: member 0's F2, moments
    and Courant limits are the same bits in every list."""
    from ramgpu import abi, workload as W
    wl = W.make_workload("tiny_pert")
    g, ns = wl.grid, len(wl.grid.species)
    first = None
    for members in (1, 3, 16, 24):
        gpu = abi.RamGpu(g, wl.fields, n_members=members)
        for m in range(members):
            for s in range(ns):
                gpu.upload_f2(m, s, np.asfortranarray(wl.f2[s]))
                gpu.set_boundary(m, s, wl.fgeos[s])
        gpu.set_kp_all([4.0] * members)
        for _ in range(3):
            gpu.ram_run(wl.dts)
        got = [gpu.download_f2(0, s) for s in range(ns)] + [np.array(gpu.moments(0, s)) for s in range(ns)] \
            + [gpu.cfl(0, s) for s in range(ns)]
        gpu.close()
        if first is None:
            first = got
        for a, b in zip(got, first):
            assert np.array_equal(a, b), members


@pytest.mark.gpu
def test_transposed_lane_counts_agree():
    """The DRIFTMU transpose shares a line among 4, 2 or 1 lanes as members
    join: member 0's misfit and dJ/dF2 are the same bits (a cell collects its
    faces in the same order), dJ/dFGEOS to the rounding of its atomics."""
    from ramgpu import abi, workload as W
    wl = W.make_workload("tiny_pert")
    g, ns = wl.grid, len(wl.grid.species)
    obs = [{"member": 0, "s": s, "call": c, "k": 10 + 3 * s, "l": 1 + c, "lshell": 3.0 + 0.5 * s, "mlt": 6.0 * c,
            "log_obs": 0.0} for s in range(ns) for c in range(2)]
    first = None
    for members in (1, 9, 24):
        gpu = abi.RamGpu(g, wl.fields, n_members=members)
        for m in range(members):
            for s in range(ns):
                gpu.upload_f2(m, s, np.asfortranarray(wl.f2[s]))
                gpu.set_boundary(m, s, wl.fgeos[s])
        j = gpu.adj_forward(2, wl.dts, np.full((2, members), 4.0), 1, obs)[0]
        gf, gb = gpu.adj_backward()
        gpu.close()
        if first is None:
            first = (j, gf[0], gb[0])
        assert j == first[0] and np.array_equal(gf[0], first[1])
        assert np.abs(gb[0] - first[2]).max() <= 1e-13 * np.abs(first[2]).max()


@pytest.mark.gpu
@pytest.mark.parametrize("beta", [1.0, 1.3, 1.5, 2.0])
@pytest.mark.parametrize("dts", [5.0, 400.0])
def test_transposes_at_the_limits(dts, beta):
    """The transposes' fixed-point weights, and at the long step the FP64
    ones of faces with Courant numbers above 1: one call's misfit and
    gradients against the oracle at the window test's bars (1e-12, 1e-9)."""
    from ramgpu import abi, workload as W
    import pyoracle
    wl = W.make_workload("tiny_pert8")
    g, ns = wl.grid, len(wl.grid.species)
    obs = [{"member": 0, "s": s, "call": 0, "k": 6 + 5 * n, "l": 1 + 9 * n, "lshell": 3.0 + 0.7 * n, "mlt": 5.0 * n,
            "log_obs": 0.0} for s in range(ns) for n in range(5)]
    gpu, o = abi.RamGpu(g, wl.fields, betalim=beta), pyoracle.Oracle(g, wl.fields, betalim=beta)
    try:
        for s in range(ns):
            gpu.upload_f2(0, s, np.asfortranarray(wl.f2[s]))
            gpu.set_boundary(0, s, wl.fgeos[s])
        j = gpu.adj_forward(1, dts, np.full((1, 1), 4.0), 1, obs)[0]
        gf, gb = gpu.adj_backward()
        gpu.ram_run(dts)  # (a recorded call keeps no limits)
        assert (gpu.cfl(0, 1).min() < 0.8 * dts) == (dts > 100.0)  # Courant numbers above 1 at the long step
    finally:
        gpu.close()
    jc, cf, cb = o.window_gradient([np.asfortranarray(a) for a in wl.f2], [np.asfortranarray(a) for a in wl.fgeos], dts,
                                   [4.0], obs)
    assert abs(j - jc) <= 1e-12 * jc
    for s in range(ns):
        assert np.abs(gf[0, s] - cf[s]).max() <= 1e-9 * np.abs(cf[s]).max(), s
        assert np.abs(gb[0, s] - cb[s]).max() <= 1e-9 * max(np.abs(cb[s]).max(), 1e-300), s

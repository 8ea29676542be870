"""The kinetic step's measured cases: what users of this framework have it do.

Every case goes through ``ramgpu.abi.RamGpu`` (or the autograd wrapper) as a
time loop does: set Kp, advance with ram_run, and hand the moments on.  A
pass of several calls stands for a coupling interval, after which SCB reads
the pressures.  ``exact`` restates the step with plain torch in 64 bits,
from the formulas of src/ModRamDrift.f90, src/ModRamLoss.f90,
src/ModRamWPI.f90 and src/ModRamRun.f90, without the library.
"""
from __future__ import annotations

import functools
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "ram-scb_gb300"))

from ramgpu import abi, autograd  # noqa: E402
from ramgpu import workload as W  # noqa: E402

# per species of the four-species configuration: kT [keV], share of the density
SPEC = {code: (kt, share) for code, kt, share in W.FOUR_SPECIES}
LETTER = {"e": "e", "H": "H", "h": "He", "O": "O"}  # a case's "species" text, one letter each


def listed():
    std = dict(gen="std", nr=20, nt=25, ne=35, npa=72, dts=5.0, members=1, field="dipole", graph=True)
    four = dict(std, species="eHhO")
    return [
        # the reduced grid with one species, one call a pass: launches and host work count
        dict(std, name="tiny_h", kind="run", species="H", nr=6, nt=9, calls=1),
        # the same grid family in a non-dipole field with magnetopause cells, direct launches
        dict(four, name="tiny_nondipole", kind="run", nr=8, nt=9, field="perturbed", calls=1, graph=False),
        # one ion on the standard grid, the plain method
        dict(std, name="single_h", kind="run", species="H", calls=6),
        # the production step: four species on the standard grid over a coupling interval
        dict(four, name="four_species", kind="run", calls=6),
        # a ragged grid in a compressed field with induced E and dB/dt, two ions
        dict(std, name="ragged_nondipole", kind="run", species="HO", nr=23, nt=30, ne=37, npa=69, dts=4.0,
             field="perturbed", calls=4),
        # the refined grid, whose working set is past L2
        dict(four, name="refined", kind="run", gen="ref", nr=40, nt=49, ne=70, npa=144, dts=2.5, calls=2),
        # an ensemble of members with uneven species sets and their own Kp
        dict(four, name="ensemble", kind="run", members=24, calls=2),
        # electrons with implicit pitch-angle diffusion beside the ions
        dict(four, name="diffusion", kind="run", diffusion=True, calls=4),
        # the SUMRC loss bookkeeping of a run that reports its loss channels
        dict(std, name="loss_books", kind="run", species="HO", losses=True, calls=4),
        # F2 kept by the host in page-locked per-species arrays, moved each call
        dict(four, name="host_arrays", kind="host", calls=1),
        # the Fortran array F2(NS,NR,NT,NE,NPA) as it is, pageable
        dict(four, name="ref_layout", kind="ref", calls=1),
        # data assimilation: misfit of an observed window and its gradients
        dict(four, name="adjoint", kind="adj", calls=6, ckpt=2, nobs=50),
    ]


def _ncell(c):
    return c["nr"] * c["nt"] * c["ne"] * c["npa"]


def _items(c):
    return sum(len(s) for s in _member_species(c))


def _cost(c):
    return _ncell(c) * _items(c) * c["calls"] * (4 if c["kind"] == "adj" else 1)


def draw(rng):
    most = max(_cost(c) for c in listed())
    logi = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    while True:
        kind = rng.choice(["run", "run", "run", "run", "host", "ref", "adj"])
        c = dict(kind=kind, members=1, graph=rng.random() < 0.8, field=rng.choice(["dipole", "perturbed"]))
        if rng.random() < 0.25:
            c.update(gen="ref", nr=rng.randint(20, 40), nt=rng.randint(19, 49), ne=rng.choice([35, 70]), npa=144)
        else:
            c.update(gen="std", nr=logi(6, 28), nt=logi(9, 40), ne=rng.randint(32, 39), npa=rng.randint(60, 72))
        c["species"] = "".join(x for x in "eHhO" if rng.random() < 0.6) or "H"
        c["dts"] = round(5.0 * min(1.0, 19.0 / (c["nr"] - 1), 24.0 / (c["nt"] - 1)), 3)
        c["calls"] = rng.randint(1, 6) if kind in ("run", "adj") else 1
        if kind == "run":
            c["members"] = rng.choice([1, 1, 1, logi(2, 16)])
            c["diffusion"] = "e" in c["species"] and rng.random() < 0.25
            c["losses"] = rng.random() < 0.2
        if kind == "adj":
            c.update(ckpt=rng.randint(1, c["calls"]), nobs=rng.randint(5, 60))
        if _cost(c) <= most:
            return c


# ------------------------------------------------------------------ inputs
def _rng(seed, *more):
    return np.random.Generator(np.random.PCG64([seed, *more]))


def _member_species(c):
    """Per member the species it carries: all of them, or uneven subsets in an ensemble."""
    ns = len(c["species"])
    r = random.Random(101 * c["members"] + ns)
    return [sorted(r.sample(range(ns), r.randint(1, ns))) if c["members"] > 1 else list(range(ns))
            for _ in range(c["members"])]


@functools.lru_cache(maxsize=32)
def _grid(gen, nr, nt, ne, npa, species):
    sp = tuple(W.SPECIES[LETTER[x]] for x in species)
    if gen == "ref":
        return W.refined_arrays(nr, nt, ne, npa, species=sp, dl1=0.125)
    return W.arrays(nr, nt, ne, npa, species=sp, mu_grid_nr=20)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a, order=None):
    """A host array on the device in 64 bits, its axes reordered."""
    a = np.asarray(a, dtype=np.float64)
    return torch.from_numpy(np.ascontiguousarray(a.transpose(order) if order else a)).to(_device())


def _inputs(c, seed):
    """(grid, fields, F2 (members, species, NPA, NE, NT, NR), FGEOS per species, Kp (calls, members))."""
    g = _grid(c["gen"], c["nr"], c["nt"], c["ne"], c["npa"], c["species"])
    f = W.perturbed_fields(g, seed=seed) if c["field"] == "perturbed" else W.dipole_fields(g, seed=seed)
    gen = torch.Generator(device=_device())
    gen.manual_seed(9000 + seed)
    nm, ns = c["members"], len(c["species"])
    radial = torch.exp(-(_t(g.lz[:g.nr]) - 4.5) ** 2 / (2.0 * 0.8 ** 2))
    azim = 1.0 + 0.2 * torch.cos(_t(g.phi))
    sin2 = 1.0 - _t(g.mu) ** 2
    fnhs = _t(f.fnhs[:g.nr], (2, 1, 0))
    f2 = torch.empty((nm, ns, g.npa, g.ne, g.nt, g.nr), dtype=torch.float64, device=_device())
    scale = _rng(seed, 1).lognormal(0.0, 0.5, size=nm) if nm > 1 else np.ones(1)
    fgeos = []
    for s, x in enumerate(c["species"]):
        kt, share = SPEC[LETTER[x]]
        je = _t(W.kappa_flux(g.ekev, kt) * share)
        shape = sin2[:, None, None, None] * je[:, None, None] * azim[:, None] * radial
        shape = shape * _t(g.ffactor[s], (2, 1, 0))[:, :, None, :] * fnhs[:, None]
        for m in range(nm):
            noise = torch.randn(shape.shape, generator=gen, dtype=torch.float64, device=_device())
            f2[m, s] = shape * scale[m] * torch.exp(0.01 * noise)
        fgeos.append(W.boundary_fgeos(g, s, kt=kt, density_scale=share))
    f2[..., g.nt - 1, :] = f2[..., 0, :]
    kp = 1.0 + 5.0 * _rng(seed, 2).random(nm)[None, :] + 0.05 * np.arange(c["calls"])[:, None]
    return g, f, f2, fgeos, kp


def _diffusion(g, f, seed):
    return W.pa_diffusion(g, f, seed=seed)


def _stencil(g, lshell, mlt):
    """Bilinear corners and upper weights of an equatorial point on the flux grid."""
    i0 = 1
    while i0 + 1 < g.nr - 1 and g.lz[i0 + 1] <= lshell:
        i0 += 1
    wi = min(1.0, max(0.0, (lshell - g.lz[i0]) / (g.lz[i0 + 1] - g.lz[i0])))
    ph = math.fmod(mlt * W.PI / 12.0, 2.0 * W.PI)
    j0 = min(int(ph / g.dphi), g.nt - 2)
    wj = min(1.0, max(0.0, (ph - g.phi[j0]) / g.dphi))
    j1 = 0 if j0 + 1 == g.nt - 1 else j0 + 1
    return [(i0, j0, (1 - wi) * (1 - wj)), (i0, j1, (1 - wi) * wj), (i0 + 1, j0, wi * (1 - wj)), (i0 + 1, j1, wi * wj)]


def _observations(c, g, f, f2, seed):
    """Equatorial samples at L = 4-6, 10-200 keV, second pitch-angle bin, about the initial flux."""
    r = _rng(seed, 3)
    ks = [k for k in range(1, g.ne) if 10.0 <= g.ekev[k] <= 200.0]
    obs = []
    for _ in range(c["nobs"]):
        o = dict(member=0, s=int(r.integers(len(c["species"]))), call=int(r.integers(c["calls"])),
                 k=int(r.choice(ks)), l=1, lshell=float(r.uniform(4.0, 6.0)), mlt=float(r.uniform(0.0, 24.0)))
        v = sum(w * float(f2[0, o["s"], o["l"], o["k"], j, i]) / g.ffactor[o["s"], i, o["k"], o["l"]]
                / f.fnhs[i, j, o["l"]] for i, j, w in _stencil(g, o["lshell"], o["mlt"]))
        o["log_obs"] = math.log(v) + float(r.normal(0.0, 0.3))
        obs.append(o)
    return obs


class _View:
    """Device memory of a context as torch sees it; the tensor keeps the context."""

    def __init__(self, gpu, ptr, shape):
        self.gpu = gpu
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr="<f8", data=(ptr, False), version=3, strides=None)


def prepare(case, seed):
    g, f, f2, fgeos, kp = _inputs(case, seed)
    gpu = abi.RamGpu(g, f, n_members=case["members"], flags=abi.FLAG_LOSSES if case.get("losses") else 0)
    state = dict(case=case, gpu=gpu, kp=kp)
    for m, sp in enumerate(_member_species(case)):
        if len(sp) < len(case["species"]):
            gpu.set_member_species(m, sp)
        for s in range(len(fgeos)):
            gpu.set_boundary(m, s, fgeos[s])
    if case["graph"]:
        gpu.set_graph(True)
    if case.get("diffusion"):
        gpu.set_pa_diffusion(0, _diffusion(g, f, seed))
    if case["kind"] == "host":
        state["f2"], state["pe"], state["pa"] = [], [], []
        for s in range(f2.shape[1]):
            for key, src in (("f2", f2[0, s].reshape(-1)), ("pe", torch.zeros(g.nr * g.nt)), ("pa", torch.zeros(g.nr * g.nt))):
                buf = torch.empty(src.numel(), dtype=torch.float64, pin_memory=True)
                buf.copy_(src)
                state[key].append(buf.numpy())
    elif case["kind"] == "ref":
        a = f2[0].cpu().numpy().transpose(0, 4, 3, 2, 1)  # (NS, NR, NT, NE, NPA)
        state["f2"] = np.asfortranarray(a).copy(order="F")
        state["pe"], state["pa"] = (np.zeros((a.shape[0], g.nr, g.nt), order="F") for _ in range(2))
    elif case["kind"] == "adj":
        state["obs"] = _observations(case, g, f, f2, seed)
        state["f2"] = f2.requires_grad_()
        state["fgeos"] = _t(np.stack([x.transpose(2, 1, 0) for x in fgeos])[None]).requires_grad_()
    else:
        state["f2"] = torch.as_tensor(_View(gpu, gpu.f2_device_ptr(0, 0), f2.shape), device="cuda")
        state["f2"].copy_(f2)
        torch.cuda.synchronize()
        if case.get("losses"):
            gpu.reset_losses()
    return state


def run(state):
    c, gpu, kp = state["case"], state["gpu"], state["kp"]
    dts = c["dts"]
    if c["kind"] == "host":
        gpu.set_kp(0, kp[0, 0])
        gpu.ram_run_host(dts, state["f2"], state["pe"], state["pa"])
        return dict(f2=state["f2"], pe=state["pe"], pa=state["pa"])
    if c["kind"] == "ref":
        gpu.set_kp(0, kp[0, 0])
        gpu.ram_run_ref(dts, [state["f2"]], [state["pe"]], [state["pa"]])
        return dict(f2=state["f2"], pe=state["pe"], pa=state["pa"])
    if c["kind"] == "adj":
        f2, fg = state["f2"], state["fgeos"]
        f2.grad = fg.grad = None
        j = autograd.window_misfit(gpu, f2, fg, c["calls"], dts, kp, c["ckpt"], state["obs"])
        j.sum().backward()
        return dict(j=j.detach(), gf2=f2.grad, gfgeos=fg.grad)
    for k in range(c["calls"]):
        gpu.set_kp_all(kp[k])
        gpu.ram_run(dts)
    pairs = [(m, s) for m in range(c["members"]) for s in gpu.member_species[m]]
    out = dict(f2=state["f2"], moments=np.array([gpu.moments(m, s) for m, s in pairs]),
               cfl=np.array([gpu.cfl(m, s) for m, s in pairs]))
    if c.get("losses"):
        out["losses"] = np.array([gpu.losses(m, s) for m, s in pairs])
    return out


def work(case):
    cells = _ncell(case) * _items(case)
    # every F2 value is read once and written once a pass (and for the
    # adjoint its gradient written); per cell, call and half step the four
    # sweeps need about 12 + 12 + 15 + 14 operations, the moments 4
    ops = cells * case["calls"] * (2 * 53 + 4)
    if case["kind"] == "adj":
        return dict(bytes=16.0 * cells, flops=3.0 * ops)
    return dict(bytes=16.0 * cells, flops=float(ops))


# ------------------------------------------------------------------- exact
# Axes are (L, K, J, I) throughout, a species' block of F2 as it is laid out.
def _limited(x, d, up, a, beta):
    """FBND of a face: upwind value plus a*LIMITER(D/X)*X (src/ModRamDrift.f90:169-183)."""
    ax, ad = x.abs(), d.abs()
    lim = torch.maximum(torch.minimum(beta * ad, ax), torch.minimum(ad, beta * ax))
    on = (ax > 1e-27) & (((d > 0) & (x > 0)) | ((d < 0) & (x < 0)))
    return up + torch.where(on, a * lim * torch.sign(x), torch.zeros_like(x))


def _clip(v):
    return torch.where(v < 0, torch.full_like(v, 1e-15), v)


class _Exact:
    def __init__(self, c, g, f, kp):
        self.c, self.g, self.f = c, g, f
        self.beta, self.fraccfl, self.dtsmin = 1.5, 0.8, 0.1
        n = g.nr
        self.f3 = {k: _t(getattr(f, k), (2, 1, 0)) for k in ("fnhs", "fnis", "bounhs", "bounis", "hdns", "didt", "dibndt")}
        self.f2d = {k: _t(getattr(f, k), (1, 0)) for k in ("bnes", "dbdt", "eir", "eip")}
        self.outside = torch.from_numpy(np.ascontiguousarray(np.asarray(f.outside).T)).to(_device()) == 1
        self.j0 = torch.tensor([g.nt - 2] + list(range(g.nt - 1)), device=_device())
        self.j1 = torch.tensor(list(range(1, g.nt)) + [1], device=_device())
        self.rlz, self.lz = _t(g.rlz), _t(g.lz)
        self.ekev, self.ebnd, self.we, self.de = (_t(getattr(g, k)) for k in ("ekev", "ebnd", "we", "de"))
        self.mu, self.wmu, self.dmu = _t(g.mu), _t(g.wmu), _t(g.dmu)
        fh, fi, b = self.f3["fnhs"], self.f3["fnis"], self.f2d["bnes"]
        mdr, dphi = g.mdr, g.dphi
        rad = slice(0, n)       # I
        nxt = slice(1, n + 1)   # I+1
        self.rad, self.nxt = rad, nxt
        j0, j1 = self.j0, self.j1
        cgr1 = fi[:, j1][..., nxt] + fi[:, j1][..., rad] - fi[:, j0][..., nxt] - fi[:, j0][..., rad]
        cgr2 = b[j1][:, nxt] + b[j1][:, rad] - b[j0][:, nxt] - b[j0][:, rad]
        cgr3 = cgr1 + (fi[..., nxt] + fi[..., rad] - 2 * fh[..., nxt] - 2 * fh[..., rad]) * cgr2 / 2 / (b[:, nxt] + b[:, rad])
        self.grt = cgr3 / (fh[..., rad] + fh[..., nxt]) / 2 / (b[:, rad] + b[:, nxt]) / (self.rlz[rad] + 0.5 * mdr)

    def potential(self, kp):
        g = self.g
        t = 1.0 - 0.159 * kp + 0.0093 * (kp * kp)
        avs = 7.05e-6 / (t * t * t) / W.RE
        return avs * (self.lz * W.RE) ** 2 * torch.sin(_t(g.phi))[:, None]  # (J, I')

    def coefficients(self, s, vt, dts):
        """Face coefficients of the four sweeps for species s."""
        g, n = self.g, self.g.nr
        mdr, dphi, R, j0, j1 = g.mdr, g.dphi, self.rlz[1:n], self.j0, self.j1
        fh, fi, bh, bi = (self.f3[k] for k in ("fnhs", "fnis", "bounhs", "bounis"))
        b, dbdt, eir, eip = (self.f2d[k] for k in ("bnes", "dbdt", "eir", "eip"))
        q = float(g.species[s].charge)
        rad, nxt = self.rad, self.nxt
        mid, up, dn = slice(1, n), slice(2, n + 1), slice(0, n - 1)  # I, I+1, I-1 for I >= 2
        gr, gb = _t(g.grel[s]), _t(g.grbnd[s])
        den = b[:, rad] + b[:, nxt]
        vr = dts / mdr / (self.rlz[rad] + 0.5 * mdr) / 2 / dphi
        cr = vr * (vt[j0][:, rad] + vt[j0][:, nxt] - vt[j1][:, rad] - vt[j1][:, nxt]) / den + (eip[:, rad] + eip[:, nxt]) / den * dts / mdr
        p4 = dts * self.ekev * 1000 * (gr + 1) / gr / dphi / mdr / q
        cR = self.grt[:, None] * p4[:, None, None] + cr
        # phi faces, J = 2..NT used
        fj, fj1 = fi, fi[:, j1]
        hj, hj1 = fh, fh[:, j1]
        denp = b[:, mid] + b[j1][:, mid]
        gpa1 = fj[..., mid] + fj1[..., mid] + (fj1[..., up] + fj[..., up] - fj[..., dn] - fj1[..., dn]) * R / 2 / mdr
        gpa2 = R / 4 / mdr * (fj[..., mid] + fj1[..., mid] - 2 * hj[..., mid] - 2 * hj1[..., mid]) * \
            (b[j1][:, up] + b[:, up] - b[:, dn] - b[j1][:, dn]) / denp
        gpt = -(gpa1 + gpa2) / (hj[..., mid] + hj1[..., mid]) / denp
        ca = ((vt[:, up] + vt[j1][:, up] - vt[:, dn] - vt[j1][:, dn]) / 2 / mdr - eir[j1][:, mid] - eir[:, mid]) / R * dts / dphi / denp \
            + 7.3e-5 * dts / dphi
        p2 = dts * self.ekev[:, None] * 1000 * ((gr + 1) / gr)[:, None] / R ** 2 / dphi / q
        cP = gpt[:, None] * p2[:, None, :] + ca
        # energy faces
        m, bm = fi[..., mid], b[:, mid]
        h = fh[..., mid]
        gpa = (1 - m / 2 / h) / bm
        dbr, dbp = b[:, up] - b[:, dn], b[j1][:, mid] - b[j0][:, mid]
        dir_, dip = fi[..., up] - fi[..., dn], fi[:, j1][..., mid] - fi[:, j0][..., mid]
        gre = gpa * dbr / 2 / mdr - m / h / R - dir_ / 2 / mdr / h
        gpe = gpa * dbp / 2 / dphi - dip / 2 / dphi / h
        drd1 = (eip[:, mid] * R - (vt[j1][:, mid] - vt[j0][:, mid]) / 2 / dphi) / bm
        dpd1 = 7.3e-5 * R + ((vt[:, up] - vt[:, dn]) / 2 / mdr - eir[:, mid]) / bm
        drd2 = dip / 2 / dphi + (m - 2 * h) * dbp / 4 / bm / dphi
        dpd2 = m + dir_ * R / 2 / mdr + R * (m - 2 * h) / 4 / mdr * dbr / bm
        ze = dbdt[:, mid] * (1 - m / 2 / h) * R / bm - self.f3["didt"][..., mid] * R / h
        ue = gre * drd1 + gpe * dpd1 + ze
        wet = (gre * drd2 * R - gpe * dpd2) / h / R / bm
        eb = self.ebnd * 1e3 * (gb + 1) / 2 / gb / q
        edot = self.ebnd[:, None] * dts / R * ((gb + 1) / gb / 2)[:, None]
        cE = edot[:, None, :] * (ue[:, None] + eb[:, None, None] * wet[:, None])
        # pitch-angle faces
        m, h = bi[..., mid], bh[..., mid]
        dir_, dip = bi[..., up] - bi[..., dn], bi[:, j1][..., mid] - bi[:, j0][..., mid]
        gmr = dbr / 4 / mdr / bm + 1 / R + dir_ / 2 / mdr / m
        gmp = dbp / 4 / dphi / bm + dip / 2 / dphi / m
        drm2 = dip / 2 / dphi + (m - 2 * h) * dbp / 4 / bm / dphi
        dpm2 = m + dir_ * R / 2 / mdr + (m - 2 * h) * R / 4 / mdr * dbr / bm
        zm = dbdt[:, mid] / 2 / bm * R + self.f3["dibndt"][..., mid] * R / m
        mub = self.mu + 0.5 * self.wmu
        mudot = ((1 - mub ** 2) * dts / 2 / mub)[:, None, None] / R
        ek = self.ekev * 1e3 * (gr + 1) / 2 / gr / q
        um = gmr * drd1 + gmp * dpd1 + zm
        hm = (gmr * drm2 * R - gmp * dpm2) / h / R / bm
        cM = -(mudot * m / h)[:, None] * (um[:, None] + ek[:, None, None] * hm[:, None])
        return cR, cP, cE, cM

    def sweep_r(self, F, fg, cc):
        """fg: FGEOS (L, K, J)."""
        g, n, c = self.g, self.g.nr, cc[0]
        inflow = c[..., n - 1] < 0
        ghost = torch.where(self.outside[:, n - 1], torch.zeros_like(fg), fg * self.f3["fnhs"][..., n - 1][:, None])
        # F(NR+1) left by the last inflow line before, in K -> L -> J order
        perm = (1, 0, 2)
        fl = inflow.permute(perm).reshape(-1)
        at = torch.where(fl, torch.arange(fl.numel(), device=fl.device), torch.full((), -1, device=fl.device))
        last = torch.cummax(at, 0).values
        gv = (ghost * g.conf1).permute(perm).reshape(-1)
        stale = torch.where(last >= 0, gv[last.clamp(min=0)], torch.zeros_like(gv))
        stale = stale.reshape(g.ne, g.npa, g.nt).permute(perm)
        g1 = torch.where(inflow, ghost * g.conf1, stale)
        g2 = torch.where(inflow, ghost * g.conf2, torch.zeros_like(ghost))
        G = torch.cat([F, g1[..., None], g2[..., None]], -1)
        x = G[..., 1:] - G[..., :-1]                   # X of face I at index I-1
        cf = c[..., 1:]                                # faces 2..NR
        neg = cf < 0
        fb = _limited(x[..., 1:n], torch.where(neg, x[..., 2:n + 1], x[..., 0:n - 1]), torch.where(neg, G[..., 2:n + 1], G[..., 1:n]),
                      0.5 * (torch.where(neg, -1.0, 1.0) - cf), self.beta)
        fb = torch.cat([fb[..., :-1], torch.where(inflow, fb[..., -1], F[..., n - 1])[..., None]], -1)
        first = torch.where(inflow, F[..., 1], torch.zeros_like(F[..., 1]))
        phi = c * torch.cat([first[..., None], fb], -1)
        return torch.cat([F[..., :1], _clip(F[..., 1:] - phi[..., 1:] + phi[..., :-1])], -1)

    def sweep_p(self, F, cc):
        n, c = self.g.nt, cc[1][..., 1:, :]            # faces J = 2..NT
        G = F[..., 1:]
        # cells J-1 .. J+2 of face J, with J = NT+1 -> 2, NT+2 -> 3 and, as
        # the reference wraps its index, D of face NT-1 from cells 1 and 2
        x = G[..., 1:, :] - G[..., :-1, :]             # F(J+1)-F(J), J = 1..NT-1
        xw = torch.cat([x, (G[..., 1, :] - G[..., n - 1, :])[..., None, :]], -2)  # and J = NT
        xf = xw[..., 1:, :]                            # X of faces 2..NT
        dm = xw[..., :-1, :]                           # D, right going
        dp = torch.cat([xw[..., 2:n - 1, :], x[..., :1, :], x[..., 1:2, :]], -2)
        # faces 2..NT-2 take X of the next face; face NT-2's is F(NT)-F(NT-1)
        neg = c < 0
        upn = torch.cat([G[..., 2:, :], G[..., 1:2, :]], -2)
        fb = _limited(xf, torch.where(neg, dp, dm), torch.where(neg, upn, G[..., 1:, :]),
                      0.5 * (torch.where(neg, -1.0, 1.0) - c), self.beta)
        phi = c * fb
        prev = torch.cat([phi[..., -1:, :], phi[..., :-1, :]], -2)
        new = _clip(G[..., 1:, :] - phi + prev)
        new = torch.cat([new[..., -1:, :], new], -2)
        return torch.cat([F[..., :1], new], -1)

    def sweep_e(self, F, cc, s):
        g, c = self.g, cc[2]
        gr = _t(g.grel[s])
        G = F[..., 1:]
        ez = self.ekev[0] - self.we[0]
        rm = float(g.rmas[s])
        grz = 1 + ez * 1000 * W.Q / rm / W.CS / W.CS
        k1 = gr[0] / gr[1] * torch.sqrt((gr[1] ** 2 - 1) / (gr[0] ** 2 - 1))
        k0 = grz / gr[0] * torch.sqrt((gr[0] ** 2 - 1) / (grz ** 2 - 1))
        e1 = k1 * G[:, 1:2]
        z = torch.zeros_like(e1)
        A = torch.cat([k0 * e1, e1, G[:, 1:], z, z], 1)  # cells 0..NE+2
        x = A[:, 1:] - A[:, :-1]
        n = g.ne
        neg = c < 0
        de = self.de[:, None, None]
        fb = _limited(x[:, 1:n + 1], torch.where(neg, x[:, 2:n + 2], x[:, 0:n]), torch.where(neg, A[:, 2:n + 2], A[:, 1:n + 1]),
                      0.5 * (torch.where(neg, -1.0, 1.0) - c / de), self.beta)
        phi = c * fb
        new = _clip(G[:, 1:] + (phi[:, :-1] - phi[:, 1:]) / self.we[1:, None, None])
        return torch.cat([F[..., :1], torch.cat([G[:, :1], new], 1)], -1)

    def sweep_mu(self, F, cc):
        g, c, n = self.g, cc[3], self.g.npa
        G = torch.cat([F[1:2, ..., 1:], F[1:, ..., 1:]], 0)
        x = G[1:] - G[:-1]
        cf = c[1:n - 2]                                # faces 2..NPA-2
        neg = cf < 0
        dm = self.dmu[1:n - 2, None, None, None]
        fb = _limited(x[1:n - 2], torch.where(neg, x[2:n - 1], x[0:n - 3]), torch.where(neg, G[2:n - 1], G[1:n - 2]),
                      0.5 * (torch.where(neg, -1.0, 1.0) - cf / dm), self.beta)
        phi = torch.cat([torch.zeros_like(G[:1]), c[1:n - 1] * torch.cat([fb, G[n - 1:]], 0)], 0)
        new = _clip(G[1:n - 1] + (phi[:-1] - phi[1:]) / self.wmu[1:n - 1, None, None, None])
        fh = self.f3["fnhs"][..., 1:g.nr]
        rho = fh[n - 1] * self.mu[n - 1] / fh[n - 2] / self.mu[n - 2]
        new = torch.cat([F[:1, ..., 1:], new, (new[-1] * rho)[None]], 0)
        return torch.cat([F[..., :1], new], -1)

    def losses(self, s, dts):
        """(CHARGE, ATLOS**(1/FNHS)) per cell (src/ModRamLoss.f90:34-170,485-507)."""
        g, n = self.g, self.g.nr
        v = _t(g.v[s])
        one = torch.ones((g.npa, g.ne, g.nt, n), dtype=torch.float64, device=_device())
        kind = g.species[s].cex_kind
        ch, at = one, one.clone()
        if kind:
            X = torch.clamp(torch.log10(self.ekev), min=-2.0)
            p = {1: (-18.767, -0.11017, -3.8173e-2, -0.1232, -5.0488e-2), 2: (-20.789, 0.92316, -0.68017, 0.66153, -0.20998),
                 3: (-18.987, -0.10613, -5.4841e-3, -1.6262e-2, -7.0554e-3)}[kind]
            y = p[0] + p[1] * X + p[2] * X ** 2 + p[3] * X ** 3 + p[4] * X ** 4
            alpha = (10.0 ** y * v)[:, None, None] * self.f3["hdns"][..., :n][:, None] * dts
            ch = one.clone()
            ch[1:, 1:, :, 1:] = torch.exp(-alpha)[1:, 1:, :, 1:]
        up = torch.from_numpy(np.asarray(g.upa).astype(np.int64)).to(_device())
        taub = 2 * self.rlz[:n] / v[:, None]
        a = torch.exp(-dts / taub)[:, None, :] ** (1 / self.f3["fnhs"][..., :n])[:, None]
        inside = torch.arange(1, g.npa + 1, device=_device())[:, None] >= up[None, :]
        on = inside[:, None, None, :] & (torch.arange(g.ne, device=_device()) >= 1)[:, None, None] & (torch.arange(n, device=_device()) >= 1)
        return ch, torch.where(on, a, at)

    def diffuse(self, F, D, dts):
        """WPADIF (src/ModRamWPI.f90:643-714) on I, K >= 2; D (L, K, J, I)."""
        g, n = self.g, self.g.npa
        fac = (self.f3["fnhs"][..., 1:g.nr] * self.mu[:, None, None])[:, None]
        G, Dm = F[:, 1:, :, 1:], D[:, 1:, :, 1:]
        f = G / torch.where(fac == 0, torch.ones_like(fac), fac)
        rk, rl = [torch.zeros_like(f[0])], [torch.full_like(f[0], -1.0)]
        for L in range(1, n - 1):
            an = Dm[L] / self.dmu[L] * dts / fac[L] / self.wmu[L]
            gn = Dm[L - 1] / self.dmu[L - 1] * dts / fac[L] / self.wmu[L]
            den = an + gn + gn * rl[-1] + 1
            rk.append((f[L] + gn * rk[-1]) / den)
            rl.append(-an / den)
        x = rk[-1] / (1 + rl[-1])
        new = [x * fac[n - 1], x * fac[n - 2]]
        for L in range(n - 3, -1, -1):
            x = rk[L] - rl[L] * x
            new.append(x * fac[L])
        F = F.clone()
        F[:, 1:, :, 1:] = torch.stack(new[::-1], 0)
        return F

    def content(self, F):
        """SETRC (src/ModRamRun.f90:231-259)."""
        w = (self.ekev * self.we)[:, None, None] * self.wmu[:, None, None, None]
        return (F * w)[1:, 1:, :self.g.nt - 1, 1:].sum()

    def courant(self, cc, dts):
        """DtDriftR/P/E/Mu from the largest face coefficients inside the magnetopause."""
        inside = ~self.outside
        tiny = lambda c, lo: torch.clamp(c.abs(), min=lo)  # noqa: E731
        de, dm = self.de[:, None, None], self.dmu[:, None, None, None]
        n = self.g.npa
        qs = ((tiny(cc[0], 1e-10), inside), (tiny(cc[1][..., 1:, :], 1e-10), inside[1:, 1:]),
              (tiny(cc[2], 1e-10) / de, inside[:, 1:]), (tiny(cc[3][1:n - 1], 1e-32) / dm[1:n - 1], inside[:, 1:]))
        init = (1e5, 1e5, 1e4, 1e4)
        return [min(i0, self.fraccfl * dts / float(torch.where(i, q, torch.zeros_like(q)).max())) for i0, (q, i) in zip(init, qs)]

    def call(self, s, F, fg, vt, dts, D=None, books=None):
        """One ram_run of species s: (F2, Courant limits); books gets the loss channels."""
        cc = self.coefficients(s, vt, dts)
        ch, at = self.losses(s, dts)
        F = self.sweep_mu(self.sweep_e(self.sweep_p(self.sweep_r(F, fg, cc), cc), cc, s), cc)
        log = []
        note = lambda F, i: log.append((i, self.content(F))) if books is not None else None  # noqa: E731
        note(F, 1)
        if D is not None:
            F = self.diffuse(F, D, dts)
            note(F, 4)
        for f, i in ((ch, 2), (at, 3), (at, 3), (ch, 2)):
            F = F * f
            note(F, i)
        if D is not None:
            F = self.diffuse(F, D, dts)
            note(F, 4)
        F = self.sweep_r(self.sweep_p(self.sweep_e(self.sweep_mu(F, cc), cc, s), cc), fg, cc)
        note(F, 1)
        for i, v in log:
            if i < 4:
                books[i] += float(books[0] - v)
            books[0] = float(v)
        F = torch.cat([F[..., :-1, :], F[..., :1, :]], -2)
        F = torch.where(self.outside, torch.full_like(F, 1e-31), F)
        low = torch.cat([F[:1, :, :, :1], F[1:2, :, :, 1:]], -1)  # ANISCH: F2(:,:,:,1) = F2(:,:,:,2) for I, K >= 2
        low = torch.cat([F[:1, :1], low[:, 1:]], 1)
        return torch.cat([low, F[1:]], 0), self.courant(cc, dts)

    def moments(self, s, F):
        """(PPERT, PPART), each (I, J) (src/ModRamRun.f90:343-404)."""
        g, n = self.g, self.g.nr
        rfac = 4 * W.PI / (W.CS * 100)
        ern = self.wmu[:, None, None, None] / _t(g.ffactor[s], (2, 1, 0))[:, :, None, :] / self.f3["fnhs"][..., :n][:, None]
        mu2 = (self.mu ** 2)[:, None, None, None]
        u = torch.from_numpy((np.asarray(g.upa) - 1).astype(np.int64)).to(_device())
        on = torch.arange(1, g.npa + 1, device=_device())[:, None, None, None] <= u
        w = torch.where(on, F * ern * _t(g.epp[s])[:, None, None] * rfac, torch.zeros_like(F))
        pe = (w * (1 - mu2))[:, 1:].sum((0, 1))
        pa = (2 * w * mu2)[:, 1:].sum((0, 1))
        pe[:, 0] = pa[:, 0] = 0.0
        return pe.T, pa.T


def exact(case, seed):
    g, f, f2, fgeos, kp = _inputs(case, seed)
    X = _Exact(case, g, f, kp)
    fgs = [_t(a.transpose(2, 1, 0)) for a in fgeos]
    dts = case["dts"]
    D = _t(_diffusion(g, f, seed), (3, 2, 1, 0)) if case.get("diffusion") else None
    if case["kind"] == "adj":
        obs = _observations(case, g, f, f2, seed)
        f2 = f2.requires_grad_()
        fgs = [x.requires_grad_() for x in fgs]
        j = torch.zeros(1, dtype=torch.float64, device=_device())
        gf, gb = torch.zeros_like(f2), []
        for s in range(len(fgs)):
            F, part = f2[0, s], torch.zeros(1, dtype=torch.float64, device=_device())
            for k in range(case["calls"]):
                F, _ = X.call(s, F, fgs[s], X.potential(kp[k, 0]), dts)
                for o in (o for o in obs if o["s"] == s and o["call"] == k):
                    v = sum(w * F[o["l"], o["k"], jj, i] / g.ffactor[s, i, o["k"], o["l"]] / f.fnhs[i, jj, o["l"]]
                            for i, jj, w in _stencil(g, o["lshell"], o["mlt"]))
                    part = part + (torch.log(v) - o["log_obs"]) ** 2
            a = torch.autograd.grad(part, (f2, fgs[s]), allow_unused=True) if part.requires_grad else (None, None)
            gf += a[0] if a[0] is not None else 0.0
            gb.append(a[1] if a[1] is not None else torch.zeros_like(fgs[s]))
            j += part.detach()
            del F, part, a
        return dict(j=j, gf2=gf, gfgeos=torch.stack(gb)[None])
    moments, cfl, books = [], [], []
    with torch.no_grad():
        for m, sp in enumerate(_member_species(case)):
            limits = []
            for s in sp:
                F = f2[m, s]
                b = [float(X.content(F)), 0.0, 0.0, 0.0]
                for k in range(case["calls"]):
                    F, lim = X.call(s, F, fgs[s], X.potential(kp[k, m]), dts, D if s == 0 else None, b if case.get("losses") else None)
                f2[m, s] = F
                moments.append(torch.stack(X.moments(s, F)))
                limits.append(lim)
                books.append(b)
            nxt = max(min(min(x) for x in limits), X.dtsmin)
            cfl += [x + [nxt] for x in limits]
    if case["kind"] == "host":
        return dict(f2=[f2[0, s].reshape(-1) for s in range(len(fgs))], pe=[x[0].T.reshape(-1) for x in moments], pa=[x[1].T.reshape(-1) for x in moments])
    if case["kind"] == "ref":
        return dict(f2=f2[0].permute(0, 4, 3, 2, 1).contiguous(), pe=torch.stack([x[0] for x in moments]), pa=torch.stack([x[1] for x in moments]))
    out = dict(f2=f2, moments=torch.stack(moments), cfl=np.array(cfl))
    if case.get("losses"):
        out["losses"] = np.array(books)
    return out

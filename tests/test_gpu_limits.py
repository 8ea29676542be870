"""GPU: the Courant limits where few cells or faces decide them."""
import dataclasses

import numpy as np
import pytest

from ramgpu import abi, workload as W
import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [1, 2, 4, None])
def test_mu_limit_leaves_face_1_out(lanes):
    """DtDriftMu counts the faces L = 2..NPA (src/ModRamDrift.f90:434-437).  Here
    face 1 has a Courant number above 1 and above every other face's, and the
    lanes that share a line form it too (None: the automatic count, 8 for this
    list).  The limit agrees with the oracle's to the parity bar."""
    wl = W.make_workload("tiny_pert8")
    f = W.perturbed_fields(wl.grid, seed=1)
    f = dataclasses.replace(f, dibndt=2.0 * f.dibndt)  # |C(1)|/DMU(1) up to 1.56, the others up to 1.18
    dts, kp = 200.0, 4.0
    o = pyoracle.Oracle(wl.grid, f)
    vt = o.vt_vols(kp)
    gpu = abi.RamGpu(wl.grid, f)
    try:
        if lanes:
            gpu.set_mu_lanes(lanes)
        gpu.set_kp(0, kp)
        for s in range(len(wl.grid.species)):
            gpu.upload_f2(0, s, np.asfortranarray(wl.f2[s]))
            gpu.set_boundary(0, s, wl.fgeos[s])
        gpu.apply_op(dts, abi.OP_DRIFTMU, cfl=True)
        for s in range(len(wl.grid.species)):
            dt = o.sweep("MU", s, np.asfortranarray(wl.f2[s]).copy(order="F"), vt, dts)
            assert abs(gpu.cfl(0, s)[3] - dt) <= 1e-12 * dt, s
    finally:
        gpu.close()


def test_limits_inside_any_outside_flag():
    """Every sweep's limit counts the cells with flag 0 alone, whatever the other
    flags are (OUTSIDE_MGNP == 0, src/ModRamDrift.f90:146): flags of 2 and -1,
    none of 1, over the cells that hold the largest |C|."""
    wl = W.make_workload("tiny_pert8")
    out = np.asfortranarray(np.zeros_like(wl.fields.outside))
    out[4:, :] = 2
    out[2, 3] = -1
    f = dataclasses.replace(wl.fields, outside=out)
    o = pyoracle.Oracle(wl.grid, f)
    vt = o.vt_vols(4.0)
    for w, op in (("R", abi.OP_DRIFTR), ("P", abi.OP_DRIFTP), ("E", abi.OP_DRIFTE), ("MU", abi.OP_DRIFTMU)):
        gpu = abi.RamGpu(wl.grid, f)
        gpu.set_kp(0, 4.0)
        for s in range(len(wl.grid.species)):
            gpu.upload_f2(0, s, np.asfortranarray(wl.f2[s]))
            gpu.set_boundary(0, s, wl.fgeos[s])
        gpu.apply_op(wl.dts, op, cfl=True)
        for s in range(len(wl.grid.species)):
            dt = o.sweep(w, s, np.asfortranarray(wl.f2[s]).copy(order="F"), vt, wl.dts, fgeos=wl.fgeos[s])
            got = gpu.cfl(0, s)["R P E MU".split().index(w)]
            assert abs(got - dt) <= 1e-12 * dt, (w, s)
        gpu.close()

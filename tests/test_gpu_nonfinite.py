"""GPU: where a non-finite cell spreads to."""
import numpy as np
import pytest

from ramgpu import abi, workload as W
import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("lanes", [1, 4])
def test_zero_coefficient_flows_up(value, lanes):
    """C = -0 is not C < 0 (src/ModRamDrift.f90:441): the face's upwind cell is
    F(L), whose NaN or infinity its flux carries to cell L+1, not the other way
    round.  A dipole's CDriftMu vanishes along a meridian, as -0 for electrons."""
    wl = W.make_workload("tiny")
    g, s = wl.grid, 0
    o = pyoracle.Oracle(g, wl.fields)
    cd = np.zeros((g.nr, g.nt, g.ne, g.npa), order="F")
    f2 = np.asfortranarray(wl.f2[s]).copy(order="F")
    o.sweep("MU", s, f2.copy(order="F"), o.vt_vols(4.0), wl.dts, cdrift=cd)
    lines = np.argwhere((cd[1:, :, :, 1:g.npa - 1] == 0).all(axis=3)) + [1, 0, 0]
    assert len(lines)
    spots = [(i, j, k, 3 + (7 * n) % (g.npa - 10)) for n, (i, j, k) in enumerate(lines)]
    for i, j, k, l in spots:
        f2[i, j, k, l] = value
    gpu = abi.RamGpu(g, wl.fields)
    try:
        gpu.set_mu_lanes(lanes)
        gpu.set_kp(0, 4.0)
        for q in range(len(g.species)):
            gpu.upload_f2(0, q, f2 if q == s else np.asfortranarray(wl.f2[q]))
            gpu.set_boundary(0, q, wl.fgeos[q])
        gpu.apply_op(wl.dts, abi.OP_DRIFTMU)
        out = gpu.download_f2(0, s)
    finally:
        gpu.close()
    for i, j, k, l in spots:
        # the flux out of the cell, 0*inf or a NaN, leaves the next cell a NaN or
        # the clip's 1e-15 (a NaN whose sign bit is set); a cell that no such
        # flux enters keeps its value, as C = 0 on the whole line
        assert out[i, j, k, l - 1] == f2[i, j, k, l - 1], (i, j, k, l)
        assert out[i, j, k, l + 1] != f2[i, j, k, l + 1], (i, j, k, l)

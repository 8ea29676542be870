"""ANISCH moments at the edges of the kernel's tiles: 32 (I,J), 8 pitch
angles and 8 energies at a time (src/ModRamRun.f90:343-404)."""
import dataclasses

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("separable", [True, False])
@pytest.mark.parametrize("nr,nt,ne,npa", [(5, 8, 32, 60), (4, 11, 33, 64), (6, 19, 34, 65), (9, 12, 35, 72)])
def test_moments_at_tile_edges(nr, nt, ne, npa, separable):
    """Both moments of every (I,J) and the F2(L=1) = F2(L=2) side effect
    against the oracle, twice in a row: positive sums of at most NE*NPA terms
    of a few roundings each, in two orders."""
    from ramgpu import abi, workload as W
    import pyoracle
    g = W.arrays(nr, nt, ne, npa, species=(W.HYDROGEN, W.SPECIES["O"]), mu_grid_nr=20)
    rng = np.random.Generator(np.random.PCG64(nr))
    if not separable:
        g = dataclasses.replace(g, ffactor=g.ffactor * rng.lognormal(0.0, 0.2, size=g.ffactor.shape))
    f = W.dipole_fields(g, seed=nr)
    gpu, o = abi.RamGpu(g, f), pyoracle.Oracle(g, f)
    try:
        for _ in range(2):
            f2 = [np.asfortranarray(rng.lognormal(0.0, 2.0, size=(nr, nt, ne, npa))) for _ in range(2)]
            for s in range(2):
                gpu.upload_f2(0, s, f2[s])
            gpu.apply_op(1.0, abi.OP_ANISCH)
            for s in range(2):
                ref = o.anisch(s, f2[s])
                assert np.array_equal(gpu.download_f2(0, s), f2[s])
                for a, b in zip(gpu.moments(0, s), ref):
                    assert np.all(np.abs(a[1:] - b[1:]) <= ne * npa * 2.0 ** -52 * np.abs(b[1:]))
    finally:
        gpu.close()

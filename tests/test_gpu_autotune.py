"""GPU: the autotuner leaves no trace but the launch shapes."""
import numpy as np
import pytest

from ramgpu import abi, workload as W

pytestmark = pytest.mark.gpu


def _gpu(wl, flags=0):
    gpu = abi.RamGpu(wl.grid, wl.fields, flags=flags)
    for s in range(len(wl.grid.species)):
        gpu.upload_f2(0, s, np.asfortranarray(wl.f2[s]))
        gpu.set_boundary(0, s, wl.fgeos[s])
    gpu.set_kp(0, 4.0)
    return gpu


def _state(gpu, ns):
    out = [gpu.download_f2(0, s) for s in range(ns)]
    out += [np.concatenate(gpu.moments(0, s)) for s in range(ns)]
    return out + [gpu.cfl(0, s) for s in range(ns)]


@pytest.mark.parametrize("flags", [0, abi.FLAG_LOSSES])
@pytest.mark.parametrize("check", [False, True])
def test_autotune_leaves_the_results_alone(flags, check):
    """F2, the loss books, the moments, the Courant limits and the status word
    are those of the last call after a tuning, and the next call's are those of
    a context that was never tuned."""
    wl = W.make_workload("tiny_pert")
    ns = len(wl.grid.species)
    ref, tun = _gpu(wl, flags), _gpu(wl, flags)
    try:
        for g in (ref, tun):
            g.set_check(check)
            if flags:
                g.reset_losses()
            g.ram_run(wl.dts)
        tun.autotune(wl.dts, reps=1)
        for step in range(2):
            for a, b in zip(_state(ref, ns), _state(tun, ns)):
                assert np.array_equal(a, b), step
            if flags:
                for s in range(ns):
                    assert np.array_equal(ref.losses(0, s), tun.losses(0, s)), (step, s)
            if check:
                assert ref.last_status() == tun.last_status(), step
            for g in (ref, tun):
                g.ram_run(wl.dts)
    finally:
        ref.close()
        tun.close()


def test_lanes_return_to_the_rule():
    """A fixed DRIFTMU lane count, and what a tuning chose, go back to the
    automatic one with 0, whose results are the same bits."""
    wl = W.make_workload("tiny_pert")
    ns = len(wl.grid.species)
    ref, gpu = _gpu(wl), _gpu(wl)
    try:
        for act in (lambda: gpu.set_mu_lanes(2), lambda: gpu.set_mu_lanes(0), lambda: gpu.autotune(wl.dts, reps=1),
                    lambda: gpu.set_mu_lanes(0)):
            act()
            ref.ram_run(wl.dts)
            gpu.ram_run(wl.dts)
            for a, b in zip(_state(ref, ns), _state(gpu, ns)):
                assert np.array_equal(a, b)
        for lanes in (3, 8, -1):
            with pytest.raises(abi.RamGpuError):
                gpu.set_mu_lanes(lanes)
    finally:
        ref.close()
        gpu.close()

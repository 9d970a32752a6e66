"""The ensemble's pool: 52 arrays an event, or 61 with a divergence set of the
y sweeps' own where a quarter of the free memory holds them."""
import numpy as np
import pytest

from conftest import rel_err
from viral_b200 import _abi as A
from viral_b200 import configs as C
from viral_b200.batch import EVENT_RUNNING, Batch
from viral_b200.hydro import Hydro

pytestmark = pytest.mark.gpu

SIDES = [24, 33, 58, 9, 27, 105]


@pytest.mark.parametrize("precision", [A.PREC_FP64, A.PREC_MIXED])
@pytest.mark.parametrize("recon", [A.RECON_WENO5, A.RECON_MINMOD])
@pytest.mark.parametrize("sets", ["1", "2"])
@pytest.mark.parametrize("variant", [0, 2, 4])
def test_both_layouts_match_single_events(precision, recon, sets, variant, monkeypatch):
    """x tiles, a barrier and y tiles that add to them, and all tiles at once,
    with both reconstructions; tolerances of the single-event comparison (the
    same source in another kernel: rounding of fused operations)"""
    monkeypatch.setenv("VH_BATCH_SETS", sets)
    cfg = C.glauber_config(nx=8, ny=8, boost_invariant=True, precision=precision)
    cfg.recon = recon
    steps = 10
    with Batch(cfg, SIDES, tau0=cfg.tau0, dtau=cfg.dtau, tau_max=100.0, t_freeze_gev=0.0) as B:
        B.init_glauber(seeds=np.arange(len(SIDES)), bimp=[2.0 + k for k in range(len(SIDES))])
        B.set_tuning(variant, steps_per_launch=4)
        B.run(steps)
        _, nst, st = B.events()
        assert np.all(st == EVENT_RUNNING) and np.all(nst == steps)
        got = [B.event_state(ev) for ev in range(len(SIDES))]
    tol = 1e-13 if precision == A.PREC_FP64 else 1e-5
    for ev, side in enumerate(SIDES):
        c = C.glauber_config(nx=side, ny=side, boost_invariant=True, precision=precision)
        c.recon = recon
        with C.make_hydro(c, C.glauber_inputs(c, b=2.0 + ev, seed=ev)) as H:
            H.step(steps)
            want = H.get_state()
        for q in range(14):
            assert rel_err(got[ev][q], want[q]) <= tol, (ev, q)


class Tight:
    """all but `free` bytes of the GPU's memory taken"""

    def __init__(self, free):
        self.free = free

    def __enter__(self):
        import torch
        torch.cuda.empty_cache()
        self.held = torch.empty(torch.cuda.mem_get_info()[0] - self.free, dtype=torch.uint8, device="cuda")
        return torch.cuda.mem_get_info

    def __exit__(self, *a):
        import torch
        del self.held
        torch.cuda.empty_cache()


def test_what_fits_with_52_arrays_is_created():
    """one event whose 52 arrays and staging fit, and whose 61 arrays alone would"""
    side = 3536
    array = 8 * (side + 6) ** 2
    cfg = C.glauber_config(nx=8, ny=8, boost_invariant=True)
    with Batch(cfg, [9], tau0=cfg.tau0, dtau=cfg.dtau):
        pass  # the context and the library's kernels are there
    with Tight(74 * array) as info:
        before = info()[0]
        with Batch(cfg, [side], tau0=cfg.tau0, dtau=cfg.dtau, tau_max=100.0, t_freeze_gev=0.0) as B:
            assert before - info()[0] < 71 * array  # 52 and the staging's 18
            e = np.full((side + 6) ** 2, 5.0)
            B.init_event(0, e, 0 * e, 0 * e)
            B.run(1)
            assert B.events()[2][0] == EVENT_RUNNING


def test_tuning_needs_room_for_the_state_alone():
    """a pool of 61 arrays and 40 arrays' memory left: the trials' copy is of
    18, and the states are as before"""
    cfg = C.glauber_config(nx=8, ny=8, boost_invariant=True)
    sides = [500] * 20
    array = 8 * sum((s + 6) ** 2 for s in sides)
    with Batch(cfg, sides, tau0=cfg.tau0, dtau=cfg.dtau, tau_max=100.0, t_freeze_gev=0.0) as B:
        c = C.glauber_config(nx=500, ny=500, boost_invariant=True)
        inp = C.glauber_inputs(c, b=4.0, seed=1)
        for ev in range(len(sides)):
            B.init_event(ev, inp["e"] * (1 + 0.01 * ev), inp["ux"], inp["uy"])
        before = [B.event_state(ev) for ev in (0, 19)]
        B.run(1)  # allocates what a run needs
        B.init_event(0, inp["e"], inp["ux"], inp["uy"])
        B.init_event(19, inp["e"] * 1.19, inp["ux"], inp["uy"])
        with Tight(40 * array):
            assert B.autotune(None, probe_steps=1) > 0
        for ev, want in zip((0, 19), before):
            assert np.array_equal(B.event_state(ev), want)

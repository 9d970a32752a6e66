"""Events that fail among healthy ones.  A failing cell raises its event's flag
while other blocks are at work on the same event; the blocks' way through the
grid-wide barriers must not depend on who has seen it.  The healthy events
therefore equal, bit for bit, the same events in an ensemble where nothing
fails."""
import numpy as np
import pytest

from viral_b200 import _abi as A
from viral_b200 import configs as C
from viral_b200.batch import EVENT_FAILED, EVENT_RUNNING, Batch

pytestmark = pytest.mark.gpu

SIDES = [96, 58, 120, 41, 96, 75, 130, 96, 33]
# of the shear noise, in units of the energy density, per event (0: healthy);
# some fail in the first step, some several steps in
NOISE = [0.2, 0, 0.22, 0, 0.3, 0, 0.25, 0.5, 0]


def run(cfg, noise, variant, steps):
    with Batch(cfg, SIDES, tau0=cfg.tau0, dtau=cfg.dtau, tau_max=100.0, t_freeze_gev=0.0) as B:
        for ev, side in enumerate(SIDES):
            c = C.glauber_config(nx=side, ny=side, boost_invariant=True)
            inp = C.glauber_inputs(c, b=4.0, seed=ev)
            e = np.asarray(inp["e"]).reshape(-1)
            pi5 = noise[ev] * e * np.random.default_rng(ev).standard_normal((5, e.size)) * np.array([[1, 1, 1, 0, 0]]).T
            B.init_event(ev, e, inp["ux"], inp["uy"], None, A.PI_GIVEN, pi5)
        B.set_tuning(variant, steps_per_launch=4, use_graph=False)
        B.run(steps)
        return (*B.events(), [B.event_state(ev) for ev in range(len(SIDES))], *B.observables())


@pytest.mark.parametrize("precision", [A.PREC_FP64, A.PREC_MIXED])
@pytest.mark.parametrize("variant", [0, 2, 4])
def test_healthy_events_do_not_notice(precision, variant):
    cfg = C.glauber_config(nx=8, ny=8, boost_invariant=True, precision=precision)
    steps = 12
    tau, nst, st, state, eps_p, eps_2 = run(cfg, NOISE, variant, steps)
    _, _, _, want, want_p, want_2 = run(cfg, [0] * len(SIDES), variant, steps)
    for ev, a in enumerate(NOISE):
        if a:
            assert st[ev] == EVENT_FAILED and nst[ev] < steps, (ev, st[ev], nst[ev])
            continue
        assert st[ev] == EVENT_RUNNING and nst[ev] == steps
        assert np.array_equal(state[ev], want[ev]), ev
        assert eps_p[ev] == want_p[ev] and eps_2[ev] == want_2[ev]

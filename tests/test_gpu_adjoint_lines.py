"""The reverse sweeps' line segments at the sizes where their number changes:
lines of three cells (one segment), of a few (segments of four centres), at
the change of the block's threads (64 cells with ghosts) and longer ones,
2+1D and 3+1D: every field of the gradient, ghost cells included, against
automatic differentiation of the same scheme in torch (perf/cases.py)."""
import numpy as np
import pytest

from perf import cases
from viral_b200.hydro import Hydro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("table", [False, True])
@pytest.mark.parametrize("nx,ny,nz", [(3, 3, 0), (4, 14, 0), (59, 6, 0), (15, 130, 0), (3, 3, 3), (5, 13, 4), (58, 7, 5),
                                      (6, 59, 3), (4, 5, 60)])
def test_gradient(nx, ny, nz, table):
    """Two steps.  Both sides differentiate the same map exactly; they differ
    by rounding, which the smoothness indicators of nearly constant stencils
    amplify by up to 1e6 (the inverse of the weights' epsilon): 1e-9 of each
    field group's 2-norm, and of the largest group's for one that vanishes."""
    c = cases._case("", "adjoint", nx, ny, nz, 2, every=1, table=table)
    cfg = cases._config(c)
    seed = nx + 3 * ny + 5 * nz
    want = cases._exact_adjoint(c, cfg, seed)
    s0 = cases._inputs(cfg, seed).reshape(18, -1).cpu().numpy()
    with Hydro(cfg) as h:
        h.set_state(s0, cfg.tau0)
        eps, gs, ge, gc = h.adjoint_eps_p(2, 1)
    assert abs(eps - want["eps_p"]) <= 1e-12
    got = {"grad_e0": ge, "grad_etas": gc, **{"grad_" + k: v for k, v in cases._fields(gs, False).items()}}
    most = max(np.linalg.norm(v) for v in got.values())
    for k, v in got.items():
        assert np.linalg.norm(v - want[k]) <= 1e-9 * max(np.linalg.norm(want[k]), 1e-6 * most), k

"""vh_step_static around the grids whose scratch just holds, or just does not,
a divergence set per direction (43 of 34 x 61,680 words a cell in 2+1D, 52 in
3+1D): the same steps as on a handle, as in test_zz_no_alloc.py."""
import numpy as np
import pytest

from test_zz_no_alloc import GROUPS, TOL, _from_inputs, _run_pair
from viral_b200 import _abi as A
from viral_b200 import configs as C

pytestmark = pytest.mark.gpu

WORDS = 34 * 61680
# ghost-inclusive 192x254 = 48768 and 193x253 = 48829 about 48769.7 cells,
# 64x45x14 = 40320 and 37x38x29 = 40774 about 40329.2; short lines
GRIDS = [(186, 248, 1), (187, 247, 1), (58, 39, 8), (31, 32, 23), (3, 3, 1), (3, 3, 3), (5, 90, 1)]


@pytest.mark.parametrize("recon", [A.RECON_WENO5, A.RECON_MINMOD])
@pytest.mark.parametrize("nx,ny,nz", GRIDS)
def test_either_layout_matches_the_handle(nx, ny, nz, recon):
    cfg = C.glauber_config(nx=nx, ny=ny, nz=nz, boost_invariant=nz == 1)
    cfg.recon = recon
    f0, tau0 = _from_inputs(cfg, C.glauber_inputs(cfg, b=4.0, seed=nx))
    ref, got, free = _run_pair(cfg, f0, tau0, steps=(2, 2))
    for r, g in zip(ref, got):
        for grp in GROUPS:
            scale = max(float(np.max(np.abs(r[q]))) for q in grp)
            for q in grp:
                assert np.max(np.abs(g[q] - r[q])) <= TOL * scale, f"field {q}"
    assert free[0] == free[1]


def test_the_grids_lie_on_both_sides():
    cells = [(nx + 6) * (ny + 6) * (1 if nz == 1 else nz + 6) for nx, ny, nz in GRIDS]
    assert 43 * cells[0] <= WORDS < 43 * cells[1] and 52 * cells[2] <= WORDS < 52 * cells[3]

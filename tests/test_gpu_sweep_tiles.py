"""The flux sweeps at the edges of their tiles: lengths at and around a
tile's 24 (FP64), 30 (FP32) and 16 cells, single-tile lines, widths that are
no multiple of a tile's 8 lines, both reconstructions, tiles by TMA and
through the cache, against the oracle; and one divergence array for all
directions against a set per direction (debug_stage_terms adds up one)."""
import numpy as np
import pytest

from helpers import interior_mask, oracle_config, smooth_inputs
from pyoracle import Oracle
from test_gpu_parity import STAGE_TOL, compare_states
from viral_b200 import _abi as A
from viral_b200.hydro import Config, Hydro

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3), (8, 9, 7), (16, 17, 5), (24, 25, 8), (48, 23, 9), (31, 49, 16), (15, 30, 33), (61, 4, 25), (5, 90, 1)]


@pytest.mark.parametrize("tma", ["1", "0"])
@pytest.mark.parametrize("recon", [A.RECON_WENO5, A.RECON_MINMOD])
@pytest.mark.parametrize("precision", [A.PREC_FP64, A.PREC_MIXED])
@pytest.mark.parametrize("nx,ny,nz", SIZES)
def test_tile_edges(nx, ny, nz, precision, recon, tma, monkeypatch):
    """Two steps.  FP64: rounding of the step's few thousand operations, the
    bound of the stage terms.  Mixed: the FP32 state's rounding (6e-8)
    through two stages of differences over 0.1 fm times dtau = 0.01: a few
    units per step; 2e-6."""
    monkeypatch.setenv("VH_TMA", tma)
    cfg = Config(nx=nx, ny=ny, nz=nz, boost_invariant=nz == 1, dx=0.1, dy=0.1, dz=0.1, tau0=1.3, dtau=0.01,
                 eos_kind=A.EOS_CONFORMAL, eos_a=13.899692864867510, etas0=1 / (4 * np.pi), precision=precision,
                 recon=recon)
    f = smooth_inputs(cfg, cfg.tau0, seed=nx + 7 * ny + 11 * nz)
    O = Oracle(oracle_config(cfg))
    O.set_state(f)
    tau = cfg.tau0
    for _ in range(2):
        assert O.step(tau, cfg.dtau) == 0
        tau += cfg.dtau
    with Hydro(cfg) as H:
        H.set_state(f, cfg.tau0)
        H.step(2)
        got = H.get_state()
    compare_states(got, O.get_state(), STAGE_TOL if precision == A.PREC_FP64 else 2e-6, fields=range(18),
                   mask=interior_mask(cfg))


@pytest.mark.parametrize("nx,ny,nz", [(25, 17, 1), (26, 31, 9)])
def test_one_divergence_array(nx, ny, nz):
    """the directions added to one array in order, as the allocation-free
    step has it, against the oracle's sum"""
    cfg = Config(nx=nx, ny=ny, nz=nz, boost_invariant=nz == 1, dx=0.1, dy=0.1, dz=0.1, tau0=1.3, dtau=0.01,
                 eos_kind=A.EOS_CONFORMAL, eos_a=13.899692864867510, etas0=1 / (4 * np.pi))
    f = smooth_inputs(cfg, cfg.tau0, seed=5)
    O = Oracle(oracle_config(cfg))
    O.set_state(f)
    _, ro, _ = O.stage_terms(cfg.tau0, cfg.dtau)
    with Hydro(cfg) as H:
        H.set_state(f, cfg.tau0)
        rg, _, _ = H.debug_stage_terms()
    m = interior_mask(cfg)
    for l in range(9):
        scale = np.max(np.abs(ro[l][m]))
        assert np.max(np.abs(rg[l][m] - ro[l][m])) <= STAGE_TOL * max(scale, 1e-300)

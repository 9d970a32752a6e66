"""Relaxation times without bound, which the configuration accepts: a constant
tau_pi of infinity (and one beyond FP32's range, in the mixed mode), and
tau_pi = 1.5 eta / P on a table whose rows hold no pressure.  The shear
source's 1 / tau_pi is then zero, as a division gives it, and the step goes on;
against the oracle."""
import numpy as np
import pytest

from helpers import interior_mask, oracle_config, smooth_inputs
from pyoracle import Oracle
from test_gpu_parity import RUN_TOL, compare_states
from viral_b200 import _abi as A
from viral_b200 import configs as C
from viral_b200.hydro import Config, Hydro

pytestmark = pytest.mark.gpu


def dust_table(e_most):
    """no pressure up to above e_most, then the usual table's, continuous"""
    t = np.array(C.eos_table())
    k = int(np.searchsorted(t[0], 2 * e_most))
    t[1] = np.maximum(t[1] - t[1][k], 0.0)
    t[2, :k] = 0.0
    return t


@pytest.mark.parametrize("precision", [A.PREC_FP64, A.PREC_MIXED])
@pytest.mark.parametrize("kind", ["infinite", "1e300", "pressureless"])
@pytest.mark.parametrize("nx,ny,nz", [(12, 9, 1), (9, 8, 7)])
def test_step_without_relaxation(nx, ny, nz, kind, precision):
    """Two steps.  FP64: the bar of runs against the oracle.  Mixed: the FP32
    state's rounding (6e-8) through four stages of differences over 0.1 fm
    times dtau = 0.01 and a table's row fraction; 1e-5."""
    cfg = Config(nx=nx, ny=ny, nz=nz, boost_invariant=nz == 1, dx=0.1, dy=0.1, dz=0.1, tau0=1.3, dtau=0.01,
                 eos_kind=A.EOS_CONFORMAL, eos_a=13.899692864867510, etas0=1 / (4 * np.pi), precision=precision)
    f = smooth_inputs(cfg, cfg.tau0, seed=3)
    if kind == "pressureless":
        cfg.eos_kind, cfg.eos_table = A.EOS_TABLE, dust_table(float(f[0].max()))
        f = smooth_inputs(cfg, cfg.tau0, seed=3)
    else:
        cfg.taupi_kind, cfg.taupi_const = A.TAUPI_CONST, float("inf") if kind == "infinite" else 1e300
    O = Oracle(oracle_config(cfg))
    O.set_state(f)
    tau = cfg.tau0
    for _ in range(2):
        assert O.step(tau, cfg.dtau) == 0
        tau += cfg.dtau
    want = O.get_state()
    assert np.all(np.isfinite(want))
    with Hydro(cfg) as H:
        H.set_state(f, cfg.tau0)
        H.step(2)
        got = H.get_state()
    compare_states(got, want, RUN_TOL if precision == A.PREC_FP64 else 1e-5, fields=range(18),
                   mask=interior_mask(cfg))

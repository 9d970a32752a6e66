"""What the tuner's cache file may decide: only a choice timed on the same
candidates, reconstruction and pool layout."""
import numpy as np
import pytest
import torch

from viral_b200 import _abi as A
from viral_b200 import configs as C
from viral_b200.batch import Batch

pytestmark = pytest.mark.gpu


def tuned(cache, precision, recon=A.RECON_WENO5):
    cfg = C.glauber_config(nx=8, ny=8, boost_invariant=True, precision=precision)
    cfg.recon = recon
    with Batch(cfg, [24, 30], tau0=cfg.tau0, dtau=cfg.dtau, tau_max=100.0, t_freeze_gev=0.0) as B:
        B.init_glauber(seeds=np.arange(2), bimp=[3.0, 5.0])
        return B.autotune(str(cache), probe_steps=8), B.tuning()


@pytest.mark.parametrize("precision,name", [(A.PREC_FP64, "fp64"), (A.PREC_MIXED, "mixed")])
def test_foreign_entries_are_not_obeyed(tmp_path, precision, name, monkeypatch):
    cache = tmp_path / "tune.txt"
    # an entry without the candidates' blocks per SM: indices of other kernels
    cache.write_text("%s|%s|2:2:0:0:0:0=1,77\n" % (torch.cuda.get_device_name(), name))
    ms, t = tuned(cache, precision)
    assert ms > 0 and t["steps_per_launch"] in (8, 32)
    assert tuned(cache, precision)[0] < 0  # now known
    assert tuned(cache, precision, A.RECON_MINMOD)[0] > 0
    monkeypatch.setenv("VH_BATCH_SETS", "1")
    assert tuned(cache, precision)[0] > 0
    if precision == A.PREC_FP64:  # variants 2 and 3 are 0 and 1 again
        assert t["variant"] in (0, 1, 4)

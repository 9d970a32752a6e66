"""Spectra with few azimuths a p_T, which a block's warps share by elements
instead of by bins, and with tiles of every number of bins: against the host
sums."""
import resource

import numpy as np
import pytest

from test_gpu_freezeout import dev
from viral_b200.hydro import cooper_frye_2d, cooper_frye_2d_device, cooper_frye_3d, cooper_frye_3d_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [0, 1, 31, 33, 128, 129, 1000])
@pytest.mark.parametrize("nphi", [1, 2, 3, 4, 5, 8, 9, 13, 18, 20, 21])
def test_tiles_of_few_bins(nphi, count):
    """Every term is positive, so the sums agree to the rounding of the
    exponents (below 100, 1e-14 each side) and of the terms' products."""
    rng = np.random.default_rng(100 * nphi + count)
    pt, phi = np.linspace(0.1, 2.0, 5), np.linspace(0, 2 * np.pi, nphi, endpoint=False)
    v = 0.3 * rng.standard_normal((3, count))
    for w, dev_fn, host_fn, rap in ((3, cooper_frye_2d_device, cooper_frye_2d, ()),
                                    (4, cooper_frye_3d_device, cooper_frye_3d, (0.3,))):
        el = np.zeros((count, 3 * w))
        el[:, 0] = 1 + rng.random(count)
        el[:, 1:w] = rng.standard_normal((count, w - 1)) * 0.5
        el[:, w] = 1 + rng.random(count)
        el[:, w + 1:2 * w] = 0.1 * rng.standard_normal((count, w - 1))
        el[:, 2 * w + 1:] = v[:w - 1].T
        el[:, 2 * w] = np.sqrt(1 + (v[:2] ** 2).sum(0) + (el[:, 0] * v[2]) ** 2 * (w == 4))
        host = host_fn(el, 0.15, 0.7, 3.0, *rap, pt, phi)
        got = dev_fn(dev(el), 0.15, 0.7, 3.0, *rap, pt, phi)
        assert np.allclose(got, host, rtol=1e-12, atol=0)


def test_host_memory_of_many_bins():
    """A million p_T at one azimuth: the call's host scratch is that of one
    launch's bins, well below 100 MB more than the bins and results in hand
    (in tiles of 16 all bins took 384 MB)."""
    npt = 1_000_000
    pt, phi = np.linspace(0.1, 2.0, npt), np.zeros(1)
    el = np.array([[1.0, 0, 0, 1.0, 0.1, 0.1, 1.0, 0, 0]])
    cooper_frye_2d_device(dev(el), 0.15, 0.7, 3.0, pt[:1000], phi)
    before = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss
    got = cooper_frye_2d_device(dev(el), 0.15, 0.7, 3.0, pt, phi)
    grown = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss - before
    pick = slice(0, npt, 9973)
    assert np.allclose(got[pick], cooper_frye_2d(el, 0.15, 0.7, 3.0, pt[pick], phi), rtol=1e-12, atol=0)
    assert grown < 100_000  # KB

"""The reciprocals and roots from the hardware's seeds (vh_device.cuh), and the
root-find's two eliminations with them, as the GPU computes them
(libvh_check.so): against CUDA's division and square root, 80-bit values, and
the oracle's exchanging solver."""
import ctypes
import math

import numpy as np
import pytest

from helpers import oracle_config
from pyoracle import Oracle
from test_adjoint3_cpu import L  # noqa: F401
from test_adjoint_cpu import P, _dp
from viral_b200 import _abi as A
from viral_b200 import configs as C
from viral_b200.hydro import Config

pytestmark = pytest.mark.gpu


def seeds(L, x):  # noqa: F811
    x = np.ascontiguousarray(x, dtype=np.float64)
    out, ref = np.zeros((7, x.size)), np.zeros((3, x.size))
    assert L.vhc_seeds_gpu(P(x), ctypes.c_longlong(x.size), P(out), P(ref)) == 0
    return out, ref


def ulps(a, exact, dtype):
    """|a - exact| in units of the last place of the larger"""
    step = np.spacing(np.maximum(np.abs(a), np.abs(exact).astype(np.float64)).astype(dtype)).astype(np.longdouble)
    return float(np.max(np.abs(a.astype(np.longdouble) - exact) / step))


def operands(lo, hi, seed):
    """magnitudes over 2^lo .. 2^hi: random, powers of two and their neighbours"""
    rng = np.random.default_rng(seed)
    k = 2.0 ** np.arange(lo + 1, hi)
    r = np.exp2(rng.uniform(lo, hi, 200_000))
    return np.concatenate([r, k, np.nextafter(k, np.inf), np.nextafter(k, 0)])


def test_fp64_reciprocal(L):  # noqa: F811
    """2^-1000 to 2^1000, both signs, which holds the products of four WENO
    sums (1e-92 where the weights' eps is all of them, 1e285 at |q| = 1e8).
    From a seed of 18 bits the step leaves 2^-54, half a unit, and rounds by
    another half."""
    x = operands(-1000, 1000, 1)
    x = np.concatenate([x, -x, [1e-92, 1e285]])
    out, ref = seeds(L, x)
    exact = 1 / x.astype(np.longdouble)
    for q in (0, 1):
        assert ulps(out[q], exact, np.float64) <= 1.0
        assert np.all(np.abs(out[q] - ref[0]) <= np.spacing(np.abs(ref[0])))


def test_fp64_roots(L):  # noqa: F811
    """s from 1 up: the root rounded once after a correction of second order;
    its reciprocal with s y's rounding (half a unit) and 5/16 of 2^-54."""
    x = np.concatenate([[1.0], operands(0, 1000, 2), 1 + operands(-52, 0, 3)])
    out, ref = seeds(L, x)
    exact = np.sqrt(x.astype(np.longdouble))
    assert ulps(out[2], exact, np.float64) <= 1.0
    assert ulps(out[3], 1 / exact, np.float64) <= 1.25
    assert np.all(np.abs(out[2] - ref[1]) <= np.spacing(ref[1]))
    assert np.all(np.abs(out[3] - ref[2]) <= 2 * np.spacing(ref[2]))


def test_fp32_reciprocal(L):  # noqa: F811
    """Normal operands with normal reciprocals: the seed within one unit, with
    a Newton step rounded once."""
    x = operands(-126, 126, 4)
    x = x[(x >= 2.0 ** -126) & (x <= 2.0 ** 126)].astype(np.float32).astype(np.float64)
    x = np.concatenate([x, -x])
    out, _ = seeds(L, x)
    exact = 1 / x.astype(np.longdouble)
    assert ulps(out[4], exact, np.float32) <= 1.0
    for q in (5, 6):
        assert ulps(out[q], exact, np.float32) <= 0.51


def test_reciprocals_of_zero_and_infinity(L):  # noqa: F811
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan])
    out, ref = seeds(L, x)
    for q in (1, 6):
        assert np.array_equal(out[q], ref[0], equal_nan=True)
        assert np.array_equal(np.signbit(out[q][:4]), np.signbit(ref[0][:4]))


@pytest.mark.parametrize("table", [False, True])
@pytest.mark.parametrize("size", [0.0, 0.3, 3.0, 30.0, 300.0])
def test_every_root_the_exchanging_solver_finds(L, size, table):  # noqa: F811
    """From ordinary velocities, where no multiplier is large, to u of 300,
    where most are above 1024 and the step is formed again with exchanges.
    T^{tau mu}'s rounding reaches the root times about u0^2."""
    cfg = Config(nx=4, ny=4, nz=4, boost_invariant=False, eos_kind=A.EOS_TABLE if table else A.EOS_CONFORMAL,
                 eos_table=C.eos_table() if table else None, tau0=1.3)
    O = Oracle(oracle_config(cfg))
    rng = np.random.default_rng(int(10 * size) + table)
    tau, n = 1.3, 300
    T, p5, g, u0 = np.zeros((n, 4)), np.zeros((n, 5)), np.zeros((n, 4)), np.zeros(n)
    for i in range(n):
        d = rng.normal(size=3)
        u1, u2, u3 = size * d / np.linalg.norm(d) * np.array([1, 1, 1 / tau])
        e = math.exp(rng.uniform(-2, 6))
        u0[i] = math.sqrt(1 + u1 * u1 + u2 * u2 + tau * tau * u3 * u3)
        ep = e + O.eos(e)[0]
        T[i] = ep * u0[i] ** 2 - (ep - e), ep * u0[i] * u1, ep * u0[i] * u2, ep * u0[i] * u3
        g[i] = np.array([e, u1, u2, u3]) * (1 + 0.02 * rng.normal(size=4))
    got, it = g.copy(), np.zeros(n, dtype=np.int32)
    assert L.vhc_con2prim4_gpu(ctypes.byref(cfg.to_c()), ctypes.c_longlong(n), P(T), P(p5), ctypes.c_double(tau),
                               P(got), it.ctypes.data_as(ctypes.POINTER(ctypes.c_int))) == 0
    found = 0
    for i in range(n):
        want = g[i].copy()
        if O.lib().vho_con2prim(O.h, P(T[i]), P(p5[i]), tau, want.ctypes.data_as(_dp)) < 0:
            continue
        found += 1
        assert it[i] > 0
        assert np.all(np.abs(got[i] - want) <= 1e-13 * (1 + u0[i] ** 2) * np.maximum(np.abs(want), 1e-3))
    assert found >= (n // 2 if size <= 30 else 1)

"""The fixed-point FP64 element updates on the GPU against the CPU oracle, on
what its scales depend on: side ratios on both sides of the rectangles' limit
of 32, open water (a pressure of zero), and neighbouring velocities of very
different size."""
import numpy as np
import pytest

from nextsimdg_gb300._lib import NsdgError
from nextsimdg_gb300.dynamics import BBMDynamicsKernel, MEVPDynamicsKernel
from test_stress_metric import _coords

pytestmark = pytest.mark.gpu


def _step(k, ratio, spread, steps=2, damage=None):
    nx, ny = 11, 9
    c = np.array(_coords("stretched", nx, ny), dtype=float)
    c[..., 1] *= ratio
    k.initialise(c, False, np.ones((ny, nx)))
    rng = np.random.default_rng(5)
    n = nx * ny
    f = {"hice": rng.uniform(0.2, 2.0, n), "cice": rng.uniform(0.7, 1.0, n), "uwind": np.full(n, 9.0),
         "vwind": rng.uniform(-3, 3, n), "uocean": np.zeros(n), "vocean": np.full(n, 0.02), "ssh": np.zeros(n)}
    f["u"], f["v"] = (rng.uniform(-0.1, 0.1, n) * 10.0 ** rng.uniform(-spread, 0, n) for _ in range(2))
    f["hice"][: n // 3] = f["cice"][: n // 3] = 0.0
    if damage is not None:
        f["damage"] = rng.uniform(damage, 1.0, n)
    for name, a in f.items():
        k.setData(name, a)
    for s in range(steps):
        k.update(10.0 * s, 10.0)
    return {name: k.getDG0Data(name) for name in ("hice", "cice", "u", "v")}


@pytest.mark.parametrize("ratio,spread", [(1 / 60, 0), (1 / 20, 0), (0.3, 12), (1.0, 300), (20.0, 3), (60.0, 0)])
def test_matches_oracle(gpu, oracle, ratio, spread):
    """1e-10 of the largest value, the bar of the FP64 path."""
    got = _step(MEVPDynamicsKernel(dg_comp=3, n_steps=60), ratio, spread)
    ref = _step(oracle.OracleKernel(0, 3, n_steps=60), ratio, spread)
    for name, r in ref.items():
        assert np.abs(got[name] - r).max() <= 1e-10 * max(np.abs(r).max(), 1e-300), name


@pytest.mark.parametrize("ratio,spread", [(1 / 60, 0), (1 / 20, 3), (20.0, 0), (60.0, 0)])
def test_bbm_matches_oracle(gpu, oracle, ratio, spread):
    """Ten sub-steps: 1e-10 of the largest value (the oracle's own response to
    h x (1 + 1e-14) is below 3e-14)."""
    got = _step(BBMDynamicsKernel(dg_comp=3, n_steps=10), ratio, spread, steps=1, damage=0.5)
    ref = _step(oracle.OracleKernel(1, 3, n_steps=10), ratio, spread, steps=1, damage=0.5)
    for name, r in ref.items():
        assert np.abs(got[name] - r).max() <= 1e-10 * max(np.abs(r).max(), 1e-300), name


@pytest.mark.parametrize("kind", ["box", "quads", "sphere"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_velocity_that_is_not_finite_is_reported(gpu, kind, bad):
    k = MEVPDynamicsKernel(dg_comp=1, n_steps=3)
    k.initialise(_coords(kind, 6, 5), kind == "sphere", np.ones((5, 6)))
    for name in ("hice", "cice", "uwind", "vwind", "uocean", "vocean", "ssh", "v"):
        k.setData(name, np.full(30, 0.5))
    u = np.zeros(30)
    u[14] = bad
    k.setData("u", u)
    with pytest.raises(NsdgError):
        k.update(0.0, 120.0)
        k.synchronize()

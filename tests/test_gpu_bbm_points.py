"""The BBM sub-cycle on Gauss-point values against the CPU oracle: tensor grids
(equal and unequal cells), sheared and general quadrilaterals, land cells, open
water, non-integer exponents, at sizes around the kernels' blocks of 32
elements."""
import numpy as np
import pytest

from nextsimdg_gb300.dynamics import BBMDynamicsKernel
from test_stress_metric import _coords

pytestmark = pytest.mark.gpu


def _step(k, kind, nx, ny, steps=2, thicker=0.0):
    rng = np.random.default_rng(9)
    mask = np.ones((ny, nx))
    mask[rng.integers(0, ny, 2), rng.integers(0, nx, 2)] = 0.0
    k.initialise(_coords(kind, nx, ny), False, mask)
    n = nx * ny
    f = {"hice": rng.uniform(0.2, 2.0, n), "cice": rng.uniform(0.7, 1.0, n), "damage": rng.uniform(0.5, 1.0, n),
         "u": np.zeros(n), "v": np.zeros(n), "uwind": np.full(n, 9.0), "vwind": rng.uniform(-3, 3, n),
         "uocean": np.zeros(n), "vocean": np.full(n, 0.02), "ssh": np.zeros(n)}
    f["hice"] *= 1.0 + thicker
    f["hice"][: n // 5] = 0.0  # open water
    f["cice"][: n // 5] = 0.0
    for name, a in f.items():
        k.setData(name, a)
    for s in range(steps):
        k.update(120.0 * s, 120.0)
    return {name: k.getDG0Data(name) for name in ("hice", "cice", "damage", "u", "v", "uiostress")}


CASES = [("box", 2, 3, 6, {}), ("stretched", 11, 3, 3, {}), ("sheared", 16, 8, 1, {}), ("quads", 33, 5, 6, {}),
         ("quads", 8, 4, 3, {}), ("box", 33, 29, 6, {}), ("box", 9, 9, 3, {"exponent_relaxation_sigma": 4.3}),
         ("sheared", 9, 9, 6, {"exponent_compression_factor": 1.2, "ocean_turning_angle": 25.0})]


def _oracle(oracle, dg, prm, kind, nx, ny, thicker=0.0):
    return _step(oracle.OracleKernel(1, dg, n_steps=60, **prm), kind, nx, ny, thicker=thicker)


@pytest.mark.parametrize("kind,nx,ny,dg,prm", CASES)
def test_fp64_matches_oracle(gpu, oracle, kind, nx, ny, dg, prm):
    """Rough fields amplify rounding through the damage thresholds (the
    oracle's own response to h x (1 + 1e-14) is 1e-14 on the smallest case and
    1e-3 on the largest): 1e-10 of the largest value, the bar of the FP64
    path, or 10x that response where it is above 1e-11."""
    got = _step(BBMDynamicsKernel(dg_comp=dg, n_steps=60, **prm), kind, nx, ny)
    ref, other = (_oracle(oracle, dg, prm, kind, nx, ny, t) for t in (0.0, 1e-14))
    for name, r in ref.items():
        sens = np.abs(other[name] - r).max()
        scale = max(np.abs(r).max(), 1e-300)
        assert np.abs(got[name] - r).max() <= (1e-10 * scale if sens < 1e-11 * scale else 10.0 * sens), name


@pytest.mark.parametrize("kind,nx,ny,dg,prm", CASES)
def test_mixed_within_the_mixed_bars(gpu, oracle, kind, nx, ny, dg, prm):
    """The mixed path's bars, velocity and damage 1e-5, h and A 1e-6 (RMS), or
    10x the oracle's response to h x (1 + 1e-7), one FP32 rounding."""
    got = _step(BBMDynamicsKernel(dg_comp=dg, n_steps=60, precision=1, **prm), kind, nx, ny)
    ref, other = (_oracle(oracle, dg, prm, kind, nx, ny, t) for t in (0.0, 1e-7))
    for name, bar in (("u", 1e-5), ("v", 1e-5), ("damage", 1e-5), ("hice", 1e-6), ("cice", 1e-6)):
        sens = np.sqrt(np.mean((other[name] - ref[name]) ** 2))
        assert np.sqrt(np.mean((got[name] - ref[name]) ** 2)) <= max(bar, 10.0 * sens), name


@pytest.mark.parametrize("precision", [0, 1])
def test_non_finite_stress_is_reported(gpu, precision):
    from nextsimdg_gb300.dynamics import NsdgError
    k = BBMDynamicsKernel(dg_comp=3, n_steps=5, precision=precision)
    _step(k, "box", 9, 8, steps=0)
    k.setData("u", np.full(72, np.inf))
    k.update(0.0, 120.0)
    with pytest.raises(NsdgError) as e:
        k.getDG0Data("u")
    assert e.value.status == 5  # NSDG_ERR_NUMERIC

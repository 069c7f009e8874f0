"""The sum-factorised mEVP element kernels on the GPU against the CPU oracle:
tensor grids (equal and unequal cells), sheared and general quadrilaterals and
a sphere, with land cells, at sizes around the kernels' blocks of 32 elements."""
import numpy as np
import pytest

from nextsimdg_gb300.dynamics import MEVPDynamicsKernel
from test_stress_metric import _coords

pytestmark = pytest.mark.gpu


def _step(k, kind, nx, ny, steps=2):
    rng = np.random.default_rng(7)
    mask = np.ones((ny, nx))
    mask[rng.integers(0, ny, 3), rng.integers(0, nx, 3)] = 0.0
    k.initialise(_coords(kind, nx, ny), kind == "sphere", mask)
    n = nx * ny
    f = {"hice": rng.uniform(0.2, 2.0, n), "cice": rng.uniform(0.7, 1.0, n), "u": rng.uniform(-0.1, 0.1, n),
         "v": rng.uniform(-0.1, 0.1, n), "uwind": np.full(n, 9.0), "vwind": rng.uniform(-3, 3, n),
         "uocean": np.zeros(n), "vocean": np.full(n, 0.02), "ssh": np.zeros(n)}
    for name, a in f.items():
        k.setData(name, a)
    for s in range(steps):
        k.update(120.0 * s, 120.0)
    return {name: k.getDG0Data(name) for name in ("hice", "cice", "u", "v", "uiostress", "viostress")}


@pytest.mark.parametrize("kind", ["box", "stretched", "sheared", "quads", "sphere"])
@pytest.mark.parametrize("nx,ny,dg", [(2, 3, 6), (8, 4, 1), (11, 3, 3), (33, 29, 6)])
def test_fp64_matches_oracle(gpu, oracle, kind, nx, ny, dg):
    """1e-10 of the largest value, the bar of the FP64 path."""
    got = _step(MEVPDynamicsKernel(dg_comp=dg, n_steps=60), kind, nx, ny)
    ref = _step(oracle.OracleKernel(0, dg, n_steps=60), kind, nx, ny)
    for name, r in ref.items():
        assert np.abs(got[name] - r).max() <= 1e-10 * max(np.abs(r).max(), 1e-300), name

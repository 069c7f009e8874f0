"""The sum-factorised mEVP element kernels on the GPU against the CPU oracle:
tensor grids (equal and unequal cells), sheared and general quadrilaterals and
a sphere, with land cells, at sizes around the kernels' blocks of 32 elements."""
import numpy as np
import pytest

from nextsimdg_gb300.dynamics import Ensemble, MEVPDynamicsKernel
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


@pytest.mark.parametrize("kind", ["box", "stretched", "sheared", "quads", "sphere"])
@pytest.mark.parametrize("nx,ny,dg", [(2, 3, 6), (11, 3, 3), (16, 8, 1), (33, 29, 6)])
def test_mixed_within_the_mixed_bars(gpu, oracle, kind, nx, ny, dg):
    """The mixed path's bars: velocity 1e-5 m/s, h and A 1e-6 (RMS)."""
    k = MEVPDynamicsKernel(dg_comp=dg, n_steps=60, precision=1)
    got = _step(k, kind, nx, ny)
    ref = _step(oracle.OracleKernel(0, dg, n_steps=60), kind, nx, ny)
    assert k.stress_variant()[0] == ("global" if kind in ("quads", "sphere") else "affine")
    for name, bar in (("u", 1e-5), ("v", 1e-5), ("hice", 1e-6), ("cice", 1e-6)):
        assert np.sqrt(np.mean((got[name] - ref[name]) ** 2)) <= bar, name


@pytest.mark.parametrize("kinds", [("quads", "box"), ("quads", "sheared"), ("stretched", "sheared")])
def test_ensemble_of_mixed_geometries(gpu, kinds):
    """An ensemble whose members have different maps: bitwise the members'
    single runs where one kernel serves all members in both, else within FP32
    rounding of them (1e-5 m/s after two steps)."""
    sizes = [(13, 11), (37, 9)]
    ref = [_step(MEVPDynamicsKernel(dg_comp=3, n_steps=60, precision=1), k, *s) for k, s in zip(kinds, sizes)]
    members = [MEVPDynamicsKernel(dg_comp=3, n_steps=60, precision=1) for _ in kinds]
    for m, k, s in zip(members, kinds, sizes):
        _step(m, k, *s, steps=0)
    ens = Ensemble(members)
    for i in range(2):
        ens.update(120.0 * i, 120.0)
    ens.synchronize()
    for m, r in zip(members, ref):
        for name in ("u", "v"):
            d = m.getDG0Data(name) - r[name]
            if "quads" not in kinds:
                assert np.all(d == 0.0), name
            assert np.sqrt(np.mean(d * d)) <= 1e-5, name


@pytest.mark.parametrize("kind", ["stretched", "quads"])
def test_one_thread_per_element_is_bitwise_three(gpu, kind):
    """From 16,384 elements the element kernels run one thread per element: an
    ensemble above that of members below it is bitwise their single runs."""
    sizes = [(127, 90), (61, 83)]
    ref = [_step(MEVPDynamicsKernel(dg_comp=3, n_steps=20, precision=1), kind, *s) for s in sizes]
    members = [MEVPDynamicsKernel(dg_comp=3, n_steps=20, precision=1) for _ in sizes]
    for m, s in zip(members, sizes):
        _step(m, kind, *s, steps=0)
    ens = Ensemble(members)
    for i in range(2):
        ens.update(120.0 * i, 120.0)
    ens.synchronize()
    assert ens.tile(0) == (64, 1)
    for m, r in zip(members, ref):
        for name in ("u", "v"):
            np.testing.assert_array_equal(m.getDG0Data(name), r[name])

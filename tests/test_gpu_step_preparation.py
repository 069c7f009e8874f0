"""What a step prepares before its sub-cycle, on the GPU against the CPU oracle:
node values of thickness and concentration, a rough sea surface's gradient,
pressures and node constants, at mesh widths down to two cells; and the batched
conversion of module_step's node fields."""
import numpy as np
import pytest

from nextsimdg_gb300.dynamics import BBMDynamicsKernel, MEVPDynamicsKernel
from test_stress_metric import _coords

pytestmark = pytest.mark.gpu


def _fields(nx, ny, bbm):
    rng = np.random.default_rng(11)
    n = nx * ny
    f = {"hice": rng.uniform(0.0, 2.0, n), "cice": rng.uniform(0.0, 1.0, n), "u": np.zeros(n), "v": np.zeros(n),
         "uwind": rng.uniform(-9, 9, n), "vwind": rng.uniform(-3, 3, n), "uocean": rng.uniform(-0.1, 0.1, n),
         "vocean": np.full(n, 0.02), "ssh": rng.uniform(-0.1, 0.1, n)}
    if bbm:
        f["damage"] = rng.uniform(0.5, 1.0, n)
    f["hice"][0] = f["cice"][0] = 0.0
    return f


def _step(k, kind, nx, ny, bbm):
    k.initialise(_coords(kind, nx, ny), False, np.ones((ny, nx)))
    for name, a in _fields(nx, ny, bbm).items():
        k.setData(name, a)
    k.update(0.0, 120.0)
    return {name: k.getDG0Data(name) for name in ("hice", "cice", "u", "v")}


@pytest.mark.parametrize("nx,ny", [(2, 2), (2, 5), (5, 2), (2, 3), (127, 2), (33, 31)])
@pytest.mark.parametrize("dg", [1, 3, 6])
@pytest.mark.parametrize("bbm", [False, True])
def test_fp64_matches_oracle(gpu, oracle, nx, ny, dg, bbm):
    """1e-10 of the largest value, the bar of the FP64 path (the oracle's own
    response to h x (1 + 1e-14) is below 1e-11 on every case)."""
    n = 40 if bbm else 3
    kind = "quads" if nx > 1 and ny > 1 else "box"
    got = _step((BBMDynamicsKernel if bbm else MEVPDynamicsKernel)(dg_comp=dg, n_steps=n), kind, nx, ny, bbm)
    ref = _step(oracle.OracleKernel(int(bbm), dg, n_steps=n), kind, nx, ny, bbm)
    for name, r in ref.items():
        assert np.abs(got[name] - r).max() <= 1e-10 * max(np.abs(r).max(), 1e-300), name


@pytest.mark.parametrize("dg", [1, 3])
@pytest.mark.parametrize("precision", [0, 1])
def test_module_step_converts_as_set_data(gpu, dg, precision):
    """Bitwise the node fields that setData leaves, with more of them than one
    launch converts."""
    nx, ny = 9, 6
    f = _fields(nx, ny, False)
    ref = _step(MEVPDynamicsKernel(dg_comp=dg, n_steps=3, precision=precision), "sheared", nx, ny, False)
    k = MEVPDynamicsKernel(dg_comp=dg, n_steps=3, precision=precision)
    k.initialise(_coords("sheared", nx, ny), False, np.ones((ny, nx)))
    out = k.module_step(0.0, 120.0, f, list(ref))
    for name, r in ref.items():
        np.testing.assert_array_equal(np.asarray(out[name]).ravel(), np.asarray(r).ravel())


@pytest.mark.parametrize("bbm", [False, True])
def test_second_initialise_takes_the_new_mesh(gpu, bbm):
    """Parallelograms (tiled transport), then general quadrilaterals on the same
    handle: bitwise a fresh handle's step."""
    new = lambda: (BBMDynamicsKernel if bbm else MEVPDynamicsKernel)(dg_comp=3, n_steps=40, precision=1)  # noqa: E731
    k = new()
    _step(k, "sheared", 9, 6, bbm)
    assert k.transport_variant()[0] == "tiled"
    again, ref = _step(k, "quads", 9, 6, bbm), _step(new(), "quads", 9, 6, bbm)
    assert k.transport_variant()[0] == "element"
    for name, r in ref.items():
        np.testing.assert_array_equal(again[name], r)

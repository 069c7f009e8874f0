"""A handle's second initialise: the step on the new mesh is bitwise that of a
fresh handle, whatever kind of mesh came before (parallelograms, general
quadrilaterals, a sphere, other sizes)."""
import numpy as np
import pytest

from nextsimdg_gb300.dynamics import BBMDynamicsKernel, MEVPDynamicsKernel
from test_gpu_step_preparation import _fields
from test_stress_metric import _coords

pytestmark = pytest.mark.gpu


def _step(k, kind, nx, ny, bbm):
    k.initialise(_coords(kind, nx, ny), kind == "sphere", np.ones((ny, nx)))
    for name, a in _fields(nx, ny, bbm).items():
        k.setData(name, a)
    k.update(0.0, 120.0)
    return {name: k.getDG0Data(name) for name in ("hice", "cice", "u", "v", "uiostress") + (("damage",) if bbm else ())}


PAIRS = [("sheared", "quads"), ("quads", "sheared"), ("box", "quads"), ("quads", "box"), ("sphere", "box"),
         ("box", "sphere"), ("sphere", "quads"), ("quads", "sphere")]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("bbm", [False, True])
@pytest.mark.parametrize("first,second", PAIRS)
def test_bitwise_a_fresh_handle(gpu, first, second, bbm, precision):
    if bbm and "sphere" in (first, second):
        pytest.skip("BBM takes no spherical meshes")
    new = lambda: (BBMDynamicsKernel if bbm else MEVPDynamicsKernel)(  # noqa: E731
        dg_comp=3, n_steps=20, precision=precision)
    k = new()
    _step(k, first, 14, 9, bbm)
    again, ref = _step(k, second, 9, 6, bbm), _step(new(), second, 9, 6, bbm)
    for name, r in ref.items():
        np.testing.assert_array_equal(again[name], r, err_msg=name)


def test_float_pair_kernel_does_not_outlive_its_mesh(gpu, monkeypatch):
    """NSDG_FP64_STRESS=pairs applies to Cartesian meshes: a sphere after one
    takes the kernel that a fresh handle takes."""
    monkeypatch.setenv("NSDG_FP64_STRESS", "pairs")
    k = MEVPDynamicsKernel(dg_comp=3, n_steps=20)
    _step(k, "quads", 14, 9, False)
    again, ref = _step(k, "sphere", 9, 6, False), _step(MEVPDynamicsKernel(dg_comp=3, n_steps=20), "sphere", 9, 6, False)
    for name, r in ref.items():
        np.testing.assert_array_equal(again[name], r, err_msg=name)

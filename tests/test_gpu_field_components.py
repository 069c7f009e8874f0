"""Node fields given with another number of components than the handle's: the
cell averages (component 0) count, as DG2CG of the reference's ma2dg takes them
(DGModelArray.hpp:20-32, CGDynamicsKernel.cpp:54-90)."""
import numpy as np
import pytest

from nextsimdg_gb300.dynamics import BBMDynamicsKernel, MEVPDynamicsKernel
from test_gpu_step_preparation import _fields
from test_stress_metric import _coords

pytestmark = pytest.mark.gpu

NODE_FIELDS = ("u", "v", "uwind", "vwind", "uocean", "vocean")


@pytest.mark.parametrize("dg,comps", [(1, 2), (1, 3), (1, 6), (3, 1), (3, 2), (3, 6), (6, 3), (6, 8), (1, 1), (3, 3), (6, 6)])
@pytest.mark.parametrize("bbm", [False, True])
@pytest.mark.parametrize("together", [False, True])
def test_as_the_oracle(gpu, oracle, dg, comps, bbm, together):
    nx, ny = 11, 7
    f = _fields(nx, ny, bbm)
    rng = np.random.default_rng(3)
    for name in NODE_FIELDS:
        f[name] = np.stack([f[name] + 0.1 * rng.standard_normal(nx * ny)]
                           + [rng.standard_normal(nx * ny) for _ in range(comps - 1)], axis=1)
    f["u"], f["v"] = 0.05 * f["u"], 0.05 * f["v"]

    def step(k):
        k.initialise(_coords("quads", nx, ny), False, np.ones((ny, nx)))
        if together and hasattr(k, "module_step"):
            k.module_step(0.0, 20.0, f, [])
        else:
            for name, a in f.items():
                k.setData(name, a)
            k.update(0.0, 20.0)
        return {name: k.getDG0Data(name) for name in ("u", "v", "hice", "cice")}

    got = step((BBMDynamicsKernel if bbm else MEVPDynamicsKernel)(dg_comp=dg, n_steps=4))
    ref = step(oracle.OracleKernel(int(bbm), dg, n_steps=4))
    for name, r in ref.items():  # the FP64 path's bar
        assert np.abs(got[name] - r).max() <= 1e-10 * max(np.abs(r).max(), 1e-300), name

"""The damage projection of the BBM sub-cycle keeps a constant: uniform damage in
calm, compact ice stays what it is through the sub-steps of several updates."""
import numpy as np
import pytest

from nextsimdg_gb300.dynamics import BBMDynamicsKernel
from test_stress_metric import _coords

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["box", "sheared", "quads"])
@pytest.mark.parametrize("dg", [1, 3, 6])
@pytest.mark.parametrize("damage", [1.0, 0.7])
def test_fp64_damage_stays(gpu, kind, dg, damage):
    """With row sums of 1 and 0 to half a unit of the centre's weight, a sub-step
    moves a constant by less than two of its units, and not at all once its
    rounded image is itself: 16 units of 2^-53 (a projection off by 2^-53 in each of
    the 300 sub-steps moves it by 300)."""
    nx, ny = 13, 9
    k = BBMDynamicsKernel(dg_comp=dg, n_steps=100)
    k.initialise(_coords(kind, nx, ny), False, np.ones((ny, nx)))
    n = nx * ny
    for name, a in {"hice": 1.0, "cice": 1.0, "damage": damage, "u": 0.0, "v": 0.0, "uwind": 0.0, "vwind": 0.0,
                    "uocean": 0.0, "vocean": 0.0, "ssh": 0.0}.items():
        k.setData(name, np.full(n, a))
    for s in range(3):
        k.update(120.0 * s, 120.0)
    assert np.abs(k.getDG0Data("damage") / damage - 1.0).max() <= 16 * 2.0 ** -53

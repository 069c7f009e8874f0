"""nsdg_kernel_time_kernel repeats one kernel on the handle's own state; a
repetition follows the one before it.  The state that many repetitions in a row
leave is bitwise that of the same number one by one, each waited for."""
import numpy as np
import pytest

from nextsimdg_gb300.dynamics import BBMDynamicsKernel, MEVPDynamicsKernel
from test_gpu_step_preparation import _fields
from test_stress_metric import _coords

pytestmark = pytest.mark.gpu

CASES = [(False, kind, precision) for kind in ("box", "quads", "sphere") for precision in (0, 1)] \
    + [(True, kind, precision) for kind in ("box", "quads") for precision in (0, 1)]


@pytest.mark.parametrize("bbm,kind,precision", CASES)
@pytest.mark.parametrize("kernel_id", [0, 1])
@pytest.mark.parametrize("nx,ny", [(23, 17), (150, 120)])
def test_repetitions_follow_each_other(gpu, bbm, kind, precision, kernel_id, nx, ny):
    def run(calls, reps):  # a call launches once more than reps
        k = (BBMDynamicsKernel if bbm else MEVPDynamicsKernel)(dg_comp=3, n_steps=10, precision=precision)
        k.initialise(_coords(kind, nx, ny), kind == "sphere", np.ones((ny, nx)))
        for name, a in _fields(nx, ny, bbm).items():
            k.setData(name, a)
        k.update(0.0, 20.0)
        for _ in range(calls):
            k.time_kernel(kernel_id, reps)
        k.update(20.0, 20.0)
        return {name: k.getDG0Data(name) for name in ("u", "v", "hice")}

    one_by_one, in_a_row = run(12, 1), run(1, 23)
    for name, a in one_by_one.items():
        np.testing.assert_array_equal(in_a_row[name], a, err_msg=name)

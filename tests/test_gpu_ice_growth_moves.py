"""Fields of the GPU growth component from and to host arrays: moved directly by
a kernel (pageable arrays on a GPU that reads them), through the pinned buffer
(NSDG_HOST_DIRECT=0) and from page-locked arrays, the same bits."""
import numpy as np
import pytest
import torch

from nextsimdg_gb300.ice_growth import IceGrowth

pytestmark = pytest.mark.gpu

INPUTS = ("hice", "cice", "hsnow", "tice", "qia", "dqia_dt", "qow", "qio", "sublim", "snowfall", "penSW", "sst", "tf",
          "mlbhc", "damage")
OUTPUTS = ("hice_updated", "cice_updated", "hsnow_updated", "tice_updated", "damage", "newice", "snow_melt", "qio")


@pytest.mark.parametrize("n", [1, 511, 4097])
def test_moves_are_bitwise_copies(gpu, monkeypatch, n):
    rng = np.random.default_rng(n)
    f = {name: rng.uniform(0.1, 1.0, n + 1)[1:] for name in INPUTS}  # not 16-byte aligned

    def outputs(locked=False):
        g = IceGrowth(n)
        for name, a in f.items():
            g.setData(name, torch.from_numpy(a.copy()).pin_memory().numpy() if locked else a)
            np.testing.assert_array_equal(g.getData(name), a)
        g.update(3600.0)
        return [g.getData(name) for name in OUTPUTS]

    direct, locked = outputs(), outputs(locked=True)
    monkeypatch.setenv("NSDG_HOST_DIRECT", "0")
    for a, b, c in zip(outputs(), direct, locked):
        np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(a, c)

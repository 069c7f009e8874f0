"""Fields in and out on both sides of the sizes from which they move by a kernel:
the same bits as through the page-locked buffer, also when a field is set, read
and set again without an update between."""
import numpy as np
import pytest

from nextsimdg_gb300.ice_growth import IceGrowth

pytestmark = pytest.mark.gpu

INPUTS = ("hice", "cice", "hsnow", "tice", "qia", "dqia_dt", "qow", "qio", "sublim", "snowfall", "penSW", "sst", "tf",
          "mlbhc", "damage")
OUTPUTS = ("hice_updated", "cice_updated", "hsnow_updated", "tice_updated", "damage", "newice")


@pytest.mark.parametrize("n", [5999, 6000, 23999, 24000, 24001])
def test_the_same_bits_either_way(gpu, monkeypatch, n):
    rng = np.random.default_rng(n)
    f = {name: rng.uniform(0.1, 1.0, n) for name in INPUTS}

    def outputs():
        g = IceGrowth(n)
        for name, a in f.items():
            g.setData(name, np.zeros(n))
            g.setData(name, a)
        got = [g.getData(name) for name in INPUTS]
        g.update(3600.0)
        return got + [g.getData(name) for name in OUTPUTS]

    direct = outputs()
    monkeypatch.setenv("NSDG_HOST_DIRECT", "0")
    for a, b in zip(outputs(), direct):
        np.testing.assert_array_equal(a, b)
    for a, name in zip(direct, INPUTS):
        np.testing.assert_array_equal(a, f[name])

"""The element maps the sum-factorised stress kernels take: the strain and
divergence operators rebuilt from them on the host against the exact ones."""
import numpy as np
import pytest

from nextsimdg_gb300.boxtest import BoxTest


def _coords(kind, nx, ny):
    if kind == "sphere":
        lon, lat = np.linspace(-0.3, 0.3, nx + 1), np.linspace(1.0, 1.3, ny + 1)
        return np.stack([a.ravel() for a in np.meshgrid(lon, lat)], axis=1)
    if kind == "stretched":  # a tensor grid of unequal cells
        x, y = np.linspace(0, 1, nx + 1) ** 1.3 * 4e5, np.linspace(0, 1, ny + 1) ** 0.8 * 3e5
        return np.stack([a.ravel() for a in np.meshgrid(x, y)], axis=1)
    c = BoxTest(nx, ny, distort=0.04 if kind == "quads" else 0.0).coords()
    if kind == "sheared":
        c[:, 0] += 0.3 * c[:, 1]
    return c


@pytest.mark.parametrize("kind", ["box", "stretched", "sheared", "quads", "sphere"])
@pytest.mark.parametrize("nx,ny", [(2, 2), (17, 9)])
def test_rebuilt_operators_match_the_exact_ones(nsdg_lib, kind, nx, ny):
    """Both are FP64 products of at most nine terms around an 8 x 8 inverse
    whose condition number is about 1e4: 1e-11 of the largest entry."""
    from nextsimdg_gb300.dynamics import metric_mismatch
    assert metric_mismatch(_coords(kind, nx, ny), nx, ny, kind == "sphere") <= 1e-11

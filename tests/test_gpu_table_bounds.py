"""Loaded tables: the exactness bound of the team kernel at its limits (in-degree 65535, and
sums of weights below 2^31 in units of 2^-16), over the edges of the parts in which the
in-degrees are counted (51,200 neurons each)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [20000, 51200, 51201, 102401])
@pytest.mark.parametrize("into,weight,fits", [(65535, 1e-3, True), (65536, 1e-3, False),
                                              (1, 20000.0, True), (2, 20000.0, False), (2, -20000.0, False)])
def test_bound(g4s, n, into, weight, fits):
    idx = np.full((n, 4), -1, dtype=np.int32)
    w = np.zeros((n, 4), dtype=np.float32)
    for target in (0, n // 2 + 1, n - 1):
        idx[:], w[:] = -1, 0.0
        idx.reshape(-1)[-into:] = target  # (the table's last slots)
        w.reshape(-1)[-into:] = weight
        w[0] = np.where(idx[0] < 0, 3e4, w[0])  # (an unused slot's weight counts for nothing)
        with g4s.Network(n, 4, seed=3, record_raster=False) as net:
            net.load_tables(idx, w)
            net.run(1)
            assert (net.geometry()[0] >= 1) == fits

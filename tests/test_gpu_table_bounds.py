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


@pytest.mark.parametrize("ran", [False, True])
@pytest.mark.parametrize("n,nsyn", [(7001, 9), (21846, 3), (20001, 300)])
def test_refused_upload_keeps_the_tables(g4s, oracle, n, nsyn, ran):
    """Uploads checked on the device (65,536 slots or more), before and after the packed rows
    exist: the first offending slot is named, the network runs on as if there had been no
    upload, and the same call with good tables is taken."""
    d = oracle.make_desc(n, nsyn, 21, drive_scale=2.0)
    idx, w = oracle.conn_philox(d)
    sim = oracle.Sim(d, idx, w)
    sim.run(40, threads=8)
    with g4s.Network(n, nsyn, seed=21, drive_scale=2.0) as net:
        own = net.tables()
        net.run(20 if ran else 0)
        for pos in (0, 3, idx.size // 2 + 1, idx.size - 1):
            bad = np.where(own[0] < 0, -5, n - 1).astype(np.int32)
            bad.flat[pos] = n
            bad.flat[idx.size - 1] = np.iinfo(np.int32).max
            with pytest.raises(g4s.G4SError) as e:
                net.load_tables(bad, np.zeros_like(own[1]))
            assert f"table entry {pos} targets neuron {bad.flat[pos]} " in str(e.value)
        net.run(20 if ran else 40)
        assert np.array_equal(np.stack(net.raster()), np.stack(sim.raster()))
        net.load_tables(idx, w)
        net.reset()
        net.run(40)
        assert np.array_equal(np.stack(net.raster()), np.stack(sim.raster()))
        assert all(np.array_equal(a, b) for a, b in zip(own, net.tables()))


@pytest.mark.parametrize("ran", [False, True])
@pytest.mark.parametrize("n,nsyn", [(2001, 9), (20001, 300)])
def test_upload_that_fails_half_way(g4s, oracle, n, nsyn, ran):
    """An upload that runs out of memory once the new tables (rows in draw order) have replaced
    the old ones, checked on the host or on the device, before and after the packed rows exist:
    no run uses what was planned for the old tables, and the next upload is taken."""
    from gpu4snn_gb300 import _lib
    d = oracle.make_desc(n, nsyn, 22, drive_scale=2.0)
    idx, w = oracle.conn_philox(d)
    sim = oracle.Sim(d, idx, w)
    sim.run(40, threads=8)
    with g4s.Network(n, nsyn, seed=23, drive_scale=2.0) as net:
        net.run(20 if ran else 0)
        assert net.geometry()[0] >= 1
        net.inject_fault(_lib.FAULT_ALLOC)
        with pytest.raises(g4s.G4SError) as e:
            net.load_tables(idx, w)
        assert e.value.code == _lib.ERR_NOMEM
        assert net.geometry() == (0, 0)
        net.run(20)
    with g4s.Network(n, nsyn, seed=22, drive_scale=2.0) as net:
        net.run(20 if ran else 0)
        net.inject_fault(_lib.FAULT_ALLOC)
        with pytest.raises(g4s.G4SError):
            net.load_tables(idx, w)
        net.load_tables(idx, w)
        assert net.geometry()[0] >= 1
        net.reset()
        net.run(40)
        assert np.array_equal(np.stack(net.raster()), np.stack(sim.raster()))

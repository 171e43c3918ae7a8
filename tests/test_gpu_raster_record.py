"""The host record of the raster: many small chunks, a stretch of steps streamed to a file
in between (not kept on the host), reads into buffers that are too short, a run long enough
to outgrow the first raster buffer."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alg", [2, 4])
@pytest.mark.parametrize("budget", [0, 4 * 2000 * 7])
def test_recorded_and_streamed_stretches(g4s, oracle, tmp_path, alg, budget):
    from gpu4snn_gb300 import _lib, formats
    n, nsyn, seed = 2000, 150, 71
    d = oracle.make_desc(n, nsyn, seed, drive_scale=1.5)
    idx, w = oracle.conn_philox(d)
    sim = oracle.Sim(d, idx, w)
    sim.run(75 + 700, threads=8)
    ot, oi = sim.raster()
    with g4s.Network(n, nsyn, seed=seed, drive_scale=1.5, raster_budget_bytes=budget) as net:
        net.run(30, alg)
        net.stream_raster(str(tmp_path / "r.bin"))
        net.run(20, alg)
        net.stream_raster(None)
        net.run(25, alg)
        net.run(700, alg)
        keep = (ot < 30) | (ot >= 50)
        t, i = net.raster()
        assert np.array_equal(t, ot[keep]) and np.array_equal(i, oi[keep])
        assert np.array_equal(net.counts(), sim.counts())
        for cap in (1, int(np.searchsorted(ot, 29)) + 3, len(t) - 1):
            a, b = np.full(cap + 4, -9, np.int32), np.full(cap + 4, -9, np.int32)
            size = C.c_int64()
            _lib.check(g4s.load().g4s_net_raster(net._h, _lib.ptr(a), _lib.ptr(b), cap, C.byref(size)))
            assert size.value == len(t)
            assert np.array_equal(a[:cap], t[:cap]) and np.array_equal(b[:cap], i[:cap])
            assert (a[cap:] == -9).all() and (b[cap:] == -9).all()
        r = formats.read_raster(str(tmp_path / "r.bin"))
        assert r.t0 == 30 and np.array_equal(r.ids, oi[~keep]) and np.array_equal(r.counts, sim.counts()[30:50])


@pytest.mark.parametrize("alg", [3, 4])
@pytest.mark.parametrize("n", [2000, 300_000, 2_500_000, 4_300_000])
def test_large_steps_in_order(g4s, n, alg):
    """Steps with a burst of a third of the neurons, whose ids the host sorts (by two or three
    digits of 11 bits): ascending, each as often as the neuron's own count of its spikes."""
    with g4s.Network(n, 4, seed=58, drive_scale=3.0) as net:
        net.run(30, alg)
        t, i = net.raster()
        c = net.counts()
        assert c.max() > n // 8
        assert np.array_equal(np.bincount(t, minlength=30), c)
        assert (np.diff(i.astype(np.int64) + t.astype(np.int64) * n) > 0).all()
        assert np.array_equal(np.bincount(i, minlength=n), net.state()["nospks"])

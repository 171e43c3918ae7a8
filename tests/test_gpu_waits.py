"""Waits of the team kernel that last a second or more.  Warps of large steps draw the next
step's drive while they poll; what they draw is bounded by the slice, however long the wait."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads,geometry", [(1024, (0, 0)), (1024, (16, 0)), (1024, (0, 1)), (768, (0, 0))])
def test_long_wait_that_times_out(g4s, oracle, threads, geometry):
    """A launch's first step waits sixteen times the limit, 1.6 s here, for a block that does not
    exist: the run reports it, and the handle goes on."""
    from gpu4snn_gb300 import _lib
    n, nsyn, seed = 150_000, 24, 61
    d = oracle.make_desc(n, nsyn, seed)
    idx, w = oracle.conn_philox(d)
    sim = oracle.Sim(d, idx, w)
    sim.run(30, threads=8)
    with g4s.Network(n, nsyn, seed=seed) as net:
        net.set_geometry(*geometry)
        net.set_block_threads(threads)
        net.set_barrier_timeout(100_000_000)
        net.inject_fault(_lib.FAULT_BARRIER_STALL)
        with pytest.raises(g4s.G4SError) as e:
            net.run(10, 4)
        assert e.value.code == _lib.ERR_TIMEOUT
        net.reset()
        net.run(30, 4)
        assert np.array_equal(np.stack(net.raster()), np.stack(sim.raster()))
        assert np.array_equal(net.currents(), sim.acc())


def test_team_that_waits_for_another(g4s):
    """Two networks whose teams do not fit the GPU together: most ranks of the second wait in
    their first step until the first network's chunk ends, about 1.5 s (1024 threads, segment
    runs, slices of 8,131 neurons), and both end as when they run alone."""
    from gpu4snn_gb300.network import run_batch
    n, nsyn, steps = 1_000_000, 100, 5000
    nets = [g4s.Network(n, nsyn, seed=62 + k, drive_scale=8.0, record_raster=False) for k in range(2)]
    run_batch(nets, steps)
    for k, net in enumerate(nets):
        with g4s.Network(n, nsyn, seed=62 + k, drive_scale=8.0, record_raster=False) as alone:
            alone.run(steps, 4)
            assert np.array_equal(alone.counts(), net.counts())
            a, b = alone.state(), net.state()
            assert all(np.array_equal(a[f].view(np.uint32), b[f].view(np.uint32)) for f in ("v", "u", "I", "nospks"))
        net.close()


@pytest.mark.parametrize("n,threads,geometry,fits", [(700, 0, (0, -1), True), (2000, 0, (0, -1), True), (2000, 0, (4, 0), True),
                                                     (2000, 0, (15, 1), True), (9000, 1024, (0, 0), True),
                                                     (2000, 0, (0, -1), False)])
def test_limit_of_nothing(g4s, oracle, n, threads, geometry, fits):
    """A time limit of 0 ends every run that waits, however short the wait would be: alone, in a
    batch, in the FP64 check, and on the global-atomic kernel (tables beyond the exactness
    bound of the team kernel)."""
    from gpu4snn_gb300 import _lib
    from gpu4snn_gb300.network import run_batch
    nsyn, seed = 100, 63
    d = oracle.make_desc(n, nsyn, seed)
    idx, w = oracle.conn_philox(d)
    if not fits:
        w = w.copy()
        idx[0, :2], w[0, :2] = (5, 6), 30000.0
        idx[1, :2], w[1, :2] = (5, 6), 30000.0
    sim = oracle.Sim(d, idx, w)
    sim.run(30, threads=8)

    def check(call):
        with pytest.raises(g4s.G4SError) as e:
            call()
        assert e.value.code == _lib.ERR_TIMEOUT

    with g4s.Network(n, nsyn, seed=seed, tables=(idx, w)) as net, g4s.Network(300, 50, seed=64) as one:
        net.set_geometry(*geometry)
        net.set_block_threads(threads)
        assert (net.geometry()[0] > 1) == fits
        net.set_barrier_timeout(0)
        check(lambda: net.run(20, 4))
        net.reset()
        check(lambda: net.fp64_check(5))
        net.reset()
        if fits and geometry[0]:
            check(lambda: run_batch([net, one], 20))
            net.reset()
            one.reset()
        net.set_barrier_timeout(2_000_000_000)
        net.run(30, 4)
        assert np.array_equal(np.stack(net.raster()), np.stack(sim.raster()))
        assert np.array_equal(net.currents(), sim.acc())
        one.set_barrier_timeout(0)  # (one CTA: no waits)
        one.run(20, 4)
        assert one.info().steps_done == 20

"""The global-memory schemes at the sizes where their step loop changes its launch shape (one
block of 256 or 512 threads per SM, two per SM), with bursts of a whole block's neurons."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7, 38_912, 38_913, 77_824, 77_825, 180_001])
def test_scheme_sizes(g4s, oracle, n):
    nsyn, seed = 5, 81
    d = oracle.make_desc(n, nsyn, seed, drive_scale=3.0)
    idx, w = oracle.conn_philox(d)
    sim = oracle.Sim(d, idx, w)
    sim.run(24, threads=8)
    ot, oi = sim.raster()
    want, cur = sim.state(), sim.acc()
    with g4s.Network(n, nsyn, seed=seed, drive_scale=3.0) as net:
        for alg in (0, 1, 2, 3):
            net.reset()
            net.run(10, alg)
            net.run(14, alg)
            t, i = net.raster()
            assert np.array_equal(t, ot) and np.array_equal(i, oi), alg
            got = net.state()
            for k in ("v", "u", "I"):
                assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), (alg, k)
            assert np.array_equal(got["nospks"], want["nospks"]) and np.array_equal(net.currents(), cur)


@pytest.mark.parametrize("nsyn", [125, 129, 511, 512, 513, 1021, 1024, 1025])
def test_row_lengths(g4s, oracle, nsyn):
    """Rows around one and four vectors a thread of N's and AP's groups (32 and 64 threads)."""
    n, seed = 1500, 82
    d = oracle.make_desc(n, nsyn, seed, drive_scale=3.0)
    idx, w = oracle.conn_philox(d)
    sim = oracle.Sim(d, idx, w)
    sim.run(30, threads=8)
    for alg in (0, 1):
        with g4s.Network(n, nsyn, seed=seed, drive_scale=3.0) as net:
            net.run(30, alg)
            assert np.array_equal(net.counts(), sim.counts())
            assert np.array_equal(net.currents(), sim.acc())


@pytest.mark.parametrize("nsyn,two", [(7000, False), (7600, True)])
def test_steps_with_many_synapses(g4s, nsyn, two):
    """Scheme S at sizes on both sides of 16 million expected synapses a step (22 Hz at drive 3
    before there is a measured rate), from which it takes two launches a step: the results of
    the SKL scheme."""
    n = 100_000
    with g4s.Network(n, nsyn, seed=83, drive_scale=3.0) as net:
        net.run(24, 4)
        want, cur, raster = net.state(), net.currents(), np.stack(net.raster())
        net.reset()
        net.run(10, 2)
        assert net.info().last_run_launches == (20 if two else 1)
        net.run(14, 2)
        assert np.array_equal(np.stack(net.raster()), raster) and np.array_equal(net.currents(), cur)
        got = net.state()
        assert all(np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)) for k in want)

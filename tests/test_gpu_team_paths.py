"""The team kernel's exchange and table layouts at their edges, against the oracle: team
sizes around the one from which warps poll source ranks of their own, ranks with more spikes
than their record lines hold, and weights too large to be packed beside their targets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run_both(g4s, oracle, n, nsyn, seed, drive, steps, geometry, threads, scale=None):
    d = oracle.make_desc(n, nsyn, seed, drive_scale=drive)
    idx, w = oracle.conn_philox(d)
    if scale is not None:  # a few weights scaled up, at the ends of rows and of the table
        w = w.copy()
        for pos in (0, n * nsyn // 2, n * w.shape[1] - 1 - (w.shape[1] - nsyn)):
            w.flat[pos] = scale
    sim = oracle.Sim(d, idx, w)
    sim.run(steps, threads=8)
    with g4s.Network(n, nsyn, seed=seed, drive_scale=drive, tables=(idx, w)) as net:
        net.set_geometry(*geometry)
        net.set_block_threads(threads)
        net.run(steps // 2, 4)
        net.run(steps - steps // 2, 4)
        assert np.array_equal(np.stack(net.raster()), np.stack(sim.raster()))
        s, o = net.state(), sim.state()
        for k in ("v", "u", "I"):
            # (a neuron whose potential overflows ends with u = NaN, whose bits differ by machine)
            a, b = s[k], o[k]
            assert np.array_equal(np.isnan(a), np.isnan(b)), k
            assert np.array_equal(a[~np.isnan(a)].view(np.uint32), b[~np.isnan(b)].view(np.uint32)), k
        assert np.array_equal(s["nospks"], o["nospks"])
        assert np.array_equal(net.currents(), sim.acc())
        return net.counts()


@pytest.mark.parametrize("threads", [768, 1024])
@pytest.mark.parametrize("p", [2, 11, 12, 13, 22, 23, 25, 33])
def test_source_ranks(g4s, oracle, p, threads):
    """A rank's few hundred neurons at drive 2 (about 60 spikes a step in the first burst):
    more ids than a record's lines hold, in teams on both sides of every split of the ranks
    over the warps."""
    counts = run_both(g4s, oracle, 3001, 203, 51, 2.0, 60, (p, 0), threads)
    assert counts.max() > 31 * 2


@pytest.mark.parametrize("threads,delivery", [(768, 1), (1024, 0), (1024, 1)])
@pytest.mark.parametrize("p", [14, 15, 16, 17, 18, 24])
def test_shared_sources(g4s, oracle, p, threads, delivery):
    """Teams around sixteen ranks, up to which the warps of large steps and of the group mapping
    share all ranks' spikes."""
    counts = run_both(g4s, oracle, 3001, 203, 56, 2.0, 60, (p, delivery), threads)
    assert counts.max() > 31 * 2


@pytest.mark.parametrize("delivery", [0, 1])
def test_single_spikes_and_bursts(g4s, oracle, delivery):
    """Steps without any spike, and a burst with more than 64 spikes a rank."""
    counts = run_both(g4s, oracle, 5003, 203, 52, 2.0, 60, (16, delivery), 0)
    assert counts.max() > 16 * 64 and counts.min() == 0


@pytest.mark.parametrize("geometry", [(0, 0), (40, 1), (9, 0)])
@pytest.mark.parametrize("scale", [16383.0, 20000.0, -20000.0])
def test_weights_at_the_packing_limit(g4s, oracle, geometry, scale):
    """70,000 targets take 17 bits of a packed word, which leaves Q32.32 weights below 2^14:
    16383 is packed, +-20000 sends the network to the separate arrays."""
    run_both(g4s, oracle, 70_000, 8, 53, 2.0, 40, geometry, 0, scale)


@pytest.mark.parametrize("n,nsyn,p", [(33, 30, 1), (640, 639, 1), (641, 30, 13), (641, 640, 27), (1000, 479, 20),
                                      (4000, 3647, 152), (4000, 3648, 77), (7904, 30, 152), (7905, 30, 152)])
def test_automatic_team(g4s, oracle, n, nsyn, p):
    """The team a network alone gets: one CTA, one per 52 neurons, as many as segment runs take,
    or one per SM (152)."""
    with g4s.Network(n, nsyn, seed=54) as net:
        assert net.geometry()[0] == p
    run_both(g4s, oracle, n, nsyn, 54, 2.0, 60, (0, -1), 0)


@pytest.mark.parametrize("n,steps,geometry", [(5003, 39, (0, -1)), (5003, 40, (0, -1)), (5003, 40, (16, 1)),
                                              (5003, 41, (3, 0)), (40_000, 320, (0, -1)), (42_000, 330, (0, -1))])
def test_segment_columns(g4s, oracle, n, steps, geometry):
    """Launches on both sides of the number of steps from which the ranks keep their columns of
    the segment table in shared memory, and sizes on both sides of the largest column."""
    run_both(g4s, oracle, n, 120, 55, 1.5, 2 * steps, geometry, 768)


@pytest.mark.parametrize("n,p", [(152 * 14896, 152), (152 * 14896 + 1, 0)])
def test_largest_automatic_slices(g4s, n, p):
    """The largest network that a team takes by itself, and the first that the global-atomic
    kernel does (also with a team, if one is asked for): the same results as scheme S."""
    with g4s.Network(n, 12, seed=57, drive_scale=1.5) as a, g4s.Network(n, 12, seed=57, drive_scale=1.5) as b:
        assert a.geometry()[0] == p
        a.run(12, 4)
        b.run(20, 2)
        a.set_geometry(152, 0)
        assert a.geometry()[0] == 152
        a.run(8, 4)
        assert np.array_equal(np.stack(a.raster()), np.stack(b.raster()))
        assert np.array_equal(a.currents(), b.currents())
        x, y = a.state(), b.state()
        assert all(np.array_equal(x[k].view(np.uint32), y[k].view(np.uint32)) for k in x)

"""Runs and reads that do not get the memory they ask for first: the raster buffer, the host
staging of the raster and of the neuron state.  They take what there is, with the same results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same(a, b):
    return all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(a, b))


def state(net):
    s = net.state()
    return [s[k] for k in ("v", "u", "I", "a", "b", "c", "d", "nospks")]


@pytest.fixture
def drive():
    return 1.5


@pytest.fixture
def pair(g4s, drive):
    from gpu4snn_gb300 import _lib
    nets = [g4s.Network(3001, 100, seed=71, drive_scale=drive) for _ in range(2)]
    for net in nets:
        net.run(1, 4)  # (the packed rows exist, the raster buffer holds one step)

    def fail():
        nets[0].inject_fault(_lib.FAULT_ALLOC)
    yield nets[0], nets[1], fail
    for net in nets:
        net.close()


@pytest.mark.parametrize("alg", [0, 1, 2, 3, 4])
def test_raster_buffer(pair, alg):
    """1.8 million ids refused, 0.9 million taken: two chunks of 300 steps."""
    a, b, fail = pair
    fail()
    for net in (a, b):
        net.run(600, alg)
    assert a.info().last_run_launches == 2 * b.info().last_run_launches
    assert same(a.raster(), b.raster()) and same([a.counts()], [b.counts()]) and same(state(a), state(b))


def test_raster_buffer_of_a_batch(g4s, pair):
    from gpu4snn_gb300.network import run_batch
    a, b, fail = pair
    with g4s.Network(500, 50, seed=72) as c, g4s.Network(500, 50, seed=72) as d:
        run_batch([a, c], 1)
        run_batch([b, d], 1)
        fail()
        run_batch([a, c], 600)
        run_batch([b, d], 600)
        assert same(a.raster(), b.raster()) and same(c.raster(), d.raster()) and same(state(a), state(b))


def test_raster_buffer_of_the_fp64_check(pair):
    a, b, fail = pair
    for net in (a, b):
        net.reset()
    fail()
    x, y = a.fp64_check(500), b.fp64_check(500)
    assert all(np.array_equal(x[k], y[k]) for k in x)
    assert same(a.raster(), b.raster())


@pytest.mark.parametrize("drive", [8.0])  # (more ids in a run than the first staging buffer holds)
def test_staging(pair):
    """The raster through pageable staging, then the state without pinned memory, and both again
    with it."""
    a, b, fail = pair
    for net in (a, b):
        net.run(40, 4)  # (the raster buffer holds 349 steps from here on)
    fail()
    for net in (a, b):
        net.run(340, 4)
    assert len(a.raster()[0]) > 65536
    assert same(a.raster(), b.raster())
    fail()
    assert same(state(a), state(b))
    for net in (a, b):
        net.run(340, 4)
    assert same(a.raster(), b.raster()) and same(state(a), state(b))


def test_state_without_staging(g4s):
    from gpu4snn_gb300 import _lib
    with g4s.Network(70_001, 20, seed=73) as net:
        net.run(30, 4)
        net.inject_fault(_lib.FAULT_ALLOC)
        a = state(net)
        assert same(a, state(net))


def test_segment_table_of_another_team(g4s):
    """No room for the segment table of a larger team, in a batch and then alone: the call reports
    it, and the next one plans anew instead of running the former team without a table."""
    from gpu4snn_gb300 import _lib
    from gpu4snn_gb300.network import run_batch
    with g4s.Network(3001, 100, seed=74, drive_scale=1.5) as a, g4s.Network(3001, 100, seed=74, drive_scale=1.5) as b, \
            g4s.Network(64, 8, seed=75) as c:
        a.set_geometry(2, -1)
        a.run(30, 4)
        a.set_geometry(0, -1)
        for call in (lambda: run_batch([a, c], 10), lambda: a.run(10, 4)):
            a.inject_fault(_lib.FAULT_ALLOC)
            with pytest.raises(g4s.G4SError) as e:
                call()
            assert e.value.code == _lib.ERR_NOMEM
            call()
        b.run(50, 4)
        assert same(a.raster(), b.raster()) and same(state(a), state(b))

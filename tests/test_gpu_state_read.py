"""Read-back of the neuron state in blocks: sizes at the edges of a block and of the threaded
copy, and every subset of the fields in turn, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("v", "u", "I", "a", "b", "c", "d", "nospks")


@pytest.mark.parametrize("n", [2, 65_536, 65_537, 131_072, 131_073, 200_003])
def test_state_fields(g4s, oracle, n):
    from gpu4snn_gb300 import _lib
    nsyn, seed = 1, 61
    d = oracle.make_desc(n, nsyn, seed, drive_scale=2.0)
    idx, w = oracle.conn_philox(d)
    sim = oracle.Sim(d, idx, w)
    sim.run(30, threads=8)
    want = sim.state()
    with g4s.Network(n, nsyn, seed=seed, drive_scale=2.0, record_raster=False) as net:
        net.run(30, 4)
        assert net.counts().sum() == want["nospks"].sum() and (n < 1000 or want["nospks"].sum() > n)
        for chosen in (FIELDS, ("u",), ("nospks",), ("v", "nospks"), ("I", "a", "d"), ("b", "c")):
            out = {k: np.full(n, -7, dtype=np.int32 if k == "nospks" else np.float32) for k in chosen}
            _lib.check(g4s.load().g4s_net_state(net._h, *(_lib.ptr(out.get(k)) for k in FIELDS)))
            for k in chosen:
                assert np.array_equal(out[k].view(np.uint32), want[k].view(np.uint32)), (chosen, k)
        _lib.check(g4s.load().g4s_net_state(net._h, *([None] * 8)))

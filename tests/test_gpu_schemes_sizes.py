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

"""The FP64 check in many chunks and at small sizes: the percentiles selected on the device, the
twin's state and the network itself equal the CPU's, whatever the chunk."""
import numpy as np
import pytest

from test_gpu_fp64_check import _cpu_lockstep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nsyn,drive,steps,chunk", [(2, 1, 3.0, 40, 0), (3, 2, 2.0, 33, 5), (999, 50, 1.5, 61, 7),
                                                      (1000, 999, 2.0, 40, 1), (40_001, 20, 2.0, 30, 11)])
def test_fp64_check_in_chunks(g4s, oracle, n, nsyn, drive, steps, chunk):
    seed = 91
    mx, p99, p50, first, v64, u64 = _cpu_lockstep(oracle, n, nsyn, seed, drive, steps)
    with g4s.Network(n, nsyn, seed=seed, drive_scale=drive, raster_budget_bytes=4 * n * chunk) as net, \
            g4s.Network(n, nsyn, seed=seed, drive_scale=drive) as ref:
        r = net.fp64_check(steps)
        assert np.array_equal(r["max"], mx) and np.array_equal(r["p99"], p99) and np.array_equal(r["median"], p50)
        assert np.array_equal(r["v64"], v64) and np.array_equal(r["u64"], u64) and r["first_divergent"] == first
        ref.run(steps, 4)
        assert np.array_equal(np.stack(net.raster()), np.stack(ref.raster()))
        a, b = net.state(), ref.state()
        for k in ("v", "u", "I"):
            assert np.array_equal(a[k].view(np.uint32), b[k].view(np.uint32)), k
        assert np.array_equal(a["nospks"], b["nospks"]) and np.array_equal(net.currents(), ref.currents())
        net.run(20, 4)
        ref.run(20, 4)
        assert np.array_equal(np.stack(net.raster()), np.stack(ref.raster()))

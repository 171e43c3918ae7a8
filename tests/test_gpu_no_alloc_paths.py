"""g4s_run_noalloc against g4s_net_run where its set-up and its kernels branch: slices on both
sides of 2048 neurons (768 and 1024 threads), rows of one to three rounds of the segment search
with empty and fully padded ones, networks of different sizes and teams that take turns on the
shared scratch, and tags that wrap."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from test_zz_no_alloc import DevNet

pytestmark = pytest.mark.gpu


class Dev:
    """A network's device arrays in the caller's hands, and the handle it was taken from."""

    def __init__(self, g4s, n, nsyn, seed, drive, tables=None):
        torch = pytest.importorskip("torch")
        self.net = g4s.Network(n, nsyn, seed=seed, drive_scale=drive, tables=tables)
        self.n, self.t, dev = n, 0, "cuda:0"
        st = self.net.state()
        idx, w = self.net.tables()
        self.vu = torch.tensor(np.stack([st["v"], st["u"]], 1), device=dev)
        self.abcd = torch.tensor(np.stack([st["a"], st["b"], st["c"], st["d"]], 1), device=dev)
        self.acc = torch.zeros(n, dtype=torch.int64, device=dev)
        self.ilast = torch.zeros(n, dtype=torch.float32, device=dev)
        self.sstat = torch.zeros((n, 8), dtype=torch.int32, device=dev)
        self.sstat[:, 1] = -1
        self.idx, self.w = torch.tensor(idx, device=dev), torch.tensor(w, device=dev)
        self.raster = torch.zeros(n * 40, dtype=torch.int32, device=dev)
        self.counts = torch.zeros(40, dtype=torch.int32, device=dev)
        self.base = torch.zeros(40, dtype=torch.int64, device=dev)
        self.status = torch.ones(1, dtype=torch.int32, device=dev)
        self.ids = []
        f = np.float32
        self.d = DevNet(n=n, nexc=n * 800 // 1000, nsyn=nsyn, stride=idx.shape[1], seed=seed,
                        ge=float(f(5.0) * f(drive)), gi=float(f(2.0) * f(drive)), vu=self.vu.data_ptr(),
                        abcd=self.abcd.data_ptr(), acc=self.acc.data_ptr(), i_last=self.ilast.data_ptr(),
                        spike_stat=self.sstat.data_ptr(), idx=self.idx.data_ptr(), w=self.w.data_ptr())
        torch.cuda.synchronize()

    def step(self, lib, team, steps):
        import torch
        rc = lib.g4s_run_noalloc(C.byref(self.d), C.c_int64(self.t), steps, team, 1, C.c_void_p(self.counts.data_ptr()),
                                 C.c_void_p(self.base.data_ptr()), C.c_void_p(self.raster.data_ptr()),
                                 C.c_int64(self.raster.numel()), C.c_void_p(self.status.data_ptr()), None)
        assert rc == 0
        torch.cuda.synchronize()
        assert int(self.status.item()) == 0
        c, r = self.counts.cpu().numpy()[:steps], self.raster.cpu().numpy()
        for b, k in zip(self.base.cpu().numpy(), c):
            self.ids.append(np.sort(r[b:b + k]))
        self.t += steps

    def check(self):
        self.net.run(self.t, 4)
        assert np.array_equal(np.concatenate(self.ids), self.net.raster()[1])
        s, got = self.net.state(), self.vu.cpu().numpy()
        assert np.array_equal(got[:, 0].view(np.uint32), s["v"].view(np.uint32))
        assert np.array_equal(got[:, 1].view(np.uint32), s["u"].view(np.uint32))
        assert np.array_equal(self.ilast.cpu().numpy().view(np.uint32), s["I"].view(np.uint32))
        assert np.array_equal(self.sstat.cpu().numpy()[:, 0], s["nospks"])
        assert np.array_equal(self.acc.cpu().numpy(), self.net.currents())
        self.net.close()


@pytest.mark.parametrize("n,nsyn,team", [(2500, 1000, t) for t in (1, 2, 3, 8)] + [
    (4096, 60, 2), (4097, 60, 2), (2048, 60, 1), (2049, 60, 1), (16384, 60, 8), (16385, 60, 8)])
def test_slices(g4s, n, nsyn, team):
    d = Dev(g4s, n, nsyn, 91, 2.0)
    for steps in (1, 1, 38, 20):
        d.step(g4s.load(), team, steps)
    d.check()


@pytest.mark.parametrize("stride", [4, 28, 32, 36, 1020, 1024, 1028, 8196, 16384])
@pytest.mark.parametrize("team", [2, 8])
def test_rows(g4s, team, stride):
    """Rows with targets at both ends of the ranks' slices: full, empty, one slot, and all of
    them in one rank's slice."""
    n = max(2501, stride + 1) if stride < 2000 else stride + 117
    rng = np.random.default_rng(stride)
    idx = np.full((n, stride), -1, dtype=np.int32)
    w = np.zeros((n, stride), dtype=np.float32)
    rc = -(-n // team)
    for i in range(n):
        k = (0, 1, stride, int(rng.integers(0, stride + 1)))[i % 4]
        edge = np.concatenate([np.arange(r * rc - 1, r * rc + 1) for r in range(team + 1)])
        pick = rng.choice(n, size=k, replace=False) if i % 8 < 4 else np.arange(min(k, rc)) + (i % team) * rc
        pick = np.unique(np.concatenate([pick, edge])) if i % 3 == 0 else pick
        pick = pick[(pick >= 0) & (pick < n)][:stride]
        idx[i, :len(pick)] = rng.permutation(pick)
        w[i, :len(pick)] = rng.normal(0, 3.0 / max(1.0, np.sqrt(stride / 30)), len(pick))
    d = Dev(g4s, n, stride, 92, 2.0, (idx, w))
    d.step(g4s.load(), team, 1)
    d.step(g4s.load(), team, 39)
    assert sum(len(x) for x in d.ids) > n // 4
    d.check()


def test_networks_in_turn(g4s):
    """Three networks of different sizes and teams, a few steps each in turn on the one scratch."""
    nets = [(Dev(g4s, 2500, 300, 93, 2.0), 8), (Dev(g4s, 9001, 100, 94, 1.5), 3), (Dev(g4s, 30_000, 40, 95, 2.0), 5)]
    for k in range(30):
        for d, team in nets:
            d.step(g4s.load(), team, 1 + (k + team) % 3)
    for d, _ in nets:
        d.check()


def test_tags_that_wrap(g4s, tmp_path):
    """After the last tags come the first ones again, whose words earlier calls left behind."""
    from gpu4snn_gb300 import build
    here = os.path.dirname(os.path.abspath(__file__))
    objs = [os.path.join(build.BUILD, os.path.basename(s)[:-3] + ".o") for s in build.sources()
            if not s.endswith("g4s_noalloc.cu")]
    path = str(tmp_path / "noalloc_tags.so")
    r = subprocess.run([build.nvcc()] + build.NVCC_FLAGS + ["-shared", os.path.join(here, "native", "noalloc_tags.cu")] +
                       objs + ["-o", path, "-cudart", "static"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(path)
    big, small = Dev(g4s, 20_000, 40, 96, 2.0), Dev(g4s, 2500, 300, 97, 2.0)
    for d, team in ((big, 5), (small, 8), (big, 5)):  # (bursts of more ids than a record holds)
        d.step(lib, team, 20)
    for left in (3, 2, 25):  # (steps + 2 tags from the end: the calls of 1, 20 and 5 steps wrap at different ones)
        assert lib.set_next_tag(C.c_uint(0xFFFFFFFF - left)) == 0
        for d, team, steps in ((small, 8, 1), (big, 5, 20), (small, 8, 5)):
            d.step(lib, team, steps)
    big.check()
    small.check()

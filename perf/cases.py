"""The work that users of this framework have it do, as cases to be measured.

A case names one use through a public entry point and its sizes:

  run      one simulation on a network that stays resident: reset, `steps` steps, then the
           raster or the spike counts and the final state
  sweep    the driver's experiment: the same network under each of the five schemes
  request  one simulation from nothing: create the network (tables generated on the GPU),
           step it, read the results back, destroy it
  upload   host tables from page-locked memory into a network, reset, steps, raster back
  batch    an ensemble of independent networks advanced together by run_batch
  tick     the allocation-free entry point on caller-owned device arrays, a few steps a call
  fp64     the on-device FP64 check of the first steps of a network

Sizes are those of bench.py, the driver's defaults and the tests; seeds come from the caller.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

import gpu4snn_gb300 as g
from gpu4snn_gb300 import _lib

SWEEP = {"AP": g.ALG_AP, "N": g.ALG_N, "S": g.ALG_S, "AB": g.ALG_AB, "SKL": g.ALG_SKL}  # the driver's schemes


def listed():
    return [
        # a real-time loop: one 1 ms step of the driver's default network per call, on the
        # caller's own arrays; latency and launches are all of it
        {"name": "tick_n2500", "kind": "tick", "n": 2500, "nsyn": 1000, "drive": 1.0, "steps": 1, "team": 8},
        # the driver's default network (N=2500, Nsyn=1000) with its raster, 2 s of model time
        {"name": "run_n2500", "kind": "run", "n": 2500, "nsyn": 1000, "drive": 1.0, "steps": 2000, "raster": True},
        # an odd middle size in the irregular regime: rows that are no multiple of 4, slices
        # that do not divide N
        {"name": "run_n33333", "kind": "run", "n": 33333, "nsyn": 777, "drive": 1.5, "steps": 1000, "raster": True},
        # bench.py's headline network, raster recorded
        {"name": "run_n100k", "kind": "run", "n": 100000, "nsyn": 1000, "drive": 1.0, "steps": 2000, "raster": True},
        # the largest neuron count: 10^9 synapses of short segments, counts and state read
        {"name": "run_n1m", "kind": "run", "n": 1000000, "nsyn": 1000, "drive": 1.0, "steps": 1000, "raster": False},
        # the same network in the quiet regime: the neuron update is most of the step
        {"name": "run_n1m_quiet", "kind": "run", "n": 1000000, "nsyn": 1000, "drive": 0.5, "steps": 1000,
         "raster": False},
        # the largest table: 2.5 x 10^9 synapses of long segments
        {"name": "run_n250k_s10k", "kind": "run", "n": 250000, "nsyn": 10000, "drive": 1.0, "steps": 500,
         "raster": False},
        # the driver's experiment on its default network: every scheme in turn
        {"name": "sweep_n2500", "kind": "sweep", "n": 2500, "nsyn": 1000, "drive": 1.0, "steps": 500},
        # one simulation from nothing at the middle of the served mix's sizes
        {"name": "request_n14k", "kind": "request", "n": 14000, "nsyn": 700, "drive": 1.0, "steps": 500},
        # bench.py's end-to-end leg: a caller's tables up, a run, the raster down
        {"name": "upload_n100k", "kind": "upload", "n": 100000, "nsyn": 1000, "drive": 1.0, "steps": 1000},
        # bench.py's batched ensemble, a quarter of its networks
        {"name": "batch_64", "kind": "batch", "count": 64, "nmax": 50000, "mix": 5, "steps": 1000},
        # the precision statement of a configuration: its first steps against an FP64 twin
        {"name": "fp64_n20k", "kind": "fp64", "n": 20000, "nsyn": 1000, "drive": 1.0, "steps": 25},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "sweep", "request", "request", "upload", "batch", "tick", "fp64"])
    drive = round(rng.uniform(0.5, 2.0), 2)
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 4, 64), "nmax": _log_int(rng, 5000, 50000),
                "mix": rng.randrange(1 << 30), "steps": _log_int(rng, 300, 1000)}
    top = {"run": 1000000, "sweep": 50000, "request": 200000, "upload": 100000, "tick": 50000, "fp64": 50000}[kind]
    n = _log_int(rng, 1000, top)
    nsyn = min(n - 1, _log_int(rng, 100, 10000 if kind == "run" else 2000))
    # at most the synapses of the largest listed case of the kind
    nsyn = max(50, min(nsyn, {"run": 10 ** 9, "upload": 10 ** 8, "sweep": 2 * 10 ** 7, "fp64": 2 * 10 ** 7}.get(kind, 2 * 10 ** 8) // n))
    c = {"kind": kind, "n": n, "nsyn": nsyn, "drive": drive}
    if kind == "tick":
        return {**c, "steps": rng.randint(1, 20), "team": rng.randint(max(1, -(-n // 16384)), 8)}
    if kind == "fp64":
        return {**c, "steps": rng.randint(5, 25)}
    if kind == "sweep":
        return {**c, "steps": rng.randint(50, 200)}
    most = int(2.5e11 / (n * nsyn))  # the delivery work of a pass stays under the listed ones'
    steps = max(100, min(_log_int(rng, 100, 2000), most))
    if kind == "run":
        return {**c, "steps": steps, "raster": n <= 100000}
    return {**c, "steps": min(steps, 1000)}


def _mix(case):
    """The ensemble's networks: N log-uniform, Nsyn uniform in [100, 2000], drive in [0.5, 2]."""
    rng = random.Random(case["mix"])
    out = []
    for _ in range(case["count"]):
        n = _log_int(rng, 1000, case["nmax"])
        out.append((n, min(rng.randint(100, 2000), n - 1), round(rng.uniform(0.5, 2.0), 3),
                    rng.randint(case["steps"] // 2, case["steps"])))
    return out


def _seed(seed, k=0):
    return (int(seed) * 0x9E3779B97F4A7C15 + 0x632BE59BD9B4E019 * (k + 1)) % (1 << 62) + 1


class DevNet(C.Structure):
    """g4s_dev_net of include/gpu4snn.h."""
    _fields_ = [
        ("n", C.c_int64), ("nexc", C.c_int64), ("nsyn", C.c_int32), ("stride", C.c_int32),
        ("seed", C.c_uint64), ("ge", C.c_float), ("gi", C.c_float),
        ("vu", C.c_void_p), ("abcd", C.c_void_p), ("acc", C.c_void_p), ("i_last", C.c_void_p),
        ("spike_stat", C.c_void_p), ("idx", C.c_void_p), ("w", C.c_void_p),
    ]


TICK_T0 = 20  # steps that a tick's network has behind it: its neurons have begun to fire


def _prepare_tick(case, seed):
    n, steps, dev = case["n"], case["steps"], "cuda:0"
    sd = _seed(seed)
    with g.Network(n, case["nsyn"], seed=sd, drive_scale=case["drive"], record_raster=False) as net:
        net.run(TICK_T0, g.ALG_SKL)
        st, cur = net.state(), net.currents()
        idx, w = net.tables()
    s = {"case": case, "t": TICK_T0, "lib": g.load(),
         "vu": torch.tensor(np.stack([st["v"], st["u"]], 1), device=dev),
         "abcd": torch.tensor(np.stack([st["a"], st["b"], st["c"], st["d"]], 1), device=dev),
         "acc": torch.tensor(cur, device=dev),
         "ilast": torch.zeros(n, dtype=torch.float32, device=dev),
         "sstat": torch.zeros((n, 8), dtype=torch.int32, device=dev),
         "idx": torch.tensor(idx, device=dev), "w": torch.tensor(w, device=dev),
         "counts": torch.zeros(steps, dtype=torch.int32, device=dev),
         "base": torch.zeros(steps, dtype=torch.int64, device=dev),
         "raster": torch.zeros(n * steps, dtype=torch.int32, device=dev),
         "status": torch.zeros(1, dtype=torch.int32, device=dev)}
    s["sstat"][:, 1] = -1
    s["net"] = DevNet(n=n, nexc=n * 800 // 1000, nsyn=case["nsyn"], stride=idx.shape[1], seed=sd,
                      ge=float(np.float32(5.0) * np.float32(case["drive"])),
                      gi=float(np.float32(2.0) * np.float32(case["drive"])),
                      vu=s["vu"].data_ptr(), abcd=s["abcd"].data_ptr(), acc=s["acc"].data_ptr(),
                      i_last=s["ilast"].data_ptr(), spike_stat=s["sstat"].data_ptr(), idx=s["idx"].data_ptr(),
                      w=s["w"].data_ptr())
    return s


class _Pinned:
    """Page-locked host tables, freed with the state that holds them."""

    def __init__(self, idx, w):
        self.idx, self.p = _lib.pinned_empty(idx.shape, "int32")
        self.w, self.q = _lib.pinned_empty(w.shape, "float32")
        self.idx[:], self.w[:] = idx, w

    def __del__(self):
        self.idx = self.w = None
        _lib.pinned_free(self.p)
        _lib.pinned_free(self.q)


def _raster_buffers(case):
    """The caller's raster arrays, sized from the expected rate with room to spare and a
    start-up transient; slots past the raster's end keep -1."""
    cap = int(case["n"] * (case["steps"] * _rate_hz(case["drive"]) * 1.4e-3 + 4))
    return np.full(cap, -1, dtype=np.int32), np.full(cap, -1, dtype=np.int32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "tick":
        return _prepare_tick(case, seed)
    if kind == "request":
        return {"case": case, "seed": _seed(seed), "raster": _raster_buffers(case)}
    if kind == "batch":
        mix = _mix(case)
        return {"case": case, "steps": [m[3] for m in mix],
                "nets": [g.Network(n, s, seed=_seed(seed, k), drive_scale=d, record_raster=False)
                         for k, (n, s, d, _) in enumerate(mix)]}
    raster = bool(case.get("raster", kind in ("upload", "sweep")))
    net = g.Network(case["n"], case["nsyn"], seed=_seed(seed), drive_scale=case["drive"], record_raster=raster)
    s = {"case": case, "net": net, "raster": _raster_buffers(case) if raster else None}
    if kind == "sweep":
        s["raster"] = {name: _raster_buffers(case) for name in SWEEP}
    if kind == "upload":
        s["tables"] = _Pinned(*net.tables())
    return s


def _results(net, raster=None):
    st = net.state()
    out = {"counts": net.counts(), "v": st["v"], "u": st["u"], "I": st["I"], "nospks": st["nospks"]}
    if raster is not None:  # into the caller's arrays (g4s_net_raster)
        t, i = raster
        size = C.c_int64()
        _lib.check(g.load().g4s_net_raster(net._h, _lib.ptr(t), _lib.ptr(i), t.size, C.byref(size)))
        out["t"], out["id"] = t, i
    return out


def run(state):
    case = state["case"]
    kind, steps = case["kind"], case.get("steps")
    if kind == "tick":
        s = state
        _lib.check(s["lib"].g4s_run_noalloc(C.byref(s["net"]), s["t"], steps, case["team"], 1, s["counts"].data_ptr(),
                                            s["base"].data_ptr(), s["raster"].data_ptr(), s["raster"].numel(),
                                            s["status"].data_ptr(), None))
        s["t"] += steps
        return {"vu": s["vu"], "ilast": s["ilast"], "acc": s["acc"], "sstat": s["sstat"], "counts": s["counts"],
                "base": s["base"], "status": s["status"]}
    if kind == "request":
        with g.Network(case["n"], case["nsyn"], seed=state["seed"], drive_scale=case["drive"]) as net:
            net.run(steps)
            return _results(net, state["raster"])
    if kind == "batch":
        for net in state["nets"]:
            net.reset()
        g.run_batch(state["nets"], state["steps"])
        got = [_results(net) for net in state["nets"]]
        return {k: np.concatenate([r[k] for r in got]) for k in got[0]}
    net = state["net"]
    if kind == "upload":
        net.load_tables(state["tables"].idx, state["tables"].w)
    if kind == "sweep":
        out = {}
        for name in SWEEP:
            net.reset()
            net.run(steps, SWEEP[name])
            out[name] = _results(net, state["raster"][name])
        return out
    net.reset()
    if kind == "fp64":
        return net.fp64_check(steps)
    net.run(steps)
    return _results(net, state["raster"])


def _rate_hz(drive):
    """The networks' mean firing rate by drive scale (measured: about 0.08, 7.2, 15, 19 Hz)."""
    return float(np.interp(drive, [0.5, 0.6, 1.0, 1.5, 2.0], [0.08, 0.5, 7.2, 15.0, 19.0]))


def _step_work(n, nsyn, drive, steps):
    """Rows of the spiking neurons (target and weight), 64 bytes of statistics a spike, v and
    u read and written once a call; about 100 operations per neuron and step (update, drive)
    and 2 per synaptic event."""
    spikes = n * steps * _rate_hz(drive) / 1000.0
    return spikes * (nsyn * 8 + 64) + n * 16.0, n * steps * 100.0 + spikes * nsyn * 2


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [_step_work(n, s, d, t) for n, s, d, t in _mix(case)]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
        return {"bytes": b + 16.0 * sum(m[0] for m in _mix(case)), "flops": f}
    n, nsyn, steps = case["n"], case["nsyn"], case["steps"]
    b, f = _step_work(n, nsyn, case["drive"], steps)
    if kind == "sweep":
        b, f = 5 * b, 5 * f
    if kind == "fp64":
        b, f = 2 * b, 2 * f
    if kind != "tick":
        b += 16.0 * n * (5 if kind == "sweep" else 1)  # the state that is read back
    if kind == "request":
        b += n * nsyn * 8.0  # the tables, written once
        f += n * nsyn * 60.0  # and their random numbers
    if kind == "upload":
        b += n * nsyn * 8.0 * 2  # read from the host, written on the device
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------------------
# The same results in 64 bits, by numpy alone: the same draws (Philox), everything after them
# in double.  A network's spike times separate from the FP32 ones after some tens of steps,
# so values exist for the short cases only.
# ---------------------------------------------------------------------------------------
def _raw(seed, stream, c1, rows):
    """The four words of Philox4x64-10 at counters (row, c1, 0, 0), key (seed, stream)."""
    ctr = np.array([0, c1, 0, 0], dtype=np.uint64)
    bg = np.random.Philox(counter=ctr, key=np.array([seed, stream], dtype=np.uint64))
    # (the generator steps its counter before each block: its first block is row 1)
    body = bg.random_raw(4 * (rows - 1)).reshape(rows - 1, 4) if rows > 1 else np.zeros((0, 4), np.uint64)
    m = (1 << 256) - 1
    prev = ((c1 << 64) - 1) & m  # the counter before (0, c1, 0, 0)
    ctr0 = np.array([(prev >> (64 * k)) & ((1 << 64) - 1) for k in range(4)], dtype=np.uint64)
    head = np.random.Philox(counter=ctr0, key=np.array([seed, stream], dtype=np.uint64)).random_raw(4)
    return np.concatenate([head.reshape(1, 4), body])


def _mulhi(a, b):
    """High 64 bits of a * b for b < 2^32."""
    lo = (a & np.uint64(0xFFFFFFFF)) * np.uint64(b)
    return ((a >> np.uint64(32)) * np.uint64(b) + (lo >> np.uint64(32))) >> np.uint64(32)


def _tables64(n, nsyn, seed):
    """Distinct targets per row in draw order, and the weights in double."""
    rows = np.arange(n)[:, None]
    blocks = -(-int(nsyn * 1.02 + 64) // 128)
    while True:
        draws = np.empty((n, blocks, 4, 32), dtype=np.int64)
        for b in range(blocks):
            for lane in range(32):
                draws[:, b, :, lane] = _mulhi(_raw(seed, 1, 32 * b + lane, n), n - 1).astype(np.int64)
        draws = draws.reshape(n, -1)
        draws += draws >= rows  # no self-loops
        order = np.argsort(draws, axis=1, kind="stable")
        s = np.take_along_axis(draws, order, 1)
        fresh = np.ones(s.shape, dtype=bool)
        fresh[:, 1:] = s[:, 1:] != s[:, :-1]
        first = np.zeros(s.shape, dtype=bool)
        np.put_along_axis(first, order, fresh, 1)
        rank = np.cumsum(first, axis=1)
        if rank[:, -1].min() >= nsyn:
            break
        blocks = blocks + max(1, blocks // 4)
    keep = first & (rank <= nsyn)
    idx = draws[keep].reshape(n, nsyn)
    w = np.empty((n, -(-nsyn // 4) * 4))
    for q in range(w.shape[1] // 4):
        w[:, 4 * q:4 * q + 4] = (_raw(seed, 2, q, n) >> np.uint64(40)).astype(np.float64) * 2.0 ** -24
    nexc = n * 800 // 1000
    w[:nexc] *= 500.0 / nsyn
    w[nexc:] *= -1000.0 / nsyn
    return idx, w[:, :nsyn]


def _philox32(k0, k1, c):
    m32 = np.uint64(0xFFFFFFFF)
    c0, c1, c2, c3 = (np.asarray(x, dtype=np.uint64) for x in c)
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
        p0, p1 = np.uint64(0xD2511F53) * c0, np.uint64(0xCD9E8D57) * c2
        c0, c1, c2, c3 = ((p1 >> np.uint64(32)) ^ c1 ^ np.uint64(k0), p1 & m32,
                          (p0 >> np.uint64(32)) ^ c3 ^ np.uint64(k1), p0 & m32)
    return c0, c1, c2, c3


def _normals64(seed, n, t):
    z, todo = np.zeros(n), np.arange(n)
    for attempt in range(16):
        o = _philox32(seed & 0xFFFFFFFF, seed >> 32, (todo, np.full(todo.size, t), np.full(todo.size, attempt),
                                                       np.full(todo.size, 4)))
        u = [((x >> np.uint64(8)).astype(np.float64) * 2 + 1 - 2.0 ** 24) * 2.0 ** -24 for x in o]
        s0, s1 = u[0] ** 2 + u[1] ** 2, u[2] ** 2 + u[3] ** 2
        x, s = np.where(s0 < 1, u[0], u[2]), np.where(s0 < 1, s0, s1)
        ok = s < 1
        z[todo[ok]] = x[ok] * np.sqrt(-2 * np.log(s[ok]) / s[ok])
        todo = todo[~ok]
        if not todo.size:
            break
    return z


def _simulate64(n, nsyn, seed, drive, steps):
    idx, w = _tables64(n, nsyn, seed)
    exc = np.arange(n) < n * 800 // 1000
    r = (_raw(seed, 3, 0, n)[:, 0] >> np.uint64(40)).astype(np.float64) * 2.0 ** -24
    a = np.where(exc, 0.02, 0.02 + 0.08 * r)
    b = np.where(exc, 0.2, 0.25 - 0.05 * r)
    c = np.where(exc, -65 + 15 * r * r, -65.0)
    d = np.where(exc, 8 - 6 * r * r, 2.0)
    v = np.full(n, -65.0)
    u = b * v
    syn, gain = np.zeros(n), np.where(exc, 5.0, 2.0) * drive
    cur = np.zeros(n)
    for t in range(steps):
        cur = gain * _normals64(seed, n, t) + syn
        for _ in range(2):
            v = v + 0.5 * (0.04 * v * v + 5 * v + 140 - u + cur)
        u = u + a * (b * v - u)
        spk = np.flatnonzero(v >= 30)
        v[spk], u[spk] = c[spk], u[spk] + d[spk]
        syn = np.bincount(idx[spk].ravel(), weights=w[spk].ravel(), minlength=n).astype(np.float64)
    return v, u, cur


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("tick", "fp64") or case["n"] * case["nsyn"] > 2.2e7:
        return None
    if kind == "tick":
        v, u, cur = _simulate64(case["n"], case["nsyn"], _seed(seed), case["drive"], TICK_T0 + case["steps"])
        return {"vu": np.stack([v, u], 1), "ilast": cur, "acc": None, "sstat": None, "counts": None, "base": None,
                "status": None}
    v, u, _ = _simulate64(case["n"], case["nsyn"], _seed(seed), case["drive"], case["steps"])
    return {"max": None, "p99": None, "median": None, "first_divergent": None, "v64": v, "u64": u}

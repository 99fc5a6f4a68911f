"""Performance cases: the calls that a program built on this framework makes.

Each case is one call sequence through the public Python binding (the C ABI
underneath): a closed control loop, whole series through a reservoir, readout
training, a batched sweep, a round of the search's surrogate. Sizes come from
the benchmark's workloads and the tests, or lie between them.

`exact` restates every case in 64 bits with numpy and torch alone: the graphs
are redrawn from the C library's rand(), the dynamics stepped with dense or
sparse products, the readouts solved by LAPACK-style solves.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import spires_b200 as sp
from spires_b200 import sweep

TOPO = {"random": sp.CONN_RANDOM, "small_world": sp.CONN_SMALL_WORLD,
        "scale_free": sp.CONN_SCALE_FREE}
NEURON = {"lif": sp.LIF_DISCRETE, "gl": sp.FLIF_GL, "caputo": sp.FLIF_CAPUTO}
SYNAPSE = {"simple": sp.SYN_SIMPLE, "frac": sp.SYN_FRAC}
FRAC = (0.6, 4.0)  # fractional synapse: alpha, tau
L2_BYTES = 126e6   # a history larger than this is read from memory every step


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # A control loop around a small reservoir: one step, one output. The
        # smallest call there is; launches and latency are all of it.
        dict(name="closed_loop_lif_1000", kind="loop", neuron="lif", n=1000, din=3, dout=2,
             topo="random", conn=0.1, steps=1),
        # The small LIF workload: a whole series through 1000 dense-ish LIF
        # neurons from reset, rasters and readouts returned.
        dict(name="run_lif_1000", kind="run", neuron="lif", synapse="simple", n=1000, din=1,
             dout=1, topo="random", conn=0.1, steps=2000, hist=0, syn_hist=0),
        # The headline stream: 20000 fractional neurons with 1024 lags in
        # steady state, 256 steps of 13 channels through spires_run, then a
        # look at the state.
        dict(name="stream_gl_20000", kind="stream", neuron="gl", synapse="simple", n=20000,
             din=13, dout=10, topo="scale_free", conn=5.0 / 19999.0, steps=256, hist=1024,
             syn_hist=0),
        # Sequence classification: one utterance of 60 frames from reset, all
        # states back (they are averaged over time by the caller).
        dict(name="sequence_gl_20000", kind="run", neuron="gl", synapse="simple", n=20000, din=13,
             dout=10, topo="scale_free", conn=5.0 / 19999.0, steps=60, hist=1024, syn_hist=0,
             states=True),
        # The same graph with fractional synapses: a second history per neuron.
        dict(name="stream_gl_frac_20000", kind="stream", neuron="gl", synapse="frac", n=20000,
             din=13, dout=10, topo="scale_free", conn=5.0 / 19999.0, steps=64, hist=1024,
             syn_hist=512),
        # Caputo neurons: each keeps a history of its own that only advances
        # when the neuron integrates.
        dict(name="stream_caputo_20000", kind="stream", neuron="caputo", synapse="simple",
             n=20000, din=13, dout=10, topo="scale_free", conn=5.0 / 19999.0, steps=64, hist=512,
             syn_hist=0),
        # Training a readout on a reservoir: reset, the whole series, ridge.
        dict(name="train_ridge_gl_2000", kind="train_ridge", neuron="gl", n=2000, din=13, dout=3,
             topo="small_world", conn=10.0 / 1999.0, steps=5000, hist=256, lam=10.0),
        # Ridge on states that the caller holds, FP64 Gram ...
        dict(name="ridge_fit_2000", kind="ridge_fit", n=2000, rows=6000, dout=4, gram=0,
             washout=200, lam=10.0),
        # ... and at the size of the ridge workload with the INT8 tensor-core Gram.
        dict(name="ridge_fit_int8_4000", kind="ridge_fit", n=4000, rows=9000, dout=1, gram=3,
             washout=500, lam=10.0),
        # Recursive least squares over a series.
        dict(name="train_rls_800", kind="rls", neuron="gl", n=800, din=2, dout=2,
             topo="scale_free", conn=0.02, steps=400, hist=64, lam=0.999),
        # A hyper-parameter sweep: uneven reservoirs in one batch, every readout
        # fitted and scored from one simulation.
        dict(name="sweep_20", kind="sweep", count=20, n_lo=300, n_hi=1600, t_lo=500, t_hi=1500,
             conn_lo=0.02, conn_hi=0.2, space=2024),
        # One round of the search's surrogate: train on the tuples so far, then
        # score the next candidates.
        dict(name="surrogate_round", kind="surrogate", rows=1500, epochs=30, batch=256,
             candidates=4096, bf16=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loop", "run", "stream", "stream", "train_ridge", "ridge_fit", "rls",
                       "sweep", "surrogate"])
    if kind == "loop":
        return dict(kind=kind, neuron=rng.choice(["lif", "gl"]), n=_log_int(rng, 100, 4000),
                    din=rng.randint(1, 13), dout=rng.randint(1, 10), topo=rng.choice(list(TOPO)),
                    conn=rng.uniform(0.01, 0.1), steps=rng.randint(1, 8))
    if kind in ("run", "stream"):
        neuron = rng.choice(["lif", "gl", "caputo"])
        synapse = "frac" if neuron == "gl" and rng.random() < 0.3 else "simple"
        n = _log_int(rng, 100, 20000)
        mean = rng.uniform(4.0, 100.0 if n < 4000 else 10.0)  # connections per neuron
        hist = 0 if neuron == "lif" else _log_int(rng, 32, 1024)
        c = dict(kind=kind, neuron=neuron, synapse=synapse, n=n, din=rng.randint(1, 13),
                 dout=rng.randint(1, 10),
                 topo=rng.choice(["random", "small_world", "scale_free"] if n <= 3000
                                 else ["small_world", "scale_free"]),
                 conn=min(0.5, mean / n), steps=_log_int(rng, 20, 256 if n > 4000 else 1000),
                 hist=hist, syn_hist=_log_int(rng, 16, 512) if synapse == "frac" else 0)
        if kind == "run":
            c["states"] = rng.random() < 0.5
        return c
    if kind == "train_ridge":
        n = _log_int(rng, 100, 2000)
        return dict(kind=kind, neuron=rng.choice(["lif", "gl"]), n=n, din=rng.randint(4, 13),
                    dout=rng.randint(1, 5), topo=rng.choice(["small_world", "scale_free"]),
                    conn=rng.uniform(4.0, 20.0) / n, steps=rng.randint(2 * n + 200, 5000),
                    hist=_log_int(rng, 32, 256), lam=rng.uniform(10.0, 100.0))
    if kind == "ridge_fit":
        n = _log_int(rng, 100, 4000)
        rows = rng.randint(2 * n + 300, 9000) if rng.random() < 0.75 else rng.randint(60, max(61, n // 2))
        return dict(kind=kind, n=n, rows=rows, dout=rng.randint(1, 10), gram=rng.choice([0, 3]),
                    washout=rng.randint(0, 20), lam=rng.uniform(10.0, 100.0))
    if kind == "rls":
        return dict(kind=kind, neuron=rng.choice(["lif", "gl"]), n=_log_int(rng, 50, 1200),
                    din=rng.randint(1, 4), dout=rng.randint(1, 4),
                    topo=rng.choice(["small_world", "scale_free"]), conn=rng.uniform(0.01, 0.05),
                    steps=rng.randint(50, 400), hist=_log_int(rng, 16, 128),
                    lam=rng.choice([1.0, 0.999]))
    if kind == "sweep":
        n_lo = rng.randint(100, 500)
        return dict(kind=kind, count=rng.randint(2, 16), n_lo=n_lo, n_hi=rng.randint(n_lo + 100, 1600),
                    t_lo=rng.randint(200, 500), t_hi=rng.randint(600, 1400), conn_lo=0.02,
                    conn_hi=rng.uniform(0.03, 0.2), space=rng.randint(0, 10**6))
    return dict(kind="surrogate", rows=_log_int(rng, 40, 1500), epochs=rng.randint(1, 30),
                batch=rng.choice([64, 128, 256]), candidates=_log_int(rng, 50, 4096),
                bf16=rng.random() < 0.7)


# ------------------------------------------------------------------- inputs

def _neuron_params(neuron, hist):
    if neuron == "lif":  # V_0, V_th, leak rate, bias
        return (0.0, 1.0, 0.3, 0.05)
    if neuron == "gl":   # V_th, V_reset, V_rest, tau_m, alpha, T_mem, bias, t_ref
        return (1.0, 0.0, 0.0, 20.0, 0.6, float(hist), 0.1, 2.0)
    return (1.0, 0.2, 0.0, 1.0, 0.0, 1.5, 0.7, 2.0, float(hist))


def _config(case):
    syn = SYNAPSE[case.get("synapse", "simple")]
    return sp.make_config(
        case["n"], case["din"], case["dout"], rho=0.9, ei=0.5, gamma=0.5, conn=case["conn"],
        topo=TOPO[case["topo"]], neuron=NEURON[case["neuron"]],
        nparams=_neuron_params(case["neuron"], case.get("hist", 64)), synapse=syn,
        sparams=FRAC + (float(case["syn_hist"]),) if syn == sp.SYN_FRAC else None)


def _fill(case):
    """Steps after which a stream's histories are full."""
    return max(case["hist"], case["syn_hist"]) + 8


def _signal(rng, T, channels):
    """Gated sums of three sinusoids per channel (bursty sensor-like input)."""
    t = np.arange(T)[:, None, None]
    f = rng.uniform(0.01, 0.2, (channels, 3))
    x = (rng.uniform(0, 1, (channels, 3)) *
         np.sin(2 * np.pi * f * t + rng.uniform(0, 2 * np.pi, (channels, 3)))).sum(axis=2)
    gate = (np.cumsum(rng.random((T, channels)) < 0.05, axis=0) % 3) != 0
    return np.ascontiguousarray(x * gate + 0.05 * rng.standard_normal((T, channels)))


def _targets(rng, u, dout):
    """Delayed mixtures of the input channels, with a little noise."""
    mix = rng.standard_normal((u.shape[1], dout)) / math.sqrt(u.shape[1])
    d = np.roll(u, 2, axis=0) @ mix
    return np.ascontiguousarray(np.tanh(d) + 0.05 * rng.standard_normal(d.shape))


def _states(rng, T, n):
    """States as a reservoir gives them: strongly correlated over neurons,
    smooth over time, with some activity of each neuron's own."""
    k = 48
    z = _signal(rng, T, k) * (0.9 ** np.arange(k))
    x = z @ rng.standard_normal((k, n)) / 3.0
    x += 0.2 * rng.standard_normal((T, n))
    return np.ascontiguousarray(x + 0.1)


def _inputs(case, seed):
    """The arrays of one case; `exact` makes the same ones again."""
    rng = np.random.default_rng([seed, 77])
    k = case["kind"]
    if k == "loop":
        return dict(u=_signal(rng, 4096, case["din"]))
    if k == "run":
        return dict(u=_signal(rng, case["steps"], case["din"]))
    if k == "stream":
        return dict(u=_signal(rng, _fill(case) + case["steps"], case["din"]))
    if k in ("train_ridge", "rls"):
        u = _signal(rng, case["steps"], case["din"])
        return dict(u=u, y=_targets(rng, u, case["dout"]))
    if k == "ridge_fit":
        x = _states(rng, case["rows"], case["n"])
        y = x[:, :32] @ rng.standard_normal((min(32, case["n"]), case["dout"])) / 8.0
        return dict(x=x, y=np.ascontiguousarray(np.tanh(y) + 0.1 * rng.standard_normal(y.shape)))
    if k == "sweep":
        insts = sweep.sweep_space(case["count"], seed=case["space"],
                                  n_range=(case["n_lo"], case["n_hi"]),
                                  t_range=(case["t_lo"], case["t_hi"]), rings=(128, 256, 512),
                                  conn_range=(case["conn_lo"], case["conn_hi"]))
        us = [0.5 + 0.5 * _signal(rng, i.T, 1) for i in insts]
        ys = [np.ascontiguousarray(_targets(rng, u, 1)) for u in us]
        seeds = [int(s) for s in rng.integers(1, 2**31 - 1, len(insts))]
        return dict(insts=insts, us=us, ys=ys, seeds=seeds,
                    heads=[int(0.8 * i.T) for i in insts])
    x = rng.standard_normal((case["rows"], 10)).astype(np.float32)
    y = np.tanh(x[:, 0]) + 0.3 * x[:, 1] * x[:, 2] + 0.1 * rng.standard_normal(case["rows"])
    p = np.concatenate([rng.uniform(-1, 1, m) / math.sqrt(f) for m, f in
                        ((1280, 10), (128, 10), (128 * 128, 128), (128, 128), (256, 128),
                         (2, 128))]).astype(np.float32)
    return dict(x=x, y=y.astype(np.float32), p=p,
                c=rng.standard_normal((case["candidates"], 10)).astype(np.float32))


# ------------------------------------------------------------ prepare and run

def prepare(case, seed):
    s = dict(case=case, **_inputs(case, seed))
    k = case["kind"]
    if k in ("loop", "run", "stream", "train_ridge", "rls"):
        s["r"] = sp.Reservoir(_config(case), seed=seed % (2**31))
    if k == "loop":
        s["pos"] = 0
    if k == "stream":  # a stream that has been running: its histories are full
        f = _fill(case)
        s["r"].run_record(s["u"][:f], phi=False, raster=False)
        s["u"] = np.ascontiguousarray(s["u"][f:])
    if k == "sweep":
        s["b"] = sp.Batch([i.cfg for i in s["insts"]], s["seeds"])
    if k == "surrogate":
        s["net"] = sp.Surrogate(seed=seed)
    return s


def run(s):
    c, k = s["case"], s["case"]["kind"]
    if k == "loop":
        out = []
        for _ in range(c["steps"]):
            s["r"].step(s["u"][s["pos"] % 4096])
            out.append(s["r"].output())
            s["pos"] += 1
        return np.stack(out)
    if k == "run":
        s["r"].reset()
        phi, raster, y = s["r"].run_record(s["u"], phi=bool(c.get("states")), raster=True, y=True)
        return [x for x in (phi, raster.view(np.int32), y) if x is not None]
    if k == "stream":
        return [s["r"].run(s["u"]), s["r"].state()]
    if k == "train_ridge":
        s["r"].train_ridge(s["u"], s["y"], c["lam"])
        return s["r"].readout()
    if k == "ridge_fit":
        return sp.ridge_fit(s["x"], s["y"], c["lam"], washout=c["washout"], gram_mode=c["gram"])[0]
    if k == "rls":
        s["r"].train_rls(s["u"], s["y"], 1.0, c["lam"])
        return s["r"].readout()
    if k == "sweep":
        y, _ = s["b"].fit_predict(s["us"], s["ys"], s["heads"], 10.0, washout=50)
        return y
    s["net"].set_params(s["p"])
    loss = s["net"].train(s["x"], s["y"], epochs=c["epochs"], batch=c["batch"], lr=1e-3, seed=3)
    m, v = s["net"].predict(s["c"], bf16=c["bf16"])
    return dict(params=s["net"].params(), loss=loss, mean=m, logvar=v)


# --------------------------------------------------------------------- work

def _sim_work(n, T, din, hist, syn_hist, nnz, full, out_bytes):
    lags = hist if full else min(hist, T) / 2.0 if T <= hist else hist - hist * hist / (2.0 * T)
    ring = 8.0 * n * hist
    b = 8.0 * T * din + 8.0 * n * din + 12.0 * nnz + 16.0 * n + out_bytes
    # a history beyond the L2 has to be read again for every step
    b += T * 8.0 * n * lags if ring > L2_BYTES else ring
    b += T * 8.0 * n * syn_hist if 8.0 * n * syn_hist > L2_BYTES else 8.0 * n * syn_hist
    f = T * n * (2.0 * lags + 2.0 * syn_hist + 2.0 * din + 8.0) + 0.2 * T * nnz
    return b, f


def _ridge_work(n, rows, dout):
    if 2 * rows <= n:
        g, m = float(rows) * rows * n, float(rows)
    else:
        g, m = float(rows) * n * n, float(n)
    return (8.0 * rows * (n + dout) + 8.0 * n * dout,
            g + m ** 3 / 3.0 + 4.0 * rows * n * dout + 2.0 * m * m * dout)


def work(case):
    k = case["kind"]
    n, T = case.get("n", 0), case.get("steps", 0)
    if k in ("loop", "run", "stream", "train_ridge", "rls"):
        nnz = n * n * case["conn"]
        hist = case.get("hist", 64) if case["neuron"] != "lif" else 0
        out = 8.0 * T * case["dout"]
        if k == "run":
            out += T * n / 8.0 + (8.0 * T * n if case.get("states") else 0.0)
        if k == "stream":
            out += 8.0 * n
        b, f = _sim_work(n, T, case["din"], hist, case.get("syn_hist", 0), nnz, k == "stream", out)
        f += 2.0 * T * n * case["dout"]
        if k == "train_ridge":
            rb, rf = _ridge_work(n, T, case["dout"])
            b, f = b + rb - 8.0 * T * n, f + rf
        if k == "rls":
            b, f = b + 8.0 * n * n, f + 5.0 * T * n * n
        return {"bytes": b, "flops": f}
    if k == "ridge_fit":
        b, f = _ridge_work(n, case["rows"] - case["washout"], case["dout"])
        return {"bytes": b, "flops": f}
    if k == "sweep":
        b = f = 0.0
        for i in sweep.sweep_space(case["count"], seed=case["space"],
                                   n_range=(case["n_lo"], case["n_hi"]),
                                   t_range=(case["t_lo"], case["t_hi"]), rings=(128, 256, 512),
                                   conn_range=(case["conn_lo"], case["conn_hi"])):
            hist = i.L if i.neuron == sp.FLIF_GL else 0
            x, y = _sim_work(i.n, i.T, 1, hist, 0, i.n * i.n * i.conn, False, 8.0 * i.T)
            rx, ry = _ridge_work(i.n, int(0.8 * i.T) - 50, 1)
            b, f = b + x + rx - 6.4 * i.T * i.n, f + y + ry
        return {"bytes": b, "flops": f}
    mac = 1280 + 16384 + 256
    seen = case["rows"] * case["epochs"]
    return {"bytes": 4.0 * (11 * case["rows"] + 12 * case["candidates"] + 2 * 18178),
            "flops": 2.0 * mac * (3 * seen + case["candidates"])}


# -------------------------------------------------- the same values in 64 bits

_libc = ctypes.CDLL("libc.so.6")
_R = 2147483647.0  # RAND_MAX


class _Draws:
    """The C library's rand() after srand(seed), drawn ahead in blocks."""

    def __init__(self, seed):
        _libc.srand(ctypes.c_uint(seed))
        self.buf, self.pos = np.empty(0), 0

    def peek(self, k):
        """The next k draws as fractions of RAND_MAX."""
        have = len(self.buf) - self.pos
        if have < k:
            f, m = _libc.rand, max(k - have, 65536)
            more = np.fromiter((f() for _ in range(m)), np.float64, m) / _R
            self.buf, self.pos = np.concatenate([self.buf[self.pos:], more]), 0
        return self.buf[self.pos:self.pos + k]

    def take(self, k):
        x = self.peek(k)
        self.pos += k
        return x

    def one(self):
        return float(self.take(1)[0])

    def weights(self, k, ei):
        d = self.take(2 * k).reshape(k, 2)
        return np.where(d[:, 1] < ei, d[:, 0], -d[:, 0])


def _edges_random(d, n, conn, ei):
    # one draw per ordered pair, two more behind each that is an edge
    need = n * (n - 1)
    x = d.peek(int(need * (1 + 2.2 * conn)) + 4096)
    pair, q, e = 0, 0, []
    for h in np.flatnonzero(x < conn).tolist():
        if h < q:
            continue  # that draw was a weight's
        if pair + h - q >= need:
            break
        pair += h - q
        e.append((pair, h))
        pair, q = pair + 1, h + 3
    d.take(q + need - pair)
    e = np.array(e, np.int64).reshape(-1, 2)
    i, jj = e[:, 0] // (n - 1), e[:, 0] % (n - 1)
    mag, sign = x[e[:, 1] + 1], x[e[:, 1] + 2]
    return i, jj + (jj >= i), np.where(sign < ei, mag, -mag)


def _edges_small_world(d, n, conn, ei):
    K = max(2, int(conn * (n - 1) + 0.5))
    K = min(K + K % 2, n - 1)
    half = K // 2
    ring = d.weights(n * half, ei).reshape(n, half)
    I, J, V = [], [], []
    for i in range(n):
        row = {(i + s) % n: ring[i, s - 1] for s in range(1, half + 1)}
        for s in range(1, half + 1):
            if d.one() < 0.1:
                row[(i + s) % n] = 0.0
                tries = 0
                while True:
                    j = min(int(d.one() * n), n - 1)
                    tries += 1
                    if tries > 10 * n or not (j == i or row.get(j, 0.0) != 0.0):
                        break
                if j != i:
                    row[j] = d.weights(1, ei)[0]
        I += [i] * len(row)
        J += list(row)
        V += list(row.values())
    return np.array(I), np.array(J), np.array(V)


def _edges_scale_free(d, n, conn, ei):
    m = min(max(1, int(conn * (n - 1) + 0.5)), n - 1)
    m0 = min(max(m, 2), n - 1)
    # roulette over deg + 1: a Fenwick tree of integer weights
    size = 1 << max(1, (n - 1).bit_length())
    tree = [0] * (size + 1)

    def add(u, x):
        u += 1
        while u <= size:
            tree[u] += x
            u += u & -u

    def pick(target):  # the first node whose inclusive prefix sum reaches target
        pos, bit = 0, size
        while bit:
            if pos + bit <= size and tree[pos + bit] < target:
                pos += bit
                target -= tree[pos]
            bit >>= 1
        return pos

    deg = [0] * n
    above = [[] for _ in range(n)]
    for u in range(m0):
        above[u] = list(range(u + 1, m0))
        deg[u] = m0 - 1
        add(u, deg[u] + 1)
    total = m0 * (m0 - 1)
    for v in range(m0, n):
        mine, guard = set(), 0
        while len(mine) < m and guard < 50 * m:
            u = pick(math.ceil(d.one() * float(total + v)))
            u = u if u < v else 0
            guard += 1
            if u not in mine:
                mine.add(u)
                deg[u] += 1
                total += 1
                add(u, 1)
                above[u].append(v)
        while len(mine) < m:
            u = min(int(d.one() * v), v - 1)
            if u not in mine:
                mine.add(u)
                deg[u] += 1
                total += 1
                add(u, 1)
                above[u].append(v)
        deg[v] += len(mine)
        add(v, deg[v] + 1)
        total += deg[v]
    a = np.repeat(np.arange(n), [len(x) for x in above])
    b = np.array([v for x in above for v in x], np.int64)
    w = d.take(3 * len(a)).reshape(-1, 3)
    fwd = w[:, 0] < 0.5
    return np.where(fwd, a, b), np.where(fwd, b, a), np.where(w[:, 2] < ei, w[:, 1], -w[:, 1])


def _model(n, din, dout, topo, conn, rho, ei, seed):
    """W_in, recurrent matrix (sparse, on the GPU), W_out of a seeded reservoir."""
    d = _Draws(seed)
    w_in = d.weights(n * din, ei).reshape(n, din)
    f = {sp.CONN_RANDOM: _edges_random, sp.CONN_SMALL_WORLD: _edges_small_world,
         sp.CONN_SCALE_FREE: _edges_scale_free}[topo]
    i, j, v = f(d, n, conn, ei)
    w_out = d.weights(n * dout, 0.5).reshape(dout, n)
    idx = torch.tensor(np.stack([i, j]), device="cuda")
    W = torch.sparse_coo_tensor(idx, torch.tensor(v, device="cuda"), (n, n)).coalesce()
    W = W.to_sparse_csr()
    x = torch.ones(n, 1, dtype=torch.float64, device="cuda")
    old = 0.0
    for _ in range(1000):
        y = W @ x
        new = float(y.abs().max())
        if new == 0.0:
            break
        x = y / new
        if abs(new - old) < 1e-6:
            break
        old = new
    if new > 1e-9:
        W = torch.sparse_csr_tensor(W.crow_indices(), W.col_indices(), W.values() * (rho / new),
                                    (n, n))
    return (torch.tensor(w_in, device="cuda"), W, torch.tensor(w_out, device="cuda"))


def _gl_coef(alpha, L):
    c = np.ones(L)
    for k in range(1, L):
        c[k] = c[k - 1] * (1.0 - (alpha + 1.0) / float(k))
    return c


def _simulate(neuron, params, w_in, W, u, gamma, synapse="simple", syn_hist=0):
    """States [T, n] and spikes [T, n] from reset, dt = 1."""
    n, T, dev = w_in.shape[0], u.shape[0], "cuda"
    ext = gamma * (torch.tensor(u, device=dev) @ w_in.T)
    f8 = dict(dtype=torch.float64, device=dev)
    S = torch.zeros(T, n, dtype=torch.bool, device=dev)
    P = torch.empty(T, n, **f8)
    spk = torch.zeros(n, **f8)
    p = params
    if synapse == "frac":
        Ls = syn_hist
        sc = torch.tensor(_gl_coef(FRAC[0], Ls), device=dev).flip(0)[:-1].contiguous()
        cur = torch.zeros(T + Ls, n, **f8)  # row t + Ls: the current of step t
    if neuron == "lif":
        V = torch.full((n,), p[0], **f8)
    elif neuron == "gl":
        L = int(p[5])
        c = torch.tensor(_gl_coef(p[4], L), device=dev).flip(0)[:-1].contiguous()
        H = torch.zeros(T + L, n, **f8)  # row t + L: the state of step t
        tprev = torch.full((n,), p[7] + 1.0, **f8)
        V = torch.full((n,), p[2], **f8)
    else:
        D = int(p[8]) - 2
        x = np.arange(D) + 2.0
        c = torch.tensor(x ** (1 - p[6]) - (x - 1) ** (1 - p[6]), device=dev)
        reg = torch.zeros(n, D, **f8)  # newest first
        kr = math.gamma(2.0 - p[6])
        tprev = torch.full((n,), 2.0 * p[7], **f8)
        V = torch.full((n,), p[4], **f8)
    for t in range(T):
        drive = spk
        if synapse == "frac":
            last = cur[t + Ls - 1]
            hist = sc @ cur[t + 1:t + Ls]
            cur[t + Ls] = (spk - last) / FRAC[1] - hist
            drive = cur[t + Ls]
        inp = ext[t] + (W @ drive[:, None])[:, 0]
        if neuron == "lif":
            V = (1.0 - p[2]) * V + inp + p[3]
            fired = V > p[1]
            V = torch.where(fired, p[0], V)
        elif neuron == "gl":
            integ = tprev > p[7]
            last = H[t + L - 1]
            hist = c @ H[t + 1:t + L]
            Vn = (-(last - p[2]) / p[3] + inp + p[6]) - hist
            fired = integ & (Vn >= p[0])
            V = torch.where(integ & ~fired, Vn, p[1])
            H[t + L] = V
            tprev = torch.where(fired, 0.0, tprev) + 1.0
        else:
            integ = tprev > p[7]
            dV = (-p[1] * (V - p[2]) + inp) / p[0]
            reg = torch.where(integ[:, None], torch.cat([(V - p[4])[:, None], reg[:, :-1]], 1), reg)
            Vn = V + kr * dV - reg @ c
            fired = integ & (Vn >= p[3])
            V = torch.where(integ & ~fired, Vn, p[4])
            tprev = torch.where(fired, 0.0, tprev) + 1.0
        spk = fired.to(torch.float64)
        S[t] = fired
        P[t] = V
    return P, S


def _words(S):
    """[T, n] spikes -> [T, ceil(n / 32)] words."""
    b = np.zeros((S.shape[0], (S.shape[1] + 31) // 32 * 32), np.uint8)
    b[:, :S.shape[1]] = S
    return np.packbits(b, axis=1, bitorder="little").view(np.int32)


def _ridge(x, y, lam):
    if 2 * x.shape[0] <= x.shape[1]:
        K = x @ x.T
        K.diagonal().add_(lam)
        return (x.T @ torch.linalg.solve(K, y)).T
    A = x.T @ x
    A.diagonal().add_(lam)
    return torch.linalg.solve(A, x.T @ y).T


def _mlp(p, x, rounded=False):
    r = (lambda a: a.to(torch.bfloat16).to(torch.float64)) if rounded else (lambda a: a)
    shapes = ((128, 10), (128,), (128, 128), (128,), (2, 128), (2,))
    w, o = [], 0
    for s in shapes:
        k = int(np.prod(s))
        w.append(p[o:o + k].reshape(s))
        o += k
    z1 = r(x) @ r(w[0]).T + w[1]
    h1 = r(torch.nn.functional.gelu(z1))
    z2 = h1 @ r(w[2]).T + w[3]
    h2 = r(torch.nn.functional.gelu(z2))
    return h2 @ r(w[4]).T + w[5]


def _shuffles(n, epochs, seed):
    """The row orders of the training epochs: Fisher-Yates on a PCG32."""
    s, M = (seed ^ 0x5DEECE66D), (1 << 64) - 1
    perm = list(range(n))
    for _ in range(epochs):
        for i in range(n - 1, 0, -1):
            old = s
            s = (old * 6364136223846793005 + 1442695040888963407) & M
            xs = (((old >> 18) ^ old) >> 27) & 0xFFFFFFFF
            rot = old >> 59
            j = ((xs >> rot) | (xs << ((32 - rot) & 31))) & 0xFFFFFFFF
            j %= i + 1
            perm[i], perm[j] = perm[j], perm[i]
        yield list(perm)


def exact(case, seed):
    k = case["kind"]
    a = _inputs(case, seed)
    cuda = lambda v: torch.tensor(v, device="cuda")  # noqa: E731
    if k == "surrogate":
        p = cuda(a["p"]).double().requires_grad_()
        x, y = cuda(a["x"]).double(), cuda(a["y"]).double()
        batch = min(case["batch"], case["rows"])
        m1, m2, t, loss = torch.zeros_like(p), torch.zeros_like(p), 0, None
        for perm in _shuffles(case["rows"], case["epochs"], 3):
            for s in range(0, case["rows"], batch):
                at = torch.tensor(perm[s:s + batch], device="cuda")
                o = _mlp(p, x[at])
                e = y[at] - o[:, 0]
                loss = (0.5 * (o[:, 1] + e * e * torch.exp(-o[:, 1]))).mean()
                g, = torch.autograd.grad(loss, p)
                t += 1
                with torch.no_grad():
                    m1 = 0.9 * m1 + 0.1 * g
                    m2 = 0.999 * m2 + 0.001 * g * g
                    p -= 1e-3 * (m1 / (1 - 0.9 ** t)) / ((m2 / (1 - 0.999 ** t)).sqrt() + 1e-8)
        # candidates are scored with the weights as training left them
        o = _mlp(p.detach(), cuda(a["c"]).double(), case["bf16"])
        return dict(params=p.detach(), loss=float(loss), mean=o[:, 0], logvar=o[:, 1])
    if k == "ridge_fit":
        w = case["washout"]
        return _ridge(cuda(a["x"][w:]), cuda(a["y"][w:]), case["lam"])
    if k == "sweep":
        if sum(i.n * i.n * i.conn for i in a["insts"]) > 2e6:
            return None  # redrawing the graphs one edge at a time takes too long
        out = []
        for i, u, y, sd, h in zip(a["insts"], a["us"], a["ys"], a["seeds"], a["heads"]):
            w_in, W, _ = _model(i.n, 1, 1, i.topo, i.conn, i.rho, 0.5, sd)
            gl = i.neuron == sp.FLIF_GL
            params = (1.0, 0.0, 0.0, 20.0, i.alpha, float(i.L), 0.1, 2.0) if gl else sweep.LIF_BASE
            P, _ = _simulate("gl" if gl else "lif", params, w_in, W, u, 0.5)
            out.append(P @ _ridge(P[50:h], cuda(y[50:h]), 10.0).T)
        return out
    n = case["n"]
    if n * n * case["conn"] > 2e6:
        return None  # redrawing the graph one edge at a time takes too long
    w_in, W, w_out = _model(n, case["din"], case["dout"], TOPO[case["topo"]], case["conn"], 0.9,
                            0.5, seed % (2**31))
    params = _neuron_params(case["neuron"], case.get("hist", 64))
    u = a["u"][:case["steps"]] if k == "loop" else a["u"]
    P, S = _simulate(case["neuron"], params, w_in, W, u, 0.5, case.get("synapse", "simple"),
                     case.get("syn_hist", 0))
    if k == "loop":
        return P @ w_out.T
    if k == "run":
        return [x for x in (P if case.get("states") else None, _words(S.cpu().numpy()),
                            P @ w_out.T) if x is not None]
    if k == "stream":
        return [P[-case["steps"]:] @ w_out.T, P[-1]]
    if k == "train_ridge":
        return _ridge(P, cuda(a["y"]), case["lam"])
    w = torch.zeros(case["dout"], n, dtype=torch.float64, device="cuda")
    Pm = torch.eye(n, dtype=torch.float64, device="cuda")
    y = cuda(a["y"])
    for t in range(case["steps"]):
        g = Pm @ P[t]
        den = case["lam"] + P[t] @ g
        w += torch.outer(y[t] - w @ P[t], g / den)
        Pm = (Pm - torch.outer(g, g) / den) / case["lam"]
    return w

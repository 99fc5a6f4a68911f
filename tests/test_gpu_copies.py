"""Large copies of the caller's host memory (staged through pinned buffers in 2 MB
pieces from 4 MB on, 4 MB from 32 MB on) against the small ones, which the driver moves as they are."""
import threading

import numpy as np
import pytest

import spires_b200 as sp

pytestmark = pytest.mark.gpu

MB = 1 << 20


def reservoir(n):
    return sp.Reservoir(sp.make_config(n, 2, 1, rho=0.9, conn=0.002, topo=sp.CONN_RANDOM,
                                       neuron=sp.FLIF_GL,
                                       nparams=(1.0, 0.0, 0.0, 20.0, 0.6, 40.0, 0.1, 2.0)), seed=5)


# around the first staged size, whole pieces and one double more, more than the buffers
@pytest.mark.parametrize("doubles", [4 * MB // 8 - 1, 4 * MB // 8, 6 * MB // 8 + 1,
                                     10 * MB // 8, 21 * MB // 8 + 77,
                                     34 * MB // 8 + 5])
def test_states_of_a_long_run_match_short_runs(doubles):
    n = 1009
    T = -(-doubles // n)
    u = np.random.default_rng(1).uniform(-1, 2, (T, 2))
    a, b = reservoir(n), reservoir(n)
    phi, ras, _ = a.run_record(u)
    parts = [b.run_record(u[t:t + 200]) for t in range(0, T, 200)]
    assert np.array_equal(phi, np.concatenate([p[0] for p in parts]))
    assert np.array_equal(ras, np.concatenate([p[1] for p in parts]))
    a.close()
    b.close()


def test_fits_from_several_threads():
    """One copy holds the buffers, the others go past them: same bits."""
    rng = np.random.default_rng(2)
    X = rng.standard_normal((9000, 120))
    Y = rng.standard_normal((9000, 2))
    ref = sp.ridge_fit(X, Y, 1.0)[0]
    small = sp.ridge_fit(X[:2000], Y[:2000], 1.0)[0]
    out = [None] * 6
    def work(k):
        out[k] = [sp.ridge_fit(X, Y, 1.0)[0], sp.ridge_fit(X[:2000], Y[:2000], 1.0)[0]]
    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in out:
        assert np.array_equal(a, ref) and np.array_equal(b, small)


@pytest.mark.parametrize("dout", [1, 30, 31])
def test_outputs_of_many_reservoirs(dout):
    """The largest output row of a mail slot and one more, more reservoirs than
    slots, and slots taken again: the outputs of a run."""
    cfg = sp.make_config(40, 1, dout, rho=0.9, conn=0.2, topo=sp.CONN_RANDOM,
                         neuron=sp.LIF_DISCRETE, nparams=(0.0, 1.0, 0.1, 0.05))
    u = np.random.default_rng(3).uniform(0, 2, (6, 1))
    one = sp.Reservoir(cfg, seed=9)
    y = one.run(u)
    rs = [sp.Reservoir(cfg, seed=9) for _ in range(260 if dout == 1 else 3)]
    for k in range(2):
        for r in rs:
            r.reset()
            for t in range(len(u)):
                r.step(u[t])
            assert np.array_equal(r.output(), y[-1])
        if k == 0:
            for r in rs[::2]:
                r.close()
            rs = rs[1::2] + [sp.Reservoir(cfg, seed=9) for _ in range(3)]
    for r in rs:
        r.close()
    one.close()

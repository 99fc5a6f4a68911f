"""Large copies of the caller's host memory (staged through pinned buffers in 2 MB
pieces from 4 MB on) against the small ones, which the driver moves as they are."""
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
                                     10 * MB // 8, 21 * MB // 8 + 77])
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

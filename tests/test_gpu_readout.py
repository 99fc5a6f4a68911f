"""GPU readouts against the oracle (and the compiled reference when present):
ridge (src/reservoir.c:573-679), RLS (:681-767), the online delta rule
(:244-280), coarse-graining (:782-967) and the readout itself (:169-192).

Readout solves are floating-point reductions in a different order than the
reference (blocked Cholesky + refinement instead of one LU per output), so they
are compared with tolerances stated per test; states feeding them are
bit-identical (tests/test_gpu_parity.py)."""
import ctypes as C

import numpy as np
import pytest

import spires_b200 as sp
from tests import _oracle as O

pytestmark = pytest.mark.gpu

GL = (1.0, 0.0, 0.0, 20.0, 0.7, 64.0, 0.1, 2.0)


def cfg_gl(n=200, din=2, dout=3, conn=0.04, topo=sp.CONN_SCALE_FREE, synapse=sp.SYN_SIMPLE):
    return sp.make_config(n, din, dout, rho=1.2, ei=0.55, gamma=1.2, conn=conn, topo=topo,
                          neuron=sp.FLIF_GL, nparams=GL, synapse=synapse,
                          sparams=O.SYNAPSE_PARAMS[synapse])


def data(T, din, dout, seed=0):
    rng = np.random.default_rng(seed)
    u = rng.uniform(-1.0, 1.5, size=(T, din))
    y = np.stack([np.sin(0.05 * np.arange(T) * (o + 1)) for o in range(dout)], axis=1)
    y = y + 0.1 * rng.standard_normal((T, dout))
    return u, np.ascontiguousarray(y)


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.mark.parametrize("lam", [1e-2, 1e-6])
def test_ridge_matches_fp64_oracle(lam):
    cfg = cfg_gl()
    u, y = data(500, 2, 3)
    r = sp.Reservoir(cfg, seed=3)
    r.train_ridge(u, y, lam)
    W = r.readout()
    r.close()
    orc = O.Oracle(cfg, sp.HostModel(cfg, seed=3))
    phi, _, _ = orc.run(u)
    Wo = O.oracle_ridge(phi, y, lam)
    # tolerance: the solution's sensitivity is cond(A) * eps; both solvers are
    # backward stable, so compare the fitted outputs tightly and W loosely
    assert rel(phi @ W.T, phi @ Wo.T) < 1e-9
    assert rel(W, Wo) < (1e-9 if lam >= 1e-2 else 1e-5)


@pytest.mark.skipif(not O.have_ref(), reason="reference build absent")
def test_ridge_matches_compiled_reference():
    cfg = cfg_gl(n=150)
    u, y = data(400, 2, 3, seed=4)
    r = sp.Reservoir(cfg, seed=8)
    r.train_ridge(u, y, 1e-3)
    W = r.readout()
    r.close()
    ref = sp.Reservoir(cfg, lib=O.ref_lib(), seed=8)
    ref.train_ridge(u, y, 1e-3)
    Wr = ref.readout()
    ref.close()
    assert rel(W, Wr) < 1e-9


def test_ridge_washout_and_report():
    cfg = cfg_gl()
    u, y = data(600, 2, 3, seed=5)
    r = sp.Reservoir(cfg, seed=3)
    opts = sp.RidgeOpts(0, 30, 1e-13, 100)
    rep = sp.RidgeReport()
    assert r.lib.spires_ext_train_ridge(r.h, sp.dptr(u), sp.dptr(y), 600, 1e-4, C.byref(opts),
                                        C.byref(rep)) == sp.SPIRES_OK
    W = r.readout()
    r.close()
    orc = O.Oracle(cfg, sp.HostModel(cfg, seed=3))
    phi, _, _ = orc.run(u)
    Wo = O.oracle_ridge(phi, y, 1e-4, washout=100)
    assert rel(phi[100:] @ W.T, phi[100:] @ Wo.T) < 1e-9
    assert rep.rel_residual < 1e-10
    assert rep.gram_mode_used == 0


def test_ridge_singular_system_keeps_going():
    """lambda = 0 with fewer samples than neurons: a singular system. The call
    returns OK as the reference does (it only prints a warning)."""
    cfg = cfg_gl(n=120)
    u, y = data(40, 2, 3, seed=6)
    r = sp.Reservoir(cfg, seed=2)
    r.train_ridge(u, y, 0.0)
    r.close()


def test_rls_matches_oracle():
    cfg = cfg_gl(n=80, conn=0.06)
    u, y = data(60, 2, 3, seed=7)
    r = sp.Reservoir(cfg, seed=12)
    r.train_rls(u, y, 1.0, 0.999)
    W = r.readout()
    r.close()
    orc = O.Oracle(cfg, sp.HostModel(cfg, seed=12))
    Wo = orc.train_rls(u, y, 1.0, 0.999)
    assert rel(W, Wo) < 1e-8


def test_online_rule_matches_oracle():
    cfg = cfg_gl(n=100)
    u, y = data(50, 2, 3, seed=9)
    hm = sp.HostModel(cfg, seed=21)
    r = sp.Reservoir(cfg, seed=21)
    orc = O.Oracle(cfg, hm)
    Wo = hm.w_out().copy()
    for t in range(50):
        r.step(u[t])
        orc.step(u[t])
        r.train_online(y[t], 0.01)
        orc.train_online(y[t], 0.01, Wo)
    assert rel(r.readout(), Wo) < 1e-12
    r.close()


def test_run_and_compute_output_agree_bitwise():
    """spires_run and spires_step + spires_compute_output use one readout
    reduction, so they return the same bits."""
    cfg = cfg_gl(n=300)
    u, _ = data(30, 2, 3)
    a = sp.Reservoir(cfg, seed=5)
    Ya = a.run(u)
    a.close()
    b = sp.Reservoir(cfg, seed=5)
    Yb = []
    for t in range(30):
        b.step(u[t])
        Yb.append(b.output())
    b.close()
    assert np.array_equal(Ya, np.array(Yb))


# ------------------------------------------------------------ coarse grain

def coarse_grain_restated(W, Win, Wout, V, thr):
    """src/reservoir.c:782-967 in plain Python (small n only)."""
    n = W.shape[0]
    W = W.copy(); Win = Win.copy(); Wout = Wout.copy(); V = V.copy()
    alive = np.ones(n, bool)
    merged = True
    while merged:
        merged = False
        for i in range(n):
            for j in range(i + 1, n):
                if W[i, j] <= thr and W[j, i] <= thr:
                    continue
                merged = True
                V[i] = (V[i] + V[j]) / 2.0
                V[j] = 0.0
                alive[j] = False
                for k in range(n):
                    if k == i or k == j:
                        continue
                    a, b = W[i, k], W[j, k]
                    nw = a + b if a * b == 0.0 else (a + b) / 2.0
                    W[i, k] = nw
                    W[k, i] = nw
                for k in range(Win.shape[1]):
                    a, b = Win[i, k], Win[j, k]
                    Win[i, k] = a + b if a * b == 0.0 else (a + b) / 2.0
                    Win[j, k] = 0.0
                Wout[:, i] += Wout[:, j]
                Wout[:, j] = 0.0
                W[j, :] = 0.0
                W[:, j] = 0.0
    idx = np.nonzero(alive)[0]
    return W[np.ix_(idx, idx)], Win[idx], Wout[:, idx], V[idx]


def test_coarse_grain_matches_restatement():
    cfg = cfg_gl(n=40, conn=0.15, topo=sp.CONN_RANDOM)
    u, _ = data(20, 2, 3)
    r = sp.Reservoir(cfg, seed=14)
    for t in range(20):
        r.step(u[t])
    W, Win, Wout, V = r.weights(), r.w_in(), r.readout(), r.state()
    h = C.c_void_p()
    assert r.lib.spires_coarse_grain(r.h, 0.05, C.byref(h)) == sp.SPIRES_OK
    Wc, Winc, Woutc, Vc = coarse_grain_restated(W, Win, Wout, V, 0.05)
    m = Wc.shape[0]
    assert r.lib.spires_num_neurons(h) == m
    nw = np.empty(m * m)
    r.lib.spires_read_weights(h, sp.dptr(nw))
    assert np.array_equal(nw.reshape(m, m), Wc)
    no = np.empty(3 * m)
    r.lib.spires_read_readout(h, sp.dptr(no))
    assert np.array_equal(no.reshape(3, m), Woutc)
    ns = np.empty(m)
    r.lib.spires_read_reservoir_state(h, sp.dptr(ns))
    assert np.array_equal(ns, Vc)
    wi = np.empty(m * 2)
    r.lib.spires_ext_read_w_in(h, sp.dptr(wi))
    assert np.array_equal(wi.reshape(m, 2), Winc)
    # the coarse reservoir steps like any other
    for t in range(5):
        r.lib.spires_step(h, sp.dptr(np.ascontiguousarray(u[t])))
    r.lib.spires_reservoir_destroy(h)
    # thresholds below zero (or NaN) would merge forever: refused
    h2 = C.c_void_p()
    for thr in (-0.5, float("nan")):
        assert r.lib.spires_coarse_grain(r.h, thr, C.byref(h2)) == sp.SPIRES_ERR_INVALID_ARG
    r.close()


@pytest.mark.parametrize("lam", [1e-2, 1e-5])
def test_ridge_dual_form_when_rows_are_few(lam):
    """Fewer fitted rows than N/2: the dual form solves the same ridge."""
    cfg = cfg_gl(n=700, conn=0.02)
    u, y = data(300, 2, 3, seed=9)
    r = sp.Reservoir(cfg, seed=5)
    opts = sp.RidgeOpts(0, 30, 1e-13, 20)
    rep = sp.RidgeReport()
    assert r.lib.spires_ext_train_ridge(r.h, sp.dptr(u), sp.dptr(y), 300, lam, C.byref(opts),
                                        C.byref(rep)) == sp.SPIRES_OK
    W = r.readout()
    r.close()
    assert rep.dual == 1
    orc = O.Oracle(cfg, sp.HostModel(cfg, seed=5))
    phi, _, _ = orc.run(u)
    Wo = O.oracle_ridge(phi, y, lam, washout=20)
    assert rel(phi[20:] @ W.T, phi[20:] @ Wo.T) < 1e-8
    assert rel(W, Wo) < (1e-6 if lam >= 1e-2 else 1e-3)
    assert rep.rel_residual < 1e-8


def test_ridge_more_than_sixteen_outputs():
    """21 outputs, as many as a caller likes in the reference: solved 16 at a
    time over the one system matrix, the FP64 oracle's solution for all of
    them, through the reservoir and through ridge_fit on host states."""
    cfg = cfg_gl(dout=21)
    u, y = data(500, 2, 21, seed=9)
    r = sp.Reservoir(cfg, seed=3)
    r.train_ridge(u, y, 1e-2)
    W = r.readout()
    r.close()
    orc = O.Oracle(cfg, sp.HostModel(cfg, seed=3))
    phi, _, _ = orc.run(u)
    Wo = O.oracle_ridge(phi, y, 1e-2)
    assert W.shape == (21, cfg.num_neurons)
    assert rel(phi @ W.T, phi @ Wo.T) < 1e-9
    assert rel(W, Wo) < 1e-9
    W2, _ = sp.ridge_fit(phi, y, 1e-2)
    assert rel(W2, Wo) < 1e-9


@pytest.mark.parametrize("n,T,dout,neuron", [(1, 5, 1, sp.LIF_DISCRETE), (33, 40, 3, sp.FLIF_GL),
                                             (300, 50, 17, sp.FLIF_GL), (1300, 24, 2, sp.LIF_DISCRETE),
                                             (1900, 10, 1, sp.LIF_DISCRETE)])
@pytest.mark.parametrize("lam", [1.0, 0.99])
def test_rls_in_one_launch_matches_oracle(n, T, dout, neuron, lam):
    """The fused recursion from one row of P to several rows per warp, with P in
    shared memory (up to 1300 here) and streamed from memory (1900), more
    outputs than CTAs or one. Tolerance as in test_rls_matches_oracle."""
    params = GL if neuron == sp.FLIF_GL else O.NEURON_PARAMS[neuron]
    cfg = sp.make_config(n, 2, dout, rho=1.2, ei=0.55, gamma=1.2, conn=min(0.5, 6.0 / max(n, 2)),
                         topo=sp.CONN_SMALL_WORLD, neuron=neuron, nparams=params)
    u, y = data(T, 2, dout, seed=7)
    r = sp.Reservoir(cfg, seed=12)
    r.train_rls(u, y, 1.0, lam)
    W = r.readout()
    v = r.state()
    r.close()
    orc = O.Oracle(cfg, sp.HostModel(cfg, seed=12))
    Wo = orc.train_rls(u, y, 1.0, lam)
    assert rel(W, Wo) < 1e-8
    phi, _, _ = O.Oracle(cfg, sp.HostModel(cfg, seed=12)).run(u)
    assert np.array_equal(v, phi[-1])  # the reservoir is left after the last step


# One 64-wide tile and its edges, several tiles, odd widths, tile pairs split over
# row parts or not, the 128-wide Gram tiles, and the dual form (few rows).
@pytest.mark.parametrize("n,T,dout", [(1, 3, 1), (63, 200, 2), (64, 130, 1), (65, 1000, 16),
                                      (129, 4099, 3), (577, 700, 5), (1000, 90, 2),
                                      (2050, 2304, 1)])
def test_ridge_solver_at_tile_edges(n, T, dout):
    """The direct solve (no refinement) against float64 LAPACK. With lambda = T the
    condition number of X^T X + lambda I is at most 1 + (1 + sqrt(n / T))^2 for
    entries in [-1, 1), and both sides' forward error is below
    2 (T + n) eps times it."""
    rng = np.random.default_rng(n)
    X = rng.uniform(-1, 1, (T, n))
    Y = rng.uniform(-1, 1, (T, dout))
    W, rep = sp.ridge_fit(X, Y, float(T), max_refine=0)
    ref = np.linalg.solve(X.T @ X + T * np.eye(n), X.T @ Y).T
    cond = 1 + (1 + np.sqrt(n / T)) ** 2
    assert rep.factor_failed == 0
    assert rel(W, ref) < 4 * (T + n) * np.finfo(float).eps * cond
    # the same bits again: the sums' order is fixed
    assert np.array_equal(W, sp.ridge_fit(X, Y, float(T), max_refine=0)[0])


# states large enough that the Gram starts on the rows that have arrived: whole and
# ragged ranges, 128-, 64- and 32-wide tiles, a washout beyond the first range
@pytest.mark.parametrize("n,T,washout", [(2050, 3001, 0), (1300, 5000, 3), (1001, 6007, 2500)])
def test_ridge_fit_overlapped_with_its_copy(n, T, washout):
    """Sixteen outputs and fewer take the overlapped way, seventeen copy first: the
    same sums, so the same bits for the outputs they share."""
    rng = np.random.default_rng(n)
    X = rng.uniform(-1, 1, (T, n))
    Y = rng.uniform(-1, 1, (T, 17))
    W, rep = sp.ridge_fit(X, Y[:, :2], float(T), washout=washout, max_refine=0)
    W17, _ = sp.ridge_fit(X, Y, float(T), washout=washout, max_refine=0)
    assert rep.factor_failed == 0 and rep.dual == 0
    assert np.array_equal(W, W17[:2])


@pytest.fixture
def filled_allocations(request):
    """New device memory holds 32.5 (0x40 in every byte) or NaN (0xff) in every
    double, as after another use of it."""
    lib = sp.load()
    lib.spires_ext_test_fill_device_allocs(request.param)
    yield
    lib.spires_ext_test_fill_device_allocs(-1)


@pytest.mark.parametrize("n,T,dout,neuron", [(1, 5, 1, sp.LIF_DISCRETE), (33, 40, 3, sp.FLIF_GL),
                                             (300, 50, 2, sp.FLIF_GL), (1900, 10, 1, sp.LIF_DISCRETE)])
@pytest.mark.parametrize("filled_allocations", [0x40], indirect=True)
def test_rls_reads_only_recorded_states(filled_allocations, n, T, dout, neuron):
    """Sizes that leave lanes of the last warp without a neuron: whatever memory held
    before, the recursion and the readout see a state of 0 there. Tolerance of the
    weights as in test_rls_matches_oracle; an output is a dot product of n terms."""
    params = GL if neuron == sp.FLIF_GL else O.NEURON_PARAMS[neuron]
    cfg = sp.make_config(n, 2, dout, rho=1.2, ei=0.55, gamma=1.2, conn=min(0.5, 6.0 / max(n, 2)),
                         topo=sp.CONN_SMALL_WORLD, neuron=neuron, nparams=params)
    u, y = data(T, 2, dout, seed=7)
    r = sp.Reservoir(cfg, seed=12)
    r.train_rls(u, y, 1.0, 1.0)
    W = r.readout()
    r.reset()
    phi, _, Y = r.run_record(u, y=True)
    r.close()
    Wo = O.Oracle(cfg, sp.HostModel(cfg, seed=12)).train_rls(u, y, 1.0, 1.0)
    assert rel(W, Wo) < 1e-8
    bound = 2 * n * np.finfo(float).eps * (np.abs(phi) @ np.abs(W).T)
    assert (np.abs(Y - phi @ W.T) <= bound).all()


@pytest.mark.parametrize("filled_allocations", [0xff], indirect=True)
@pytest.mark.parametrize("n,conn", [(33, 0.2), (300, 0.002)])
def test_outputs_of_recorded_rows_ignore_empty_lanes(filled_allocations, n, conn):
    """Outputs from recorded rows, of one reservoir and of a batch with and without
    column blocks. Bound of a dot product of n terms."""
    cfg = sp.make_config(n, 2, 2, rho=1.2, ei=0.55, gamma=1.2, conn=conn, topo=sp.CONN_RANDOM,
                         neuron=sp.LIF_DISCRETE, nparams=O.NEURON_PARAMS[sp.LIF_DISCRETE])
    u, _ = data(30, 2, 2, seed=4)
    r = sp.Reservoir(cfg, seed=8)
    phi, _, Y = r.run_record(u, y=True)
    W = r.readout()
    r.close()
    bound = 2 * n * np.finfo(float).eps * (np.abs(phi) @ np.abs(W).T)
    assert (np.abs(Y - phi @ W.T) <= bound).all()
    b = sp.Batch([cfg], [8])
    Yb = b.predict([u])[0][0]
    b.close()
    assert np.array_equal(Yb, Y)


def test_ridge_pivots_over_the_exponent_range():
    """One neuron, one row: w = x y / x^2, through the reciprocal root of the pivot
    twice. rsqrt is good to 1 ulp (2 eps / 2 at most, relative), the four roundings
    around it to eps / 2 each: 4 eps in all."""
    rng = np.random.default_rng(0)
    for e in range(-500, 505, 5):
        x = np.ldexp(rng.uniform(1.0, 2.0), e)
        y = rng.uniform(1.0, 2.0)
        W, rep = sp.ridge_fit(np.array([[x]]), np.array([[y]]), 0.0, max_refine=0)
        assert rep.factor_failed == 0
        exact = np.longdouble(y) / np.longdouble(x)
        assert abs(np.longdouble(W[0, 0]) - exact) <= 4 * np.finfo(float).eps * exact, e

"""Batched multi-reservoir path: every instance of a batch of uneven
reservoirs (size, model, ring length, topology, series length, inputs) must
reproduce, bit for bit, the spike raster and final states of the same
reservoir created and run on its own -- and through it the oracle.

All calls go through the C ABI of libspires.so."""
import ctypes as C

import numpy as np
import pytest

import spires_b200 as sp
from tests import _oracle as O

pytestmark = pytest.mark.gpu


def gl_params(alpha, L):
    # [V_th, V_reset, V_rest, tau_m, alpha, T_mem, bias, t_ref] at dt = 1
    return (1.0, 0.0, 0.0, 20.0, alpha, float(L), 0.1, 2.0)


def mixed_batch(count, seed, n_lo=60, n_hi=3000, t_lo=40, t_hi=300):
    """Uneven instances in the spirit of a hyper-parameter sweep."""
    rng = np.random.default_rng(seed)
    cfgs, seeds, us = [], [], []
    topos = [sp.CONN_RANDOM, sp.CONN_SMALL_WORLD, sp.CONN_SCALE_FREE]
    for k in range(count):
        n = int(np.exp(rng.uniform(np.log(n_lo), np.log(n_hi))))
        din = int(rng.integers(1, 4))
        topo = topos[k % 3]
        conn = float(rng.uniform(0.02, 0.2)) if topo == sp.CONN_RANDOM else 6.0 / (n - 1)
        if k % 2 == 0:
            L = int(rng.choice([16, 64, 128, 256]))
            cfg = sp.make_config(n, din, 2, rho=float(rng.uniform(0.5, 1.5)), ei=0.5,
                                 gamma=float(rng.uniform(0.5, 2.0)), conn=conn, topo=topo,
                                 neuron=sp.FLIF_GL,
                                 nparams=gl_params(float(rng.uniform(0.3, 1.0)), L))
        else:
            cfg = sp.make_config(n, din, 2, rho=float(rng.uniform(0.5, 1.5)), ei=0.5,
                                 gamma=float(rng.uniform(0.5, 2.0)), conn=conn, topo=topo,
                                 neuron=sp.LIF_DISCRETE, nparams=(0.0, 1.0, 0.1, 0.05))
        cfgs.append(cfg)
        seeds.append(int(rng.integers(1, 2**31 - 1)))
        T = int(rng.integers(t_lo, t_hi))
        us.append(rng.uniform(-1.0, 1.5, size=(T, din)))
    return cfgs, seeds, us


def same_bits(a, b):
    return np.array_equal(np.asarray(a).view(np.uint64), np.asarray(b).view(np.uint64))


def solo(cfg, seed, u):
    r = sp.Reservoir(cfg, seed=seed)
    _, R, _ = r.run_record(u, phi=False)
    V = r.state()
    r.close()
    return R, V


def test_batch_matches_single_reservoirs():
    cfgs, seeds, us = mixed_batch(14, seed=11)
    b = sp.Batch(cfgs, seeds)
    R, V, ms = b.run(us)
    assert ms > 0.0
    spiking = 0
    for k, (cfg, s, u) in enumerate(zip(cfgs, seeds, us)):
        R1, V1 = solo(cfg, s, u)
        bad = np.nonzero((R[k] != R1).any(axis=1))[0]
        assert bad.size == 0, f"instance {k}: raster differs first at step {bad[0]}"
        assert same_bits(V[k], V1), f"instance {k}: final states differ"
        spiking += int(np.unpackbits(R1.view(np.uint8)).sum() > 0)
    assert spiking >= 4  # the comparison is not only over silent rasters
    info = b.info()
    assert info["groups"] >= 2 and info["ctas"] >= info["groups"]
    b.close()


def test_batch_matches_oracle():
    cfgs, seeds, us = mixed_batch(4, seed=5, n_hi=400, t_hi=120)
    b = sp.Batch(cfgs, seeds)
    R, V, _ = b.run(us)
    for k, (cfg, s, u) in enumerate(zip(cfgs, seeds, us)):
        orc = O.Oracle(cfg, sp.HostModel(cfg, seed=s))
        phi_o, ras_o, _ = orc.run(u, y=False)
        ras = sp.unpack_raster(R[k], cfg.num_neurons)
        assert np.array_equal(ras, ras_o), f"instance {k}: raster differs from the oracle"
        assert same_bits(V[k], phi_o[-1]), f"instance {k}: states differ from the oracle"
    b.close()


def test_batch_repeat_replays_graph_and_is_deterministic():
    cfgs, seeds, us = mixed_batch(6, seed=21)
    b = sp.Batch(cfgs, seeds)
    R1, V1, _ = b.run(us)
    R2, V2, _ = b.run(us)
    assert b.info()["graph"] in (1, -1)
    for k in range(len(cfgs)):
        assert np.array_equal(R1[k], R2[k])
        assert same_bits(V1[k], V2[k])
    # other series lengths re-plan the schedule
    us3 = [u[: max(1, u.shape[0] // 2)] for u in us]
    R3, _, _ = b.run(us3)
    for k in range(len(cfgs)):
        assert np.array_equal(R3[k], R1[k][: us3[k].shape[0]])
    b.close()


def test_batch_zero_input_and_zero_length():
    cfgs, seeds, us = mixed_batch(3, seed=8, t_hi=80)
    b = sp.Batch(cfgs, seeds)
    T = [us[0].shape[0], 0, us[2].shape[0]]
    R, V, _ = b.run(None, T=T)
    for k in (0, 2):
        r = sp.Reservoir(cfgs[k], seed=seeds[k])
        _, R1, _ = r.run_record(np.zeros((T[k], cfgs[k].num_inputs)), phi=False)
        V1 = r.state()
        r.close()
        assert np.array_equal(R[k], R1)
        assert same_bits(V[k], V1)
    assert R[1].shape[0] == 0
    b.close()


def test_batch_ridge_and_predict_match_single():
    cfgs, seeds, us = mixed_batch(5, seed=31, n_hi=800, t_lo=150, t_hi=260)
    rng = np.random.default_rng(4)
    ys = [rng.standard_normal((u.shape[0], 2)) for u in us]
    b = sp.Batch(cfgs, seeds)
    W, ms = b.train_ridge(us, ys, 1e-4, washout=20)
    Yb, _ = b.predict(us)
    for k, (cfg, s, u) in enumerate(zip(cfgs, seeds, us)):
        r = sp.Reservoir(cfg, seed=s)
        o = sp.RidgeOpts(0, 30, 1e-13, 20)
        rep = sp.RidgeReport()
        st = r.lib.spires_ext_train_ridge(r.h, sp.dptr(u), sp.dptr(ys[k]), u.shape[0], 1e-4,
                                          sp.C.byref(o), sp.C.byref(rep))
        assert st == sp.SPIRES_OK
        W1 = r.readout()
        assert same_bits(W[k], W1), f"instance {k}: W_out differs"
        r.reset()
        Y1 = r.run(u)
        r.close()
        assert same_bits(Yb[k][:, :2], Y1), f"instance {k}: readouts differ"
    b.close()


def test_batch_rejects_unsupported_models():
    cfg = sp.make_config(64, 1, 1, neuron=sp.FLIF_CAPUTO,
                         nparams=O.NEURON_PARAMS[sp.FLIF_CAPUTO])
    with pytest.raises(RuntimeError):
        sp.Batch([cfg], [1])
    cfg2 = sp.make_config(64, 1, 1, neuron=sp.LIF_DISCRETE, synapse=sp.SYN_PSC_HOM,
                          sparams=(5.0,))
    with pytest.raises(RuntimeError):
        sp.Batch([cfg2], [1])


def test_fit_predict_equals_train_then_predict():
    cfgs, seeds, us = mixed_batch(4, seed=41, n_hi=600, t_lo=200, t_hi=300)
    rng = np.random.default_rng(2)
    ys = [rng.standard_normal((u.shape[0], 2)) for u in us]
    T_fit = [int(0.7 * u.shape[0]) for u in us]
    b = sp.Batch(cfgs, seeds)
    Y, _ = b.fit_predict(us, ys, T_fit, 1e-3, washout=10)
    b2 = sp.Batch(cfgs, seeds)
    b2.train_ridge([u[:t] for u, t in zip(us, T_fit)], [y[:t] for y, t in zip(ys, T_fit)], 1e-3,
                   washout=10)
    Y2, _ = b2.predict(us)
    for k in range(len(cfgs)):
        assert same_bits(Y[k][:, :2], Y2[k][:, :2]), f"instance {k}"


def test_autotuned_schedule_keeps_results():
    """spires_ext_batch_autotune times every schedule family and grid size on
    a sample of the series and keeps the fastest; whichever it keeps, every
    instance's raster and final state stay bit-identical to the same
    reservoir run on its own."""
    cfgs, seeds, us = mixed_batch(12, seed=77)
    b = sp.Batch(cfgs, seeds)
    sample = [u[:30] for u in us]
    tuned = b.autotune(sample)
    assert 0 <= tuned["schedule"] <= 3 and tuned["ctas"] > 0 and tuned["ms"] > 0
    R, V, _ = b.run(us)
    assert b.info()["ctas"] == tuned["ctas"]
    b.close()
    for k in range(len(cfgs)):
        Rs, Vs = solo(cfgs[k], seeds[k], us[k])
        assert np.array_equal(R[k], Rs), k
        assert same_bits(V[k], Vs), k


def test_batch_runs_after_a_smaller_batch_was_built():
    """The batch kernel's shared-memory limit is one attribute for the whole
    process. A batch with long rings (large shared memory) must still launch
    after a second batch with short rings (less shared memory, still above the
    48 KB default) was built, and re-plan for new
    series lengths (a search builds the next chunk's batch on another thread
    while the current one runs)."""
    big_cfg = sp.make_config(1500, 1, 1, rho=0.9, ei=0.5, gamma=1.0, conn=0.05,
                             topo=sp.CONN_RANDOM, neuron=sp.FLIF_GL,
                             nparams=gl_params(0.6, 1024))
    small_cfg = sp.make_config(300, 1, 1, rho=0.9, ei=0.5, gamma=1.0, conn=0.05,
                               topo=sp.CONN_RANDOM, neuron=sp.FLIF_GL,
                               nparams=gl_params(0.6, 128))
    rng = np.random.default_rng(5)
    big = sp.Batch([big_cfg, big_cfg], [11, 12])
    small = sp.Batch([small_cfg], [13])
    try:
        for T in (60, 140):
            us = [rng.uniform(-1.0, 1.5, size=(T, 1)) for _ in range(2)]
            R, V, _ = big.run(us)
            for k, seed in enumerate((11, 12)):
                Rs, Vs = solo(big_cfg, seed, us[k])
                assert np.array_equal(R[k], Rs)
                assert same_bits(V[k], Vs)
        small.run([rng.uniform(-1.0, 1.5, size=(50, 1))])
    finally:
        big.close()
        small.close()


# (neurons, ring, connectivity) per instance: the smallest rings and sizes, odd
# ring lengths, rings that fit shared memory beside the column blocks, alone, and
# not at all, edges walked as column blocks (dense) or CSR rows.
@pytest.mark.parametrize("shapes", [
    [(1, 1, 0.5), (2, 2, 0.5), (33, 3, 0.3), (64, 17, 0.1)],
    [(300, 0, 0.2), (700, 0, 0.002), (257, 0, 0.0)],
    [(300, 129, 0.1), (1100, 64, 0.15), (500, 300, 0.003)],
    [(4200, 40, 0.02), (96, 1500, 0.1)],
    [(60, 0 if k % 3 else 20 + k, 0.2) for k in range(160)],
])
def test_batch_forms_match_single_reservoirs(shapes):
    """Bit for bit, for batches spread one instance per group and, with more
    instances than SMs, in turns."""
    rng = np.random.default_rng(len(shapes))
    cfgs, seeds, us = [], [], []
    for n, L, conn in shapes:
        neuron = dict(neuron=sp.FLIF_GL, nparams=gl_params(0.6, L)) if L else \
            dict(neuron=sp.LIF_DISCRETE, nparams=(0.0, 1.0, 0.1, 0.05))
        cfgs.append(sp.make_config(n, 2, 1, rho=1.2, ei=0.5, gamma=1.5, conn=conn,
                                   topo=sp.CONN_RANDOM, **neuron))
        seeds.append(int(rng.integers(1, 2**31 - 1)))
        us.append(rng.uniform(-1.0, 2.0, size=(int(rng.integers(20, 90)), 2)))
    b = sp.Batch(cfgs, seeds)
    R, V, _ = b.run(us)
    fired = 0
    for k in range(0, len(cfgs), 1 if len(cfgs) < 20 else 16):
        R1, V1 = solo(cfgs[k], seeds[k], us[k])
        assert np.array_equal(R[k], R1), f"instance {k}: raster differs"
        assert same_bits(V[k], V1), f"instance {k}: final states differ"
        fired += int(R1.any())
    assert fired > 0
    assert b.info()["groups"] == len(cfgs) or len(cfgs) > 148
    b.close()


def test_fits_of_a_batch_share_their_launches():
    """More fits than one factorisation takes (32): sizes around the solver's tiles,
    a fit in the dual form, systems that are singular -- each the single
    reservoir's W_out."""
    rng = np.random.default_rng(4)
    ns = [1, 2, 63, 64, 65, 128, 129, 200, 700, 500] + [40 + k for k in range(26)]
    cfgs = [sp.make_config(n, 1, 1 + k % 3, rho=1.2, ei=0.5, gamma=1.5, conn=0.2,
                           topo=sp.CONN_RANDOM, neuron=sp.LIF_DISCRETE,
                           nparams=(0.0, 1.0, 0.3, 0.05)) for k, n in enumerate(ns)]
    seeds = [int(s) for s in rng.integers(1, 2**31 - 1, len(ns))]
    Ts = [90 if n == 500 else 260 + n for n in ns]  # 500: the dual form
    us = [rng.uniform(-1.0, 2.0, size=(T, 1)) for T in Ts]
    ys = [rng.standard_normal((T, 1 + k % 3)) for k, T in enumerate(Ts)]
    b = sp.Batch(cfgs, seeds)
    b.run(us)
    W, _ = b.train_ridge(us, ys, 1e-2, washout=20)
    for k, n in enumerate(ns):
        r = sp.Reservoir(cfgs[k], seed=seeds[k])
        o = sp.RidgeOpts(0, 30, 1e-13, 20)
        rep = sp.RidgeReport()
        assert r.lib.spires_ext_train_ridge(r.h, sp.dptr(us[k]), sp.dptr(ys[k]), Ts[k], 1e-2,
                                            C.byref(o), C.byref(rep)) == sp.SPIRES_OK
        assert np.allclose(W[k], r.readout(), rtol=1e-9, atol=1e-12), f"instance {k} (n={n})"
        assert rep.dual == (n == 500)
        r.close()
    # the same fits beside singular ones (no rows to tell 700 neurons apart)
    lam = np.array([0.0 if n == 700 else 1e-2 for n in ns])
    short = [u[:300] if n == 700 else u for n, u in zip(ns, us)]
    W2, _ = b.train_ridge(short, [y[:len(u)] for y, u in zip(ys, short)], lam, washout=20)
    for k, n in enumerate(ns):
        if n != 700:
            assert np.array_equal(W2[k], W[k]), f"instance {k} (n={n})"
    b.close()


def test_groups_wider_than_an_instance():
    """Instances of one warp beside wide ones: the schedules that autotune times put
    them on groups with CTAs that have no neurons of theirs, several in turn."""
    rng = np.random.default_rng(6)
    ns = [20, 32, 7, 1] * 40 + [2300, 1200, 600]
    cfgs = [sp.make_config(n, 2, 1, rho=1.2, ei=0.5, gamma=1.5, conn=0.1, topo=sp.CONN_RANDOM,
                           neuron=sp.LIF_DISCRETE, nparams=(0.0, 1.0, 0.1, 0.05)) for n in ns]
    seeds = [int(s) for s in rng.integers(1, 2**31 - 1, len(ns))]
    us = [rng.uniform(-1.0, 2.0, size=(200, 2)) for _ in ns]
    b = sp.Batch(cfgs, seeds)
    b.autotune(us)
    R, V, _ = b.run(us)
    b.close()
    for k in list(range(0, len(ns), 23)) + [160, 161, 162]:
        Rs, Vs = solo(cfgs[k], seeds[k], us[k])
        assert np.array_equal(R[k], Rs), f"instance {k} (n={ns[k]})"
        assert same_bits(V[k], Vs), f"instance {k} (n={ns[k]})"


def test_singular_fits_in_a_batch():
    """Fits without a ridge term whose Cholesky fails, beside one that is solved: an
    exactly singular system (every state 0) keeps the instance's W_out, one with
    fewer rows than neurons takes the way that the single reservoir takes."""
    rng = np.random.default_rng(8)
    lif = lambda bias: dict(neuron=sp.LIF_DISCRETE, nparams=(0.0, 1.0, 0.3, bias))
    cfgs = [sp.make_config(40, 1, 2, conn=0.2, gamma=0.0, topo=sp.CONN_RANDOM, **lif(0.0)),
            sp.make_config(700, 1, 1, rho=1.2, gamma=1.5, conn=0.2, topo=sp.CONN_RANDOM, **lif(0.05)),
            sp.make_config(90, 1, 3, rho=1.2, gamma=1.5, conn=0.2, topo=sp.CONN_RANDOM, **lif(0.05)),
            sp.make_config(64, 1, 2, conn=0.2, gamma=0.0, topo=sp.CONN_RANDOM, **lif(0.0))]
    seeds = [5, 6, 7, 8]
    us = [rng.uniform(-1.0, 2.0, size=(300, 1)) for _ in cfgs]
    ys = [rng.standard_normal((300, int(c.num_outputs))) for c in cfgs]
    b = sp.Batch(cfgs, seeds)
    W, _ = b.train_ridge(us, ys, np.array([0.0, 0.0, 1e-2, 0.0]), washout=20)
    Y, _ = b.predict(us)
    b.close()
    for k, cfg in enumerate(cfgs):
        r = sp.Reservoir(cfg, seed=seeds[k])
        before = r.readout()
        o, rep = sp.RidgeOpts(0, 30, 1e-13, 20), sp.RidgeReport()
        st = r.lib.spires_ext_train_ridge(r.h, sp.dptr(us[k]), sp.dptr(ys[k]), 300,
                                          1e-2 if k == 2 else 0.0, C.byref(o), C.byref(rep))
        after = r.readout()
        r.reset()
        Y1 = r.run(us[k])
        r.close()
        assert st == sp.SPIRES_OK
        if k != 1:
            assert rep.factor_failed == (k != 2)
        if k in (0, 3):
            assert np.array_equal(after, before) and np.count_nonzero(before) == before.size
        assert np.allclose(W[k], after, rtol=1e-9, atol=1e-12), f"instance {k}"
        assert np.allclose(Y[k], Y1, rtol=1e-9, atol=1e-9), f"instance {k}"

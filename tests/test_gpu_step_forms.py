"""The step kernel's forms against the oracle, bit for bit: the cluster launch
and its spike exchange, the history kept in shared memory, the recurrent rows
as slots and tails and as column blocks, and FLIF_CAPUTO's 32-byte blocks --
each at the sizes where it can go wrong, over several launches in a row."""
import ctypes as C

import numpy as np
import pytest

import spires_b200 as sp
from tests import _oracle as O

pytestmark = pytest.mark.gpu

GL = lambda L: (1.0, 0.0, 0.0, 20.0, 0.7, float(L), 0.1, 2.0)


def check(n, neuron, ctas, T, nparams=None, synapse=sp.SYN_SIMPLE, topo=sp.CONN_RANDOM, conn=0.05,
          dt=1.0):
    cfg = sp.make_config(n, 2, 2, rho=1.3, ei=0.55, gamma=1.2, conn=conn, dt=dt, topo=topo,
                         neuron=neuron, nparams=nparams or O.NEURON_PARAMS[neuron],
                         synapse=synapse, sparams=O.SYNAPSE_PARAMS[synapse])
    u = np.random.default_rng(3).uniform(-1.0, 1.5, (T, 2))
    r = sp.Reservoir(cfg, seed=11)
    nw = (n + 31) // 32
    assert r.set_launch(ctas=ctas, warps_max=-(-nw // ctas), variant=0) == sp.SPIRES_OK
    h = T // 3
    parts = [r.run_record(x) for x in (u[:h], u[h:h + 1], u[h + 1:])]
    r.close()
    phi = np.concatenate([p[0] for p in parts])
    ras = sp.unpack_raster(np.concatenate([p[1] for p in parts]), n)
    phi_o, ras_o, _ = O.Oracle(cfg, sp.HostModel(cfg, seed=11)).run(u)
    assert np.array_equal(ras, ras_o)
    assert np.array_equal(phi.view(np.uint64), phi_o.view(np.uint64))


@pytest.mark.parametrize("neuron", [sp.LIF_DISCRETE, sp.LIF_BIO, sp.FLIF_CAPUTO, sp.FLIF_GL,
                                    sp.FLIF_DIFFUSIVE])
@pytest.mark.parametrize("synapse", [sp.SYN_SIMPLE, sp.SYN_PSC_HET])
@pytest.mark.parametrize("ctas", [2, 16, 3])
def test_exchange(neuron, synapse, ctas):
    """Clusters of 2 and 16 CTAs, and 3 CTAs exchanging through the L2."""
    check(600, neuron, ctas, 60, synapse=synapse, dt=0.5 if ctas == 2 else 1.0)


def test_largest_cluster():
    check(8192, sp.LIF_DISCRETE, 16, 16, topo=sp.CONN_SMALL_WORLD, conn=0.001)


@pytest.mark.parametrize("L", [1, 2, 3, 33, 64, 201])
@pytest.mark.parametrize("ctas", [1, 5, 8])
def test_history_in_shared_memory(L, ctas):
    """Odd and even ring lengths below and above a block, through ramp-up and wrap."""
    check(200 if ctas == 1 else 250, sp.FLIF_GL, ctas, 2 * L + 40, nparams=GL(L))


@pytest.mark.parametrize("n,conn,ctas", [(250, 0.2, 1), (1000, 0.1, 16), (1000, 0.3, 5),
                                         (1025, 0.06, 33), (500, 0.9, 4)])
def test_dense_rows_as_column_blocks(n, conn, ctas):
    check(n, sp.LIF_DISCRETE, ctas, 40, conn=conn)


@pytest.mark.parametrize("topo,conn", [(sp.CONN_SCALE_FREE, 0.003), (sp.CONN_SCALE_FREE, 0.0005),
                                       (sp.CONN_SMALL_WORLD, 0.004), (sp.CONN_RANDOM, 0.0005)])
@pytest.mark.parametrize("ctas", [16, 63])
def test_sparse_rows_as_slots_and_tails(topo, conn, ctas):
    """Hubs with tails of several 32-edge blocks, even rows, empty rows."""
    check(2000, sp.LIF_DISCRETE, ctas, 40, topo=topo, conn=conn)


@pytest.mark.parametrize("D", [1, 2, 3, 4, 5, 31, 32, 33, 64, 65, 66, 67, 130])
@pytest.mark.parametrize("ctas", [1, 4])
def test_caputo_blocks(D, ctas):
    """Shift registers of every alignment, shorter and longer than the blocks in
    flight, with each neuron's head at its own place after the first spikes."""
    check(100, sp.FLIF_CAPUTO, ctas, 2 * D + 40, conn=0.06,
          nparams=(1.0, 0.2, 0.0, 1.0, 0.0, 1.5, 0.7, 2.0, float(D + 2)))


@pytest.mark.parametrize("conn", [0.002, 0.1])
def test_cluster_wait_runs_out(conn):
    """A CTA of a cluster that withholds its spike words once: the launch ends
    with an error naming the micro-step, and the reservoir works after a reset."""
    cfg = sp.make_config(2000, 2, 2, rho=1.2, ei=0.55, gamma=1.2, conn=conn,
                         topo=sp.CONN_SCALE_FREE, neuron=sp.LIF_DISCRETE,
                         nparams=O.NEURON_PARAMS[sp.LIF_DISCRETE])
    u = np.random.default_rng(0).uniform(-1.0, 1.5, (30, 2))
    r = sp.Reservoir(cfg, seed=17)
    assert r.set_launch(ctas=16, warps_max=4, variant=0) == sp.SPIRES_OK
    assert r.lib.spires_ext_set_wait_limit(r.h, 50.0) == sp.SPIRES_OK
    r.run_record(u[:12])
    assert r.lib.spires_ext_test_withhold_arrival(r.h, 1, 5) == sp.SPIRES_OK
    P = np.empty((10, r.n))
    st = r.lib.spires_ext_run_record(r.h, sp.dptr(np.ascontiguousarray(u[12:22])), 10, sp.dptr(P),
                                     None, None)
    assert st == sp.SPIRES_ERR_INTERNAL
    code, step = C.c_int(-1), C.c_longlong(-1)
    assert r.lib.spires_ext_last_device_error(r.h, C.byref(code), C.byref(step)) == sp.SPIRES_OK
    assert (code.value, step.value) == (1, 17)
    r.reset()
    phi, R, _ = r.run_record(u)
    r.close()
    phi_o, ras_o, _ = O.Oracle(cfg, sp.HostModel(cfg, seed=17)).run(u)
    assert np.array_equal(sp.unpack_raster(R, 2000), ras_o)
    assert np.array_equal(phi.view(np.uint64), phi_o.view(np.uint64))


# synapse lags: fewer than a stage holds (read by the consumers), a stage, one more,
# several with a ragged last one; the neuron's ring shorter and longer than that
@pytest.mark.parametrize("Ls", [3, 16, 17, 40, 75])
@pytest.mark.parametrize("L", [16, 90])
@pytest.mark.parametrize("rows,stages", [(16, 2), (8, 5)])
def test_fractional_history_through_the_pipeline(Ls, L, rows, stages):
    """FLIF_GL with the FRACTIONAL synapse, both rings in the pipeline's stages,
    through ramp-up and wrap and over several launches."""
    n, T = 230, 2 * max(L, Ls) + 30
    cfg = sp.make_config(n, 2, 2, rho=1.3, ei=0.55, gamma=1.2, conn=0.05, dt=1.0,
                         topo=sp.CONN_RANDOM, neuron=sp.FLIF_GL, nparams=GL(L),
                         synapse=sp.SYN_FRAC, sparams=(0.6, 4.0, float(Ls)))
    u = np.random.default_rng(3).uniform(-1.0, 1.5, (T, 2))
    r = sp.Reservoir(cfg, seed=11)
    assert r.set_launch(ctas=4, warps_max=2, variant=1, rows=rows, stages=stages) == sp.SPIRES_OK
    parts = [r.run_record(x) for x in (u[:7], u[7:8], u[8:10], u[10:])]
    r.close()
    phi = np.concatenate([p[0] for p in parts])
    phi_o, _, _ = O.Oracle(cfg, sp.HostModel(cfg, seed=11)).run(u)
    assert np.array_equal(phi.view(np.uint64), phi_o.view(np.uint64))


@pytest.mark.parametrize("L,rows", [(16, 32), (40, 64), (64, 256)])
@pytest.mark.parametrize("Ls", [64, 75, 300])
def test_fractional_history_with_stages_taller_than_the_ring(L, rows, Ls):
    """A stage holds as many rows as the neuron's ring has, also for the synapse's
    longer ring."""
    n, T = 230, 2 * Ls + 30
    cfg = sp.make_config(n, 2, 2, rho=1.3, ei=0.55, gamma=1.2, conn=0.05, dt=1.0,
                         topo=sp.CONN_RANDOM, neuron=sp.FLIF_GL, nparams=GL(L),
                         synapse=sp.SYN_FRAC, sparams=(0.6, 4.0, float(Ls)))
    u = np.random.default_rng(3).uniform(-1.0, 1.5, (T, 2))
    r = sp.Reservoir(cfg, seed=11)
    assert r.set_launch(ctas=8, warps_max=1, variant=1, rows=rows, stages=2) == sp.SPIRES_OK
    parts = [r.run_record(x) for x in (u[:7], u[7:8], u[8:])]
    r.close()
    phi = np.concatenate([p[0] for p in parts])
    phi_o, _, _ = O.Oracle(cfg, sp.HostModel(cfg, seed=11)).run(u)
    assert np.array_equal(phi.view(np.uint64), phi_o.view(np.uint64))


# 7 warps of neurons: more CTAs than warps (clusters of 8 and 16, the L2's exchange on
# 12); 25 warps on 16 CTAs and 19 on 4: CTAs with a warp less than the others
@pytest.mark.parametrize("n,ctas", [(200, 8), (200, 16), (200, 12), (800, 16), (600, 4)])
@pytest.mark.parametrize("neuron,synapse", [(sp.LIF_DISCRETE, sp.SYN_SIMPLE),
                                            (sp.LIF_DISCRETE, sp.SYN_PSC_HET),
                                            (sp.FLIF_GL, sp.SYN_SIMPLE),
                                            (sp.FLIF_CAPUTO, sp.SYN_SIMPLE)])
@pytest.mark.parametrize("conn", [0.005, 0.1])
def test_ctas_and_warps_without_neurons(n, ctas, neuron, synapse, conn):
    """They publish no spike words and read none; rows as slots and as column blocks."""
    check(n, neuron, ctas, 300, synapse=synapse, conn=conn)


@pytest.mark.parametrize("variant", [0, 1])
def test_more_ctas_than_warps_with_a_gather_warp(variant):
    """FLIF_GL with its history in shared memory and through the stages."""
    n, T = 200, 120
    cfg = sp.make_config(n, 2, 2, rho=1.3, ei=0.55, gamma=1.2, conn=0.05,
                         topo=sp.CONN_RANDOM, neuron=sp.FLIF_GL, nparams=GL(64))
    u = np.random.default_rng(3).uniform(-1.0, 1.5, (T, 2))
    r = sp.Reservoir(cfg, seed=11)
    assert r.set_launch(ctas=40, warps_max=1, variant=variant, rows=16, stages=2) == sp.SPIRES_OK
    phi, _, _ = r.run_record(u)
    r.close()
    phi_o, _, _ = O.Oracle(cfg, sp.HostModel(cfg, seed=11)).run(u)
    assert np.array_equal(phi.view(np.uint64), phi_o.view(np.uint64))


def run_against_oracle(r, cfg, T, seed):
    u = np.random.default_rng(3).uniform(-1.0, 1.5, (T, 2))
    phi, _, _ = r.run_record(u)
    r.close()
    phi_o, _, _ = O.Oracle(cfg, sp.HostModel(cfg, seed=seed)).run(u)
    assert np.array_equal(phi.view(np.uint64), phi_o.view(np.uint64))


@pytest.mark.parametrize("n,edges,D", [(6000, 128, 7400), (4000, 505, 8180)])
def test_caputo_table_beside_dense_rows(n, edges, D):
    """Column blocks and memory coefficients that fit a CTA's shared memory one by one
    and not together: the default launch keeps what fits."""
    cfg = sp.make_config(n, 2, 2, rho=1.3, ei=0.55, gamma=1.2, conn=edges / n, dt=1.0,
                         topo=sp.CONN_RANDOM, neuron=sp.FLIF_CAPUTO,
                         nparams=(1.0, 0.2, 0.0, 1.0, 0.0, 1.5, 0.7, 2.0, float(D + 2)))
    run_against_oracle(sp.Reservoir(cfg, seed=11), cfg, 24, 11)


@pytest.mark.parametrize("n,conn,stages", [(1000, 0.1, 13), (2000, 0.004, 13)])
def test_stages_that_leave_the_rows_no_room(n, conn, stages):
    """A pipeline that takes all the shared memory: the rows are read from global
    memory, as column blocks or edge by edge."""
    nw = (n + 31) // 32
    cfg = sp.make_config(n, 2, 2, rho=1.3, ei=0.55, gamma=1.2, conn=conn, dt=1.0,
                         topo=sp.CONN_RANDOM, neuron=sp.FLIF_GL, nparams=GL(64))
    r = sp.Reservoir(cfg, seed=11)
    assert r.set_launch(ctas=nw, warps_max=1, variant=1, rows=64, stages=stages) == sp.SPIRES_OK
    run_against_oracle(r, cfg, 150, 11)


def test_pipeline_with_coefficients_in_global_memory():
    """More coefficients than the launch stages (8192), a chain of stages and a
    ragged one by the end."""
    n = 70
    cfg = sp.make_config(n, 2, 2, rho=1.3, ei=0.55, gamma=1.2, conn=0.2, dt=1.0,
                         topo=sp.CONN_RANDOM, neuron=sp.FLIF_GL, nparams=GL(8300))
    r = sp.Reservoir(cfg, seed=11)
    assert r.set_launch(ctas=3, warps_max=1, variant=1, rows=16, stages=3) == sp.SPIRES_OK
    run_against_oracle(r, cfg, 90, 11)


@pytest.mark.parametrize("n,L", [(30000, 1024), (37500, 600)])
def test_wide_ctas_keep_the_pipeline(n, L):
    """Rings beyond the L2 on CTAs of seven and eight warps, where two stages take more
    than the share that narrower CTAs keep to."""
    cfg = sp.make_config(n, 1, 1, rho=0.0, conn=2.0 / n, topo=sp.CONN_SMALL_WORLD,
                         neuron=sp.FLIF_GL, nparams=GL(L))
    r = sp.Reservoir(cfg, seed=1)
    l = r.launch()
    r.close()
    assert l.variant == 1 and l.stages >= 2


@pytest.mark.parametrize("n,L,syn,prm", [(20000, 1024, sp.SYN_PSC_HOM, (3.0,)),
                                         (12000, 2000, sp.SYN_FRAC, (0.6, 4.0, 100.0)),
                                         (30000, 700, sp.SYN_PSC_HET, (1.0, 10.0))])
def test_stages_beside_a_drive_are_few(n, L, syn, prm):
    """The synapses that read memory in the serial phase: at most three stages in 160 KB
    beside a ring beyond the L2, and the pipeline all the same where two take more."""
    cfg = sp.make_config(n, 1, 1, rho=0.0, conn=2.0 / n, topo=sp.CONN_SMALL_WORLD,
                         neuron=sp.FLIF_GL, nparams=GL(L), synapse=syn, sparams=prm)
    r = sp.Reservoir(cfg, seed=1)
    l = r.launch()
    r.close()
    width = (n + l.ctas - 1) // l.ctas
    assert l.variant == 1 and l.stages >= 2
    if 2 * 48 * width * 8 <= 160 * 1024:
        assert l.stages <= 3 and l.stages * l.rows * width * 8 <= 160 * 1024


@pytest.mark.parametrize("n,edges,clustered", [(1000, 100, True), (2000, 12, True), (2000, 40, False),
                                               (4000, 4, False)])
def test_heterogeneous_synapses_leave_the_cluster(n, edges, clustered):
    """PSC_HETEROGENEOUS walks every edge in every step: a cluster where its CTAs have few
    warps and edges, else the wide launch; both as the oracle."""
    cfg = sp.make_config(n, 2, 2, rho=1.3, ei=0.55, gamma=1.2, conn=edges / n, dt=1.0,
                         topo=sp.CONN_SMALL_WORLD, neuron=sp.LIF_DISCRETE,
                         nparams=O.NEURON_PARAMS[sp.LIF_DISCRETE], synapse=sp.SYN_PSC_HET,
                         sparams=(1.0, 10.0))
    r = sp.Reservoir(cfg, seed=11)
    assert (r.launch().ctas == 16) == clustered
    run_against_oracle(r, cfg, 12, 11)


def test_stages_leave_the_coefficients_an_l1():
    """More coefficients than are staged (8192): the stages leave the L1 room for them, and
    the sums through them are the oracle's."""
    n = 70
    cfg = sp.make_config(n, 2, 2, rho=1.3, ei=0.55, gamma=1.2, conn=0.2, dt=1.0,
                         topo=sp.CONN_RANDOM, neuron=sp.FLIF_GL, nparams=GL(8300))
    r = sp.Reservoir(cfg, seed=11)
    l = r.launch()
    assert l.variant == 1 and 2 <= l.stages
    assert l.stages * l.rows * 32 * l.warps_max * 8 <= 144 * 1024
    run_against_oracle(r, cfg, 90, 11)

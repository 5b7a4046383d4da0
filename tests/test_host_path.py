"""The host code without a GPU, on a stand-in for the CUDA runtime that takes
what CUDA leaves open at its worst (tests/cpp/fake_cuda.cpp)."""
import ctypes as C

import numpy as np
import pytest

import fake_gpu
from moose_gb300 import models
from moose_gb300.abi import HS_PREC_FP64, HS_PREC_MIXED
from moose_gb300.batch import Batch
from moose_gb300.hsolve import HSolve, Tick

DT = 25e-6
KCA = models.kca_2d_tables(vdivs=30, cadivs=30)


@pytest.fixture
def gpu():
    with fake_gpu.load() as L:
        yield L


def _cell(n=40, seed=3, **kw):
    rng = np.random.default_rng([seed, n])
    parent, d, length = models.branched_morphology(rng, n, 0.5, 4)
    return models.active_cell(parent, d, length, rng=rng, kca_tables=KCA, **kw)


def test_reads_wait_for_their_copy(gpu):
    """Vm and Ca of a read whose copy is still under way when the call that
    queued it returns, as one to pageable memory may be."""
    m = _cell()
    h = HSolve(m, dt=DT)
    h.target = m.seed
    h.reinit(DT)
    gpu.fake_lazy(1, 0)
    assert np.array_equal(h.vm(), m.initVm)
    assert np.array_equal(h.ca(), m.pool_CaBasal)
    h.close()


def test_batch_shares_rate_tables_of_one_shape_only(gpu):
    """Two cells of an FP64 batch whose rate tables hold the same numbers, in
    30 rows of one gate and in 10 of three: each gets the rows and differences
    of its own shape (in the other's, the last rows are out of range)."""
    cells = []
    for species, divs in ((1, 28), (3, 8)):
        m = models.config1_cell(n_cable=3)          # Na (gates 0, 1) and K (gate 2) in turn
        m.gates = [(models.VMIN, models.VMAX, np.full(divs + 1, 2.0), np.full(divs + 1, 4.0))] * 3
        if species == 1:
            for name in [a for a in vars(m) if a.startswith("chan_")]:
                setattr(m, name, getattr(m, name)[1::2].copy())
        cells.append(m)
    b = Batch(cells, DT, HS_PREC_FP64)
    b.reinit(DT)
    shape = (C.c_uint32 * 2)()
    at = []
    for k, (cols, rows) in enumerate([(2, 30), (6, 10)]):
        p = gpu.fake_table(k, shape)
        assert tuple(shape) == (cols, rows)
        got = np.ctypeslib.as_array(p, (rows - 1, cols, 2))
        assert np.array_equal(got, np.tile([[2.0, 0.0], [4.0, 0.0]], (rows - 1, cols // 2, 1)))
        at.append(C.addressof(p.contents))
    assert at[0] != at[1]
    b.close()


def test_shared_memory_limit_is_the_devices_and_stays(gpu):
    """A kernel's limit of dynamic shared memory belongs to the function: it
    is set to all that the device has beside the kernel's own arrays, per
    kernel and device, and no later launch lowers it."""
    room = 232448
    for kernel in (0x10000, 0x20400):           # without and with 1,024 bytes of its own
        for dev in (0, 1):
            assert gpu.fake_limit(kernel, dev) == 48 * 1024
            for _ in range(2):
                assert gpu.fake_allow(kernel, dev) == 0
                assert gpu.fake_limit(kernel, dev) == room - (kernel & 0xFFFF)


@pytest.mark.parametrize("kind", ["dropin", "batch"])
def test_uploads_read_their_source_late(gpu, kind):
    """What creating a solver or an FP64 batch leaves on the device is the same
    when the copies to it read the host's memory only at the next wait."""
    # (tables, programs and parameters on both sides of the size sent by itself)
    cells = [models.config1_cell(n_cable=200), _cell(60), _cell(1500, n_syn=30)]

    def digest(lazy):
        gpu.fake_digest(0)
        gpu.fake_lazy(0, lazy)
        if kind == "dropin":
            made = []
            for m in cells:
                made.append(HSolve(m, dt=DT))
                made[-1].target = m.seed
        else:
            made = [Batch(cells, DT, HS_PREC_FP64)]
        h = gpu.fake_digest(len(cells) * gpu.fake_cell_bytes())
        gpu.fake_lazy(0, 0)
        for x in made:
            x.close()
        return h
    now = digest(0)
    assert digest(0) == now
    assert digest(1) == now


def test_reads_after_a_group_wait_once_and_query_nothing(gpu):
    """Of a group's solvers the first is on the launch's stream, the second's
    read waits for the launch, and the others' know that it is over; none asks
    by a query, which a thread that captures a graph may not make."""
    cells = [_cell(20 + i) for i in range(6)]
    solvers = []
    for m in cells:
        solvers.append(HSolve(m, dt=DT))
        solvers[-1].target = m.seed
        solvers[-1].reinit(DT)
    tick = Tick(solvers)
    for _ in range(2):
        tick.process(3)
        q, w = gpu.fake_queries(), gpu.fake_waits()
        for h, m in zip(solvers, cells):
            assert np.array_equal(h.vm(), m.initVm)
        assert (gpu.fake_queries() - q, gpu.fake_waits() - w) == (0, 1)
    for h in solvers:
        h.close()


@pytest.mark.parametrize("n", [300, 3000, 9001])
@pytest.mark.parametrize("asked, warps", [(0, 8), (3, 6), (6, 12)])
def test_eliminators_of_a_cluster(gpu, n, asked, warps):
    """Twice the batch's eliminator warps, whatever the cell's size: the rule of
    one CTA's forests, which have a CTA's threads and no more, is not theirs."""
    b = Batch([_cell(n)], DT, HS_PREC_MIXED, cluster_ctas=4, max_ctas=4, elim_warps=asked)
    b.reinit(DT)
    b.process(1)
    assert gpu.fake_elim_warps() == warps
    b.close()


def test_pairs_are_as_few_as_the_nodes_need(gpu):
    """One cell nearly as large as a pair of forests may be, and many small
    ones: a lone forest and one pair, not a pair per handful of small cells."""
    cells = [_cell(10700)] + [_cell(5 + i % 7, seed=i) for i in range(400)]
    b = Batch(cells, DT, HS_PREC_MIXED, max_ctas=1)
    assert (b.info()["n_forests"], b.info()["n_shared_forests"]) == (3, 3)
    b.close()


# a CTA's cells: one shared forest, a pair of forests, one merged in global memory
CTAS = {"shared": ([2000, 900], (1, 1)), "pair": ([5000, 4000], (2, 2)), "merged": ([12000, 9000, 8000], (1, 0))}


def _forests(b):
    return b.info()["n_forests"], b.info()["n_shared_forests"]


@pytest.mark.parametrize("kind", CTAS)
def test_layout_does_not_depend_on_the_tunings_before(gpu, kind):
    """threads_per_cta and elim_warps change without a new layout, so the same
    one is made for all of them, whichever came first."""
    sizes, forests = CTAS[kind]
    cells = [_cell(n) for n in sizes]
    tunings = [dict(), dict(elim_warps=4), dict(elim_warps=8), dict(threads_per_cta=512), dict(threads_per_cta=128)]
    for t in tunings:
        b = Batch(cells, DT, HS_PREC_MIXED, max_ctas=1, **t)
        assert _forests(b) == forests, t
        for t2 in tunings:
            b.tune(max_ctas=1, **t2)
            assert _forests(b) == forests, (t, t2)
            b.tune(max_ctas=2, **t2)
            b.tune(max_ctas=1, **t)             # laid out again
            assert _forests(b) == forests, (t, t2)
        b.close()


@pytest.mark.parametrize("kind, asked, warps", [("shared", 0, 7), ("shared", 3, 3), ("pair", 0, 6), ("pair", 2, 4),
                                                ("pair", 5, 5), ("pair", 9, 6), ("merged", 0, 10), ("merged", 4, 10),
                                                ("merged", 12, 12)])
@pytest.mark.parametrize("stops", [False, True])
def test_eliminators_by_layout(gpu, kind, asked, warps, stops):
    cells = [_cell(n) for n in CTAS[kind][0]]
    b = Batch(cells, DT, HS_PREC_MIXED, max_ctas=1, elim_warps=asked)
    if stops:
        b.set_stop_steps([100] * len(cells))
    b.reinit(DT)
    b.process(1)
    assert gpu.fake_elim_warps() == warps
    b.close()


def test_one_very_large_cell_leaves_the_others_in_shared_memory(gpu):
    b = Batch([_cell(22000)] + [_cell(900, seed=i) for i in range(4)], DT, HS_PREC_MIXED, max_ctas=3)
    assert _forests(b) == (3, 2)
    b.close()


@pytest.mark.parametrize("n", [1, 2, 3, 40, 300])
def test_every_cell_has_its_forward_program(gpu, n):
    """A cell of one compartment has waves, but none of them."""
    for m in ([models.config1_cell(n_cable=n - 1)] if n > 1 else []) + [_cell(n)]:
        h = HSolve(m, dt=DT)
        h.target = m.seed
        h.reinit(DT)
        assert gpu.fake_has_forward(0) == 1
        h.close()


@pytest.mark.parametrize("p, nodes, warps", [(0.03, 3500, 4), (0.5, 3500, 7), (0.5, 200, 4)])
def test_eliminators_by_the_width_of_the_levels(gpu, p, nodes, warps):
    """A shared forest's eliminators by its nodes per level: a long sparse tree of
    many nodes has narrow levels."""
    rng = np.random.default_rng(nodes)
    parent, d, length = models.branched_morphology(rng, nodes, p, 3)
    b = Batch([models.active_cell(parent, d, length, rng=rng, kca_tables=KCA)], DT, HS_PREC_MIXED)
    b.reinit(DT)
    b.process(1)
    assert gpu.fake_elim_warps() == warps
    b.close()


@pytest.mark.parametrize("n, count, tuning, teams", [(30, 3000, {}, (16, 32)), (100, 300, {}, (4, 128)),
                                                     (900, 40, {}, (4, 128)), (30, 3000, dict(threads_per_cta=64, ctas_per_sm=2), (4, 32)),
                                                     (30, 3000, dict(threads_per_cta=96, ctas_per_sm=2), (2, 96)),
                                                     (12, 3000, dict(threads_per_cta=32, ctas_per_sm=8), (8, 32))])
def test_teams_of_the_fp64_batch(gpu, n, count, tuning, teams):
    """Small cells, many to a block, are stepped by more and smaller teams of as
    many threads."""
    b = Batch([_cell(n)] * count, DT, HS_PREC_FP64, **tuning)
    b.reinit(DT)
    b.process(1)
    got = (C.c_uint32 * 2)()
    gpu.fake_teams(C.byref(got), C.byref(got, 4))
    assert tuple(got) == teams
    b.close()


@pytest.mark.parametrize("n, warps", [(1700, 4), (9000, 10)])
def test_eliminators_of_global_forests_by_the_width_of_the_levels(gpu, n, warps):
    """Five CTAs an SM leave shared memory for ~1,400 nodes."""
    rng = np.random.default_rng(n)
    parent, d, length = models.branched_morphology(rng, n, 0.06 if warps == 4 else 0.5, 3)
    b = Batch([models.active_cell(parent, d, length, rng=rng, kca_tables=KCA)], DT, HS_PREC_MIXED, ctas_per_sm=5)
    b.reinit(DT)
    b.process(1)
    assert _forests(b) == (1, 0)
    assert gpu.fake_elim_warps() == warps
    b.close()

"""The host code without a GPU, on a stand-in for the CUDA runtime that takes
what CUDA leaves open at its worst (tests/cpp/fake_cuda.cpp)."""
import numpy as np
import pytest

import fake_gpu
from moose_gb300 import models
from moose_gb300.hsolve import HSolve

DT = 25e-6


@pytest.fixture
def gpu():
    with fake_gpu.load() as L:
        yield L


def _cell(n=40, seed=3, **kw):
    rng = np.random.default_rng([seed, n])
    parent, d, length = models.branched_morphology(rng, n, 0.5, 4)
    return models.active_cell(parent, d, length, rng=rng, kca_tables=models.kca_2d_tables(vdivs=30, cadivs=30), **kw)


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

"""Host threads with a solver or a batch each: a launch must not depend on what
another thread launches between its calls (a kernel's limit of dynamic shared
memory is the function's).  Each thread steps cells of its own size; results
are those of the same cells stepped by one thread, bit for bit."""
import threading

import numpy as np
import pytest

from moose_gb300 import models
from moose_gb300.abi import HS_PREC_FP64, HS_PREC_MIXED
from moose_gb300.batch import Batch
from moose_gb300.hsolve import HSolve

pytestmark = pytest.mark.gpu

DT = 25e-6
ROUNDS = 60


def _cell(n):
    rng = np.random.default_rng([91, n])
    parent, d, L = models.branched_morphology(rng, n, 0.5, 4)
    return models.active_cell(parent, d, L, inject=0.7e-9, rng=rng, kca_tables=models.kca_2d_tables(vdivs=100, cadivs=100))


def _dropin(n):
    h = HSolve(_cell(n), dt=DT)
    h.target = h.model.seed
    h.reinit(DT)
    return h, h.vm


def _batch(n, precision):
    b = Batch([_cell(n)], DT, precision, steps_per_launch=2)
    b.reinit(DT)
    return b, lambda: b.vm(0)


MAKERS = {
    "dropin": _dropin,
    "fp64": lambda n: _batch(n, HS_PREC_FP64),
    "mixed": lambda n: _batch(n, HS_PREC_MIXED),
}


@pytest.mark.parametrize("kind, sizes", [("dropin", (3500, 5000)), ("fp64", (1500, 4500)),
                                         ("mixed", (2000, 6000))])
def test_threads_step_cells_of_two_sizes(kind, sizes):
    def steps(n, out, go=None):
        try:
            s, vm = MAKERS[kind](n)
            if go:
                go.wait()
            for _ in range(ROUNDS):
                s.process(3)
            out[n] = vm().copy()
            s.close()
        except Exception as e:            # a refused launch
            out[n] = e
    alone, both = {}, {}
    for n in sizes:
        steps(n, alone)
    go = threading.Barrier(2, timeout=60)
    threads = [threading.Thread(target=steps, args=(n, both, go)) for n in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for n in sizes:
        assert not isinstance(both[n], Exception), both[n]
        assert np.array_equal(both[n], alone[n])

"""Forests of a CTA stepped in pairs (the mixed batch's layout where a CTA's
cells do not fit one shared-memory forest): two groups of eliminator warps,
the others assembling the one forest, then the other.  Every node's arithmetic
is that of the unsplit step, so the results must be those of the same cells
stepped so in global memory, bit for bit: Vm, Ca, traces and spikes, with stop
steps, synapses and step currents."""
import numpy as np
import pytest

from moose_gb300 import models
from moose_gb300.abi import HS_PREC_MIXED
from moose_gb300.batch import Batch

pytestmark = pytest.mark.gpu

DT = 25e-6
OFF = 0xFFFFFFFF


def _cells(sizes):
    kca = models.kca_2d_tables(vdivs=200, cadivs=200)
    cells = []
    for i, n in enumerate(sizes):
        if n < 0:                  # an unbranched cable
            cells.append(models.config1_cell(n_cable=-n))
            continue
        rng = np.random.default_rng([73, n, i])
        parent, d, L = models.branched_morphology(rng, n, 0.5, 4)
        cells.append(models.active_cell(parent, d, L, inject=float(rng.uniform(0.4e-9, 1.2e-9)), n_syn=min(n, 30),
                                        rng=rng, t_end=0.02, kca_tables=kca, syn_rate=60.0))
    return cells


def _run(cells, stops, tune=None, **tuning):
    n = len(cells)
    b = Batch(cells, DT, HS_PREC_MIXED, max_ctas=1, forest_nodes=8, steps_per_launch=70, **tuning)
    if tune:
        b.tune(max_ctas=1, forest_nodes=8, **tune)
    b.record(np.arange(n), np.zeros(n, np.uint32), 10, 60)
    if stops:
        b.set_stop_steps([400 - 90 * (i % 3) for i in range(n)])
    b.reinit(DT)
    for k in (1, 249, 150):
        b.process(k)
    b.sync()
    out = dict(vm=[b.vm(i) for i in range(n)], ca=[b.ca(i) for i in range(n)], trace=b.trace()[0],
               spikes=b.spikes(), forests=b.info()["n_forests"])
    b.close()
    return out


# sizes (negative: a cable), forests of the paired layout
LAYOUTS = [
    ((8000,), 1),                           # a lone forest
    ((5000, 4000), 2),
    ((8000, 40, 25, 3), 2),                 # the second far smaller, narrower than a warp
    ((9000, 6000, 2000), 3),                # more than one pair's shared memory: a pair, then a lone forest
    ((12000, 9000, 8000), 1),               # more than two pairs' nodes: one forest in global memory
    ((8000, -260), 1),                      # 256 levels or more: no pairs
]


@pytest.mark.parametrize("sizes, forests", LAYOUTS)
@pytest.mark.parametrize("stops", [False, True])
def test_paired_forests_bit_identical_to_global_forests(sizes, forests, stops):
    cells = _cells(sizes)
    ref = _run(cells, stops, elim_warps=OFF)
    _same(_run(cells, stops), ref, forests)


@pytest.mark.parametrize("tune", [dict(threads_per_cta=640), dict(threads_per_cta=160), dict(threads_per_cta=64),
                                  dict(elim_warps=1), dict(elim_warps=OFF)])
def test_paired_layout_steps_with_any_tuning(tune):
    cells = _cells((5000, 4000, 20))
    _same(_run(cells, True, tune=tune), _run(cells, True, elim_warps=OFF), 2)


def _same(got, ref, forests):
    assert got["forests"] == forests
    for i in range(len(ref["vm"])):
        assert np.array_equal(got["vm"][i], ref["vm"][i]), i
        assert np.array_equal(got["ca"][i], ref["ca"][i]), i
    assert np.array_equal(got["trace"], ref["trace"])
    spikes = lambda sp: sorted(zip(sp[0].tolist(), sp[1].tolist(), sp[2].tolist()))
    assert spikes(got["spikes"]) == spikes(ref["spikes"])

"""Long cables around the sizes where their matrix and the runs' scratch no
longer fit one CTA's shared memory (2 N words and 2 N of scratch: ~7,200
compartments; the 16-bit programs end at 32,700): bit-identical to the oracle
alone, in a group and in an FP64 batch."""
import numpy as np
import pytest

from moose_gb300 import models
from moose_gb300.abi import HS_PREC_FP64
from moose_gb300.batch import Batch
from moose_gb300.hsolve import HSolve, process_group
from oracle import OracleCell

pytestmark = pytest.mark.gpu

DT = 25e-6
STEPS = 12


@pytest.mark.parametrize("n", [3600, 7100, 7350, 14600, 33000])
def test_long_cable_bit_identical_to_oracle(n):
    cells = [models.config1_cell(n_cable=k - 1, inject=0.7e-9, t_on=0.0, t_off=1.0) for k in (n, 300)]
    want = []
    for m in cells:
        o = OracleCell(m, DT)
        o.reinit(DT)
        o.step(STEPS)
        want.append(o.vm())
    solvers = []
    for m in cells * 2:
        h = HSolve(m, dt=DT)
        h.target = m.seed
        h.reinit(DT)
        solvers.append(h)
    solvers[0].process(STEPS)
    solvers[1].process(STEPS)
    process_group(solvers[2:], STEPS)
    b = Batch(cells, DT, HS_PREC_FP64)
    b.reinit(DT)
    b.process(STEPS)
    for k, h in enumerate(solvers):
        assert np.array_equal(h.vm(), want[k % 2]), k
        h.close()
    for k in range(2):
        assert np.array_equal(b.vm(k), want[k])
    b.close()

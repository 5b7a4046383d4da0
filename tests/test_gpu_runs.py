"""Cable runs shared by the lanes of a warp (csrc/hs_fp64.cu, forwardWarpRun
and backwardWarpRun) on the GPU: bit-identical to the oracle's serial sweeps
at the lengths where the pieces change (around 64 rows and multiples of 32),
with segments so short that a pivot's error hardly shrinks from row to row
(every piece is then walked again and again), so long that rows hardly
couple, and on long tails of a branched cell; the FP64 batch steps the same
cells bit-identically."""
import numpy as np
import pytest

from moose_gb300 import models
from moose_gb300.abi import HS_PREC_FP64
from moose_gb300.batch import Batch
from moose_gb300.hsolve import HSolve
from oracle import OracleCell

pytestmark = pytest.mark.gpu

DT = 25e-6


def hh_cell(parent, d, L):
    m = models.config1_cell(n_cable=len(parent) - 1, inject=0.7e-9, t_on=0.0, t_off=1.0)
    m.parent = np.ascontiguousarray(parent, np.int32)
    m.Ra, m.Rm, m.Cm, area = models.passive(d, L)
    m.chan_Gbar[0::2] = 1200.0 * area
    m.chan_Gbar[1::2] = 360.0 * area
    return m


def cable(n, seg_len, seed=0):
    parent, d, L = models.cable_morphology(n - 1, seg_len=seg_len)
    d = d * np.random.default_rng(seed).uniform(0.7, 1.4, n)
    return hh_cell(parent, d, L)


@pytest.mark.parametrize("seg_len", [0.2e-6, 10e-6, 400e-6])
@pytest.mark.parametrize("n", [64, 65, 66, 97, 201, 1000])
def test_cable_bit_identical_to_oracle(n, seg_len):
    m = cable(n, seg_len, n)
    h, o = HSolve(m, dt=DT), OracleCell(m, DT)
    h.target = m.seed
    h.reinit(DT)
    o.reinit(DT)
    for k in (1, 3, 56):
        h.process(k)
        o.step(k)
        assert np.array_equal(h.vm(), o.vm())
    h.close()


def test_tails_of_a_branched_cell():
    # a soma with a 150-row and a 70-row tail and a fork half way down the first
    parent = [-1] + list(range(0, 150)) + [0] + list(range(151, 220)) + [75]
    m = hh_cell(parent, np.full(len(parent), 2e-6), np.full(len(parent), 8e-6))
    cells = [m, cable(130, 10e-6), cable(300, 3e-6)]
    b = Batch(cells, DT, HS_PREC_FP64)
    b.reinit(DT)
    b.process(80)
    for seed in (0, 150, 220):
        m.seed = seed
        h, o = HSolve(m, dt=DT), OracleCell(m, DT, seed=seed) if seed else OracleCell(m, DT)
        h.target = seed
        h.reinit(DT)
        o.reinit(DT)
        h.process(80)
        o.step(80)
        assert np.array_equal(h.vm(), o.vm())
        h.close()
    for i, c in enumerate(cells):
        c.seed = 0
        o = OracleCell(c, DT)
        o.reinit(DT)
        o.step(80)
        assert np.array_equal(b.vm(i), o.vm())
    b.close()

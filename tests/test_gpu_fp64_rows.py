"""FP64 product rows by 4 to 32 lanes (spmv_row, csrc/step_rows.cuh): rows of an odd
number of bonds, fewer bonds than lanes, one and two bonds in flight, a single
row per block, Dirichlet and contact rows, bonds broken -- against the oracle's
assembled matrix.  A row sums at most 122 products of three in 64 bits: within
(3 * 122 + 10) * 2^-53 = 4e-14 of the largest value, and its matrix entries
within a few more: 1e-12, the bound of the other FP64 operator test."""
import numpy as np
import pytest

from helpers import apply_on_device, make_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [0, 4, 8, 16, 32])
@pytest.mark.parametrize("n_side,expansion", [(1, 150.0), (2, 150.0), (3, 300.0), (8, 300.0), (13, 150.0)])
def test_fp64_rows(pdgb, scenes, n_side, expansion, lanes):
    sc = scenes.reference_block(n_side=n_side, integrator=pdgb.NEWMARK_BETA, adaptive=1, expansion=expansion, cg_tol=1e-10)
    sc.opt.precision = pdgb.PRECISION_FP64
    sc.opt.lanes_per_particle = lanes
    sim = scenes.make_simulator(sc)
    sim.makeReady()
    ora = make_oracle(sc)
    sim.advance(33)
    ora.advance(33)
    x = np.zeros((sc.n, 4))
    x[:, :3] = np.random.default_rng(5).standard_normal((sc.n, 3))
    y, dot, xs = apply_on_device(pdgb, sim, x)
    ref = ora.apply_A(xs)
    assert np.abs(y[:, :3] - ref[:, :3]).max() <= 1e-12 * np.abs(ref[:, :3]).max()
    assert np.all(y[:, 3] == 0.0)
    assert abs(dot - float(np.sum(xs[:, :3] * ref[:, :3]))) <= 1e-12 * abs(dot)

"""Stretch limits sampled on the device (csrc/stretch.cu) against the host's
serial generator, bit for bit: sizes around a thread's run of 8 particles, a
block's 2048 and several blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 2047, 2048, 2049, 4097, 70001])
def test_sampled_limits_are_the_serial_ones(pdgb, scenes, n):
    sc = scenes.cube_lattice(n_side=2)
    sc.pos = np.zeros((n, 4))
    sc.pos[:, 0] = np.arange(n) * 0.02
    sc.vel = np.zeros((n, 4))
    sc.act = np.full(n, scenes.ACTIVE, np.int32)
    sc.sim.num_pd_particle = n
    sc.run.pd_stretch_limit_s0 = 0.0173
    sim = scenes.make_simulator(sc)
    sim.makeReady()
    np.testing.assert_array_equal(sim.get(pdgb.VAR_ORIGINAL_STRETCH).ravel(), pdgb.sample_stretch_limits(0.0173, n))

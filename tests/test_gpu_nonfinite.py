"""Non-finite entries of a caller's vector reach the rows that are bonded to them
and no others: in the products by tiles a broken bond's partner (its slot stays in
the row, beyond the live ones) takes no part, as in the gather product."""
import numpy as np
import pytest

from helpers import apply_on_device

pytestmark = pytest.mark.gpu


def _body(scenes, n, jitter):
    """A clamped-base cube of n^3 sites that one step of stretching breaks bonds of."""
    sc = scenes.cube_lattice(n_side=2, coeff=5.0)
    z, y, x = np.meshgrid(*[np.arange(n)] * 3, indexing="ij")
    g = np.stack([x.ravel(), y.ravel(), z.ravel()], axis=1)
    sc.pos = np.zeros((n ** 3, 4))
    sc.pos[:, :3] = (g + np.random.default_rng(1).uniform(-jitter, jitter, g.shape)) * 0.02
    sc.vel = np.zeros((n ** 3, 4))
    sc.vel[:, 0] = 300.0 * sc.pos[:, 0]
    sc.act = np.where(g[:, 2] == 0, scenes.CLAMPED, scenes.ACTIVE).astype(np.int32)
    sc.sim.num_pd_particle = n ** 3
    sc.run.pd_stretch_limit_s0 = 0.005
    sc.run.integrator = scenes.NEWMARK_BETA
    sc.opt.phase_in_steps = 0
    return sc


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("n,jitter", [(35, 0.05), (56, 0.4)])
@pytest.mark.parametrize("lanes", [0, 8])
def test_broken_bonds_partner(pdgb, scenes, n, jitter, value, lanes):
    """The tiles of the one-launch solve and larger ones (lanes 0), and the gather."""
    sc = _body(scenes, n, jitter)
    sc.opt.lanes_per_particle = lanes
    sim = scenes.make_simulator(sc)
    sim.makeReady()
    sim.advance(3)
    count = np.diff(sim.get(pdgb.VAR_BOND_ROW_PTR))
    live = sim.get(pdgb.VAR_BOND_COUNT)
    broken = np.flatnonzero(live < count)
    assert len(broken) > 200
    at = np.random.default_rng(4).choice(broken, 100, replace=False)
    x = np.zeros((sc.n, 4))
    x[:, :3] = np.random.default_rng(5).standard_normal((sc.n, 3))
    x[at, :3] = value
    y, _, _ = apply_on_device(pdgb, sim, x)
    reached = np.zeros(sc.n, bool)
    reached[at] = True
    sets = sim.alive_sets()
    for p in at:
        reached[sets[p]] = True
    np.testing.assert_array_equal(~np.isfinite(y[:, :3]).all(axis=1), reached & (sc.act == scenes.ACTIVE))

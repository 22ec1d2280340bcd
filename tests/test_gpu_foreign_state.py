"""A state of another body with the same particle and bond-slot counts: the handle
takes it and goes on as the body that it belongs to, on routes that hold its
rows.  (This body's one-launch solve keeps a block's bonds in shared memory
sized by this body's longest row, its stencil product a table of this body's
bond offsets.)"""
import numpy as np
import pytest

from helpers import apply_on_device, rel_err, same_sets

pytestmark = pytest.mark.gpu
H = 0.02
TOL = {0: 1e-5, 1: 1e-9}   # (the bounds of the parity tests: the two solves sum in other orders)


def _scene(scenes, sites, coeff, precision, path, folder):
    """Pieces at lattice sites, every piece far from the others."""
    sc = scenes.cube_lattice(n_side=2, coeff=coeff)
    g = np.concatenate(sites).astype(np.float64)
    n = len(g)
    sc.pos = np.zeros((n, 4))
    sc.pos[:, :3] = (g + np.random.default_rng(3).uniform(-0.05, 0.05, (n, 3))) * H
    sc.vel = np.zeros((n, 4))
    sc.vel[:, 0] = sc.pos[:, 0] % 0.37
    sc.act = np.full(n, scenes.ACTIVE, np.int32)
    sc.sim.num_pd_particle = n
    sc.run.saving_path = str(folder).encode()
    sc.opt.precision = precision
    sc.opt.spmv_path = path
    sc.opt.cg_relative_tolerance = 1e-10 if precision else 1e-6
    return sc


def _goes_on(pdgb, scenes, own, other, path_after):
    """The other body's state in a handle of this body against its own handle."""
    a, b = scenes.make_simulator(own), scenes.make_simulator(other)
    a.makeReady()
    b.makeReady()
    a.advance(1)
    b.advance(2)
    b.dataIO_saveState(2)
    a.dataIO_loadState(2)
    assert a.params()[2].spmv_path == path_after
    for s in (a, b):
        s.advance(3)
        assert s.stats().cg_converged == 1
    assert same_sets(a.alive_sets(), b.alive_sets())
    np.testing.assert_array_equal(a.get(pdgb.VAR_ORIGINAL_POSITION), b.get(pdgb.VAR_ORIGINAL_POSITION))
    p = own.opt.precision
    assert rel_err(a.get(pdgb.VAR_POSITION), b.get(pdgb.VAR_POSITION)) < TOL[p]
    return a


@pytest.mark.parametrize("precision", [0, 1])
def test_longer_rows_in_a_block(pdgb, scenes, precision, tmp_path):
    """34 pieces of 9 (rows of 8 slots) against 9 of 17 (16 slots) and 153 single
    particles: 306 particles and 2448 slots each."""
    plate = np.array([(x, y, 0) for y in range(3) for x in range(3)])
    brick = np.array([(x, y, z) for z in range(2) for y in range(3) for x in range(3)])[:17]
    far = np.array([20, 0, 0])
    own = _scene(scenes, [plate + k * far for k in range(34)], 10.0, precision, 2, tmp_path)
    other = _scene(scenes, [brick + k * far for k in range(9)] + [[k * far] for k in range(9, 162)], 10.0, precision, 2,
                   tmp_path)
    assert own.n == other.n == 306
    _goes_on(pdgb, scenes, own, other, 2)


@pytest.mark.parametrize("apart", [4, 7])
def test_bond_offsets_off_the_stencil(pdgb, scenes, apart, tmp_path):
    """Pieces of two groups of four in the same slot order, rows of 8 slots; the
    groups are bonded with each other in the other body only.  By this body's
    sites those bonds reach three sites and more, where its stencil reaches one."""
    far = np.array([16, 0, 0])
    group = np.array([(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)])

    def pieces(shift):
        return [group + k * far + np.array(d) for k in range(40) for d in ((0, 0, 0), (shift, 0, 0))]

    own = _scene(scenes, pieces(apart), 5.0, 0, 3, tmp_path)
    other = _scene(scenes, pieces(3), 5.0, 0, 3, tmp_path)
    s = scenes.make_simulator(own)
    s.makeReady()
    o = scenes.make_simulator(other)
    o.makeReady()
    assert s.params()[2].spmv_path == o.params()[2].spmv_path == 3
    np.testing.assert_array_equal(s.get(pdgb.VAR_SLOT_PERMUTATION), o.get(pdgb.VAR_SLOT_PERMUTATION))
    s.advance(1)
    s.dataIO_saveState(1)
    same = scenes.make_simulator(own)
    same.makeReady()
    same.dataIO_loadState(1)
    assert same.params()[2].spmv_path == 3      # (its own state keeps the stencil)
    _goes_on(pdgb, scenes, own, other, 2)


def test_contact_rows_in_another_slot_order(pdgb, scenes, tmp_path):
    """A state saved in the bricks' slot order, taken by a handle with the builder's:
    the rest positions that the contact term of a row reads follow it."""
    sc = scenes.impact_body(9000, "ball", coeff=5.0, speed=5.0, seed=2)   # (the sphere touches it)
    sc.run.saving_path = str(tmp_path).encode()
    x = np.zeros((sc.n, 4))
    x[:, :3] = np.random.default_rng(2).standard_normal((sc.n, 3))
    y = {}
    for path in (3, 2):
        sc.opt.spmv_path = path
        s = scenes.make_simulator(sc)
        s.makeReady()
        if path == 3:
            s.advance(2)
            s.dataIO_saveState(2)
        else:
            s.dataIO_loadState(2)
        s.advance(1)
        y[path] = apply_on_device(pdgb, s, x)[0]
    # (sums of at most 122 terms in 32 bits: each within 132 * 2^-24 of the largest value)
    assert np.abs(y[2] - y[3]).max() <= 2e-5 * np.abs(y[3]).max()

"""The products that make_ready chooses by size and shape, each against the
gather product of a fixed shape (spmv_path 2, 8 lanes, 1 bond at a time): the
lattice stencil at the edges of its bricks and at horizons of one to three
sites, and the tiles of the one-launch solve (csrc/cg_persist.cu) on either side
of the size where they take over, for lattice fills and scattered bodies, with
bonds broken.  Both sum a row's bonds (at most 122) in 32 bits: each is within
(122 + 10) * 2^-24 = 8e-6 of the largest value, so the two within 2e-5."""
import numpy as np
import pytest

from helpers import apply_on_device

pytestmark = pytest.mark.gpu
TOL = 2e-5


def _body(scenes, nx, ny, nz, coeff, jitter=0.05, seed=1):
    """A clamped-base block of nx * ny * nz sites (ragged ends: its last row along x is cut)."""
    sc = scenes.cube_lattice(n_side=2, coeff=coeff)
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    g = np.stack([x.ravel(), y.ravel(), z.ravel()], axis=1)[:-1 if nx * ny * nz > 2 else None]
    rng = np.random.default_rng(seed)
    n = len(g)
    sc.pos = np.zeros((n, 4))
    sc.pos[:, :3] = (g + rng.uniform(-jitter, jitter, (n, 3))) * 0.02
    sc.vel = np.zeros((n, 4))
    sc.vel[:, 0] = 300.0 * sc.pos[:, 0]       # 3 % of strain a step: some bonds break
    sc.act = np.where(g[:, 2] == 0, scenes.CLAMPED, scenes.ACTIVE).astype(np.int32)
    sc.sim.num_pd_particle = n
    sc.run.pd_stretch_limit_s0 = 0.005
    sc.run.integrator = scenes.NEWMARK_BETA
    sc.opt.phase_in_steps = 0                 # (limits in force from the first step)
    return sc


def _handle(scenes, sc, path, load=None):
    """path 2: the gather product of the fixed shape."""
    sc.opt.spmv_path = path
    sc.opt.lanes_per_particle, sc.opt.spmv_unroll = (8, 1) if path == 2 else (0, 0)
    sim = scenes.make_simulator(sc)
    sim.makeReady()
    if load is None:
        sim.advance(1)   # (the operator of a step, at the positions that it began with)
    else:
        sim.dataIO_loadState(load)
    return sim


def _compare(pdgb, sim, gather, n):
    """Both handles' products of the same state."""
    x = np.zeros((n, 4))
    x[:, :3] = np.random.default_rng(2).standard_normal((n, 3))
    (y, dot, _), (y2, dot2, _) = (apply_on_device(pdgb, s, x) for s in (sim, gather))
    np.testing.assert_array_equal(sim.get(pdgb.VAR_BOND_COUNT), gather.get(pdgb.VAR_BOND_COUNT))
    assert np.abs(y[:, :3] - y2[:, :3]).max() <= TOL * np.abs(y2[:, :3]).max()
    assert abs(dot - dot2) <= TOL * abs(dot2)


@pytest.mark.parametrize("coeff", [3.0, 4.0, 5.0, 6.0])
@pytest.mark.parametrize("dims", [(16, 8, 4), (17, 9, 5), (33, 15, 7), (3, 50, 11), (2, 2, 90), (1, 1, 40), (7, 6, 1), (2, 1, 1)])
def test_stencil_at_brick_edges(pdgb, scenes, dims, coeff):
    """Whole and partial bricks of 16 x 8 x 4 sites, bodies thinner than one, and
    those that the stencil leaves to the gather."""
    sc = _body(scenes, *dims, coeff)
    sim = _handle(scenes, sc, 3)
    assert sim.params()[2].spmv_path in (2, 3)
    if min(dims) >= 4:
        assert sim.params()[2].spmv_path == 3
    _compare(pdgb, sim, _handle(scenes, sc, 2), sc.n)


@pytest.mark.parametrize("jitter", [0.05, 0.4])
@pytest.mark.parametrize("n,coeff", [(24, 6.0), (29, 6.0), (38, 4.0), (35, 5.0), (48, 5.0), (50, 4.0)])
def test_tiles_of_the_one_launch_solve(pdgb, scenes, n, coeff, jitter, tmp_path):
    """14k to 125k rows: bonds kept in shared memory or not, products by the
    gather or the tiles, a ragged last block; and a state with broken bonds that
    both handles load."""
    sc = _body(scenes, n, n, n, coeff, jitter)
    sc.run.saving_path = str(tmp_path).encode()
    sim, gather = _handle(scenes, sc, 0), _handle(scenes, sc, 2)
    assert sim.params()[2].spmv_path == 2
    _compare(pdgb, sim, gather, sc.n)
    sim.advance(2)
    st = sim.stats()
    assert st.cg_graph_solves == 3 and st.cg_converged == 1
    assert st.bonds_alive < st.bonds_initial
    sim.dataIO_saveState(3)
    _compare(pdgb, _handle(scenes, sc, 0, load=3), _handle(scenes, sc, 2, load=3), sc.n)


def test_a_tile_of_two_distant_pieces(pdgb, scenes, tmp_path):
    """Rows of two blocks 300 spacings apart in one tile: more than 64 supercells,
    where a block keeps the decoded positions (kFixedReach, csrc/cg_persist.cu)."""
    a, b = _body(scenes, 27, 27, 27, 6.0), _body(scenes, 26, 26, 26, 6.0, seed=5)
    a.pos = np.concatenate([a.pos, b.pos + np.array([6.0, 0.0, 0.0, 0.0])])
    a.vel, a.act = np.concatenate([a.vel, b.vel]), np.concatenate([a.act, b.act])
    a.sim.num_pd_particle = len(a.pos)
    a.vel[:] = 0.0
    rows = -(-a.n // 152)
    assert 0 < 27 ** 3 % rows < rows   # (a tile of both, with 152 blocks)
    sim, gather = _handle(scenes, a, 0), _handle(scenes, a, 2)
    _compare(pdgb, sim, gather, a.n)
    sim.advance(2)
    st = sim.stats()
    assert st.cg_graph_solves == 3 and st.cg_converged == 1


@pytest.mark.parametrize("n,coeff,jitter", [(56, 5.0, 0.05), (61, 5.0, 0.4), (48, 6.0, 0.4), (80, 4.0, 0.4)])
def test_tiles_of_larger_bodies(pdgb, scenes, n, coeff, jitter, tmp_path):
    """110k to 512k rows that take no one-launch solve (or do, at 48 and 6.0):
    one or more tiles per SM in the products and in the CG's graph, a ragged last
    tile, and a state that both handles load."""
    sc = _body(scenes, n, n, n, coeff, jitter)
    sc.run.saving_path = str(tmp_path).encode()
    sim, gather = _handle(scenes, sc, 0), _handle(scenes, sc, 2)
    assert sim.params()[2].spmv_path == 2
    _compare(pdgb, sim, gather, sc.n)
    for s in (sim, gather):
        s.advance(1)
        assert s.stats().cg_converged == 1
    x, x2 = sim.get(pdgb.VAR_POSITION), gather.get(pdgb.VAR_POSITION)
    assert np.abs(x - x2).max() <= 1e-5 * np.abs(x2).max()   # (the bound of the mixed-precision parity tests)
    sim.dataIO_saveState(2)
    _compare(pdgb, _handle(scenes, sc, 0, load=2), _handle(scenes, sc, 2, load=2), sc.n)

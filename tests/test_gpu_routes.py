"""Which route a body takes (pd_get_routes, pd_batch_get_gangs), and the CUDA graph of
separate launches on bodies small enough for the one-launch solve: kept off it, they
run the gather product's while node and host-checked batches (one set of kernels, so
the two runs agree bit for bit), through bond breaking, rollbacks and the iteration
limit, and so do bodies that a preconditioner keeps off it.  The reference's solve is
the CUSP cg of Simulator::solveLinearSystem (src/core/simulator.cu:735-799)."""
import numpy as np
import pytest

from helpers import apply_on_device, assert_positions, make_oracle, same_sets

pytestmark = pytest.mark.gpu


def _ready(scenes, sc, one_launch=True):
    sim = scenes.make_simulator(sc)
    sim.set_one_launch(one_launch)
    sim.makeReady()
    return sim


def _cube(scenes, n, coeff, jitter=0.05, precision=0):
    """A clamped-base cube of n^3 sites."""
    sc = scenes.cube_lattice(n_side=2, coeff=coeff)
    z, y, x = np.meshgrid(*[np.arange(n)] * 3, indexing="ij")
    g = np.stack([x.ravel(), y.ravel(), z.ravel()], axis=1)
    sc.pos = np.zeros((n ** 3, 4))
    sc.pos[:, :3] = (g + np.random.default_rng(1).uniform(-jitter, jitter, g.shape)) * 0.02
    sc.vel = np.zeros((n ** 3, 4))
    sc.act = np.where(g[:, 2] == 0, scenes.CLAMPED, scenes.ACTIVE).astype(np.int32)
    sc.sim.num_pd_particle = n ** 3
    sc.opt.precision = precision
    return sc


@pytest.mark.parametrize("n,coeff,jitter,precision,one_launch,bonds_kept,tiles,lattice", [
    (17, 5.0, 0.05, 0, True, True, False, False),
    (24, 6.0, 0.05, 0, True, False, False, False),
    (35, 5.0, 0.05, 0, True, False, True, False),
    (48, 6.0, 0.4, 0, False, False, True, False),
    (56, 5.0, 0.05, 0, False, False, True, False),
    (56, 5.0, 0.4, 0, False, False, True, False),
    (64, 5.0, 0.05, 0, False, False, False, True),
    (64, 5.0, 0.4, 0, False, False, True, False),
    (14, 5.0, 0.05, 1, True, True, False, False),
    (23, 5.0, 0.05, 1, True, False, False, False),
    (40, 5.0, 0.05, 1, True, False, False, False),
    (56, 5.0, 0.05, 1, False, False, False, False)])
def test_route_by_size(pdgb, scenes, n, coeff, jitter, precision, one_launch, bonds_kept, tiles, lattice):
    sim = _ready(scenes, _cube(scenes, n, coeff, jitter, precision))
    r = sim.routes()
    assert (r.one_launch_blocks > 0, r.one_launch_bonds > 0, r.tile_blocks > 0, r.lattice == 1) == \
        (one_launch, bonds_kept, tiles, lattice)
    sim.advance(2)
    assert sim.routes().one_launch_solves == (2 if one_launch else 0)
    assert sim.stats().cg_graph_solves == 2


def test_route_by_option(pdgb, scenes):
    sc = _cube(scenes, 35, 5.0)
    assert _ready(scenes, sc, False).routes().one_launch_blocks == 0
    for field, value, tiles in (("preconditioner", 1, True), ("lanes_per_particle", 8, False), ("spmv_path", 3, False)):
        sc = _cube(scenes, 35, 5.0)
        setattr(sc.opt, field, value)
        r = _ready(scenes, sc).routes()
        assert (r.one_launch_blocks > 0) == (field == "lanes_per_particle")
        assert (r.tile_blocks > 0, r.lattice == 1) == (tiles, field == "spmv_path")


@pytest.mark.parametrize("sizes,gangs", [((500,), True), ((40, 3000, 9, 700), True), ((40000, 300, 52000, 9000), True),
                                         ((220000, 2000), False)])
def test_gangs_by_size(pdgb, scenes, sizes, gangs):
    b = pdgb.Batch(0)
    for k, n in enumerate(sizes):
        scenes.add_to_batch(b, scenes.impact_body(n, "block", coeff=5.0, speed=4.0, seed=k, steps=10))
    b.makeReady()
    count, blocks = b.gangs()
    assert (count > 0) == (blocks > 0) == gangs
    assert count <= len(sizes)


def test_no_gangs_in_fp64(pdgb, scenes):
    b = pdgb.Batch(0)
    scenes.add_to_batch(b, scenes.impact_body(600, "block", precision=1))
    b.makeReady()
    assert b.gangs() == (0, 0)


def _steps(sim, steps):
    iters, retries = [], 0
    for _ in range(steps):
        sim.advance(1)
        st = sim.stats()
        iters.append(st.last_cg_iterations)
        retries += st.retries_last_step
    return iters, retries


@pytest.mark.parametrize("preconditioner", [0, 2])
@pytest.mark.parametrize("precision", [0, 1])
def test_graph_equals_host_batches_on_the_gather_product(pdgb, scenes, precision, preconditioner):
    """Newmark with bond breaking and rollbacks (the time step halves and doubles)."""
    runs = {}
    for loop in (0, 1):
        sc = scenes.reference_block(n_side=9, seed=5, integrator=pdgb.NEWMARK_BETA, adaptive=1, expansion=150.0,
                                    cg_tol=1e-10)
        sc.opt.precision = precision
        sc.opt.preconditioner = preconditioner
        sc.opt.cg_loop = loop
        sim = _ready(scenes, sc, False)
        runs[loop] = (sim, *_steps(sim, 70))
    (g, ig, rg), (h, ih, rh) = runs[0], runs[1]
    assert ig == ih and rg == rh > 0
    sg, sh = g.stats(), h.stats()
    assert sg.bonds_alive < sg.bonds_initial
    assert sg.cg_graph_solves == 70 and sh.cg_graph_solves == 0
    assert g.routes().one_launch_solves == h.routes().one_launch_solves == 0
    # per integrate call the adaptive test; per kept step the solve's read-back
    assert sg.host_syncs == (70 + rg) + 70 < sh.host_syncs
    assert sg.time_step_ticks == sh.time_step_ticks
    assert same_sets(g.alive_sets(), h.alive_sets())
    np.testing.assert_array_equal(g.get(pdgb.VAR_POSITION), h.get(pdgb.VAR_POSITION))
    np.testing.assert_array_equal(g.get(pdgb.VAR_VELOCITY), h.get(pdgb.VAR_VELOCITY))
    if preconditioner == 0:
        ora = make_oracle(sc)
        ora.advance(70)
        assert same_sets(g.alive_sets(), ora.alive_sets())
        assert_positions(g.get(pdgb.VAR_POSITION), ora.position, sc.pos, precision, "graph of the gather product")


@pytest.mark.parametrize("interval", [1, 4, 16])
def test_one_wait_per_step_and_odd_intervals(pdgb, scenes, interval):
    """Implicit Euler without adaptivity: one host wait per step, whatever the body's length."""
    sc = scenes.cube_lattice(n_side=10, seed=2)
    sc.opt.cg_check_interval = interval
    sim = _ready(scenes, sc, False)
    sim.advance(20)
    st = sim.stats()
    assert st.cg_graph_solves == 20 and st.host_syncs == 20
    assert sim.routes().one_launch_solves == 0


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("loop", [0, 1])
def test_iteration_limit_ends_the_graph(pdgb, scenes, loop, precision):
    """The while node ends on the device's limit test; the handle stops advancing."""
    sc = scenes.cube_lattice(n_side=8, seed=1)
    sc.opt.precision = precision
    sc.opt.cg_max_iterations = 5
    sc.opt.cg_loop = loop
    sim = _ready(scenes, sc, False)
    sim.advance(3)
    st = sim.stats()
    assert st.last_cg_iterations == 5 and st.cg_converged == 0 and st.current_step == 1
    assert st.cg_graph_solves == (1 if loop == 0 else 0)
    assert sim.routes().one_launch_solves == 0


def test_a_tile_of_two_distant_pieces(pdgb, scenes):
    """A tile of the two cubes, 300 spacings apart, on any number of SMs: more than 64
    supercells, where a block keeps the decoded positions (kFixedReach)."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    a, b = _cube(scenes, 27, 6.0), _cube(scenes, 26, 6.0)
    while 27 ** 3 % -(-(a.n + b.n) // sms) == 0:   # (whole tiles of the first: drop a particle of the second)
        b.pos, b.vel, b.act = b.pos[:-1], b.vel[:-1], b.act[:-1]
        b.sim.num_pd_particle = len(b.pos)
    first = a.n
    a.pos = np.concatenate([a.pos, b.pos + np.array([6.0, 0.0, 0.0, 0.0])])
    a.vel, a.act = np.concatenate([a.vel, b.vel]), np.concatenate([a.act, b.act])
    a.sim.num_pd_particle = len(a.pos)
    sim = _ready(scenes, a)
    r = sim.routes()
    rows = -(-len(a.pos) // sms)
    assert r.one_launch_blocks > 0 and r.tile_blocks == -(-len(a.pos) // rows) and first % rows
    a.opt.lanes_per_particle, a.opt.spmv_unroll = 8, 1
    gather = _ready(scenes, a)
    assert gather.routes().tile_blocks == 0
    x = np.zeros((len(a.pos), 4))
    x[:, :3] = np.random.default_rng(2).standard_normal((len(a.pos), 3))
    for s in (sim, gather):
        s.advance(1)
    y, y2 = (apply_on_device(pdgb, s, x)[0] for s in (sim, gather))
    # (sums of at most 122 terms in 32 bits: each within 132 * 2^-24 of the largest value)
    assert np.abs(y - y2).max() <= 2e-5 * np.abs(y2).max()

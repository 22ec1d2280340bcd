"""A kernel whose wait runs out (csrc/lattice.cu, csrc/cg_persist.cu) ends the
solve and reports it.  The wait is made to run out by its limit (0: at once); the
copies it waited for arrive all the same and are waited for before the kernel
returns, so the handle works again after the next makeReady."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
PD_ERR_CUDA = 2


def _fails(pdgb, call):
    t0 = time.perf_counter()
    with pytest.raises(pdgb.PdError) as e:
        call()
    assert e.value.status == PD_ERR_CUDA and "ran out of time" in str(e.value)
    assert time.perf_counter() - t0 < 2.0   # (the waits' own limits are 1 and 5 s, a solve some hundred products)


def _recovers(pdgb, sim, steps, expected):
    sim.set_wait_limit(-1)
    _fails(pdgb, lambda: sim.advance(1))    # until the next makeReady
    sim.makeReady()
    sim.advance(steps)
    np.testing.assert_array_equal(sim.get(pdgb.VAR_POSITION), expected)


def _run(scenes, pdgb, sc, steps):
    sim = scenes.make_simulator(sc)
    sim.makeReady()
    sim.makeReady()   # (as _recovers: the bonds of a row stand in another order after the first)
    sim.set_wait_limit(10.0)
    sim.advance(steps)
    return sim, sim.get(pdgb.VAR_POSITION)


def _lattice_body(scenes, loop=0, warm_start=0):
    sc = scenes.ellipsoid_impact(target_n=30_000, gap=0.0, dt=5e-5 * (1e6 / 30_000) ** (1 / 3), steps=10)
    sc.opt.spmv_path = 3
    sc.opt.cg_loop = loop
    sc.opt.warm_start = warm_start
    return sc


@pytest.mark.parametrize("loop,warm_start", [(0, 0), (1, 0), (0, 2)])
def test_stencil_product_of_a_solve(pdgb, scenes, loop, warm_start):
    sim, x = _run(scenes, pdgb, _lattice_body(scenes, loop, warm_start), 2)
    assert sim.params()[2].spmv_path == 3
    sim.set_wait_limit(0)
    _fails(pdgb, lambda: sim.advance(3))
    _recovers(pdgb, sim, 2, x)


@pytest.mark.parametrize("asks", ["synchronize", "get", "advance"])
def test_stencil_product_of_a_caller(pdgb, scenes, asks):
    """apply_operator only enqueues: the next call that waits reports it."""
    import torch
    sim, x = _run(scenes, pdgb, _lattice_body(scenes), 1)
    v = torch.ones((sim.n, 4), device="cuda")
    y = torch.empty_like(v)
    torch.cuda.synchronize()
    sim.set_wait_limit(0)
    sim.apply_operator(v.data_ptr(), y.data_ptr())
    sim.set_wait_limit(-1)
    sim.apply_operator(v.data_ptr(), y.data_ptr())
    _fails(pdgb, {"synchronize": sim.synchronize, "get": lambda: sim.get(pdgb.VAR_POSITION),
                  "advance": lambda: sim.advance(1)}[asks])
    _recovers(pdgb, sim, 1, x)


@pytest.mark.parametrize("loop", [0, 1])
@pytest.mark.parametrize("n,precision", [(20, 0), (5000, 0), (30000, 0), (20, 1), (3000, 1), (12000, 1)])
def test_one_launch_solve(pdgb, scenes, n, precision, loop):
    """One block and many, bonds in shared memory and from global memory."""
    sc = scenes.impact_body(n, "block", coeff=5.0, speed=5.0, seed=2)
    sc.opt.precision = precision
    sc.opt.cg_loop = loop
    sc.opt.spmv_path = 2
    sc.opt.lanes_per_particle, sc.opt.spmv_unroll = 8, 1 if precision else 2   # (one shape: nothing is timed)
    sim, x = _run(scenes, pdgb, sc, 2)
    sim.set_wait_limit(0)
    _fails(pdgb, lambda: sim.advance(3))
    _recovers(pdgb, sim, 2, x)


@pytest.mark.parametrize("graph", [0, 1])
def test_gangs_of_a_batch(pdgb, scenes, graph):
    opt = pdgb.Batch(0).options
    opt.use_graph = graph
    opt.item_rows, opt.lanes_per_particle, opt.spmv_unroll = 128, 8, 2   # (one shape: nothing is timed)
    b = pdgb.Batch(0, opt)
    sizes = (700, 3000, 1500)
    for k, n in enumerate(sizes):
        scenes.add_to_batch(b, scenes.impact_body(n, "block", coeff=5.0, speed=4.0, seed=k, steps=10))
    b.makeReady()
    b.makeReady()   # (as below: the bonds of a row stand in another order after the first)
    b.advance(3)
    x = [b.get(k, pdgb.VAR_POSITION) for k in range(len(sizes))]
    b.set_wait_limit(0)
    b.makeReady()
    _fails(pdgb, lambda: b.advance(3))
    b.set_wait_limit(-1)
    with pytest.raises(pdgb.PdError):
        b.advance(1)
    b.makeReady()
    b.advance(3)
    for k, xk in enumerate(x):
        np.testing.assert_array_equal(b.get(k, pdgb.VAR_POSITION), xk)

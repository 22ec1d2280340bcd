"""Handles of different shared-memory needs alive together.  The limit of a kernel's
dynamic shared memory belongs to the kernel: a handle that sets it for itself takes
it from the others.  Two batches whose shares differ (csrc/cg_persist.cu) and
two simulators whose tiles differ (csrc/tiles.cu) step in turn and from a thread
each, and end where each ends alone (the kernels sum in a fixed order: the same
bits)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
STEPS = 30


def _batch(pdgb, scenes, sizes, graph):
    opt = pdgb.Batch(0).options
    opt.use_graph = graph
    opt.item_rows, opt.lanes_per_particle, opt.spmv_unroll = 128, 8, 2   # (one shape: nothing is timed)
    b = pdgb.Batch(0, opt)
    for k, n in enumerate(sizes):
        scenes.add_to_batch(b, scenes.impact_body(n, "block", coeff=5.0, speed=4.0, seed=k, steps=STEPS))
    b.makeReady()
    return b


def _positions(pdgb, b, count):
    return [b.get(k, pdgb.VAR_POSITION) for k in range(count)]


def _same(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("graph", [0, 1])
def test_two_batches_in_turn_and_from_two_threads(pdgb, scenes, graph):
    sizes = [(20000, 30000), (600, 900, 700)]
    alone = []
    for s in sizes:
        b = _batch(pdgb, scenes, s, graph)
        b.advance(STEPS)
        alone.append(_positions(pdgb, b, len(s)))
        b.close()
    pair = [_batch(pdgb, scenes, s, graph) for s in sizes]
    for _ in range(STEPS):
        for b in pair:
            b.advance(1)
    for b, s, x in zip(pair, sizes, alone):
        _same(_positions(pdgb, b, len(s)), x)
        b.close()

    pair = [_batch(pdgb, scenes, s, graph) for s in sizes]
    failed = []

    def work(b):
        try:
            for _ in range(STEPS):
                b.advance(1)
        except Exception as e:   # noqa: BLE001 (reported by the test)
            failed.append(e)

    threads = [threading.Thread(target=work, args=(b,)) for b in pair]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for b, s, x in zip(pair, sizes, alone):
        _same(_positions(pdgb, b, len(s)), x)


def test_tiles_of_two_simulators(pdgb, scenes):
    """spmv_path 1: the second handle's halos are the smaller ones."""
    def body(n, coeff):
        sc = scenes.impact_body(n, "block", coeff=coeff, speed=4.0, seed=1, steps=4)
        sc.opt.spmv_path = 1
        sc.opt.lanes_per_particle, sc.opt.spmv_unroll = 8, 2
        sim = scenes.make_simulator(sc)
        sim.makeReady()
        return sim
    large = body(20000, 6.0)
    large.advance(4)
    x = large.get(pdgb.VAR_POSITION)
    large, small = body(20000, 6.0), body(200, 3.0)
    assert large.params()[2].spmv_path == small.params()[2].spmv_path == 1
    for _ in range(4):
        small.advance(1)
        large.advance(1)
    np.testing.assert_array_equal(large.get(pdgb.VAR_POSITION), x)

"""The gangs' solve of a batch (k_gang_solve32, csrc/cg_persist.cu) at the sizes
where its plan changes: fewer gangs than scenes, shares with the bonds in shared
memory and read from global memory, blocks without rows, a scene that stops
early, and a batch with a scene too large for it (the phases between grid
barriers).  Each scene against its own Simulator, with the bounds of the other
batch tests (bond sets equal, positions within 1e-5 relative)."""
import pytest

from helpers import rel_err, same_sets

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _check(pdgb, scenes, lst, steps, stops=()):
    b = pdgb.Batch(0)
    for sc in lst:
        scenes.add_to_batch(b, sc)
    b.makeReady()
    b.advance(steps)
    for k, sc in enumerate(lst):
        s = scenes.make_simulator(sc)
        s.makeReady()
        s.advance(steps)
        sb, ss = b.stats(k), s.stats()
        assert sb.current_step == ss.current_step == (1 if k in stops else steps), f"scene {k}"
        assert sb.cg_converged == ss.cg_converged == (k not in stops)
        assert sb.time_step_ticks == ss.time_step_ticks
        assert same_sets(b.alive_sets(k), s.alive_sets()), f"scene {k}"
        assert rel_err(b.get(k, pdgb.VAR_POSITION), s.get(pdgb.VAR_POSITION)) < TOL, f"scene {k}"
    return b


def _body(scenes, n, shape, coeff, seed):
    return scenes.impact_body(n, shape, coeff=coeff, speed=4.0, seed=seed, steps=10)


@pytest.mark.parametrize("sizes", [(1, 2, 33), (500,), (40, 3000, 9, 700, 2500, 64, 1200), (40000, 300, 52000, 9000),
                                   (7000,) * 20 + (8,) * 5])
def test_scenes_of_a_batch(pdgb, scenes, sizes):
    lst = [_body(scenes, n, "ball" if k % 2 else "block", (4.0, 5.0, 6.0)[k % 3], k) for k, n in enumerate(sizes)]
    _check(pdgb, scenes, lst, 5)


def test_a_scene_that_does_not_converge_stops_alone(pdgb, scenes):
    lst = [_body(scenes, n, "block", 5.0, n) for n in (900, 2000, 600)]
    lst[1].opt.cg_max_iterations = 3
    _check(pdgb, scenes, lst, 4, stops=(1,))


def test_a_scene_too_large_for_the_gangs(pdgb, scenes):
    lst = [_body(scenes, n, "block", 5.0, n) for n in (220000, 2000)]
    _check(pdgb, scenes, lst, 3)

"""Small bodies solve in one cooperative launch (csrc/cg_persist.cu).  The sizes
where its plan changes -- a single block, a last block that is not full, the
bonds' geometry in shared memory or read from global memory -- against the
oracle, through bond breaking and rollbacks (a broken bond's halo index moves
with it) and after a checkpoint in another slot order.  Bounds: those of every
parity test (helpers.POS_TOL / DISP_TOL)."""
import numpy as np
import pytest

from helpers import assert_positions, make_oracle, same_sets

pytestmark = pytest.mark.gpu


def _check(pdgb, scenes, sc, steps, label):
    sim = scenes.make_simulator(sc)
    sim.makeReady()
    sim.advance(steps)
    ora = make_oracle(sc)
    ora.advance(steps)
    st = sim.stats()
    assert st.cg_graph_solves == steps and st.cg_converged == 1
    assert same_sets(sim.alive_sets(), ora.alive_sets()), label
    assert st.time_step_ticks == ora.dt_ticks
    assert_positions(sim.get(pdgb.VAR_POSITION), ora.position, sc.pos, sc.opt.precision, label)
    return sim


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n_side", [2, 3, 4, 7])
def test_small_blocks_with_breaking_bonds(pdgb, scenes, n_side, precision):
    """8 to 343 rows: one block up to 32 rows (FP64: 8), a ragged last one after."""
    sc = scenes.reference_block(n_side=n_side, seed=3, integrator=pdgb.NEWMARK_BETA, adaptive=1, expansion=300.0,
                                cg_tol=1e-10)
    sc.opt.precision = precision
    _check(pdgb, scenes, sc, 40, f"block {n_side}, precision {precision}")


@pytest.mark.parametrize("n,precision", [(5001, 0), (26000, 0), (3001, 1), (12000, 1)])
def test_bonds_in_shared_memory_and_from_global(pdgb, scenes, n, precision):
    """Either side of what fits in a block's shared memory."""
    sc = scenes.impact_body(n, "ball", coeff=5.0, speed=5.0, seed=2)
    sc.opt.precision = precision
    sc.opt.spmv_path = 2
    if precision == 1:
        sc.opt.cg_relative_tolerance = 1e-10
    _check(pdgb, scenes, sc, 5, f"ball {n}, precision {precision}")


def test_checkpoint_in_another_slot_order(pdgb, scenes, tmp_path):
    """A state saved by a handle on the lattice product (slots in brick order)
    goes on in a handle on the gather product: its blocks' halos are rebuilt
    for the loaded order."""
    runs = {}
    for path in (3, 2):
        sc = scenes.reference_block(n_side=9, seed=11, integrator=pdgb.NEWMARK_BETA, adaptive=1, expansion=300.0,
                                    cg_tol=1e-10)
        sc.opt.spmv_path = path
        sc.run.saving_path = str(tmp_path).encode()
        sim = scenes.make_simulator(sc)
        sim.makeReady()
        if path == 3:
            sim.advance(25)
            sim.dataIO_saveState(25)
        else:
            sim.dataIO_loadState(25)
        sim.advance(10)
        runs[path] = sim
    assert runs[2].stats().bonds_alive < runs[2].stats().bonds_initial
    assert same_sets(runs[2].alive_sets(), runs[3].alive_sets())
    ora = make_oracle(sc)
    ora.advance(35)
    assert same_sets(runs[2].alive_sets(), ora.alive_sets())
    assert_positions(runs[2].get(pdgb.VAR_POSITION), ora.position, sc.pos, 0, "loaded in brick order")
    np.testing.assert_array_equal(runs[2].get(pdgb.VAR_BOND_COUNT), runs[3].get(pdgb.VAR_BOND_COUNT))

"""The sums over all rows in a one-launch solve (csrc/cg_persist.cu) are as accurate
as those of separate launches, which are FP64 from the warp on.  A first solve
of no iterations leaves <b, b> twice: sqrt of the solve's own sum as its residual
(x = 0), and the separate launch's in the tolerance.  The two round at most some
ten times in 53 bits after sums within warps in 48: for rows of like size (a body
under no contact) 4e-16 apart, root mean square over bodies, in an emulation of
both; 1.6e-15 with the sums in 48 bits throughout.  The bound lies between, at
9e-16."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [2500, 12000, 30000])
def test_two_sums_of_one_vector(pdgb, scenes, size):
    apart = []
    for seed in range(24):
        sc = scenes.impact_body(size, "block", coeff=5.0, speed=5.0, seed=seed)
        sc.opt.spmv_path = 2
        sc.opt.lanes_per_particle, sc.opt.spmv_unroll = 8, 2   # (one shape: nothing is timed)
        sc.opt.cg_max_iterations = 0
        sc.opt.cg_relative_tolerance = 2.0 ** -20
        sc.vel[:, :3] = np.random.default_rng(seed).standard_normal((sc.n, 3))
        sim = scenes.make_simulator(sc)
        sim.makeReady()
        sim.advance(1)
        st = sim.stats()
        assert st.last_cg_iterations == 0 and st.cg_graph_solves == 1
        apart.append((st.last_cg_residual / (st.last_cg_tolerance * 2.0 ** 20)) ** 2 - 1.0)
        sim.close()
    rms = float(np.sqrt(np.mean(np.square(apart))))
    print(f"[sums] {size}: {rms:.2e}")
    assert rms < 9e-16

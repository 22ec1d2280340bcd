"""A state loaded in another bond order (csrc/tiles.cu, k_bank_order) is put into the
products' own, which halves their shared-memory conflicts, and the run goes on as the
saver's does.  Without it the body here takes 24.7 us per product after a load in the
reference's layout and 28.8 after one in the bricks' slot order, with it 20.0 and
22.7 (bricks make longer halos), 20.0 before.  The bounds stand between."""
import numpy as np
import pytest

from helpers import apply_on_device, rel_err, same_sets

pytestmark = pytest.mark.gpu


def _product_us(sim):
    import torch
    x = torch.randn((sim.n, 4), device="cuda")
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    stream = torch.cuda.ExternalStream(sim.stream_handle())
    best = 1e30
    for _ in range(30):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        for _ in range(20):
            sim.apply_operator(x.data_ptr(), y.data_ptr())
        b.record(stream)
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 50.0)
    return best


@pytest.mark.parametrize("layout,most", [("own", 1.25), ("reference", 1.1)])
def test_products_after_a_load(pdgb, scenes, layout, most, tmp_path):
    sc = scenes.impact_body(97_000, "ball", coeff=5.0, speed=5.0, seed=2)
    sc.run.saving_path = str(tmp_path).encode()
    runs = {}
    for path in (3, 0):
        sc.opt.spmv_path = path
        runs[path] = scenes.make_simulator(sc)
        runs[path].makeReady()
        runs[path].advance(2)
    saver, sim = runs[3], runs[0]
    fresh = _product_us(sim)
    if layout == "own":
        saver.dataIO_saveState(2)
        sim.dataIO_loadState(2)
    else:
        saver.dataIO_saveStateReference(2)
        sim.dataIO_loadStateReference(2)
    loaded = _product_us(sim)
    print(f"[order] {layout}: {fresh:.2f} us, after the load {loaded:.2f} us")
    assert loaded < most * fresh
    x = np.zeros((sc.n, 4))
    x[:, :3] = np.random.default_rng(2).standard_normal((sc.n, 3))
    for s in (saver, sim):
        s.advance(1)
    (y, _, _), (y2, _, _) = (apply_on_device(pdgb, s, x) for s in (sim, saver))
    assert np.abs(y[:, :3] - y2[:, :3]).max() <= 2e-5 * np.abs(y2[:, :3]).max()   # (test_gpu_product_routes.py)
    saver.advance(3)
    sim.advance(3)
    assert same_sets(sim.alive_sets(), saver.alive_sets())
    assert rel_err(sim.get(pdgb.VAR_POSITION), saver.get(pdgb.VAR_POSITION)) < 1e-5

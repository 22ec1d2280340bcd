"""The stencil product (csrc/lattice.cu) against 64 bits: no further off than the
same sum formed in 32 bits offset by offset, z, y, x, with the bond vector as
h v + (d_q - d_p) -- what the product was before it walked the stencil by columns.
Both are sums of some hundred rounded terms per row; their root-mean-square errors
over 80,000 entries are known to 0.3 %."""
import itertools

import numpy as np
import pytest
import torch

from helpers import apply_on_device

pytestmark = pytest.mark.gpu
F, D = np.float32, np.float64


def _fma(a, b, c):
    return (a.astype(D) * b.astype(D) + c.astype(D)).astype(F)


def _sums(pos, sites, w, h, horizon):
    """sum_q J (w_p - w_q) over the bonds, in 64 bits and in 32 bits."""
    dims = sites.max(0) + 1
    at = np.full(dims, -1)
    at[tuple(sites.T)] = np.arange(len(sites))
    d32 = (pos - h * sites).astype(F)
    exact, acc = np.zeros_like(pos), np.zeros(pos.shape, F)
    reach = range(-3, 4)
    for dz, dy, dx in itertools.product(reach, reach, reach):
        q0 = sites + (dx, dy, dz)
        p = np.flatnonzero((q0 >= 0).all(1) & (q0 < dims).all(1) & ((dx, dy, dz) != (0, 0, 0)))
        q = at[tuple(q0[p].T)]
        xi = pos[q] - pos[p]
        d = np.linalg.norm(xi, axis=1)
        on = d < horizon
        p, q, xi, d = p[on], q[on], xi[on], d[on]
        exact[p] += ((xi * (w[p].astype(D) - w[q])).sum(1) / d ** 3)[:, None] * xi
        g = (d32[q] - d32[p]) + (h * np.array([dx, dy, dz])).astype(F)
        dw = w[q] - w[p]
        dd = _fma(g[:, 0], g[:, 0], _fma(g[:, 1], g[:, 1], g[:, 2] * g[:, 2]))
        inv = torch.rsqrt(torch.from_numpy(dd).cuda()).cpu().numpy()   # (the device's own, two roundings)
        a1 = (1 / d).astype(F) - inv
        t = _fma(g[:, 0], dw[:, 0], _fma(g[:, 1], dw[:, 1], g[:, 2] * dw[:, 2])) * ((inv * inv) * inv)
        for k in range(3):
            acc[p, k] = _fma(a1, dw[:, k], _fma(t, g[:, k], acc[p, k]))
    return exact, -acc


@pytest.mark.parametrize("coeff", [4.0, 5.0, 6.0])
@pytest.mark.parametrize("h", [0.02, 0.0061, 2.0 ** -6])
def test_error_against_64_bits(pdgb, scenes, coeff, h):
    sc = scenes.impact_body(27000, "block", coeff=coeff, spacing=h, jitter=0.05, seed=1)
    sc.opt.spmv_path = 3
    sim = scenes.make_simulator(sc)
    sim.makeReady()
    sim.advance(1)      # (the operator of a step, at the positions that it began with)
    assert sim.params()[2].spmv_path == 3
    x = np.zeros((sc.n, 4))
    x[:, :3] = np.random.default_rng(5).standard_normal((sc.n, 3)).astype(F)
    y, _, _ = apply_on_device(pdgb, sim, x)
    v = sim.operator_view()
    sites = np.rint(sc.pos[:, :3] / h).astype(int)
    s64, s32 = _sums(sc.pos[:, :3], sites - sites.min(0), x[:, :3].astype(F), h, sc.sim.pd_horizon)
    free = sc.act == scenes.ACTIVE
    truth = v.mass * x[free, :3] + v.t2 * v.bond_coeff * s64[free]
    w = x[free, :3].astype(F)
    plain = F(v.mass) * w + F(v.t2) * (F(v.bond_coeff) * s32[free])
    rms = [np.sqrt(((a.astype(D) - truth) ** 2).mean()) / np.abs(truth).max() for a in (y[free, :3], plain)]
    print(f"[accuracy] coeff {coeff}, h {h:.4f}: stencil {rms[0]:.3e}, plain sum {rms[1]:.3e}")
    assert rms[0] <= rms[1]

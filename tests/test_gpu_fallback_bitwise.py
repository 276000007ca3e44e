"""GPU suite: the bins that a mixed call hands to FP64 come back bit for bit as the
FP64 call returns them, below and from the 64 microphones of the FP64 solve's
Jacobi start, for an operator, its own monopoles, spherical harmonics and a
boundary mesh.  A regularisation at 1e-6 of the smallest s_1 is below what the mixed path
resolves, so every bin is handed over."""
import numpy as np
import pytest

from inverseacoustics_gb300 import geometry as g
from oracle import ia_oracle as O

pytestmark = pytest.mark.gpu


def _compare(ctx, run):
    from inverseacoustics_gb300 import _lib
    import torch
    x, lam, s, info = run(0)
    xm, lamm, sm, infom = run(1)
    torch.cuda.synchronize()
    assert _lib.lib().ia_last_fallback_bins(ctx.handle) == x.shape[0]
    assert not bool(info.any()) and not bool(infom.any())
    assert torch.equal(xm, x) and torch.equal(lamm, lam) and torch.equal(sm, s)


def _cfg(prec, lam):
    from inverseacoustics_gb300 import api
    return api.default_config(precision=prec, method=2, lambda_fixed=lam)


@pytest.mark.parametrize("side", [6, 8, 9])
def test_esm_and_operator_fallback(cuda, ctx, side):
    from inverseacoustics_gb300 import api
    import torch
    rng = np.random.default_rng(side)
    l, F = side * side, 5
    mics = g.planar_array(side, side, 0.03, 0.10)
    src, _ = g.icosphere(2, 0.05)
    ks = 2 * np.pi * np.linspace(400, 2400, F) / 343.0
    H = np.stack([O.monopole_matrix(mics, src, k) for k in ks])
    lam = 1e-6 * np.linalg.norm(H[0], 2)
    p = torch.as_tensor(g.complex_normal(rng, (F, 1, l)), device=cuda)
    md, sd, kd = (torch.as_tensor(np.ascontiguousarray(a), device=cuda) for a in (mics, src, ks))
    _compare(ctx, lambda prec: api.esm_solve_batch(ctx, md, sd, kd, p, _cfg(prec, lam)))
    Hd = torch.as_tensor(np.ascontiguousarray(H.transpose(0, 2, 1)), device=cuda)
    _compare(ctx, lambda prec: api.solve_batch(ctx, Hd, l, src.shape[1], p, _cfg(prec, lam)))


@pytest.mark.parametrize("order,side", [(5, 6), (8, 8)])
def test_hels_fallback(cuda, ctx, order, side):
    from inverseacoustics_gb300 import api
    import torch
    rng = np.random.default_rng(order)
    F = 3
    P = g.planar_array(side, side, 0.04, 0.15)
    r = np.sqrt((P ** 2).sum(0))
    sph = np.ascontiguousarray(np.stack([np.mod(np.arctan2(P[1], P[0]), 2 * np.pi), np.arccos(P[2] / r), r]))
    ks = 2 * np.pi * np.linspace(800, 2000, F) / 343.0
    p = torch.as_tensor(g.complex_normal(rng, (F, 1, side * side)), device=cuda)
    pd, kd = torch.as_tensor(sph, device=cuda), torch.as_tensor(ks, device=cuda)
    s1 = float(api.hels_solve_batch(ctx, pd, order, kd, p, _cfg(0, 1.0))[2][:, 0].min())
    _compare(ctx, lambda prec: api.hels_solve_batch(ctx, pd, order, kd, p, _cfg(prec, 1e-6 * s1)))


@pytest.mark.parametrize("l", [40, 80])
def test_ibem_fallback(cuda, ctx, l):
    from inverseacoustics_gb300 import api
    import torch
    rng = np.random.default_rng(l)
    nodes, elems = g.icosphere(2, 0.1)
    F = 4
    mics = torch.as_tensor(g.hemisphere_array(rng, l, 0.3), device=cuda)
    k = torch.as_tensor(2 * np.pi * np.linspace(300.0, 1500.0, F) / 343.0, device=cuda)
    p = torch.as_tensor(g.complex_normal(rng, (F, 1, l)), device=cuda)
    mesh = api.Mesh(ctx, nodes, elems)
    s1 = float(api.ibem_solve_batch(ctx, mesh, mics, k, p, _cfg(0, 1.0))[2][:, 0].min())
    _compare(ctx, lambda prec: api.ibem_solve_batch(ctx, mesh, mics, k, p, _cfg(prec, 1e-6 * s1)))
    mesh.close()

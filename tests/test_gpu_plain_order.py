"""GPU suite: the FP64 IBEM inversion keeps one operation order: its results do
not depend on how the batch spreads over clusters (QR columns, LU rows and
Jacobi pairs over 1 to 8 CTAs), bit for bit, also with a regularisation at
the rounding level, where any change of rounding would show."""
import numpy as np
import pytest

from inverseacoustics_gb300 import geometry as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("subdiv,l", [(1, 17), (1, 42), (2, 64), (2, 96), (3, 40)])
def test_ibem_solution_is_bitwise_the_same_alone_and_in_a_batch(cuda, ctx, subdiv, l):
    from inverseacoustics_gb300 import api
    import torch
    nodes, elems = g.icosphere(subdiv, 0.1)
    rng = np.random.default_rng(l)
    mics = torch.as_tensor(g.hemisphere_array(rng, l, 0.3), device=cuda)
    F = 84
    k = torch.as_tensor(2 * np.pi * np.repeat(np.linspace(200.0, 1900.0, F // 4), 4) / 343.0, device=cuda)
    p = torch.as_tensor(g.complex_normal(rng, (F, 1, l)), device=cuda)
    cfg = api.default_config(method=2, lambda_fixed=1e-9)
    mesh = api.Mesh(ctx, nodes, elems)
    x, _, s, info = api.ibem_solve_batch(ctx, mesh, mics, k, p, cfg)
    assert int(info.abs().sum()) == 0
    for f0, n in ((0, 4), (40, 4), (8, 36)):
        x1, _, s1, _ = api.ibem_solve_batch(ctx, mesh, mics, k[f0:f0 + n].contiguous(), p[f0:f0 + n].contiguous(), cfg)
        assert torch.equal(x1, x[f0:f0 + n]) and torch.equal(s1, s[f0:f0 + n])
    mesh.close()

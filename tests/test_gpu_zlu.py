"""GPU suite: the FP64 LU and solves at the edges of their panels (64 columns),
half blocks (32 rows) and clusters, through the entry points that use them.

ESM systems with deep sources (r_i 0.5) are far from diagonally dominant, so
rows interchange; the computed Me D = M_sq, He D = M_hq is checked by its
residual, which a backward stable solver keeps near n eps |Me| |D|: bound
1e-12 |Me| |D| (Frobenius) for n <= 330."""
import numpy as np
import pytest

from conftest import relerr
from inverseacoustics_gb300 import geometry as g
from inverseacoustics_gb300 import quadrature as Q
from oracle import ia_oracle as O

pytestmark = pytest.mark.gpu
C, RHO = 343.0, 1.21


@pytest.mark.parametrize("m,l", [(1, 1), (2, 3), (31, 5), (32, 1), (33, 9), (63, 2), (64, 7), (65, 30), (96, 4),
                                 (127, 3), (128, 16), (129, 1), (257, 5), (330, 40)])
def test_esm_system_residual(cuda, m, l):
    from inverseacoustics_gb300 import api
    rng = np.random.default_rng(m)
    v = rng.normal(size=(3, m))
    P = 0.1 * v / np.linalg.norm(v, axis=0)
    F = g.hemisphere_array(rng, l, 0.3)
    k, ri = 12.0, 0.5
    Me, He = api.esm(P, F, k, ri, C, RHO)
    D, Msq, Mhq = O.esm_matrices(P, F, k, ri, C, RHO)
    for X, B in ((Me, Msq), (He, Mhq)):
        assert np.linalg.norm(X @ D - B) <= 1e-12 * np.linalg.norm(X) * np.linalg.norm(D)


@pytest.mark.parametrize("subdiv,l,F", [(0, 1, 1), (1, 7, 3), (1, 60, 40), (2, 5, 9), (2, 33, 20), (2, 3, 77), (1, 2, 160)])
def test_transfer_over_cluster_sizes(cuda, ctx, subdiv, l, F):
    """Batches that give the panel clusters of 8, 4, 2 and 1 CTAs: against the
    oracle at 1e-10, and against the same bins solved alone (the assembly's
    phase recurrence over a block of four bins differs) at 1e-12."""
    from inverseacoustics_gb300 import api
    import torch
    nodes, elems = g.icosphere(subdiv, 0.1)
    rng = np.random.default_rng(3)
    mics = g.hemisphere_array(rng, l, 0.3)
    k = 2 * np.pi * np.linspace(150.0, 1900.0, F) / C
    mesh = api.Mesh(ctx, nodes, elems)
    md = torch.as_tensor(mics, device=cuda)
    H, info = api.ibem_transfer_batch(ctx, mesh, md, torch.as_tensor(k, device=cuda))
    one = [api.ibem_transfer_batch(ctx, mesh, md, torch.as_tensor(k[f:f + 1].copy(), device=cuda))[0]
           for f in (0, F - 1)]
    torch.cuda.synchronize()
    assert int(info.abs().sum()) == 0
    for f in {0, F // 2, F - 1}:
        Ho = O.ibem_transfer(nodes, elems, mics, k[f], *Q.builtin(), C, RHO)
        assert relerr(H[f].cpu().numpy().T, Ho) < 1e-10
    for f, o in zip((0, F - 1), one):
        assert relerr(H[f].cpu().numpy(), o[0].cpu().numpy()) < 1e-12
    mesh.close()

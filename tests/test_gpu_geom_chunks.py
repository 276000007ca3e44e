"""GPU suite: the double-float assembly with its geometry table filled and read
in chunks of rows (2571 rows x 5120 elements: 2.2 GB, three chunks) against the
form that computes the geometry inline; surface, CHIEF and field rows.  The same
double-float operations: 1e-13 of each row's largest entry, as for a table that
holds every row."""
import numpy as np
import pytest

from inverseacoustics_gb300 import geometry as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins", [2, 3])
def test_chunked_geometry_table_matches_inline(cuda, ctx, monkeypatch, bins):
    from inverseacoustics_gb300 import api
    import torch
    nodes, elems = g.icosphere(4, 0.1)
    rng = np.random.default_rng(4)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=cuda)
    mics = t(0.2 + 0.1 * rng.random((3, 7)))
    cp = t(np.array([[0.01, -0.02, 0.015], [-0.03, 0.0, 0.02]]).T)
    ks = t(np.linspace(5.0, 40.0, bins))
    mesh = api.Mesh(ctx, nodes, elems)
    cfg = api.default_config(precision=1)
    monkeypatch.delenv("IA_ASM_GEOM_TABLE", raising=False)
    tab = api.ibem_assemble_batch(ctx, mesh, mics, ks, cfg, cp=cp)
    monkeypatch.setenv("IA_ASM_GEOM_TABLE", "0")
    inl = api.ibem_assemble_batch(ctx, mesh, mics, ks, cfg, cp=cp)
    torch.cuda.synchronize()
    for a, b in zip(tab, inl):
        scale = b.abs().amax(dim=-1, keepdim=True)
        assert float(((a - b).abs() / scale).max()) < 1e-13
    mesh.close()

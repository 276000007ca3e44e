"""GPU suite: the FP64 radiation modes' subspace products on the tensor cores
(10 BF16 slices), at the sizes where the rule and the tiles change: below and
from 96 radiators, around a 128-row tile, odd sizes, more bins than one group
of slice planes holds; and operators far from 1 or not finite.

Bounds as for the plate (FP64): eigenvalues 1e-12 lambda_1, residuals 1e-12
lambda_1, orthonormality 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrices(n, F, scale=1.0):
    """Symmetric positive matrices with eigenvalues 0.6^j."""
    rng = np.random.default_rng(n)
    out = []
    for _ in range(F):
        Q = np.linalg.qr(rng.normal(size=(n, n)))[0]
        w = np.maximum(0.6 ** np.arange(n), 1e-18)
        R = (Q * w) @ Q.T
        out.append(scale * 0.5 * (R + R.T))
    return np.stack(out)


@pytest.mark.parametrize("scale", [1.0, 1e-100, 1e100])
@pytest.mark.parametrize("n", [24, 95, 96, 97, 128, 129, 255])
def test_modes_at_tile_edges(cuda, ctx, n, scale):
    from inverseacoustics_gb300 import api
    import torch
    if n < 96 and scale != 1.0:
        pytest.skip("the CUDA-core product")
    nm, F = 5, 3
    R = _matrices(n, F, scale)
    lam, modes, info = api.radiation_modes_batch(ctx, torch.as_tensor(R, device=cuda), nm, api.default_config())
    torch.cuda.synchronize()
    assert int(info.abs().sum()) == 0
    lam, modes = lam.cpu().numpy(), modes.cpu().numpy()
    for f in range(F):
        w = np.linalg.eigvalsh(R[f])[::-1]
        X = modes[f].T
        assert np.max(np.abs(lam[f] - w[:nm])) <= 1e-12 * w[0]
        assert np.max(np.abs(X.T @ X - np.eye(nm))) < 1e-12
        assert np.max(np.linalg.norm(R[f] @ X - X * lam[f], axis=0)) <= 1e-12 * w[0]


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_modes_flag_a_non_finite_operator(cuda, ctx, value):
    from inverseacoustics_gb300 import api
    import torch
    R = _matrices(130, 2)
    R[1, 3, 100] = R[1, 100, 3] = value
    lam, _, info = api.radiation_modes_batch(ctx, torch.as_tensor(R, device=cuda), 4, api.default_config())
    torch.cuda.synchronize()
    assert int(info[0]) == 0 and int(info[1]) & 4
    assert bool(torch.isfinite(lam[0]).all())


def test_modes_over_more_than_one_group_of_bins(cuda, ctx):
    """Slice planes of 320 bins of 1024 radiators pass the 6 GiB of one group:
    the results are bitwise those of single-bin calls."""
    from inverseacoustics_gb300 import api
    import torch
    base = torch.as_tensor(_matrices(1024, 1)[0], device=cuda)
    scale = 1.0 + torch.arange(320, dtype=torch.float64, device=cuda) / 320
    R = base[None] * scale[:, None, None]
    lam, modes, info = api.radiation_modes_batch(ctx, R, 3, api.default_config())
    assert int(info.abs().sum()) == 0
    for f in (0, 159, 160, 319):
        l1, m1, _ = api.radiation_modes_batch(ctx, R[f:f + 1].contiguous(), 3, api.default_config())
        assert torch.equal(l1[0], lam[f]) and torch.equal(m1[0], modes[f])

"""GPU suite: the 96-column tiles of the FP64-level products, through the array
design and the radiation modes at batches on both sides of the rule that picks
them: a bin's results do not depend on the tile's width, bit for bit (the level
sums are exact integers)."""
import numpy as np
import pytest

from test_gpu_adjoint import _case, _dev_args

pytestmark = pytest.mark.gpu


# 31 / 100 / 129 microphones: partial row tiles, one and two of them, K of the
# solves 31 .. 129, partial 96- and 48-column tiles
@pytest.mark.parametrize("l,subdiv", [(31, 1), (100, 2), (129, 2)])
def test_wide_tiles_do_not_change_a_bin(cuda, ctx, l, subdiv):
    from inverseacoustics_gb300 import api
    import torch
    F = 220
    case = _case(7, l, subdiv, 2, 8)
    mics, surf, d, k, ll, q, noise = _dev_args(case, cuda)
    rep = lambda t: t.repeat((F // 2,) + (1,) * (t.dim() - 1)).contiguous()
    one = api.esm_design_batch(ctx, mics, surf, d, k, ll, q, noise)
    many = api.esm_design_batch(ctx, mics, surf, d, rep(k), rep(ll), rep(q), rep(noise))
    torch.cuda.synchronize()
    assert int(many[4].abs().sum()) == 0
    err1, errF = one[0].reshape(2, -1), many[0].reshape(F, -1)
    assert torch.equal(errF, err1.repeat(F // 2, 1))


@pytest.mark.parametrize("n", [130, 200])
def test_wide_real_tiles_do_not_change_a_bin(cuda, ctx, n):
    from inverseacoustics_gb300 import api
    import torch
    rng = np.random.default_rng(n)
    x = torch.as_tensor(rng.random((3, n)), device=cuda)
    k = torch.as_tensor(np.array([6.0, 11.0]), device=cuda)
    R = api.sinc_resistance_batch(ctx, x, k, 0.01)
    R = R[0] if isinstance(R, (tuple, list)) else R
    many = R.repeat(90, 1, 1).contiguous()
    a = api.radiation_modes_batch(ctx, R, 60)
    b = api.radiation_modes_batch(ctx, many, 60)
    torch.cuda.synchronize()
    assert torch.equal(b[0], a[0].repeat(90, 1))
    assert torch.equal(b[1].reshape(180, -1), a[1].reshape(2, -1).repeat(90, 1))

"""GPU suite: the 10-slice products past one group: contractions longer than the
768 that one product sums exactly (four of them, accumulated in FP64), and
more bins than the 2 GiB of slice planes held at once.

Bounds of the first as for the array design's other shapes (cond(K) <= 1e5: 1e-10
loss, 1e-9 gradients); the second is bitwise."""
import numpy as np
import pytest

from oracle import ia_oracle as O
from test_gpu_adjoint import _case, _dev_args

pytestmark = pytest.mark.gpu


def test_design_with_more_sources_than_one_product_sums(cuda, ctx):
    from inverseacoustics_gb300 import api
    import torch
    case = _case(21, 20, 4, 1, 2)                       # 2562 sources
    mics, surf, d, k, ll, q, noise = case
    err, gm, gd, gl, info = api.esm_design_batch(ctx, *_dev_args(case, cuda))
    torch.cuda.synchronize()
    assert int(info.abs().sum()) == 0
    eo = O.esm_design_terms(mics, surf, d, k, ll, q, noise)
    gmo, gdo, glo = O.esm_design_grad(mics, surf, d, k, ll, q, noise)
    assert np.max(np.abs(err.cpu().numpy() - eo)) <= 1e-10 * np.max(eo)
    assert np.max(np.abs(gm.cpu().numpy() - gmo)) <= 1e-9 * np.max(np.abs(gmo))
    assert abs(gd.item() - gdo) <= 1e-9 * max(abs(gdo), np.max(np.abs(gmo)))
    assert np.max(np.abs(gl.cpu().numpy() - glo)) <= 1e-9 * np.max(np.abs(glo))


def test_design_over_more_than_one_group_of_bins(cuda, ctx):
    from inverseacoustics_gb300 import api
    import torch
    mics, surf, d, k, ll, q, noise = _case(22, 16, 2, 4, 1)
    rep = 1800                                          # 7200 bins of 315 KB of planes
    kk = np.concatenate([k + 1e-3 * i for i in range(rep)])
    case = mics, surf, d, kk, np.tile(ll, rep), np.tile(q, (rep, 1, 1)), np.tile(noise, (rep, 1, 1))
    M, S, D, K, LL, Q, N = _dev_args(case, cuda)
    err, _, _, gl, info = api.esm_design_batch(ctx, M, S, D, K, LL, Q, N)
    assert int(info.abs().sum()) == 0
    for f in (0, 3599, 3600, 6700, 7199):
        s = slice(f, f + 1)
        e1, _, _, gl1, _ = api.esm_design_batch(ctx, M, S, D, K[s].contiguous(), LL[s].contiguous(),
                                                Q[s].contiguous(), N[s].contiguous())
        assert torch.equal(e1[0], err[f])
        assert abs(gl1.item() / len(kk) - gl[f].item()) <= 1e-13 * abs(gl[f].item())   # (a mean over the bins)

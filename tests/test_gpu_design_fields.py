"""GPU suite: the array-design loss and gradient with source fields of unequal
strength, which the normalised loss weighs equally, against the FP64 oracle.
Bounds as for fields of one strength (1e-10 loss, 1e-9 gradients, cond(K) <=
1e5): scaling a field leaves every digit of its loss and of its share of the
gradient."""
import numpy as np
import pytest

from oracle import ia_oracle as O
from test_gpu_adjoint import _case, _dev_args

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weak,noise_too", [([1e-6, 1.0, 1.0, 1.0], True), ([1.0, 1e-12, 3e7, 1e-3], True),
                                            ([1e60, 1.0, 1.0, 1e-60], True), ([1e-4, 1.0, 1.0, 1.0], False)])
def test_design_fields_of_unequal_strength(cuda, ctx, weak, noise_too):
    from inverseacoustics_gb300 import api
    import torch
    mics, surf, d, k, ll, q, noise = _case(7, 32, 1, 2, 4)
    q = q * np.array(weak)
    if noise_too:
        noise = noise * np.array(weak)
    case = mics, surf, d, k, ll, q, noise
    err, gm, gd, gl, info = api.esm_design_batch(ctx, *_dev_args(case, cuda))
    torch.cuda.synchronize()
    assert int(info.abs().sum()) == 0
    eo = O.esm_design_terms(mics, surf, d, k, ll, q, noise)
    gmo, gdo, glo = O.esm_design_grad(mics, surf, d, k, ll, q, noise)
    assert np.max(np.abs(err.cpu().numpy() - eo) / eo) <= 1e-10
    assert np.max(np.abs(gm.cpu().numpy() - gmo)) <= 1e-9 * np.max(np.abs(gmo))
    assert abs(gd.item() - gdo) <= 1e-9 * max(abs(gdo), np.max(np.abs(gmo)))
    assert np.max(np.abs(gl.cpu().numpy() - glo)) <= 1e-9 * np.max(np.abs(glo))


def test_design_a_zero_field_is_flagged_in_its_bin_only(cuda, ctx):
    from inverseacoustics_gb300 import api
    import torch
    mics, surf, d, k, ll, q, noise = _case(8, 16, 1, 3, 2)
    q[1, :, 0] = 0
    err, gm, gd, gl, info = api.esm_design_batch(ctx, *_dev_args((mics, surf, d, k, ll, q, noise), cuda))
    torch.cuda.synchronize()
    assert [int(i) != 0 for i in info] == [False, True, False]
    eo = O.esm_design_terms(mics, surf, d, k, ll, q, noise)[[0, 2]]
    assert np.max(np.abs(err.cpu().numpy()[[0, 2]] - eo)) <= 1e-10 * np.max(eo)

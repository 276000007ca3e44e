"""GPU suite: the array-design loss and gradient at the edges of its tiles (32
microphones per CTA of the geometry adjoint, 64-column panels, 128-row product
tiles, one to 32 fields, as many microphones as sources) against the FP64
oracle.  cond(K) <= 1e5 (lambda = 5 % of G's rms), so 1e-10 on the loss and 1e-9
on the gradients, as at the sizes of the other test."""
import numpy as np
import pytest

from oracle import ia_oracle as O
from test_gpu_adjoint import _case, _dev_args

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("l,subdiv,F,R", [(1, 1, 1, 1), (31, 1, 2, 3), (32, 1, 2, 32), (33, 1, 1, 5), (42, 1, 2, 1),
                                          (65, 2, 1, 16), (128, 2, 1, 7), (129, 2, 2, 2)])
def test_design_shapes(cuda, ctx, l, subdiv, F, R):
    from inverseacoustics_gb300 import api
    import torch
    case = _case(100 + l, l, subdiv, F, R)
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

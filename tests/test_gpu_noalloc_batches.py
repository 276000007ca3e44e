"""GPU suite: ia_solve_batch_noalloc gives a bin the same digits whatever number of
bins the call holds, up to the most that its scratch takes, with the Jacobi start
(64 to ~230 microphones) and without (below, and where the start does not fit),
and those of ia_solve_batch where that runs the same operations."""
import numpy as np
import pytest

from test_zz_no_alloc import _noalloc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,nrhs,same", [(40, 60, 1, True), (64, 162, 1, True), (64, 64, 3, True),
                                           (100, 120, 1, True), (160, 200, 2, True), (256, 300, 1, False)])
def test_noalloc_digits_do_not_depend_on_the_batch(cuda, ctx, m, n, nrhs, same):
    from inverseacoustics_gb300 import api
    import torch
    rng = np.random.default_rng(m + n)
    F = 160
    H = torch.as_tensor(rng.normal(size=(F, n, m)) + 1j * rng.normal(size=(F, n, m)), device=cuda)
    b = torch.as_tensor(rng.normal(size=(F, nrhs, m)) + 1j * rng.normal(size=(F, nrhs, m)), device=cuda)
    cfg = api.default_config(method=2, lambda_fixed=0.5)
    accepted = [f for f in range(1, F + 1) if _noalloc(ctx, H[:f], b[:f], m, n, cfg)[0] == 0] if m > 150 else None
    if accepted is None:   # the most bins, by bisection (a refusal does nothing)
        lo, hi = 1, F
        while lo < hi:
            mid = (lo + hi + 1) // 2
            lo, hi = (mid, hi) if _noalloc(ctx, H[:mid], b[:mid], m, n, cfg)[0] == 0 else (lo, mid - 1)
        accepted = [1, 2, lo // 2, lo - 1, lo]
    x1, _, s1, i1 = api.solve_batch(ctx, H, m, n, b, cfg)
    for f in accepted:
        st, x, lam, s, info = _noalloc(ctx, H[:f], b[:f], m, n, cfg)
        torch.cuda.synchronize()
        assert st == 0 and not bool(info.any())
        ref = (x1, s1)
        if not same:
            ref = _noalloc(ctx, H[:1], b[:1], m, n, cfg)[1::2]
        k = f if same else 1
        assert torch.equal(x[:k], ref[0][:k]) and torch.equal(s[:k], ref[1][:k])

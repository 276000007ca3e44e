"""GPU suite: the FP64 wide solve's pivoted QR over a cluster, at the sizes
where its row groups (32, 128), register forms (256, 768, 1280 rows, beyond)
and clusters (8 bins, 40, 160) change, and on operators with zero, equal and
dependent columns; against the oracle's SVD solve.

Random operators with a fixed lambda of 0.3 s_1: x and s are determined to a
few eps, bound 1e-12 (s relative to s_1)."""
import numpy as np
import pytest

from conftest import relerr
from oracle import ia_oracle as O

pytestmark = pytest.mark.gpu


def _solve(ctx, cuda, H, b, lam):
    from inverseacoustics_gb300 import api
    import torch
    Hc = torch.as_tensor(np.ascontiguousarray(H.transpose(0, 2, 1)), device=cuda)
    bd = torch.as_tensor(np.ascontiguousarray(b), device=cuda)
    cfg = api.default_config(method=2, lambda_fixed=lam)
    x, _, s, info = api.solve_batch(ctx, Hc, H.shape[1], H.shape[2], bd, cfg)
    torch.cuda.synchronize()
    return x.cpu().numpy(), s.cpu().numpy(), info.cpu().numpy()


def _check(ctx, cuda, H, b, lam):
    x, s, info = _solve(ctx, cuda, H, b, lam)
    assert not info.any()
    for f in {0, len(H) // 2, len(H) - 1}:
        U, so, V = O.csvd(H[f])
        assert np.max(np.abs(s[f] - so)) <= 1e-12 * so[0]
        for r in range(b.shape[1]):
            assert relerr(x[f, r], O.tikhonov(U, so, V, b[f, r], lam)) < 1e-12


@pytest.mark.parametrize("m,n,F", [(1, 1, 2), (1, 9, 3), (2, 2, 1), (7, 31, 5), (8, 32, 8), (16, 33, 40), (15, 127, 3),
                                   (33, 129, 2), (64, 256, 160), (65, 257, 3), (40, 768, 2), (24, 769, 20),
                                   (10, 1280, 3), (12, 1281, 2), (100, 100, 4)])
def test_wide_solve_qr_shapes(cuda, ctx, m, n, F):
    rng = np.random.default_rng(m * 10000 + n)
    H = (rng.normal(size=(F, m, n)) + 1j * rng.normal(size=(F, m, n))) * np.exp(rng.normal(size=(F, m, 1)))
    b = rng.normal(size=(F, 2, m)) + 1j * rng.normal(size=(F, 2, m))
    _check(ctx, cuda, H, b, 0.3 * np.linalg.norm(H[0], 2))


@pytest.mark.parametrize("kind", ["zero_row", "equal_rows", "rank_one", "zero", "real", "tiny", "huge"])
def test_wide_solve_qr_degenerate_columns(cuda, ctx, kind):
    rng = np.random.default_rng(5)
    H = rng.normal(size=(3, 24, 70)) + 1j * rng.normal(size=(3, 24, 70))
    b = rng.normal(size=(3, 1, 24)) + 1j * rng.normal(size=(3, 1, 24))
    lam = 0.3 * np.linalg.norm(H[0], 2)
    if kind == "zero_row":
        H[:, 5] = 0
    elif kind == "equal_rows":
        H[:, 9] = H[:, 3]
    elif kind == "rank_one":
        H = H[:, :, :1] * H[:, :1, :]
    elif kind == "zero":
        H[:] = 0
    elif kind == "real":
        H.imag = 0
    elif kind == "tiny":
        H, lam = H * 1e-60, lam * 1e-60
    else:
        H, lam = H * 1e60, lam * 1e60
    if kind == "zero":
        x, s, info = _solve(ctx, cuda, H, b, lam)
        assert not x.any() and not s.any() and not info.any()
        return
    _check(ctx, cuda, H, b, lam)


# batches whose clusters run in several waves or two CTAs to an SM
@pytest.mark.parametrize("m,n,F", [(64, 160, 49), (40, 200, 101), (48, 800, 61), (100, 642, 80), (16, 20, 400)])
def test_wide_solve_qr_waves(cuda, ctx, m, n, F):
    rng = np.random.default_rng(m * 1000 + F)
    H = rng.normal(size=(F, m, n)) + 1j * rng.normal(size=(F, m, n))
    b = rng.normal(size=(F, 1, m)) + 1j * rng.normal(size=(F, 1, m))
    _check(ctx, cuda, H, b, 0.3 * np.linalg.norm(H[0], 2))

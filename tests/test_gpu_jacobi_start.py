"""GPU suite: the FP64 wide solve's Jacobi start (FP32 rotations, first-order
steps as tensor-core products, flagged sweeps) at the edges of its sizes (64 to
256 microphones, pairs padded to clusters of 8, row forms of 128, 192 and 256
rows), on operators that leave it nothing to rotate with, and over the batch;
against the oracle's SVD solve.

Random operators with rows graded over two decades and a fixed lambda of
0.3 s_1: x and s are determined to a few eps, bound 1e-12 (s relative to s_1)."""
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


def _operator(rng, F, m, n):
    H = (rng.normal(size=(F, m, n)) + 1j * rng.normal(size=(F, m, n))) * np.exp(rng.normal(size=(F, m, 1)))
    b = rng.normal(size=(F, 1, m)) + 1j * rng.normal(size=(F, 1, m))
    return H, b


def _check(ctx, cuda, H, b, lam):
    x, s, info = _solve(ctx, cuda, H, b, lam)
    assert not info.any()
    for f in {0, len(H) - 1}:
        U, so, V = O.csvd(H[f])
        assert np.max(np.abs(s[f] - so)) <= 1e-12 * so[0]
        assert relerr(x[f, 0], O.tikhonov(U, so, V, b[f, 0], lam)) < 1e-12


@pytest.mark.parametrize("m,n,F", [(63, 100, 20), (64, 64, 2), (65, 80, 1),
                                   (80, 130, 3), (97, 120, 2), (127, 140, 2), (128, 128, 3), (129, 160, 2),
                                   (191, 200, 2), (193, 250, 1), (255, 260, 1), (256, 256, 1), (257, 260, 1)])
def test_jacobi_start_sizes(cuda, ctx, m, n, F):
    rng = np.random.default_rng(m * 1000 + n)
    H, b = _operator(rng, F, m, n)
    _check(ctx, cuda, H, b, 0.3 * np.linalg.norm(H[0], 2))


@pytest.mark.parametrize("kind", ["orthogonal", "equal_rows", "rank_ten", "steep", "zero", "tiny", "huge"])
def test_jacobi_start_degenerate(cuda, ctx, kind):
    rng = np.random.default_rng(11)
    H, b = _operator(rng, 3, 68, 80)
    lam = 0.3 * np.linalg.norm(H[0], 2)
    if kind == "orthogonal":          # one singular value, 68 times
        H = np.stack([np.linalg.qr(h.T)[0].T for h in H])
        lam = 0.3
    elif kind == "equal_rows":
        H[:, 9] = H[:, 3]
    elif kind == "rank_ten":
        H = H[:, :, :10] @ H[:, :10, :]
    elif kind == "steep":             # singular values over 27 decades
        H = H * 10.0 ** (-0.4 * np.arange(68))[None, :, None]
    elif kind == "zero":
        H[:] = 0
        x, s, info = _solve(ctx, cuda, H, b, lam)
        assert not x.any() and not s.any() and not info.any()
        return
    elif kind == "tiny":
        H, lam = H * 1e-60, lam * 1e-60
    elif kind == "huge":
        H, lam = H * 1e60, lam * 1e60
    if kind == "rank_ten":
        lam = 0.3 * np.linalg.norm(H[0], 2)
    _check(ctx, cuda, H, b, lam)


def test_jacobi_start_batch_independent(cuda, ctx):
    """A bin's result does not depend on the bins beside it, nor on a bin whose
    entries are not finite."""
    rng = np.random.default_rng(12)
    H, b = _operator(rng, 50, 66, 72)
    x, s, info = _solve(ctx, cuda, H, b, 1.0)
    assert not info.any()
    for f in (0, 49):
        x1, s1, _ = _solve(ctx, cuda, H[f:f + 1], b[f:f + 1], 1.0)
        assert np.array_equal(x1[0], x[f]) and np.array_equal(s1[0], s[f])
    H[7, 3, 5] = np.nan
    xn, sn, infon = _solve(ctx, cuda, H, b, 1.0)
    keep = np.arange(50) != 7
    assert infon[7] != 0 and not infon[keep].any()
    assert np.array_equal(xn[keep], x[keep]) and np.array_equal(sn[keep], s[keep])

"""GPU suite: every singular value of a graded operator to its own size.

The FP64 wide solve is a one-sided Jacobi SVD of a pivoted triangular factor,
which keeps the small singular values of H = D B and H = B D (D diagonal, B
well-conditioned) to rounding relative to themselves, and so has its start from
64 microphones on (the odd sizes are padded to clusters of 8; 63 has no start).

With B unitary the singular values are D's entries, to the rounding of H's
entries; graded columns fall in size (what a QR without row interchanges needs).
Each step's error is a few N eps relative to its column: bound 1e-11, where an
error of eps s_1 would leave 1e-4 of the smallest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["columns", "rows"])
@pytest.mark.parametrize("m", [63, 64, 81, 130, 200, 256])
def test_small_singular_values_of_a_graded_operator(cuda, ctx, m, kind):
    from inverseacoustics_gb300 import api
    import torch
    rng = np.random.default_rng(m)
    H = np.linalg.qr(rng.normal(size=(m, m)) + 1j * rng.normal(size=(m, m)))[0]
    d = 10.0 ** (-12.0 * np.arange(m) / (m - 1))
    H = H * d if kind == "columns" else H * rng.permutation(d)[:, None]
    b = torch.ones((1, 1, m), dtype=torch.complex128, device=cuda)
    Hc = torch.as_tensor(np.ascontiguousarray(H.T)[None], device=cuda)
    _, _, s, info = api.solve_batch(ctx, Hc, m, m, b, api.default_config(method=2, lambda_fixed=0.3))
    torch.cuda.synchronize()
    assert int(info[0]) == 0
    assert np.max(np.abs(s.cpu().numpy()[0] - d) / d) < 1e-11

"""GPU suite: the sinc resistance matrix at the edges of its tiles (16 x 16
entries) and of its frequency blocks (9 around a centre, 72 per chunk; direct
phases below 4 bins and for uneven wavenumbers), against the oracle.

Bound: the phase k r carries a few roundings of size 2^-53 k r (k r <= 47
here), so |R - R_oracle| <= 8 (1 + 47) 2^-53 max|R| < 1e-13 max|R|."""
import numpy as np
import pytest

from oracle import ia_oracle as O

pytestmark = pytest.mark.gpu
C, RHO = 343.0, 1.21


@pytest.mark.parametrize("spacing", ["linear", "octave"])
@pytest.mark.parametrize("n,F", [(1, 1), (15, 3), (16, 4), (17, 5), (33, 9), (31, 10), (48, 72), (19, 73), (7, 145)])
def test_sinc_resistance_tile_and_block_edges(cuda, ctx, n, F, spacing):
    from inverseacoustics_gb300 import api
    import torch
    rng = np.random.default_rng(n * 1000 + F)
    x = np.ascontiguousarray(rng.uniform(-0.35, 0.35, (3, n)))
    if n > 16:
        x[:, 16] = x[:, 2]                      # coincident radiators: the limit value off the diagonal too
    f = np.linspace(50.0, 2100.0, F) if spacing == "linear" else 50.0 * 42.0 ** (np.arange(F) / max(1, F - 1))
    k = 2 * np.pi * f / C
    R = api.sinc_resistance_batch(ctx, torch.as_tensor(x, device=cuda), torch.as_tensor(k, device=cuda), 2.5e-4)
    torch.cuda.synchronize()
    R = R.cpu().numpy()
    for i in range(F):
        Ro = O.sinc_resistance(x, k[i], C, RHO, 2.5e-4)
        assert np.max(np.abs(R[i] - Ro)) <= 1e-13 * np.max(np.abs(Ro))
        assert np.array_equal(R[i], R[i].T)


def test_sinc_resistance_keeps_a_bad_wavenumber_to_its_bin(cuda, ctx):
    from inverseacoustics_gb300 import api
    import torch
    x = np.ascontiguousarray(np.random.default_rng(1).uniform(-0.3, 0.3, (3, 20)))
    k = np.linspace(1.0, 30.0, 12)
    k[7] = np.nan
    R = api.sinc_resistance_batch(ctx, torch.as_tensor(x, device=cuda), torch.as_tensor(k, device=cuda), 1e-3)
    torch.cuda.synchronize()
    bad = torch.isnan(R).flatten(1).any(1).cpu().numpy()
    assert bad.tolist() == [i == 7 for i in range(12)]

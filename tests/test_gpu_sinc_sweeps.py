"""GPU suite: every bin of the sinc resistance matrix to its own size, over
sweeps whose ends are decades apart, upwards, downwards and across k = 0,
against the oracle.

Bound: 1e-13 max|R| of the bin, as for the other sweeps (k r <= 100 here at the
top of the 10 kHz sweep, rounded a few times: 8 (1 + 100) 2^-53 < 1e-13)."""
import numpy as np
import pytest

from oracle import ia_oracle as O

pytestmark = pytest.mark.gpu
C, RHO = 343.0, 1.21


@pytest.mark.parametrize("n", [35, 290])   # chunks of 9 bins, of 72
@pytest.mark.parametrize("f0,f1,F", [(1.0, 2000.0, 64), (2000.0, 1.0, 64), (10000.0, 20.0, 64), (0.01, 2000.0, 30),
                                     (2000.0, 20.0, 200), (20.0, 2000.0, 150), (0.0, 900.0, 9), (900.0, 0.0, 9),
                                     (-100.0, 2000.0, 70), (-1.0, -2000.0, 40), (3000.0, 1.0, 4), (5.0, 5.0, 12)])
def test_sinc_resistance_each_bin_to_its_size(cuda, ctx, f0, f1, F, n):
    from inverseacoustics_gb300 import api
    import torch
    rng = np.random.default_rng(F)
    x = np.ascontiguousarray(rng.uniform(-0.16, 0.16, (3, n)))
    x[:, 20] = x[:, 4]
    x[:, 21] = x[:, 5] + 1e-4
    k = 2 * np.pi * np.linspace(f0, f1, F) / C
    R = api.sinc_resistance_batch(ctx, torch.as_tensor(x, device=cuda), torch.as_tensor(k, device=cuda), 2.5e-4)
    torch.cuda.synchronize()
    R = R.cpu().numpy()
    for i in range(F):
        Ro = O.sinc_resistance(x, k[i], C, RHO, 2.5e-4) if k[i] != 0.0 else np.zeros((n, n))
        assert np.max(np.abs(R[i] - Ro)) <= 1e-13 * np.max(np.abs(Ro)), i
        assert np.array_equal(R[i], R[i].T)

"""GPU suite: calls on a device with little free memory.  The slice planes, the
Jacobi starts and the geometry tables of a call are scratch that it can do with
less of: where the device has no more, it works through the bins in smaller groups
and returns the same bits.  `leave` (GB) lies between what a call needs and what
it would take on an empty device."""
import contextlib

import numpy as np
import pytest

from inverseacoustics_gb300 import geometry as g

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _only(leave):
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - int(leave * 1e9), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        torch.cuda.synchronize()
        del hog
        torch.cuda.empty_cache()


def _compare(leave, call):
    """call(context, outputs or None) -> tensors, in a fresh context each"""
    from inverseacoustics_gb300 import api
    import torch
    out = []
    for limit in (None, leave):
        c = api.Context(0)
        with (_only(limit) if limit else contextlib.nullcontext()):
            out.append([t.cpu() for t in call(c)])
        c.close()
    for a, b in zip(*out):
        assert torch.equal(a, b)


def test_operator_solve(cuda):
    from inverseacoustics_gb300 import api
    import torch
    rng = np.random.default_rng(1)
    m, n, F = 128, 130, 1200
    H = torch.as_tensor(rng.normal(size=(8, n, m)) + 1j * rng.normal(size=(8, n, m)), device=cuda).repeat(F // 8, 1, 1)
    b = torch.as_tensor(rng.normal(size=(F, 1, m)) + 1j * rng.normal(size=(F, 1, m)), device=cuda)
    cfg = api.default_config(method=2, lambda_fixed=0.5)
    _compare(2.0, lambda c: api.solve_batch(c, H, m, n, b, cfg))


@pytest.fixture(scope="module")
def sphere(cuda):
    import torch
    nodes, elems = g.icosphere(3, 0.1)
    rng = np.random.default_rng(2)
    F = 64
    mics = torch.as_tensor(g.hemisphere_array(rng, 120, 0.3), device=cuda)
    k = torch.as_tensor(2 * np.pi * np.linspace(200.0, 1900.0, F) / 343.0, device=cuda)
    p = torch.as_tensor(g.complex_normal(rng, (F, 1, 120)), device=cuda)
    return nodes, elems, mics, k, p


def _with_mesh(sphere, fn):
    from inverseacoustics_gb300 import api

    def call(c):
        mesh = api.Mesh(c, sphere[0], sphere[1])
        out = fn(c, mesh)
        mesh.close()
        return out
    return call


@pytest.mark.parametrize("prec,F,leave", [(0, 64, 1.6), (1, 16, 0.72)])
def test_ibem_transfer(cuda, sphere, prec, F, leave):
    from inverseacoustics_gb300 import api
    cfg = api.default_config(precision=prec)
    k = sphere[3][:F].contiguous()
    _compare(leave, _with_mesh(sphere, lambda c, mesh: api.ibem_transfer_batch(c, mesh, sphere[2], k, cfg)))


def test_ibem_solve(cuda, sphere):
    from inverseacoustics_gb300 import api
    cfg = api.default_config(method=2, lambda_fixed=1e-3)
    _compare(1.7, _with_mesh(sphere, lambda c, mesh: api.ibem_solve_batch(c, mesh, sphere[2], sphere[3], sphere[4],
                                                                          cfg)))


def test_radiation_modes(cuda):
    from inverseacoustics_gb300 import api
    import torch
    rng = np.random.default_rng(3)
    n, F = 512, 160
    Q = np.linalg.qr(rng.normal(size=(n, n)))[0]
    R = torch.as_tensor((Q * 0.7 ** np.arange(n)) @ Q.T, device=cuda)[None]
    R = (R + R.transpose(1, 2)) * (1 + torch.arange(F, device=cuda, dtype=torch.float64) / F)[:, None, None]
    _compare(0.6, lambda c: api.radiation_modes_batch(c, R, 6, api.default_config()))


def test_bem_modes(cuda):
    from inverseacoustics_gb300 import api
    import torch
    nodes, elems = g.icosphere(2, 0.1)
    rng = np.random.default_rng(4)
    mics = torch.as_tensor(g.hemisphere_array(rng, 16, 0.3), device=cuda)
    k = torch.as_tensor(2 * np.pi * np.linspace(200.0, 1900.0, 128) / 343.0, device=cuda)
    call = _with_mesh((nodes, elems), lambda c, mesh: [t for t in api.bem_modes_batch(c, mesh, mics, k, 6)
                                                       if t is not None])
    _compare(0.6, call)


def test_array_design(cuda):
    from inverseacoustics_gb300 import api
    from test_gpu_adjoint import _case, _dev_args
    args = _dev_args(_case(5, 16, 2, 800, 2), cuda)
    _compare(0.2, lambda c: api.esm_design_batch(c, *args))

"""A kernel's dynamic shared memory limit belongs to the function, not to a launch: a
limit set to each launch's own size is lowered by another host thread between the
setting and the launch, which then fails.  So it is set in one place, to one value
per kernel (CPU: the sources), and two threads with a context each, whose sizes ask
the same kernels for different amounts, get what one thread gets (GPU)."""
import glob
import os
import threading

import pytest

from conftest import ROOT


def test_the_limit_is_set_in_one_place():
    files = glob.glob(os.path.join(ROOT, "inverseacoustics_gb300", "csrc", "*"))
    assert [os.path.basename(f) for f in files if "cudaFuncAttributeMaxDynamicSharedMemorySize" in open(f).read()] == [
        "ia_internal.h"]


@pytest.mark.gpu
def test_two_threads_of_different_sizes(cuda):
    from inverseacoustics_gb300 import api
    import torch
    cfg = api.default_config(method=2, lambda_fixed=0.5)
    gen = torch.Generator(device=cuda).manual_seed(1)
    out, errors = {}, []

    def problem(m):
        return [torch.randn(s, dtype=torch.complex128, device=cuda, generator=gen) for s in ((1, m, m), (1, 1, m))]

    def solve(m, H, b, count):
        try:
            stream = torch.cuda.Stream()
            c = api.Context(0, stream)
            with torch.cuda.stream(stream):
                for _ in range(count):
                    x = api.solve_batch(c, H, m, m, b, cfg)[0]
            stream.synchronize()
            out.setdefault(m, []).append(x)
            c.close()
        except Exception as e:   # noqa: BLE001 -- a thread's failure is the test's
            errors.append(e)

    sizes = {m: problem(m) for m in (150, 192)}
    torch.cuda.synchronize()
    for m, (H, b) in sizes.items():
        solve(m, H, b, 1)
    threads = [threading.Thread(target=solve, args=(m, H, b, 150)) for m, (H, b) in sizes.items()]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert all(torch.equal(a, b) for a, b in out.values())

"""The first solve on a new engine, with work queued on the default stream and
without: the solvers' workspaces are prepared on the solve's own stream, so the
results are the same bit for bit (the engine's stream does not wait for the
default one, and a clear that did would land in the middle of the solve)."""
import numpy as np
import pytest

from conftest import sphere

pytestmark = pytest.mark.gpu


def _solve(call, busy):
    import torch
    from hacapk_b200 import abi, configs
    from hacapk_b200.engine import Engine
    engines = []

    def E(*a, batch=False, **k):
        engines.append(Engine.batch(*a, **k) if batch else Engine(*a, **k))
        return engines[-1]
    if "batch" in call:
        inst = configs.c5(count=5, seed=5, max_level=3)
        Hs, b = [H for H, _ in inst], np.concatenate([x for _, x in inst])
        hi = E(Hs, batch=True)
        lo = E(Hs, batch=True, precision=abi.HBX_BF16)
    else:
        H = sphere(3)
        b = np.random.default_rng(3).standard_normal((H.nd, 64))
        hi = E(H.st, H.nd)
        lo = E(H.st, H.nd, precision=abi.HBX_FP32, nrhs=64)
    torch.cuda.synchronize()
    if busy:  # one resident thread for some 0.2 s
        torch.cuda._sleep(400_000_000)
    if call == "batch":
        u, info = hi.bicgstab_batch_host(b, tol=1e-8)
    elif call == "batch_refined":
        u, info = hi.bicgstab_batch_refined_host(lo, b, tol=1e-10, inner_tol=1e-2)
    elif call == "multi":
        u, info = hi.bicgstab_multi_host(lo, b, tol=1e-10)
    else:
        f = hi.bicgstab_pipe_host if call == "pipe" else hi.gcr_host
        u, i = f(b[:, 0].copy(), tol=1e-8)
        info = [i]
    torch.cuda.synchronize()
    for e in engines:
        e.close()
    assert all(i["status"] == 0 for i in info)
    return u, [i["iterations"] for i in info]


@pytest.mark.parametrize("call", ["batch", "batch_refined", "multi", "pipe", "gcr"])
def test_first_solve_ignores_the_default_stream(gpu, build_libs, call):
    u0, n0 = _solve(call, False)
    u1, n1 = _solve(call, True)
    assert n0 == n1
    assert np.array_equal(u0, u1)

"""A grid barrier that cannot complete in the first product of a solve
(hbx_debug_stall_next_barrier; the waits are bounded by HBX_TIMEOUT_MS and give
up): the step kernels find the error word set, the solve ends with
HBX_ERR_TIMEOUT, and the next solve on the engine is right."""
import numpy as np
import pytest

from conftest import sphere

pytestmark = pytest.mark.gpu

SOLVES = [("bicgstab_host", 0), ("bicgstab_host", 1), ("bicgstab_pipe_host", 0), ("bicgstab_pipe_host", 1)]


@pytest.mark.parametrize("solver,precision", SOLVES)
def test_expired_wait_ends_the_solve(gpu, build_libs, monkeypatch, solver, precision):
    from hacapk_b200.engine import Engine
    monkeypatch.setenv("HBX_TIMEOUT_MS", "100")
    H = sphere(3)
    E = Engine(H.st, H.nd, precision=precision)
    b = np.random.default_rng(1).standard_normal(H.nd)
    solve = getattr(E, solver)
    u0, i0 = solve(b, tol=1e-6, check=False)  # (the FP32 pipelined recurrence stalls above 1e-6 on this b)
    assert E.lib.hbx_debug_stall_next_barrier(E._h) == 0
    _, i = solve(b, tol=1e-6, max_iter=64, check=False)
    assert i["status"] == 4
    u1, i1 = solve(b, tol=1e-6, check=False)
    assert [i1[k] for k in ("status", "iterations", "relres")] == [i0[k] for k in ("status", "iterations", "relres")]
    assert np.array_equal(u0, u1)
    E.close()


@pytest.mark.parametrize("solver,precision", SOLVES)
def test_expired_wait_ends_the_solve_at_once(gpu, build_libs, monkeypatch, solver, precision):
    """A large step limit queues no more launches than the steps under way."""
    from hacapk_b200.engine import Engine
    monkeypatch.setenv("HBX_TIMEOUT_MS", "100")
    H = sphere(3)
    E = Engine(H.st, H.nd, precision=precision)
    b = np.random.default_rng(1).standard_normal(H.nd)
    assert E.lib.hbx_debug_stall_next_barrier(E._h) == 0
    _, i = getattr(E, solver)(b, tol=1e-6, max_iter=4000, batch=8, check=False)
    assert i["status"] == 4
    assert i["launches"] <= 2 * 4 * 8 + 7  # two batches of steps, four launches a step at most, and the ends
    E.close()

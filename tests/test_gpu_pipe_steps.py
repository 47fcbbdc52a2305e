"""Pipelined BiCGSTAB with several steps in a launch (k_pipe_steps): the
replay's bits wherever the solve ends within a launch or at its edge, with one
and two blocks of the dots' grid per CTA, at the last row that the launch takes
(512 per CTA) and the first that goes to the graph, on matrices that leave most
CTAs without work too."""
import ctypes as C
from types import SimpleNamespace

import numpy as np
import pytest

from conftest import pipe_replay, sphere

pytestmark = pytest.mark.gpu

BATCHES = (1, 2, 3, 8, 1 << 20)


def _dense(nd):
    """nd x nd, I + 0.4 E/||E||, in up to four leaves."""
    import test_plan as tp
    E = np.random.default_rng(nd).standard_normal((nd, nd))
    A = np.eye(nd) + 0.4 * E / np.linalg.norm(E, 2)
    half = max(1, nd // 2)
    leaves = [(2, 0, r0 + 1, r1 - r0, c0 + 1, c1 - c0, np.ascontiguousarray(A[r0:r1, c0:c1]).ravel())
              for r0, r1 in ((0, half), (half, nd)) for c0, c1 in ((0, half), (half, nd)) if r1 > r0 and c1 > c0]
    P, keep = tp._custom(leaves, nd)
    return SimpleNamespace(st=C.pointer(P), nd=nd, keep=(P, keep))


@pytest.mark.parametrize("nd,num_ctas", [(33, 1), (256, 5), (257, 148), (512, 1), (513, 1), (769, 2), (1280, 3)])
def test_launch_length_does_not_show(gpu, build_libs, nd, num_ctas):
    from hacapk_b200.engine import Engine
    H = sphere(3) if nd == 1280 else _dense(nd)
    assert H.nd == nd
    E = Engine(H.st, nd, num_ctas=num_ctas)
    b = np.random.default_rng(7).standard_normal(nd)
    _, steps, _, status = pipe_replay(H, b, tol=1e-8, max_iter=200, num_ctas=num_ctas)
    assert status == 0
    for max_iter in sorted({1, 2, 3, 8, steps - 1, steps, steps + 1} - {0}):
        ur, nr, rel, status = pipe_replay(H, b, tol=1e-8, max_iter=max_iter, num_ctas=num_ctas)
        for batch in BATCHES:
            u, i = E.bicgstab_pipe_host(b, tol=1e-8, max_iter=max_iter, batch=batch, check=False)
            assert (i["iterations"], i["relres"], i["status"]) == (nr, rel, status)
            assert np.array_equal(u, ur)
    E.close()
    del H


@pytest.mark.parametrize("batch", BATCHES)
def test_exact_solution_breaks_down_with_u_kept(gpu, build_libs, batch):
    """A = I: the first step's y is zero, zeta is not a number, u stays."""
    import test_plan as tp
    from hacapk_b200.engine import Engine
    nd = 40
    P, keep = tp._custom([(2, 0, 1, nd, 1, nd, np.eye(nd).ravel())], nd)
    E = Engine(C.pointer(P), nd)
    u0 = np.full(nd, 2.0)
    u, i = E.bicgstab_pipe_host(np.arange(1.0, nd + 1), u0=u0, batch=batch, check=False)
    assert i["status"] == 5 and i["iterations"] == 0 and np.array_equal(u, u0)
    v, i = E.bicgstab_pipe_host(u0, u0=u0, batch=batch)  # the engine still answers
    assert i["status"] == 0 and np.array_equal(v, u0)
    E.close()

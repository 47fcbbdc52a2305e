"""BiCGSTAB with several steps in a launch (k_bicg_steps): where the solve
ends within a launch, at its edge or in the next, the result is the same bit
for bit, on matrices that leave most CTAs without work too."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BATCHES = (1, 2, 3, 8, 64)


def _dense(nd, seed):
    """nd x nd, I + 0.4 E/||E||: every singular value in [0.6, 1.4]."""
    E = np.random.default_rng(seed).standard_normal((nd, nd))
    return np.eye(nd) + 0.4 * E / np.linalg.norm(E, 2)


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("nd,num_ctas", [(1, 0), (33, 0), (33, 1), (257, 0), (257, 5)])
def test_launch_length_does_not_show(gpu, build_libs, nd, num_ctas, precision):
    import test_plan as tp
    from hacapk_b200.engine import Engine
    A = _dense(nd, nd)
    half = max(1, nd // 2)
    leaves = [(2, 0, r0 + 1, r1 - r0, c0 + 1, c1 - c0, np.ascontiguousarray(A[r0:r1, c0:c1]).ravel())
              for r0, r1 in ((0, half), (half, nd)) for c0, c1 in ((0, half), (half, nd)) if r1 > r0 and c1 > c0]
    P, keep = tp._custom(leaves, nd)
    E = Engine(C.pointer(P), nd, precision=precision, num_ctas=num_ctas)
    b = A @ np.random.default_rng(7).standard_normal(nd)
    tol = 1e-8
    full, info = E.bicgstab_host(b, tol=tol, max_iter=200, batch=1)
    steps = info["iterations"]
    assert info["status"] == 0 and info["relres"] < tol
    if precision == 0:
        # ||u - A^-1 b|| <= ||b|| relres / 0.6, with the rounding of the recurrence well below tol
        assert np.linalg.norm(full - np.linalg.solve(A, b)) <= 2.0 * tol / 0.6 * np.linalg.norm(b)
    for max_iter in sorted({0, 1, 2, 3, 7, 8, 9, steps - 1, steps, steps + 1} - {-1}):
        first = None
        for batch in BATCHES:
            u, i = E.bicgstab_host(b, tol=tol, max_iter=max_iter, batch=batch, check=False)
            assert i["iterations"] == min(max_iter, steps)
            assert (i["status"] == 0) == (max_iter >= steps)
            first = first or (u, i["relres"], i["true_relres"])
            assert np.array_equal(u, first[0]) and (i["relres"], i["true_relres"]) == first[1:]
        if max_iter >= steps:
            assert np.array_equal(first[0], full)
        if max_iter == 0:
            assert np.array_equal(first[0], np.zeros(nd))
    E.close()


@pytest.mark.parametrize("batch", BATCHES)
def test_guess_that_solves_takes_no_step(gpu, build_libs, batch):
    import test_plan as tp
    from hacapk_b200.engine import Engine
    nd = 40
    A = np.diag(2.0 ** (np.arange(nd) % 5))  # every product exact
    P, keep = tp._custom([(2, 0, 1, nd, 1, nd, A.ravel())], nd)
    E = Engine(C.pointer(P), nd)
    u0 = np.arange(1.0, nd + 1)
    u, info = E.bicgstab_host(A @ u0, u0=u0, batch=batch)
    assert info["iterations"] == 0 and info["true_relres"] == 0.0 and np.array_equal(u, u0)
    E.close()

"""The batched and multi-RHS solvers queue a batch of steps while the flag of the
one before is read: the batch length shows in no bit of the result, at step
limits below, at and just past it; instances that break down end alone; and a
plain engine is a batch of one."""
import ctypes as C
from types import SimpleNamespace

import numpy as np
import pytest

from conftest import sphere

pytestmark = pytest.mark.gpu

BATCHES = (1, 2, 3, 8, 64)


def _leaf(A):
    import test_plan as tp
    nd = A.shape[0]
    P, keep = tp._custom([(2, 0, 1, nd, 1, nd, np.ascontiguousarray(A).ravel())], nd)
    return SimpleNamespace(st=C.pointer(P), nd=nd, A=A, keep=(P, keep))


def _dense(nd, seed):
    """I + 0.4 E/||E||."""
    E = np.random.default_rng(seed).standard_normal((nd, nd))
    return _leaf(np.eye(nd) + 0.4 * E / np.linalg.norm(E, 2))


@pytest.mark.parametrize("precision", [0, 1, 2])
def test_batch_length_does_not_show(gpu, build_libs, precision):
    from hacapk_b200.engine import Engine
    Hs = [_dense(33, 1), _dense(2500, 2), _dense(257, 3), _dense(1, 4)]
    E = Engine.batch(Hs, precision=precision)
    b = np.concatenate([H.A @ np.random.default_rng(H.nd).standard_normal(H.nd) for H in Hs])
    full, infos = E.bicgstab_batch_host(b, tol=1e-8, max_iter=200, batch=1)
    steps = [i["iterations"] for i in infos]
    assert all(i["status"] == 0 and i["relres"] < 1e-8 for i in infos)
    top = max(steps)
    for max_iter in sorted({0, 1, 2, 3, 7, 8, 9, top - 1, top, top + 1}):
        first = None
        for batch in BATCHES:
            u, infos = E.bicgstab_batch_host(b, tol=1e-8, max_iter=max_iter, batch=batch)
            assert [i["iterations"] for i in infos] == [min(max_iter, s) for s in steps]
            assert [i["status"] for i in infos] == [0 if max_iter >= s else 6 for s in steps]
            got = (u, [(i["relres"], i["true_relres"]) for i in infos])
            first = first or got
            assert np.array_equal(u, first[0]) and got[1] == first[1]
        if max_iter >= top:
            assert np.array_equal(first[0], full)
    assert top > 3
    E.close()


def test_multi_rhs_batch_length_does_not_show(gpu, build_libs):
    from hacapk_b200.engine import Engine
    H = sphere(3)
    E, M = Engine(H.st, H.nd), Engine(H.st, H.nd, precision=1, nrhs=64)
    B = np.random.default_rng(5).standard_normal((H.nd, 64))
    B[:, 7] = 0.0
    B[:, 11] = 1.0  # fewer steps than the others
    for max_iter in (1, 2, 3, 4, 5, 8, 9, 500):
        first = None
        for batch in BATCHES:
            U, infos = E.bicgstab_multi_host(M, B, tol=1e-8, max_iter=max_iter, batch=batch)
            got = [(i["iterations"], i["status"], i["relres"]) for i in infos]
            first = first or (U, got)
            assert np.array_equal(U, first[0]) and got == first[1]
        assert infos[7]["iterations"] == 0 and infos[7]["status"] == 0 and not U[:, 7].any()
        assert all((i["status"] == 0) == (i["true_relres"] <= 1e-8) for i in infos)
        assert max(i["iterations"] for i in infos) >= min(max_iter, 8)
    assert all(i["status"] == 0 for i in infos)
    for X in (E, M):
        X.close()


@pytest.mark.parametrize("batch", BATCHES)
def test_broken_instances_end_alone(gpu, build_libs, batch):
    """Skew-symmetric: rh . Ap = 0 in the first step, u stays.  A = e0 e0^T + e1 e0^T
    with b = e0: At = 0, the first step's u = e0 is kept."""
    import oracle
    from hacapk_b200.engine import Engine
    nd = 64
    S, N = np.zeros((nd, nd)), np.zeros((nd, nd))
    for k in range(0, nd, 2):
        S[k, k + 1], S[k + 1, k] = 1.0, -1.0
    N[0, 0] = N[1, 0] = 1.0
    e0 = np.eye(nd)[0]
    Hs = [sphere(3), _leaf(S), sphere(2), _leaf(N), _leaf(2.0 * np.eye(nd))]
    bs = [np.ones(Hs[0].nd), e0, np.ones(Hs[2].nd), e0, np.arange(1.0, nd + 1)]
    E = Engine.batch(Hs)
    u, infos = E.bicgstab_batch_host(np.concatenate(bs), tol=1e-8, max_iter=300, batch=batch)
    us = [u[E.offsets[k]:E.offsets[k + 1]] for k in range(len(Hs))]
    assert [i["status"] for i in infos] == [0, 5, 0, 5, 0]
    assert infos[1]["iterations"] == 0 and not us[1].any()
    assert infos[3]["iterations"] == 1 and np.array_equal(us[3], e0)
    assert np.array_equal(us[4], bs[4] / 2.0)
    for k in (0, 2):
        rel = np.linalg.norm(bs[k] - oracle.matvec(Hs[k].st, us[k])) / np.linalg.norm(bs[k])
        assert rel < 1.05e-8
    E.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_plain_engine_is_a_batch_of_one(gpu, build_libs, precision):
    import oracle
    from hacapk_b200.engine import Engine
    H = sphere(3)
    b = 1.0 + 1e-3 * np.random.default_rng(9).standard_normal(H.nd)
    E, B = Engine(H.st, H.nd, precision=precision), Engine.batch([H], precision=precision)
    u, infos = E.bicgstab_batch_host(b, tol=1e-8)
    v, ref = B.bicgstab_batch_host(b, tol=1e-8)
    assert infos[0]["status"] == 0 and infos[0]["iterations"] == ref[0]["iterations"]
    assert np.array_equal(u, v)
    if precision == 0:
        rel = np.linalg.norm(b - oracle.matvec(H.st, u)) / np.linalg.norm(b)
        assert rel < 1.05e-8
    w, infos = E.bicgstab_batch_host(b, u0=u, tol=1e-8)  # solved already
    assert infos[0]["iterations"] == 0 and np.array_equal(w, u)
    E.close()
    B.close()

"""Batched BiCGSTAB where the instances take groups of 1, 2, 4 and 8 CTAs of the
vector kernels in one launch, the smaller groups sharing clusters: every
instance solves as it does alone, whatever lies beside it."""
import numpy as np
import pytest

from conftest import sphere

pytestmark = pytest.mark.gpu


def _dense(nd, seed):
    """nd x nd, I + 0.4 E/||E||, one leaf."""
    import ctypes as C
    from types import SimpleNamespace
    import test_plan as tp
    E = np.random.default_rng(seed).standard_normal((nd, nd))
    A = np.eye(nd) + 0.4 * E / np.linalg.norm(E, 2)
    P, keep = tp._custom([(2, 0, 1, nd, 1, nd, A.ravel())], nd)
    return SimpleNamespace(st=C.pointer(P), nd=nd, keep=(P, keep, A))


# rows of the instances: at the edges of the groups (2,048 rows a CTA), more
# small ones than a cluster holds, and an odd last cluster
MIXES = {
    "one": [1],
    "edges": [2048, 2049, 1, 33],
    "eight": [20480, 320, 320, 1280],
    "all_sizes": [320, 5120, 20480, 1280, 2049, 320, 320, 4097, 7, 320, 320],
}


@pytest.mark.parametrize("mix", MIXES)
def test_mixed_groups_solve_every_instance(gpu, build_libs, mix):
    import oracle
    from hacapk_b200.engine import Engine
    levels = {320: 2, 1280: 3, 5120: 4, 20480: 5}
    Hs = [sphere(levels[n]) if n in levels else _dense(n, n) for n in MIXES[mix]]
    rng = np.random.default_rng(11)
    bs = [1.0 + 1e-3 * rng.standard_normal(H.nd) for H in Hs]
    E = Engine.batch(Hs)
    u, infos = E.bicgstab_batch_host(np.concatenate(bs), tol=1e-8, max_iter=300)
    for k, (H, b) in enumerate(zip(Hs, bs)):
        _, n_ref, _, _ = oracle.bicgstab(H.st, b, tol=1e-8, max_iter=300, kind="restated")
        uk = u[E.offsets[k]:E.offsets[k + 1]]
        rel = np.linalg.norm(b - oracle.matvec(H.st, uk)) / np.linalg.norm(b)
        assert infos[k]["status"] == 0 and rel < 1.05e-8, (k, H.nd, infos[k], rel)
        if H.nd > 1:  # (one row is exact after half a step, where the oracle, like the reference, goes on to 0 / 0)
            assert abs(infos[k]["iterations"] - n_ref) <= 3, (k, H.nd, infos[k]["iterations"], n_ref)
        assert abs(infos[k]["bnorm"] - np.linalg.norm(b)) <= 1e-14 * np.linalg.norm(b)
        assert abs(rel - infos[k]["true_relres"]) <= 1e-3 * rel + 1e-15
    E.close()

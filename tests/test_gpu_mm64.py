"""The FP64 product with 64 right-hand sides (hbx_mm64.cu) inside
hbx_bicgstab_multi: with no steps allowed the call returns ||B - H U|| / ||B||
of the given U, and with B = A U that is the product's rounding alone."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _leaves(widths, seed):
    rng = np.random.default_rng(seed)
    nd = sum(widths)
    A = np.zeros((nd, nd))
    leaves = []
    cuts = np.cumsum([0, *widths])
    ranks = [1, 7, 8, 9, 33, 64, 65]
    for a in range(len(widths)):
        for b in range(len(widths)):
            r0, r1, c0, c1 = (int(v) for v in (cuts[a], cuts[a + 1], cuts[b], cuts[b + 1]))
            if a != b and (a + b) % 2:
                kt = ranks[(3 * a + b) % len(ranks)]
                U, V = rng.standard_normal((r1 - r0, kt)), rng.standard_normal((c1 - c0, kt))
                leaves.append((1, kt, r0 + 1, r1 - r0, c0 + 1, c1 - c0, np.concatenate([V.T.ravel(), U.T.ravel()])))
                A[r0:r1, c0:c1] = U @ V.T
            else:
                D = rng.standard_normal((r1 - r0, c1 - c0))
                leaves.append((2, 0, r0 + 1, r1 - r0, c0 + 1, c1 - c0, D.ravel()))
                A[r0:r1, c0:c1] = D
    return leaves, A


@pytest.mark.parametrize("merge", [0, -1, 1])
@pytest.mark.parametrize("widths", [(1, 5, 8), (9, 31, 33), (64, 65, 100), (15, 16, 17, 400), (1025, 30)])
def test_residual_is_rounding(gpu, build_libs, widths, merge):
    import test_plan as tp
    from hacapk_b200 import abi
    from hacapk_b200.engine import Engine
    leaves, A = _leaves(widths, sum(widths))
    nd = A.shape[0]
    P, keep = tp._custom(leaves, nd)
    E = Engine(C.pointer(P), nd, merge=merge)
    Em = Engine(C.pointer(P), nd, precision=abi.HBX_FP32, nrhs=abi.HBX_NRHS)
    U = np.random.default_rng(3).standard_normal((nd, 64))
    B = A @ U
    # a low-rank entry takes two products and both sides round: (nd + rank + 4) units each, to first order
    absA = np.zeros_like(A)
    for lt, kt, r0, n, c0, m, data in leaves:
        blk = (slice(r0 - 1, r0 - 1 + n), slice(c0 - 1, c0 - 1 + m))
        absA[blk] = (np.abs(data[m * kt:]).reshape(kt, n).T @ np.abs(data[:m * kt]).reshape(kt, m) if lt == 1
                     else np.abs(data).reshape(n, m))
    bound = 2 * (nd + 70) * 2.0 ** -53 * np.linalg.norm(absA @ np.abs(U), axis=0) / np.linalg.norm(B, axis=0)
    _, infos = E.bicgstab_multi_host(Em, B, U0=U, tol=0.0, max_iter=0)
    rel = np.array([i["true_relres"] for i in infos])
    assert np.all(rel <= bound)
    # a wrong U shows: one entry of one column off by a half
    U2 = U.copy()
    U2[nd // 2, 5] += 0.5
    _, infos = E.bicgstab_multi_host(Em, B, U0=U2, tol=0.0, max_iter=0)
    want = 0.5 * np.linalg.norm(A[:, nd // 2]) / np.linalg.norm(B[:, 5])
    assert abs(infos[5]["true_relres"] - want) <= 1e-10 * want
    assert all(infos[j]["true_relres"] <= bound[j] for j in range(64) if j != 5)
    E.close()
    Em.close()


def test_vectors_off_a_16_byte_boundary(gpu, build_libs):
    """U on any double: the single-vector products take over, the same residual to rounding."""
    import test_plan as tp
    import torch
    from hacapk_b200 import abi
    from hacapk_b200.engine import Engine
    leaves, A = _leaves((30, 41, 50), 4)
    nd = A.shape[0]
    P, keep = tp._custom(leaves, nd)
    E = Engine(C.pointer(P), nd)
    Em = Engine(C.pointer(P), nd, precision=abi.HBX_FP32, nrhs=abi.HBX_NRHS)
    rng = np.random.default_rng(5)
    U, B = rng.standard_normal((nd, 64)), rng.standard_normal((nd, 64))
    got = []
    for off in (0, 1):
        b = torch.from_numpy(B).cuda()
        buf = torch.zeros(nd * 64 + 2, dtype=torch.float64, device="cuda")
        buf[off:off + nd * 64] = torch.from_numpy(U.ravel()).cuda()
        infos = E.bicgstab_multi_dev(Em, b.data_ptr(), buf.data_ptr() + 8 * off, tol=0.0, max_iter=0, check=False)
        got.append([i["true_relres"] for i in infos])
    want = np.linalg.norm(B - A @ U, axis=0) / np.linalg.norm(B, axis=0)
    assert np.allclose(got[0], want, rtol=1e-12, atol=0) and np.allclose(got[1], want, rtol=1e-12, atol=0)
    E.close()
    Em.close()

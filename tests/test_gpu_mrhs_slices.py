"""The multi-RHS product (k_matmat) at the edges of its slices, tiles and
blocks: with one-hot right-hand sides every entry of Y is one factor in TF32
(10 mantissa bits: at most 2^-10 off), and a dense leaf's neighbours stay out."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(leaves, nd, num_ctas):
    import test_plan as tp
    from hacapk_b200 import abi
    from hacapk_b200.engine import Engine
    P, keep = tp._custom(leaves, nd)
    return Engine(C.pointer(P), nd, precision=abi.HBX_FP32, nrhs=abi.HBX_NRHS, num_ctas=num_ctas)


def _product(E, X, offset):
    """Y = H X with X lying `offset` floats past a 256-byte boundary."""
    import torch
    buf = torch.zeros(X.size + 64, dtype=torch.float32, device="cuda")
    buf[offset:offset + X.size] = torch.from_numpy(X.ravel()).cuda()
    y = torch.full((X.shape[0], 64), np.nan, dtype=torch.float64, device="cuda")
    E.matmat_dev(buf.data_ptr() + 4 * offset, y.data_ptr())
    E.sync()
    return y.cpu().numpy()


@pytest.mark.parametrize("num_ctas", [0, 3])
@pytest.mark.parametrize("widths", [(1, 3, 4), (7, 8, 9), (31, 32, 33), (63, 64, 65), (127, 128, 129), (255, 257, 700)])
def test_one_hot_columns(gpu, build_libs, widths, num_ctas):
    rng = np.random.default_rng(sum(widths))
    nd = 1 + sum(widths)
    A = np.zeros((nd, nd))
    leaves = []
    rows = [0, 1, nd // 3, nd]  # blocks of 1 row, and of more than one row atom
    cuts = np.cumsum([0, 1, *widths])
    for a in range(3):
        r0, r1 = rows[a], rows[a + 1]
        if r1 <= r0:
            continue
        for b in range(4):
            c0, c1 = int(cuts[b]), int(cuts[b + 1])
            if (a + b) % 3 == 2 and r1 - r0 > 1:  # low rank: one power of two per column of V
                kt = min(r1 - r0, 1 + 20 * b)
                U = rng.standard_normal((r1 - r0, kt)).astype(np.float32).astype(np.float64)
                V = np.zeros((c1 - c0, kt))
                V[np.arange(c1 - c0), np.arange(c1 - c0) % kt] = rng.choice([1.0, -2.0, 0.5], c1 - c0)
                leaves.append((1, kt, r0 + 1, r1 - r0, c0 + 1, c1 - c0, np.concatenate([V.T.ravel(), U.T.ravel()])))
                A[r0:r1, c0:c1] = U @ V.T
            else:
                D = rng.standard_normal((r1 - r0, c1 - c0))
                leaves.append((2, 0, r0 + 1, r1 - r0, c0 + 1, c1 - c0, D.ravel()))
                A[r0:r1, c0:c1] = D
    E = _engine(leaves, nd, num_ctas)
    for c0 in range(0, nd, 64):
        X = np.zeros((nd, 64), np.float32)
        n = min(64, nd - c0)
        X[c0 + np.arange(n), np.arange(n)] = 1.0
        for offset in (0, 1, 6):
            Y = _product(E, X, offset)
            # float storage (2^-24) and TF32 (2^-10) of the factor, both in one bound
            assert np.all(np.abs(Y[:, :n] - A[:, c0:c0 + n]) <= 1.01 * 2.0 ** -10 * np.abs(A[:, c0:c0 + n]))
            assert np.all(Y[:, n:] == 0.0)
    E.close()

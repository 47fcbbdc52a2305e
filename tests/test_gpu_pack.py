"""The packed stream formed on the device (hbx_pack.cu): the product with a
unit vector returns one column of H, each entry the stored factor times a power
of two plus zeros, so it equals the rounded factor exactly."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rounded(v, prec):
    """v in the storage precision: double, float, or bfloat16 (nearest, ties to even)."""
    if prec == 0:
        return v
    if prec == 1:
        return v.astype(np.float32).astype(np.float64)
    import torch
    return torch.from_numpy(v).to(torch.bfloat16).to(torch.float64).numpy()


def _lowrank(rng, ndl, ndt, kt):
    """U (ndl x kt) arbitrary, V (ndt x kt) with one power of two per column t: row t mod kt."""
    U = rng.standard_normal((ndl, kt))
    V = np.zeros((ndt, kt))
    V[np.arange(ndt), np.arange(ndt) % kt] = rng.choice([1.0, -2.0, 0.5], ndt)
    return U, V


def _columns(E, cols):
    out = []
    for j in cols:
        e = np.zeros(E.nd)
        e[j] = 1.0
        out.append(E.matvec_host(e)[0])
    return np.stack(out, 1)


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("num_ctas", [0, 1])
def test_columns_equal_the_stored_factors(gpu, build_libs, prec, num_ctas):
    """Ragged leaves beside one dense leaf that takes the stream past the 32 MB
    from which the device packs."""
    import test_plan as tp
    from hacapk_b200.engine import Engine
    rng = np.random.default_rng(11)
    # row and column cuts at the edges of a tile (32 columns), a row atom (32)
    # and a slab (64 rows): 1, 31, 32, 33, 64, 65 and a ragged rest
    cuts = np.cumsum([0, 1, 31, 32, 33, 64, 65, 27])
    pad = [2100, 2960, 4180][prec]  # rows and columns of the large leaf: over 32 MB at 8, 4, 2 bytes a word
    small = int(cuts[-1])
    nd = small + pad
    leaves, want = [], np.zeros((nd, nd))
    B = rng.standard_normal((pad, pad))
    leaves.append((2, 0, small + 1, pad, small + 1, pad, B.ravel()))
    want[small:, small:] = _rounded(B, prec)
    ranks = [1, 3, 31, 32, 33, 63, 64, 65]
    for a in range(len(cuts) - 1):
        for b in range(len(cuts) - 1):
            r0, ndl, c0, ndt = cuts[a], cuts[a + 1] - cuts[a], cuts[b], cuts[b + 1] - cuts[b]
            if (a + b) % 2:
                kt = ranks[(3 * a + b) % len(ranks)]
                U, V = _lowrank(rng, ndl, ndt, kt)
                data = np.concatenate([V.T.ravel(), U.T.ravel()])
                leaves.append((1, kt, r0 + 1, ndl, c0 + 1, ndt, data))
                want[r0:r0 + ndl, c0:c0 + ndt] = _rounded(U, prec) @ V.T
            else:
                A = rng.standard_normal((ndl, ndt)) * 10.0 ** rng.integers(-30, 30, (ndl, ndt))
                A[rng.random((ndl, ndt)) < 0.05] = 0.0
                leaves.append((2, 0, r0 + 1, ndl, c0 + 1, ndt, A.ravel()))
                want[r0:r0 + ndl, c0:c0 + ndt] = _rounded(A, prec)
    P, keep = tp._custom(leaves, nd)
    E = Engine(C.pointer(P), nd, precision=prec, num_ctas=num_ctas)
    assert E.info["stream_bytes"] >= 32 << 20
    cols = [*range(small), small, small + 31, small + 32, nd - 1]
    assert np.array_equal(_columns(E, cols), want[:, cols])
    E.close()


def test_leaves_past_the_staging_buffers(gpu, build_libs):
    """More words than the plain copy takes: several buffers, pieces across their ends."""
    import test_plan as tp
    from hacapk_b200.engine import Engine
    rng = np.random.default_rng(12)
    nd, cut = 2100, 1999
    leaves, want = [], np.zeros((nd, nd))
    for r0, r1 in ((0, cut), (cut, nd)):
        for c0, c1 in ((0, cut), (cut, nd)):
            A = rng.standard_normal((r1 - r0, c1 - c0))
            leaves.append((2, 0, r0 + 1, r1 - r0, c0 + 1, c1 - c0, A.ravel()))
            want[r0:r1, c0:c1] = A
    P, keep = tp._custom(leaves, nd)
    E = Engine(C.pointer(P), nd)
    cols = [0, 1, 31, 32, cut - 1, cut, nd - 1]
    assert np.array_equal(_columns(E, cols), want[:, cols])
    E.close()

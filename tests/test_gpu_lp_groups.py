"""FP32 and BF16 products whose blocks alternate between consumer groups: blocks
of one and of several runs, an odd number of blocks, CTAs with no block for one
of the groups, P slabs on both sides of 32 rows."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("num_ctas", [0, 1, 2, 3])
@pytest.mark.parametrize("nd", [1, 33, 95, 2049, 4500])
def test_blocks_alternate(gpu, build_libs, nd, num_ctas, precision):
    import test_plan as tp
    from hacapk_b200.engine import Engine
    rng = np.random.default_rng(nd + num_ctas)
    A = np.zeros((nd, nd))
    leaves = []
    rows = sorted({0, min(nd, 7), min(nd, 40), min(nd, 73), nd})
    cuts = sorted({0, min(nd, 33), min(nd, 96), min(nd, 2100), nd})
    for a, (r0, r1) in enumerate(zip(rows, rows[1:])):
        for b, (c0, c1) in enumerate(zip(cuts, cuts[1:])):
            # powers of two: exact in every storage, products exact; the sums of
            # up to 4500 of them in floats and doubles are whole numbers below 2^24
            if (a + b) % 2 and r1 - r0 > 1 and c1 - c0 > 1:
                kt = min(r1 - r0, c1 - c0, 1 + 31 * a)
                U = np.zeros((r1 - r0, kt))
                U[np.arange(r1 - r0), np.arange(r1 - r0) % kt] = rng.choice([1.0, -2.0], r1 - r0)
                V = np.zeros((c1 - c0, kt))
                V[np.arange(c1 - c0), np.arange(c1 - c0) % kt] = rng.choice([1.0, -1.0], c1 - c0)
                leaves.append((1, kt, r0 + 1, r1 - r0, c0 + 1, c1 - c0, np.concatenate([V.T.ravel(), U.T.ravel()])))
                A[r0:r1, c0:c1] = U @ V.T
            else:
                D = rng.choice([1.0, -1.0, 2.0], (r1 - r0, c1 - c0))
                leaves.append((2, 0, r0 + 1, r1 - r0, c0 + 1, c1 - c0, D.ravel()))
                A[r0:r1, c0:c1] = D
    P, keep = tp._custom(leaves, nd)
    E = Engine(C.pointer(P), nd, precision=precision, num_ctas=num_ctas)
    x = rng.integers(-8, 9, nd).astype(np.float64)
    yin = rng.integers(-8, 9, nd).astype(np.float64)
    assert np.array_equal(E.matvec_host(x)[0], A @ x)
    assert np.array_equal(E.matvec_host(x, yin)[0], A @ x + yin)
    E.close()

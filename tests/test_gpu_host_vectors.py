"""Products with host vectors on both sides of the size up to which they go
through page-locked memory (524,288 rows), and of the copy kernel's blocks."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nd", [1, 2, 255, 257, 37889, 524288, 524289])
def test_host_product(gpu, build_libs, nd):
    import test_plan as tp
    from hacapk_b200.engine import Engine
    # block diagonal: u v^T of ones
    leaves, step = [], 1024
    for r in range(0, nd, step):
        m = min(step, nd - r)
        leaves.append((1, 1, r + 1, m, r + 1, m, np.ones(2 * m)) if m > 1 else (2, 0, r + 1, 1, r + 1, 1, np.ones(1)))
    P, keep = tp._custom(leaves, nd)
    E = Engine(C.pointer(P), nd)
    rng = np.random.default_rng(nd)
    for _ in range(2):  # whole numbers: every sum exact
        x, y0 = rng.integers(-9, 10, (2, nd)).astype(np.float64)
        ref = np.repeat([x[r:r + step].sum() for r in range(0, nd, step)], step)[:nd]
        assert np.array_equal(E.matvec_host(x)[0], ref)
        assert np.array_equal(E.matvec_host(x, y0)[0], ref + y0)
    E.close()

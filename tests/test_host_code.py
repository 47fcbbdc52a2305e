"""The engine's host code on the CPU, its object files linked with a stand-in
for the CUDA runtime (tests/emu/fake_cuda.cpp: launches do nothing, every call
is logged with its stream, any call can be made to fail)."""
import ctypes as C
import glob
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, sphere

PKG = os.path.join(ROOT, "hacapk-magma_b200")


EMU = os.path.join(ROOT, "tests", "emu")
LIB = os.path.join(EMU, "_build", "libfakecuda.so")


def _load():
    from hacapk_b200 import abi
    L = abi._load(LIB, abi.ENGINE_SYMBOLS)
    L.fake_fail.argtypes = [C.c_char_p, C.c_int, C.c_int]
    L.fake_op.argtypes = [C.c_int, C.POINTER(C.c_ulonglong), C.POINTER(C.c_int)]
    L.fake_op.restype = C.c_char_p
    L.fake_device_bytes.restype = C.c_longlong
    L.fake_device_blocks.argtypes = [C.c_longlong]
    L.fake_op_memory.argtypes = [C.c_int, C.POINTER(C.c_ulonglong)]
    L.fake_op_memory.restype = C.c_void_p
    return L


@pytest.fixture(scope="module")
def fake(build_libs):
    os.makedirs(os.path.dirname(LIB), exist_ok=True)
    objs = sorted(glob.glob(os.path.join(PKG, "_build", "hbx_*.o")))
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I/usr/local/cuda/include", "-o", LIB,
                    os.path.join(EMU, "fake_cuda.cpp"), *objs, "-fopenmp",
                    f"-Wl,--version-script={os.path.join(EMU, 'fake_cuda.map')}"], check=True)
    return _load()


@pytest.fixture
def engine(fake, monkeypatch):
    """The Engine class on the stand-in library."""
    from hacapk_b200 import abi
    from hacapk_b200.engine import Engine
    monkeypatch.setattr(abi, "engine_lib", lambda: fake)
    fake.fake_clear()
    return Engine


def _ops(L):
    """(call, stream, complete on return) of every logged operation."""
    out = []
    for i in range(L.fake_ops()):
        s, w = C.c_ulonglong(), C.c_int()
        out.append((L.fake_op(i, C.byref(s), C.byref(w)).decode(), s.value, w.value))
    return out


DEVICE_WORK = ("launch", "cudaMemcpy", "cudaMemcpyAsync", "cudaMemset", "cudaMemsetAsync")


def _unordered(ops, streams):
    """Operations that a launch on one of `streams` (none of them ordered after
    the default stream) may overtake: queued elsewhere, and neither complete on
    return nor waited for by the host before the call's end."""
    bad, waiting = [], {}
    for what, s, done in ops:
        if what in ("cudaStreamSynchronize", "cudaDeviceSynchronize"):
            for k in [s] if what == "cudaStreamSynchronize" else list(waiting):
                waiting.pop(k, None)
        elif what == "launch" and s in streams:
            bad += [x for k, v in waiting.items() if k != s for x in v]
        elif what in DEVICE_WORK:
            if done:  # and with it all that its stream held
                waiting.pop(s, None)
            else:
                waiting.setdefault(s, []).append((what, s))
    return bad


USER = 0xbeef0  # a stream of the caller's


@pytest.mark.parametrize("call", ["batch", "batch_host", "plain_batch", "batch_refined", "multi", "multi_host",
                                  "multi_unaligned", "pipe", "gcr", "bicgstab"])
def test_first_solves_queue_nothing_on_another_stream(engine, fake, call):
    """A solver's first call on a new engine prepares its workspace.  All of it
    is queued on the solve's own stream, or complete before the solve's first
    launch: a non-blocking stream does not wait for the default one, where a
    clear queued behind the caller's own work would land in the middle of the
    solve."""
    H = sphere(2)
    n = H.nd
    b = np.ones(n)
    if "batch" in call and call != "plain_batch":
        E, low = engine.batch([H, H]), engine.batch([H, H], precision=1)
    else:
        E, low = engine(H.st, n), engine(H.st, n, precision=1)
    n = E.nd
    M = engine(H.st, H.nd, precision=1, nrhs=64) if call.startswith("multi") else None
    buf = np.zeros((2 * n + 1) * 64)
    p = buf.ctypes.data + (-buf.ctypes.data) % 16
    create = _ops(fake)
    fake.fake_clear()
    if call in ("batch", "plain_batch"):
        E.bicgstab_batch_dev(p, p + 8 * n, stream=USER, check=False)
    elif call == "batch_host":
        E.bicgstab_batch_host(np.ones(n))
    elif call == "batch_refined":
        E.bicgstab_batch_refined_host(low, np.ones(n))
    elif call == "multi":
        E.bicgstab_multi_dev(M, p, p + 8 * 64 * n, stream=USER, check=False)
    elif call == "multi_unaligned":
        E.bicgstab_multi_dev(M, p, p + 8 * 64 * n + 8, stream=USER, check=False)
    elif call == "multi_host":
        E.bicgstab_multi_host(M, np.ones((n, 64)))
    elif call == "pipe":
        E.bicgstab_pipe_host(b, check=False, max_iter=8)
    elif call == "gcr":
        E.gcr_host(b, check=False, max_iter=8)
    else:
        E.bicgstab_host(b, check=False, max_iter=8)
    ops = _ops(fake)
    streams = {s for what, s, _ in ops if what == "launch"}
    assert streams and 0 not in streams
    assert _unordered(create + ops, streams) == []
    for X in (E, low, M):
        if X is not None:
            X.close()


def _big_dense(n=2100):
    """One dense leaf of 35 MB: packed on the device, through the page-locked buffers."""
    import test_plan as tp
    P, keep = tp._custom([(2, 0, 1, n, 1, n, np.ones(n * n))], n)
    return P, keep, n


NO_MEMORY = 2  # cudaErrorMemoryAllocation
REFUSALS = [("cudaHostAlloc", 0), ("cudaHostAlloc", 1), ("cudaEventCreate", 0), ("cudaStreamCreate", 0)]


@pytest.mark.parametrize("what,nth", REFUSALS)
def test_create_without_page_locked_memory(engine, fake, what, nth):
    """The device packing goes on with plain copies where page-locked memory (or
    a stream or event) is refused, and leaves no error behind for the next
    launch to report."""
    P, keep, n = _big_dense()
    # the engine's own stream and events come before the packing's
    first = {"cudaHostAlloc": 0, "cudaEventCreate": 6, "cudaStreamCreate": 1}[what]
    fake.fake_fail(what.encode(), first + nth, NO_MEMORY)
    E = engine(C.pointer(P), n)
    assert fake.fake_last_error() == 0
    E.close()


@pytest.mark.parametrize("what,nth", REFUSALS)
def test_fill_without_page_locked_memory(fake, engine, what, nth):
    """The same for the leaves' copy from the device."""
    from hacapk_b200 import hmatrix
    first = {"cudaHostAlloc": 0, "cudaEventCreate": 0, "cudaStreamCreate": 6}[what]  # after the fill's own streams
    fake.fake_fail(what.encode(), first + nth, NO_MEMORY)
    H = hmatrix.HostHMatrix(hmatrix.icosphere(4), leaf_size=3000, eta=2.0, aca_eps=1e-5, fill="gpu")
    assert fake.fake_last_error() == 0
    H.close()


def test_a_reported_error_is_reported_once(engine, fake):
    """The runtime keeps a failed call's error until it is asked for: the next
    call's first launch must not report it again."""
    from hacapk_b200.engine import HbxError
    H = sphere(2)
    E = engine(H.st, H.nd)
    fake.fake_fail(b"cudaMalloc", 0, NO_MEMORY)
    with pytest.raises(HbxError) as ei:
        E.matvec_host(np.ones(H.nd))
    assert ei.value.status == 2
    E.matvec_host(np.ones(H.nd))
    E.close()


def _multi(engine):
    H = sphere(2)
    E, M = engine(H.st, H.nd), engine(H.st, H.nd, precision=1, nrhs=64)
    buf = np.zeros((2 * H.nd + 1) * 64)
    p = buf.ctypes.data + (-buf.ctypes.data) % 16
    return E, M, buf, lambda: E.bicgstab_multi_dev(M, p, p + 8 * 64 * H.nd, stream=USER)


def test_unit_table_is_published_once_it_is_on_the_device(engine, fake):
    """A failed upload of the multi-RHS product's units leaves no table behind:
    the next solve uploads it."""
    from hacapk_b200.engine import HbxError

    def uploads():
        return sum(what == "cudaMemcpyAsync" and s != USER for what, s, _ in _ops(fake))
    E, M, buf, solve = _multi(engine)
    fake.fake_clear()
    fake.fake_fail(b"cudaMemcpyAsync", 0, 1)  # the first of the call
    with pytest.raises(HbxError):
        solve()
    assert uploads() == 0
    solve()
    assert uploads() == 1
    solve()  # kept
    assert uploads() == 1
    for X in (E, M):
        X.close()


def _fail_allocations():
    """In a child: every host allocation of a first multi-RHS solve fails once."""
    import test_host_code as t
    from hacapk_b200 import abi
    from hacapk_b200.engine import Engine
    L = t._load()
    abi.engine_lib = lambda: L
    for n in range(100000):
        E, M, buf, solve = t._multi(Engine)
        L.fake_fail_new(n)
        solve()  # an exception that leaves the C entry ends this process
        left = L.fake_fail_new(-1)
        E.close()
        M.close()
        if left >= 0:
            print(f"{n} allocations")
            return


def test_no_exception_leaves_the_multi_rhs_solve(fake):
    code = "import conftest, test_host_code as t; t._fail_allocations()"
    r = subprocess.run([sys.executable, "-c", code], cwd=os.path.dirname(os.path.abspath(__file__)),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, (r.returncode, r.stderr[-500:])
    assert int(r.stdout.split()[0]) > 5


@pytest.mark.parametrize("refined", [False, True])
def test_batch_host_solve_holds_two_vectors_of_its_own(engine, fake, refined):
    """The host-vector form of a batch solve holds b and u on the device beside
    what the device-vector form holds, and no other solver's workspace."""
    H = sphere(2)
    held = []
    for host in (False, True):
        E, low = engine.batch([H, H]), engine.batch([H, H], precision=1)
        before = fake.fake_device_bytes()
        b = np.ones(2 * E.nd)
        if host:
            E.bicgstab_batch_refined_host(low, b[:E.nd]) if refined else E.bicgstab_batch_host(b[:E.nd])
        elif refined:
            E.bicgstab_batch_refined_dev(low, b.ctypes.data, b.ctypes.data + 8 * E.nd)
        else:
            E.bicgstab_batch_dev(b.ctypes.data, b.ctypes.data + 8 * E.nd)
        held.append(fake.fake_device_bytes() - before)
        nd = E.nd
        E.close()
        low.close()
    assert held[1] - held[0] == 2 * 8 * nd


@pytest.mark.parametrize("precision,nrhs", [(0, 0), (1, 0), (2, 0), (1, 64)])
def test_only_fp64_engines_hold_zbu_in_doubles(engine, fake, precision, nrhs):
    """The other engines' V^T x segments are floats, in a buffer of their own."""
    H = sphere(3)
    E = engine(H.st, H.nd, precision=precision, nrhs=nrhs)
    assert E.info["zbu_len"] > 0
    assert fake.fake_device_blocks(2 * 8 * E.info["zbu_len"]) == (1 if precision == 0 else 0)
    E.close()


def test_fill_workspace_is_cleared_before_the_kernels(fake, engine):
    """ACA+ reads a column of its workspace that it never set when it stops in
    one, so the workspace must not hold what another allocation left there."""
    from hacapk_b200 import hmatrix
    H = hmatrix.HostHMatrix(hmatrix.icosphere(3), leaf_size=32, eta=2.0, aca_eps=1e-5, fill="gpu")
    mem = []
    for i in range(fake.fake_ops()):
        n = C.c_ulonglong()
        mem.append((fake.fake_op_memory(i, C.byref(n)), n.value))
    names = [what for what, _, _ in _ops(fake)]
    mallocs = [i for i, w in enumerate(names) if w == "cudaMalloc"]
    work = max(mallocs, key=lambda i: mem[i][1])  # the largest by far: U and V of every leaf at 64 columns
    launch = next(i for i in range(work, len(names)) if names[i] == "launch")
    assert [i for i in range(work, launch) if names[i] == "cudaMemset" and mem[i] == mem[work]]
    H.close()

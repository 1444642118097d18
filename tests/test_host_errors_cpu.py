"""Error paths of the host runtime, on the CPU: the library's own objects linked
against a CUDA runtime without a GPU (fake_cudart.cpp) whose calls can be made
to fail and which checks what the launches name."""
import ctypes
import glob
import os
import subprocess

import numpy as np
import pytest

from sonicsolver_b200 import build, capi, cases

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    build.build()
    out = str(tmp_path_factory.mktemp("fake") / "libsfg_fake.so")
    cuda = os.path.dirname(os.path.dirname(build._nvcc()))
    objs = sorted(glob.glob(os.path.join(build.OBJ, "*.o")))
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-fvisibility=hidden", "-I", os.path.join(cuda, "include"),
                    "-I", build.CSRC, "-I", os.path.join(build.ROOT, "include"), os.path.join(HERE, "fake_cudart.cpp"),
                    *objs, "-o", out, "-Wl,-Bsymbolic"], check=True)
    return out


@pytest.fixture
def fake(fake_lib, monkeypatch):
    """capi on the fake library."""
    monkeypatch.setattr(capi, "LIB_PATH", fake_lib)
    monkeypatch.setattr(capi, "_lib", None)
    lib = capi.lib()
    lib.fake_violation.restype = ctypes.c_char_p
    lib.fake_alloc.restype = lib.fake_residual.restype = ctypes.c_void_p
    lib.fake_alloc.argtypes = [ctypes.c_size_t, ctypes.c_int]
    lib.fake_reset()
    yield lib
    assert lib.fake_violations() == 0, lib.fake_violation().decode()


def _grid(side, laws=False):
    b = capi.BC_LAW if laws else capi.BC_PERIODIC
    n = (side, side, 1)
    return cases.Case("g", 2, n, (0.01, 0.01, 1.0), (b, b, 0), (b, b, 0), np.ones((1, side, side, 5)), 1.4, 1.0, 0.4,
                      "weno5Rusanov", "SSPRK3")


WALLS = {(a, e): dict(velocity=capi.LAW_SYMMETRY) for a in range(2) for e in range(2)}


@pytest.mark.parametrize("laws,skip", [(False, 0), (False, 1), (True, 0), (True, 1), (True, 2)])
def test_batch_list_that_cannot_grow(fake, laws, skip):
    """A grid whose tiles (or law points) need a longer device list than can be
    allocated is refused by the add, as one beyond the budget is; the grids
    already there step on from a list that is theirs, and the same grid is
    taken once there is memory.  First list: 1024 tiles or 256 law runs; `skip`:
    allocations that still succeed (the staging array, one list of the two)."""
    b = capi.Batch(800 << 20, 4, recipe="weno5Rusanov")
    first = b.add(_grid(40, laws), laws=WALLS if laws else None)
    b.step(3, graph_steps=2)
    side = 20000 if laws else 750
    big = _grid(60, laws)
    big.n = (side, 40, 1) if laws else (side, side, 1)
    big.q = np.ones((1, big.n[1], side, 5))
    b.add(_grid(30, laws), laws=WALLS if laws else None)
    fake.fake_fail(b"cudaMalloc", skip, 1000)
    with pytest.raises(capi.SolverError):
        b.add(big, laws=WALLS if laws else None)
    for _ in range(2):
        b.step(3, graph_steps=2)
    fake.fake_fail(b"cudaMalloc", 0, 0)
    before = b.info()["items"]
    slot = b.add(big, laws=WALLS if laws else None)
    b.step(3, graph_steps=2)
    assert b.info()["items"] > before
    b.remove(slot)
    b.remove(first)
    b.step(3, graph_steps=2)
    assert b.info()["items"] == fake.fake_tiles() == 2


def test_batch_list_that_cannot_be_published(fake):
    """A step whose list does not reach the device fails, and so does every
    step after it until the list has."""
    b = capi.Batch(16 << 20, 4, recipe="weno5Rusanov")
    b.add(_grid(40))
    b.step(3, graph_steps=2)
    b.add(_grid(60))
    tiles = [6, 14]
    for k in range(2):
        assert fake.fake_tiles() == tiles[0]
        fake.fake_fail(b"cudaMemcpy", k, 1)
        with pytest.raises(capi.SolverError):
            b.step(3, graph_steps=2)
    b.step(3, graph_steps=2)
    assert fake.fake_tiles() == tiles[1]


@pytest.mark.parametrize("dim,precision", [(1, capi.PREC_FP64), (2, capi.PREC_FP64), (2, capi.PREC_FP32_FLUX),
                                           (3, capi.PREC_FP64)])
def test_noalloc_residual_goes_only_where_kernels_can_write(fake, dim, precision):
    """The kernels get the caller's result array when it is this device's memory
    on an 8-byte boundary, all of it; any other gets a copy, which refuses what
    is not there."""
    n = (20, 20 if dim > 1 else 1, 20 if dim > 2 else 1)
    nodes = n[0] * n[1] * n[2]
    bc = tuple(1 if d < dim else 0 for d in range(3))

    def call(q, r):
        capi.residual_noalloc(dim, n, (0.1, 0.1, 0.1), bc, bc, q, r, recipe="weno5Rusanov", precision=precision)
        return fake.fake_residual()

    q = fake.fake_alloc(40 * nodes, 0)
    r, wide = fake.fake_alloc(40 * nodes, 0), fake.fake_alloc(40 * nodes + 8, 0)
    assert call(q, r) == r and call(q, wide + 8) == wide + 8
    for other in (fake.fake_alloc(40 * nodes, 1), wide + 4, q):
        assert call(q, other) not in (other, r, q)
        assert not any(ctypes.string_at(other, 40 * nodes))  # the fixed array's zeros, copied
    host = np.ones(5 * nodes)
    for missing in (fake.fake_alloc(40 * nodes - 8, 0), host.ctypes.data):
        with pytest.raises(capi.SolverError) as e:
            call(q, missing)
        assert e.value.code == capi.ERR_CUDA and fake.fake_residual() != missing
    assert host.all()


@pytest.mark.parametrize("call", [b"cudaStreamBeginCapture", b"cudaStreamEndCapture", b"cudaGraphInstantiate"])
def test_run_without_a_graph(fake, call):
    """A run whose graph cannot be had is a run all the same, and its failed
    capture is not the next call's error."""
    s = _grid(40).solver()
    fake.fake_fail(call, 0, 1000)
    for _ in range(2):
        s.advance(1e30, max_steps=9, graph_steps=4)
    assert fake.cudaGetLastError() == 0

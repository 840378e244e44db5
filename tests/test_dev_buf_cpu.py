"""The context's device buffers near the end of the memory (csrc/dev_buf.h, the
functions capi.cu uses), over an allocator with a fixed amount of it: optional
buffers leave room, give way to required ones, and do not come and go from call
to call."""
import ctypes as C
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "dm-annihilation-cxx_gb300", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("buf") / "libdevbuf.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC,
                    os.path.join(REPO, "tests", "cpp", "dev_buf_shim.cpp"), "-o", so], check=True)
    d = C.CDLL(so)
    L = C.c_longlong
    d.reset.argtypes, d.reset.restype = [L, C.c_int], None
    for f in (d.grow_opt, d.grow_req):
        f.argtypes = [C.c_int, L]
    d.share.argtypes, d.share.restype = [C.c_int, L, L, L], L
    d.held.argtypes, d.held.restype = [C.c_int], L
    for f in (d.used, d.changes, d.calls):
        f.restype = L
    return d


def test_a_required_buffer_takes_the_optional_ones_place(lib):
    lib.reset(1000, 3)
    assert lib.grow_opt(1, 400) and lib.grow_opt(2, 400)
    assert lib.grow_req(0, 900)                      # fits alone
    assert lib.held(0) >= 900 and lib.held(1) == lib.held(2) == 0
    assert not lib.grow_req(0, 1001) and lib.used() == 0


def test_a_failed_optional_buffer_changes_nothing(lib):
    lib.reset(1000, 2)
    assert lib.grow_opt(0, 600)
    n = lib.changes()
    for _ in range(3):
        assert not lib.grow_opt(1, 500)              # kept graphs stay valid
    assert lib.changes() == n


@pytest.mark.parametrize("size,least,most", [(10000, 100, 1000), (10000, 100, 100000), (1000, 300, 100000)])
def test_a_share_leaves_three_quarters(lib, size, least, most):
    lib.reset(size, 2)
    got = lib.share(0, least, most, 0)
    assert got == lib.held(0) and got <= size // 4 and got <= most + most // 8
    assert got >= least or got == 0
    assert (got == 0) == (size // 4 < least)


def test_a_share_is_kept_while_the_free_memory_moves(lib):
    lib.reset(10000, 2)
    first = lib.share(0, 100, 100000, 0)
    n = lib.changes()
    for taken in (500, 0, 900, 100):
        lib.free_buf(1)
        assert taken == 0 or lib.grow_opt(1, taken)
        m = lib.changes()
        assert lib.share(0, 100, 100000, 0) == first and lib.changes() == m
    assert lib.share(0, first + 1, 100000, 0) == 0   # fewer than it takes now
    assert lib.changes() >= n


def test_azimuth_tables_are_bounded(lib):
    """A context that renders the plain form at every Nside."""
    lib.trig_cap.argtypes, lib.trig_cap.restype = [C.c_int, C.c_longlong], C.c_longlong
    assert all(lib.trig_cap(n, 0) == 32 * n * (n - 1) for n in (1, 64, 512, 1024, 1448))
    held = 0
    for nside in range(1, 8193):
        held += lib.trig_cap(nside, held)
    assert held <= 256 << 20

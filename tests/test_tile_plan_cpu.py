"""The choice between the renders of a large chunk (csrc/tile_plan.h, the
functions capi.cu and k_seg_decide use), built for the host: a chunk is
rendered by tiles only when its (disc, tile) pairs are known to fit the pair
list, whatever other buffers there are.  And the order of a tile's discs: by
octaves of the deposit scale, such that no deposit is lost on the FP32 sum of the
ones before it."""
import ctypes as C
import itertools
import math
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "dm-annihilation-cxx_gb300", "csrc")
TILE, SEG, COUNT = 1, 2, 4


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("plan") / "libtileplan.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC,
                    os.path.join(REPO, "tests", "cpp", "tile_plan_shim.cpp"), "-o", so], check=True)
    d = C.CDLL(so)
    for f in (d.pairs_bound, d.capacity):
        f.restype, f.argtypes = C.c_longlong, [C.c_longlong, C.c_int]
    d.always_fits.argtypes = [C.c_longlong, C.c_int]
    d.mode.argtypes = [C.c_longlong] * 7
    return d


def chunk_mode(lib, n, nside, have_tile, have_seg, pairs, items):
    """The mode that a chunk's launches and the device's decision come to."""
    p = lib.plan(have_tile, lib.always_fits(n, nside), have_seg)
    return lib.mode(1 << 40, 1 << 28, n, pairs if p & COUNT else 0, lib.capacity(n, nside) if p & TILE else 0,
                    items if p & SEG else 0, 4 * n + (1 << 20) if p & SEG else 0)


# a chunk whose pairs always fit, and two that can overflow
@pytest.mark.parametrize("n,nside", [(1000, 64), (10000, 1024), (1 << 20, 4096)])
def test_no_chunk_overflows_the_pair_list(lib, n, nside):
    bound, cap = lib.pairs_bound(n, nside), lib.capacity(n, nside)
    for tile, seg, pairs in itertools.product((0, 1), (0, 1), (1, cap, min(cap + 1, bound), bound)):
        mode = chunk_mode(lib, n, nside, tile, seg, pairs, n)
        if tile and pairs <= cap:
            assert mode == 2
        else:
            assert mode == (1 if seg else 0), (tile, seg, pairs, cap)


def test_no_deposit_is_lost_on_the_ones_before(lib):
    """For every range of octaves: classes ascend with the octaves and there are
    64 of them; with the discs of one class in any order, the smallest addend
    (the class's smallest scale, times a weight of exp(-6)) is above half an ulp
    of the largest total before it (a unit's discs at the class's largest scale)."""
    for omax in range(256):
        for omin in range(omax + 1):
            c = [lib.cls(o, omax, omin) for o in range(omin, omax + 1)]
            assert c[0] >= 0 and c[-1] == 63 and all(a <= b for a, b in zip(c, c[1:]))
            width = max(c.count(k) for k in set(c))
            least, total = math.exp(-6.0), lib.unit_max() * 2.0 ** width   # in the class's smallest scale
            assert least > 2.0 ** -24 * total


def test_the_units_of_all_lists_fit(lib):
    """The lists' units, one behind the other, however the pairs are dealt to the
    four lists and to the tiles (one pair in every tile but one makes the most)."""
    L = C.c_longlong
    lib.units_of.argtypes, lib.units_of.restype = [L, L], L
    lib.unit_capacity.argtypes, lib.unit_capacity.restype = [L, C.c_int], L
    lib.unit_len.argtypes = [L]
    for nside in (64, 1024, 4096):
        nt = ((4 * nside + 30) // 32) * ((4 * nside + 63) // 64)
        for slots in (1, 1000, 1 << 19, 3 << 20, 1 << 24, 1 << 31):
            for split in ((1, 0, 0, 0), (0.25, 0.25, 0.25, 0.25), (0.7, 0.1, 0.1, 0.1), (0.97, 0.01, 0.01, 0.01)):
                pairs = [int(slots * f) for f in split]
                room = [lib.units_of(p, nt) for p in pairs]
                assert sum(room) <= lib.unit_capacity(slots, nside)
                for p, have in zip(pairs, room):
                    n = lib.unit_len(p)
                    assert 32 <= n <= lib.unit_max()
                    spread = min(p, nt)               # tiles with a pair
                    most = (spread - 1 + (p - spread + 1 + n - 1) // n) if p else 0
                    assert most <= have

"""The staging rule of phase A (mpart_gb300/csrc/mpgb_stage.h), built for the
host: whole components or nothing in FP64, chunks with limbs, and no lower
occupancy for FP64."""
import ctypes
import math
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "mpart_gb300", "csrc")


@pytest.fixture(scope="module")
def room(tmp_path_factory):
    d = tmp_path_factory.mktemp("st")
    (d / "s.cpp").write_text('#include "mpgb_stage.h"\nextern "C" int room(const int* s, const int* n, int k, int limbs, '
                             'long base, long sm, long blocks) { mpgb::StageNeed q; for (int i = 0; i < k; ++i) '
                             'q.add(s[i], n[i]); return mpgb::stageRoom(q, limbs != 0, base, sm, blocks); }\n')
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "s.so"), str(d / "s.cpp")],
                   check=True)
    lib = ctypes.CDLL(str(d / "s.so"))

    def f(dim, order, limbs, blocks=4):
        # every component of a triangular total-order map; 128-point tiles
        nodes = [math.comb(d - 1 + order, order) for d in range(1, dim + 1)]
        slots = [math.comb(d + order, order) for d in range(1, dim + 1)]
        arr = lambda v: (ctypes.c_int * len(v))(*v)  # noqa: E731
        n_basis = (dim - 1) * order
        base = 8 * (dim * 128 + ((n_basis * 129 + 1) & ~1) + (min(order, dim - 1) + 1 if order < dim else order + 1) * 128)
        base += 2048 if limbs else 1024
        return lib.room(arr(slots), arr(nodes), dim, int(limbs), ctypes.c_long(base), ctypes.c_long(228 * 1024),
                        ctypes.c_long(blocks)), base
    return f


@pytest.mark.parametrize("dim,order,want", [(8, 4, 825), (6, 5, 714), (4, 3, 55), (11, 3, 650), (2, 2, 9)])
def test_fp64_stages_whole_components(room, dim, order, want):
    got, base = room(dim, order, False)
    assert got == want == math.comb(dim + order, order) + math.comb(dim - 1 + order, order)


@pytest.mark.parametrize("dim,order", [(12, 3), (16, 3), (20, 3), (12, 5)])
def test_fp64_keeps_its_blocks(room, dim, order):
    got, base = room(dim, order, False)
    blocks = lambda b: min(4, 228 * 1024 // b)  # noqa: E731
    assert got == 0 or blocks(base + 8 * got) == blocks(base)
    # (of the components the cap of 2,048 lets in, the largest)
    need = [math.comb(d + order, order) + math.comb(d - 1 + order, order) for d in range(1, dim + 1)]
    assert got in (0, max(n for n in need if n <= 2048))


@pytest.mark.parametrize("dim,order", [(2, 1), (8, 4), (12, 3), (20, 3), (30, 3)])
def test_limbs_have_their_smallest(room, dim, order):
    got, base = room(dim, order, True)
    assert 256 <= got <= 2048 or base + 256 * 8 > 227 * 1024

"""The rules that decide how a host buffer travels (gpumhd_hostmem.cuh),
compiled for the host."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "gpumhd_hostmem.cuh"
extern "C" int covers(uint64_t s, uint64_t n, uint64_t p, uint64_t b) { return hostmem::covers(s, n, p, b); }
extern "C" int moves_directly(int nf, int s, uint64_t a, int d) { return hostmem::moves_directly(nf, s, a, d != 0); }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("hostmem")
    (d / "r.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "muram_main_gb300", "csrc"), str(d / "r.cpp"), "-o", str(d / "r.so")], check=True)
    lib = C.CDLL(str(d / "r.so"))
    lib.covers.argtypes = [C.c_uint64] * 4
    lib.moves_directly.argtypes = [C.c_int, C.c_int, C.c_uint64, C.c_int]
    return lib


def test_range_within_one_pinned_piece(rules):
    base, size = 0x7f0000000000, 1 << 20
    inside = [(base, size), (base, 1), (base + 64, size - 64), (base + size - 8, 8)]
    outside = [(base - 8, 16), (base - 8, size), (base, size + 1), (base + 64, size), (base + size, 8),
               (base + size - 8, 16), (0, base + size), (base, (1 << 64) - 1), (base + 64, (1 << 64) - 64)]
    assert all(rules.covers(base, size, p, n) for p, n in inside)
    assert not any(rules.covers(base, size, p, n) for p, n in outside)


def test_two_pieces_with_a_gap(rules):
    """Both ends pinned and as far apart as the host addresses are, but pageable
    memory between them: neither piece covers the range."""
    lo, hi, piece = 0x7f0000000000, 0x7f0000400000, 0x100000
    p, n = lo + 4096, hi + 4096 - (lo + 4096)
    assert rules.covers(lo, piece, p, 1) and rules.covers(hi, piece, p + n - 1, 1)
    assert not rules.covers(lo, piece, p, n) and not rules.covers(hi, piece, p, n)


def test_nothing_is_covered_by_an_unknown_piece(rules):
    assert not rules.covers(0, 0, 0x7f0000000000, 8)


@pytest.mark.parametrize("size", [4, 8])
@pytest.mark.parametrize("download", [0, 1])
def test_records_move_directly_only_in_whole_pieces(rules, size, download):
    """Unaligned records go through the staging buffer, but for float uploads."""
    at = 0x7f0000000000
    assert all(rules.moves_directly(8, size, at + 16 * k, download) for k in range(4))
    assert all(rules.moves_directly(8, size, at + k, download) == (size == 4 and not download)
               for k in (4, 8, 12, 20, 24))
    assert all(rules.moves_directly(1, size, at + k, download) for k in (0, 4, 8, 16))
    assert not rules.moves_directly(3, size, at, download)

"""The pieces that a stream is cut into for the latest positions (rosa_heads.cuh), compiled for the host."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def pieces(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("rosa_pieces") / "librosa_host.so")
    src = os.path.join(ROOT, "tests", "host_harness", "rosa_host.cpp")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", src, "-o", out], check=True)
    lib = C.CDLL(out)

    def of(T, wanted):
        row0, row1 = (np.full(wanted, 0xFFFF, np.uint32) for _ in range(2))
        n = lib.rosa_host_pieces(C.c_uint32(T), C.c_uint32(wanted), C.c_void_p(row0.ctypes.data), C.c_void_p(row1.ctypes.data))
        return n, row0[:n], row1[:n]

    return of


@pytest.mark.parametrize("wanted", [1, 2, 4])
def test_every_piece_has_rows(pieces, wanted):
    """All rows, once each, in at most as many pieces as are wanted, none of which is there for nothing."""
    for T in range(1, 2049):
        n, row0, row1 = pieces(T, wanted)
        assert 1 <= n <= wanted and row0[0] == 0 and row1[-1] == (T + 31) // 32, T
        assert np.array_equal(row0[1:], row1[:-1]) and (row0 < row1).all(), T

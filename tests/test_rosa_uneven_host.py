"""Which streams the latest positions give up by their runs alone (rosa_heads.cuh), compiled for the host: those whose walks along the runs of
11 equal bits, counted here one by one, are too long, and no even ones."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, pack_streams

DEPTH = 11


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("rosa_uneven") / "librosa_host.so")
    src = os.path.join(ROOT, "tests", "host_harness", "rosa_host.cpp")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", src, "-o", out], check=True)
    return C.CDLL(out)


def too_long(host, q, k, most):
    """Per stream; q and k [n, words]."""
    n, words = q.shape
    return np.array([host.rosa_host_runs_too_long(C.c_void_p(q[i].ctypes.data), C.c_void_p(k[i].ctypes.data), C.c_uint32(words), C.c_uint32(most))
                     for i in range(n)], bool)


def walk_along_runs(q, k):
    """Over the rows of 32 steps the longest walk of each: the positions before its queries that end a run of DEPTH bits which theirs ends."""
    T, total = len(q), 0
    ends = []
    for x in (k, q):
        run = np.ones(T, int)
        for t in range(1, T):
            run[t] = run[t - 1] + 1 if x[t] == x[t - 1] else 1
        ends.append([(run >= DEPTH) & (x == z) for z in (0, 1)])
    before = [np.concatenate([[0], np.cumsum(e)]) for e in ends[0]]
    for row in range(0, T, 32):
        total += max([int(before[z][t]) for t in range(row, min(row + 32, T)) for z in (0, 1) if ends[1][z][t]], default=0)
    return total


@pytest.mark.parametrize("T", [320, 704, 2048])
def test_streams_with_long_runs_are_told_from_even_ones(host, T):
    rng = np.random.default_rng(T)
    n, words = 24, T // 32
    most = 128 + 16 * words
    flagged = 0
    for kind in ("even", 0.65, 0.75, 0.85, 0.9, 0.97, "slow"):
        if kind == "slow":
            q, k = ((np.cumsum(rng.random((n, T)) < 0.05, axis=1) & 1).astype(np.uint8) for _ in range(2))
        else:
            p = 0.5 if kind == "even" else kind
            q, k = ((rng.random((n, T)) < p).astype(np.uint8) for _ in range(2))
        got = too_long(host, *(pack_streams(x) for x in (q, k)), most)
        walks = np.array([walk_along_runs(a, b) for a, b in zip(q, k)])
        # Only positions that end a run inside a word are counted, half of the keys are taken to lie before a row.
        assert not got[walks < most / 2].any() and got[walks > 4 * most].all(), (kind, walks, got)
        flagged += got.sum()
        if kind == "even":
            assert not got.any()
    assert flagged >= n * (1 if T == 320 else 3)


@pytest.mark.parametrize("run", [10, 11, 12, 31, 32])
def test_the_ends_of_a_run(host, run):
    """`run` equal bits and alternating ones behind them, as queries and as keys: their product is held against twice the limit."""
    bits = np.array([1 if i < run else (i - run) % 2 for i in range(32)], np.uint8)[None, :]
    ends = max(0, run - DEPTH + 1)
    for x in (pack_streams(bits), pack_streams(1 - bits)):
        for most in range(0, 14):
            assert too_long(host, x, x, most).all() == (ends > 2 * most), (run, most)
    assert not too_long(host, pack_streams(bits), pack_streams(1 - bits), 0).any()   # runs of ones against runs of zeros

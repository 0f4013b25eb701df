"""The automaton-free ROSA match (rosa_context.cuh, rosa_match.cuh), compiled for the host, against the oracle's pushes:
every input of a few steps, every key history of a few more under chosen queries, and long streams of the families that
each of its ways has to take."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, pack_streams
from test_sam_core_host import _streams

BY_BITS, BY_ALL_BITS, BY_RUNS = 0, 1, 2      # otherwise: sets of lags in pieces of so many steps
UNEVEN_BY_BITS, UNEVEN_BY_RUNS = 3, 4        # BY_ALL_BITS and BY_RUNS with the wider buckets of uneven streams


@pytest.fixture(scope="module")
def rosa_host(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("rosa_host") / "librosa_host.so")
    src = os.path.join(ROOT, "tests", "host_harness", "rosa_host.cpp")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fsanitize=undefined,bounds", "-fno-sanitize-recover=all",
                    "-static-libubsan", src, "-o", out], check=True)
    lib = C.CDLL(out)

    def run(way, q, k, v, n, T):
        q, k, v = (np.ascontiguousarray(a, np.uint32) for a in (q, k, v))
        res = np.full((n, (T + 31) // 32), 0xA5A5A5A5, np.uint32)
        rc = lib.rosa_host_batch(C.c_uint32(way), C.c_void_p(q.ctypes.data), C.c_void_p(k.ctypes.data), C.c_void_p(v.ctypes.data),
                                 C.c_size_t(n), C.c_uint32(T), C.c_void_p(res.ctypes.data))
        assert rc == 0, "wrote past its memory"
        if T % 32:
            res[:, -1] &= np.uint32((1 << T % 32) - 1)
        return res

    return run


@pytest.mark.parametrize("T", [1, 2, 3, 4, 5])
def test_every_input_of_a_few_steps(oracle, rosa_host, T):
    n = 1 << (3 * T)
    a = np.arange(n, dtype=np.uint32)
    m = (1 << T) - 1
    q, k, v = a & m, (a >> T) & m, (a >> (2 * T)) & m
    ref = oracle.rosa_qkv_streams(q, k, v, n, T)
    for way in (BY_BITS, 32):
        assert np.array_equal(rosa_host(way, q, k, v, n, T), ref), way


@pytest.mark.parametrize("tail", range(3))
def test_every_history_of_ten_steps_behind_a_prefix(oracle, rosa_host, tail):
    """Steps beyond the brute-force ones: a prefix of 64 steps (one key, two alternating, a rare one), then every pair of
    five query and five key bits, in buckets and in pieces that begin behind the prefix."""
    T, n = 69, 1 << 10
    a = np.arange(n)
    prefix = [np.zeros(64, np.uint8), np.arange(64, dtype=np.uint8) & 1, (np.arange(64) % 37 == 5).astype(np.uint8)][tail]
    q, k, v = (np.tile(np.concatenate([prefix, np.zeros(5, np.uint8)]), (n, 1)) for _ in range(3))
    for i in range(5):
        q[:, 64 + i], k[:, 64 + i] = a >> i & 1, a >> (5 + i) & 1
    v[:] = np.random.default_rng(tail).integers(0, 2, T)
    q, k, v = (pack_streams(x) for x in (q, k, v))
    ref = oracle.rosa_qkv_streams(q, k, v, n, T)
    for way in (BY_BITS, BY_ALL_BITS, BY_RUNS, UNEVEN_BY_BITS, UNEVEN_BY_RUNS, 32, 64):
        assert np.array_equal(rosa_host(way, q, k, v, n, T), ref), way


@pytest.mark.parametrize("kind,n", [("iid", 24), ("qk_same", 16), ("biased", 16), ("periodic", 16), ("periodic_clean", 8), ("q_const", 16),
                                    ("k_const", 8)])
@pytest.mark.parametrize("T", [65, 97, 777, 1024, 2048, 2081, 4097, 8192])
def test_long_streams(oracle, rosa_host, kind, T, n):
    if T > 2081:
        n //= 8
    rng = np.random.default_rng([T, n])
    q, k, v = (pack_streams(np.asarray(b, np.uint8)) for b in _streams(kind, n, T, rng))
    ref = oracle.rosa_qkv_streams(q, k, v, n, T)
    for way in (BY_BITS, BY_ALL_BITS, BY_RUNS, UNEVEN_BY_BITS, UNEVEN_BY_RUNS, 32, 256, 1024, 8192):
        if way == 32 and T > 2081:
            continue
        assert np.array_equal(rosa_host(way, q, k, v, n, T), ref), (kind, way)


@pytest.mark.parametrize("flips", [0, 1, 3])
@pytest.mark.parametrize("T", [97, 1000, 1024, 2047, 4100])
def test_streams_that_repeat_themselves_but_for_a_few_flips(oracle, rosa_host, T, flips):
    """Windows that reach back to the first key, and ones that stop doing so in the middle of a piece; the queries repeat
    the keys at once or a few steps later."""
    n = 24 if T <= 2047 else 6
    rng = np.random.default_rng([T, flips])
    base = rng.integers(0, 2, (n, 100), dtype=np.uint8)
    shift, period = rng.integers(0, 5, (n, 1)), rng.integers(2, 100, (n, 1))
    steps = np.arange(T)[None, :]
    q, k = (np.take_along_axis(base, (steps + s) % period, 1) for s in (shift, 0 * shift))
    for x in (q, k):
        for _ in range(flips):
            x[np.arange(n), rng.integers(0, T, n)] ^= 1
    v = rng.integers(0, 2, (n, T), dtype=np.uint8)
    q, k, v = (pack_streams(x) for x in (q, k, v))
    ref = oracle.rosa_qkv_streams(q, k, v, n, T)
    for way in (32, 64, 512, 8192):
        assert np.array_equal(rosa_host(way, q, k, v, n, T), ref), way

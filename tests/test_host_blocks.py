"""The register of page-locked blocks (host_blocks.hpp), compiled for the host: kernels write results only into memory that is there."""
import ctypes as C
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture
def blocks(tmp_path):
    out = str(tmp_path / "libblocks_host.so")
    src = os.path.join(ROOT, "tests", "host_harness", "blocks_host.cpp")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", src, "-o", out], check=True)
    lib = C.CDLL(out)
    for f in (lib.blocks_add, lib.blocks_hold):
        f.argtypes = [C.c_uint64, C.c_uint64]
    lib.blocks_remove.argtypes = [C.c_uint64]
    return lib


def test_only_whole_ranges_of_one_block_are_held(blocks):
    a, b, size = 0x7f0000010000, 0x7f0000020000, 0x10000      # b right behind a
    assert not blocks.blocks_hold(a, 1)
    assert blocks.blocks_add(a, size) and blocks.blocks_add(b, size)
    assert blocks.blocks_hold(a, size) and blocks.blocks_hold(a + 5, size - 5) and blocks.blocks_hold(b + size - 1, 1)
    assert not blocks.blocks_hold(a - 1, 1) and not blocks.blocks_hold(b + size, 1)
    assert not blocks.blocks_hold(a, size + 1) and not blocks.blocks_hold(b - 1, 2) and not blocks.blocks_hold(b, size + 1)
    assert not blocks.blocks_hold(b + 8, (1 << 64) - 8)       # the end wraps around


def test_a_freed_block_is_held_no_longer(blocks):
    a, size = 0x7f0000010000, 1 << 16
    assert blocks.blocks_add(a, size) and blocks.blocks_add(a + size, size)
    blocks.blocks_remove(a)
    assert not blocks.blocks_hold(a, 1) and not blocks.blocks_hold(a + size - 1, 1) and blocks.blocks_hold(a + size, size)
    blocks.blocks_remove(a)                                   # not there: nothing happens
    assert blocks.blocks_add(a, 16) and blocks.blocks_hold(a, 16) and not blocks.blocks_hold(a, 17)


def test_a_block_that_finds_no_entry_is_refused_and_not_held(blocks):
    a, size = 0x7f0000010000, 1 << 16
    blocks.blocks_no_memory(1)
    refused = not blocks.blocks_add(a, size)
    blocks.blocks_no_memory(0)
    assert refused and not blocks.blocks_hold(a, 1)
    assert blocks.blocks_add(a, size) and blocks.blocks_hold(a, size)

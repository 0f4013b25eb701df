"""When the Python layer page-locks memory for results, and when it gives it back (host side, the library's two calls
stood in for)."""
import threading

import numpy as np
import pytest

from ullis_b200 import cuda

BIG = 1 << 20


class Library:
    """ullis_cuda_host_alloc / _free over ordinary memory, counting."""

    def __init__(self):
        self.blocks, self.locks = {}, 0
        self._lib, self._h = self, None

    def ullis_cuda_host_alloc(self, _, size, out):
        block = np.zeros(size.value, np.uint8)
        self.blocks[block.ctypes.data] = block
        self.locks += 1
        out._obj.value = block.ctypes.data
        return cuda.OK

    def ullis_cuda_host_free(self, p):
        del self.blocks[p.value]


@pytest.fixture
def lib():
    return Library()


def test_kept_results_lock_little_and_dropped_ones_are_reused(lib):
    pool = cuda._ResultPool(unproven=3 * BIG)
    kept = [pool.empty(lib, BIG, np.uint8) for _ in range(20)]
    assert lib.locks == 3
    for i, a in enumerate(kept):
        a[:] = i
    assert all((a == i).all() for i, a in enumerate(kept))
    del kept[5:], a
    for _ in range(50):
        pool.empty(lib, BIG, np.uint8)
    assert lib.locks == 4                                              # the three are under live arrays
    kept += [pool.empty(lib, BIG, np.uint8) for _ in range(100)]       # as many blocks as results came back before, no more
    assert lib.locks <= 3 + 15 and pool._held == lib.locks * pool._block_size(BIG)


def test_results_that_live_in_batches_are_all_reused(lib):
    pool = cuda._ResultPool(unproven=BIG)
    for _ in range(4):
        batch = [pool.empty(lib, (2, BIG // 8), np.float32) for _ in range(10)]
        del batch
    assert lib.locks == 10


def test_one_result_larger_than_the_trial_is_locked_the_second_time(lib):
    pool = cuda._ResultPool(unproven=BIG)
    for locks in (0, 1, 1):
        pool.empty(lib, 2 * BIG, np.uint8)
        assert lib.locks == locks


def test_idle_memory_is_given_back_on_request_and_with_the_last_runtime(lib):
    pool = cuda._ResultPool()
    pool.attach()
    pool.attach()
    a = pool.empty(lib, 1000, np.float32)
    pool.empty(lib, 5000, np.float32)
    pool.release()
    assert len(lib.blocks) == 1                                        # the one under `a`
    pool.empty(lib, 5000, np.float32)
    pool.detach()
    assert len(lib.blocks) == 2
    pool.detach()
    assert len(lib.blocks) == 1
    view = a[3:7]
    del a
    assert len(lib.blocks) == 1
    del view
    assert not lib.blocks and pool._held == 0


@pytest.mark.parametrize("unproven", [0, 1 << 28])
def test_sizes_that_do_not_fit_together_do_not_take_turns_at_every_call(lib, unproven):
    pool = cuda._ResultPool(limit=3 * BIG, unproven=unproven)
    for _ in range(10):
        pool.empty(lib, 2 * BIG, np.uint8)
        pool.empty(lib, 2 * BIG + BIG // 2, np.uint8)
    assert lib.locks <= 12 and pool._held <= pool.limit                # of 20 calls
    held = pool._held
    assert pool.empty(lib, 4 * BIG, np.uint8).size == 4 * BIG and pool._held == held   # never fits: nothing goes for it


def test_threads_share_the_pool(lib):
    pool = cuda._ResultPool()
    errors = []

    def work(value):
        for _ in range(200):
            a = pool.empty(lib, 3000, np.uint8)
            a[:] = value
            if not (a == value).all():
                errors.append(value)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    # the name lets go of the last result after the next one is made: two blocks per thread
    assert not errors and lib.locks <= 8 and pool._held == sum(b.size for b in lib.blocks.values())

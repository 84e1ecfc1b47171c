"""CPU tests of the budget on a resident run's waits (gpu_bpf_debug_wait_budget): it counts time spent
polling, so a clock that jumps while the whole grid is held up does not end a wait, and polling without
an answer always does."""
from __future__ import annotations

import ctypes as C

import pytest

LIMIT = 2_000_000_000
T0 = 1_700_000_000_000_000_000
UNIT = 1024


@pytest.fixture(scope="module")
def budget(bpf):
    lib = bpf.load()

    def call(looks, limit=LIMIT):
        return lib.gpu_bpf_debug_wait_budget((C.c_ulonglong * len(looks))(*looks), len(looks), limit)
    return call


@pytest.mark.parametrize("step", [1_000, 150_000, 10_000_000, 100_000_000])
def test_steady_polling_gives_up_at_the_limit(budget, step):
    n = -(-(LIMIT + UNIT) // step)                   # the first look at which n steps reach the limit,
    looks = [T0 + i * step for i in range(n + 5)]    # to a unit of the clock
    assert -(-(LIMIT - UNIT) // step) <= budget(looks) <= n


def test_a_grid_held_up_goes_on_waiting(budget):
    """One look before a hold of a minute, then polling as usual: the wait has most of its limit left."""
    looks = [T0 + i * 150_000 for i in range(100)]
    held = looks[-1] + 60_000_000_000
    looks += [held + i * 150_000 for i in range(1000)]
    assert budget(looks) == len(looks)
    more = [looks[-1] + (i + 1) * 150_000 for i in range(20_000)]
    at = budget(looks + more)
    assert at < len(looks + more)                    # and still ends
    assert (looks + more)[at] - held >= LIMIT * 15 // 16 - 100 * 150_000 - 150_000 - 2 * UNIT


def test_ends_however_long_the_looks_are_apart(budget):
    assert budget([T0 + i * 60_000_000_000 for i in range(40)]) == 16
    assert budget([T0 + i * 2048 for i in range(9)], 4096) == 4      # 1 of 4 units counted of each 2
    assert budget([T0] * 1000) == 1000               # a clock that stands still spends nothing


def test_rejects_bad_arguments(bpf):
    from gpubpf import _lib
    lib = bpf.load()
    one = (C.c_ulonglong * 1)(T0)
    assert lib.gpu_bpf_debug_wait_budget(None, 1, LIMIT) == -_lib.BPF_ERR_ARG
    assert lib.gpu_bpf_debug_wait_budget(one, -1, LIMIT) == -_lib.BPF_ERR_ARG
    assert lib.gpu_bpf_debug_wait_budget(one, 1, 1023) == -_lib.BPF_ERR_ARG
    assert lib.gpu_bpf_debug_wait_budget(one, 1, LIMIT + 1) == -_lib.BPF_ERR_ARG

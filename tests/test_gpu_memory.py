"""What the library does when device memory runs out, and what it keeps idle.  Needs a B200."""
from __future__ import annotations

import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GIB = 1 << 30


@pytest.fixture(scope="module")
def z(zntt):
    zntt.init(0)
    return zntt


@pytest.fixture
def fresh(z):
    """The library with nothing cached, before and after."""
    import torch
    z.shutdown()
    z.init(0)
    torch.cuda.empty_cache()
    yield z
    z.shutdown()
    z.init(0)
    torch.cuda.empty_cache()


def _fill(leave):
    """Torch buffers that take all free device memory but `leave` bytes (memory just freed may
    turn up late, so until none does)."""
    import torch
    taken = []
    for _ in range(20):
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        if free > leave + (64 << 20):
            taken.append(torch.empty(free - leave, dtype=torch.uint8, device="cuda"))
        time.sleep(0.05)
    return taken


def _roundtrip(z, F, log_n):
    import torch
    x = torch.zeros(4 << log_n, dtype=torch.int64, device="cuda")
    y, w = torch.zeros_like(x), torch.zeros_like(x)
    torch.cuda.synchronize()
    with z.DeviceTwiddles(F, log_n, z.primitiveRootOfUnity(F, log_n)) as tw:
        z.random_elements(F, 9, x.data_ptr(), 1 << log_n)
        z.ntt_device(tw, x.data_ptr(), y.data_ptr(), z.FORWARD)
        z.ntt_device(tw, y.data_ptr(), w.data_ptr(), z.INVERSE)
        torch.cuda.synchronize()
    assert torch.equal(x, w) and not torch.equal(x, y)


def test_a_refused_allocation_is_not_the_next_calls_error(fresh):
    z, F = fresh, fresh.BN254_FR
    _roundtrip(z, F, 10)  # the slabs of small buffers are there before memory is taken
    filler = _fill(2 * GIB)
    try:
        with pytest.raises(z.OutOfMemory):
            z.DeviceTwiddles(F, 27, z.primitiveRootOfUnity(F, 27))
        _roundtrip(z, F, 10)
    finally:
        del filler


def test_caller_tables_leave_two_vectors_in_the_pool(fresh):
    """A host call with the caller's own table keeps what any host call does: its two vectors."""
    z, F, log_n = fresh, fresh.BN254_FR, 18
    tab = z.precomputeTwiddles(F, log_n, z.primitiveRootOfUnity(F, log_n))
    own = [np.array(s, copy=True) for s in tab]
    z.freeTwiddles(F, tab)
    z.shutdown()
    z.init(0)
    before = z.pool_stats()
    data = np.zeros((1 << log_n, 4), dtype=np.uint64)
    data[:, 0] = np.arange(1 << log_n)
    keep = data.copy()
    for _ in range(3):
        z.nttWithTwiddles(F, data, log_n, own)
        z.inttWithTwiddles(F, data, log_n, own)
    assert np.array_equal(data, keep)
    after = z.pool_stats()
    assert after["cached_bytes"] - before["cached_bytes"] == 2 * (32 << log_n)
    assert after["device_mallocs"] - before["device_mallocs"] == 2


def test_idle_tables_of_a_large_size_stay(fresh):
    """A program that takes and returns the tables of 2^28 for a forward and an inverse root in
    turn builds each once."""
    import oracle as O
    z, F, log_n = fresh, fresh.BN254_FR, 28
    root = z.primitiveRootOfUnity(F, log_n)
    roots = [root, O.pow_(O.BN254_FR, root, (1 << log_n) - 1)]
    took = []
    for _ in range(3):
        for r in roots:
            t0 = time.perf_counter()
            with z.DeviceTwiddles(F, log_n, r):
                took.append(time.perf_counter() - t0)
    assert max(took[2:]) < 0.2 * min(took[:2]), took


def test_idle_tables_make_room(fresh):
    """On a full device the library's idle tables go before a call is refused."""
    import torch
    z, F, log_n = fresh, fresh.BN254_FR, 26
    x = torch.zeros(4 << log_n, dtype=torch.int64, device="cuda")
    x[:4096] = torch.arange(4096, device="cuda")
    first = x[:4096].clone()
    with z.DeviceTwiddles(F, log_n, z.primitiveRootOfUnity(F, log_n)) as tw:
        z.DeviceTwiddles(F, 27, z.primitiveRootOfUnity(F, 27)).close()  # 8 GiB, idle
        filler = _fill(GIB)
        try:
            for mode in (z.FORWARD, z.INVERSE):
                z.ntt_device(tw, x.data_ptr(), x.data_ptr(), mode)  # borrows 2 GiB
            torch.cuda.synchronize()
        finally:
            del filler
    assert torch.equal(x[:4096], first)

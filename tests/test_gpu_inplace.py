"""In-place transforms of at most 2^11 elements are one pass: no scratch, no wait, no memory
shared between calls.  Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def z(zntt):
    zntt.init(0)
    return zntt


def _fields(z):
    return [(z.BN254_FR, O.BN254_FR), (z.BLS12_381_FR, O.BLS12_381_FR)]


def _vec(z, F, seed, n):
    import torch
    x = torch.empty(n * 4, dtype=torch.int64, device="cuda")
    z.random_elements(F, seed, x.data_ptr(), n)
    return x


def _host(t):
    return t.cpu().numpy().view(np.uint64).reshape(-1, 4).copy()


@pytest.mark.parametrize("log_n", [2, 3, 5, 7, 8, 9, 10, 11])
def test_allocation_free_calls_match_oracle(z, log_n):
    import torch
    for F, fid in _fields(z):
        _, root = O.primitive_root(fid, log_n)
        _, stages = O.precompute_twiddles(fid, log_n, root)
        with z.DeviceTwiddles(F, log_n, z.primitiveRootOfUnity(F, log_n)) as tw:
            for mode, inverse in ((z.FORWARD, False), (z.INVERSE, True)):
                x = _vec(z, F, 60 + log_n, 1 << log_n)
                torch.cuda.synchronize()
                want = _host(x)
                O.ntt_with_twiddles(fid, want, log_n, stages, inverse=inverse)
                z.ntt_device_inplace_noalloc(tw, x.data_ptr(), mode)
                torch.cuda.synchronize()
                np.testing.assert_array_equal(_host(x), want, err_msg=f"{F.name} 2^{log_n} mode {mode}")


@pytest.mark.parametrize("log_n", [8, 9, 10, 11])
def test_allocation_free_calls_may_overlap(z, log_n):
    """Calls on several streams, which run side by side, agree with single ones."""
    import torch
    streams = [torch.cuda.Stream() for _ in range(8)]
    for F, _ in _fields(z):
        with z.DeviceTwiddles(F, log_n, z.primitiveRootOfUnity(F, log_n)) as tw:
            xs = [_vec(z, F, 70 + i, 1 << log_n) for i in range(64)]
            wants = [torch.empty_like(x) for x in xs]
            for x, w in zip(xs, wants):
                z.ntt_device(tw, x.data_ptr(), w.data_ptr(), z.FORWARD)
            torch.cuda.synchronize()
            for i, x in enumerate(xs):
                z.ntt_device_inplace_noalloc(tw, x.data_ptr(), z.FORWARD, stream=streams[i % 8].cuda_stream)
            torch.cuda.synchronize()
            for i, (x, w) in enumerate(zip(xs, wants)):
                assert torch.equal(x, w), (F.name, i)


@pytest.mark.parametrize("log_n", [8, 9, 10, 11])
def test_no_wait_under_the_shipped_tuning_table(z, log_n):
    """Whatever plan the tuning table holds, an in-place call without scratch neither waits nor
    allocates up to 2^11, so a caller's graph can hold it."""
    import os

    import torch
    z.tune_load(os.path.join(os.path.dirname(z.__file__), "tune", "b200.json"))
    stream = torch.cuda.Stream()
    try:
        for F, fid in _fields(z):
            _, root = O.primitive_root(fid, log_n)
            _, stages = O.precompute_twiddles(fid, log_n, root)
            with z.DeviceTwiddles(F, log_n, z.primitiveRootOfUnity(F, log_n)) as tw, torch.cuda.stream(stream):
                for mode, inverse in ((z.FORWARD, False), (z.INVERSE, True)):
                    x = _vec(z, F, 80 + log_n, 1 << log_n)
                    torch.cuda.synchronize()
                    want = _host(x)
                    O.ntt_with_twiddles(fid, want, log_n, stages, inverse=inverse)
                    before = z.pool_stats()["acquires"]
                    graph = torch.cuda.CUDAGraph()
                    with torch.cuda.graph(graph, stream=stream):
                        z.ntt_device(tw, x.data_ptr(), x.data_ptr(), mode, stream=stream.cuda_stream)
                    graph.replay()
                    stream.synchronize()
                    assert z.pool_stats()["acquires"] == before
                    np.testing.assert_array_equal(_host(x), want, err_msg=f"{F.name} 2^{log_n} mode {mode}")
    finally:
        z.tune_clear()

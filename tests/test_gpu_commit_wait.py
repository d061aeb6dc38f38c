"""How a commitment that returns its root waits for it.  Needs a B200."""
from __future__ import annotations

import os
import subprocess
import sys
import time

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def z(zntt):
    zntt.init(0)
    return zntt


_BLOCKING = """
import ctypes, sys, time
sys.path.insert(0, {tests!r})
cu = ctypes.CDLL("libcuda.so.1")
assert cu.cuInit(0) == 0 and cu.cuDevicePrimaryCtxSetFlags_v2(0, 4) == 0  # CU_CTX_SCHED_BLOCKING_SYNC
import torch
from conftest import load_package
z = load_package()
z.init(0)
L = 26
layer = torch.zeros(1 << L, dtype=torch.int64, device="cuda")
nodes = torch.empty(32 << L, dtype=torch.uint8, device="cuda")
z.fri_commit_layer(z.GOLDILOCKS, layer.data_ptr(), L, nodes.data_ptr())
wall, cpu = time.perf_counter(), time.thread_time()
for _ in range(30):
    z.fri_commit_layer(z.GOLDILOCKS, layer.data_ptr(), L, nodes.data_ptr())
print(time.perf_counter() - wall, time.thread_time() - cpu)
"""


def test_a_long_wait_leaves_the_core(z):
    """In a process that asks for blocking waits a long commitment sleeps: its thread is on a core
    for less than half of the time (the launches, and a wait of at most 0.2 ms before it sleeps)."""
    code = _BLOCKING.format(tests=os.path.join(ROOT, "tests"))
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    wall, cpu = map(float, out.stdout.split())
    assert wall > 30 * 1e-3  # milliseconds each, so that the bound says something
    assert cpu < 0.5 * wall, (wall, cpu)


def test_a_larger_commitment_does_not_wait_for_other_streams(z):
    """A commitment larger than any before it neither frees nor allocates: it returns while
    another stream is still busy."""
    import torch
    z.shutdown()
    z.init(0)
    F, L = z.GOLDILOCKS, 26
    layer = torch.zeros(1 << L, dtype=torch.int64, device="cuda")
    nodes = torch.empty(32 << L, dtype=torch.uint8, device="cuda")
    mine, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    z.fri_commit_layer(F, layer.data_ptr(), 22, nodes.data_ptr(), stream=mine.cuda_stream)  # the same kernels
    with torch.cuda.stream(other):
        torch.cuda._sleep(2_000_000_000)  # about a second
        busy = torch.cuda.Event()
        busy.record()
    t0 = time.perf_counter()
    root = z.fri_commit_layer(F, layer.data_ptr(), L, nodes.data_ptr(), stream=mine.cuda_stream)
    took = time.perf_counter() - t0
    assert not busy.query() and took < 0.5, took
    torch.cuda.synchronize()
    assert root == z.fri_commit_layer(F, layer.data_ptr(), L, nodes.data_ptr(), stream=mine.cuda_stream)

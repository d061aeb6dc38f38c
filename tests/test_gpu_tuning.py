"""The tuning table decides the plan of a transform at every size it holds, the radix-2 passes
among its candidates.  Plans are told apart by the launches that a captured call holds.
Needs a B200."""
from __future__ import annotations

import json

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def z(zntt):
    zntt.init(0)
    return zntt


def _launches(z, F, log_n):
    """How many launches one out-of-place transform of 2^log_n elements makes."""
    import torch
    from cuda.bindings import runtime as rt
    stream = torch.cuda.Stream()
    with z.DeviceTwiddles(F, log_n, z.primitiveRootOfUnity(F, log_n)) as tw, torch.cuda.stream(stream):
        x = torch.zeros(4 << log_n, dtype=torch.int64, device="cuda")
        y = torch.zeros_like(x)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph, stream=stream):
            z.ntt_device(tw, x.data_ptr(), y.data_ptr(), z.FORWARD, stream=stream.cuda_stream)
        err, _, count = rt.cudaGraphGetNodes(graph.raw_cuda_graph(), 64)
        assert int(err) == 0
        return count


def _table(z, tmp_path, **extra):
    import torch
    row = {"gpu": torch.cuda.get_device_name(0), "field": 0, "log_n": 11, "shape": 3, "kmax": 4, "us": 20.0, **extra}
    path = tmp_path / "tune.json"
    path.write_text("[\n " + json.dumps(row) + "\n]\n")
    return str(path)


def test_a_loaded_table_decides(z, tmp_path):
    F = z.BN254_FR
    z.tune_clear()
    try:
        assert _launches(z, F, 11) == 2  # the radix-2 plan
        z.tune_load(_table(z, tmp_path))
        assert _launches(z, F, 11) == 3  # four stages a pass
        assert _launches(z, F, 12) == 2 and _launches(z, z.BLS12_381_FR, 11) == 2  # sizes it does not hold
        z.tune_load(_table(z, tmp_path, radix2_us=30.0))
        assert _launches(z, F, 11) == 3
        z.tune_load(_table(z, tmp_path, radix2_us=10.0))
        assert _launches(z, F, 11) == 2
    finally:
        z.tune_clear()


def test_the_tuner_times_the_radix2_passes(z, tmp_path):
    z.tune_clear()
    path = str(tmp_path / "tune.json")
    try:
        z.autotune(z.BLS12_381_FR, 12, 12)
        z.tune_save(path)
        rows = json.load(open(path))
        assert rows and all(r["radix2_us"] > 0 for r in rows)
        best = min(rows, key=lambda r: r["us"])
        made = _launches(z, z.BLS12_381_FR, 12)
        assert made == 2 if best["radix2_us"] <= best["us"] else made >= 2
        z.tune_clear()
        z.tune_load(path)
        assert _launches(z, z.BLS12_381_FR, 12) == made
    finally:
        z.tune_clear()

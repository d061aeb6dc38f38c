"""The radix-4 passes on partial tiles and odd stage counts, which plain transforms of these sizes
reach through the tuning table, in batches and in place: values and tables at the ends of the
range, bit-exact against the oracle.  Needs a B200."""
from __future__ import annotations

import json
import os

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
WORKERS = min(os.cpu_count() or 1, 64)
LOG_TILE = {0: 11, 1: 10, 2: 9, 3: 8, 4: 9}  # kShapes in csrc/kernels.cuh


@pytest.fixture(scope="module")
def z(zntt):
    zntt.init(0)
    return zntt


def _fields(z):
    return [(z.BN254_FR, O.BN254_FR), (z.BLS12_381_FR, O.BLS12_381_FR)]


def _edge_elements(fid, n, seed):
    """Values at the ends of the range among random ones."""
    p = O.MODULI[fid]
    edge = O.from_ints([p - 1, 0, 1, p - 2, ((p >> 224) << 224) - 1, p >> 1, (p >> 1) + 1, (1 << 224) - 1])
    a = O.random_elements(fid, seed, n)
    pos = np.random.default_rng(seed).permutation(n)[:max(1, n // 2)]
    a[pos] = edge[np.arange(len(pos)) % len(edge)]
    return a


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int64).reshape(-1)).cuda()


def _host(t):
    return t.cpu().numpy().view(np.uint64).reshape(-1, 4).copy()


def _want(fid, a, log_n, stages, inverse):
    want = a.copy()
    assert O.ntt_with_twiddles(fid, want, log_n, stages, inverse=inverse, workers=WORKERS, inplace4=True) == O.OK
    return want


@pytest.mark.parametrize("shape", sorted(LOG_TILE))
def test_forced_plans_on_small_sizes(z, tmp_path, shape):
    """Every stage count per pass of a shape, out of place and in place with scratch."""
    import torch
    name = torch.cuda.get_device_name(0)
    path = tmp_path / "tune.json"
    for F, fid in _fields(z):
        for log_n in (1, 2, 3, 4, 6, 7, 8, 9, 10, 11, 12, 13):
            _, root = O.primitive_root(fid, log_n)
            _, stages = O.precompute_twiddles(fid, log_n, root)
            a = _edge_elements(fid, 1 << log_n, 10 * log_n + shape)
            wants = [_want(fid, a, log_n, stages, inverse) for inverse in (False, True)]
            x = _dev(a)
            with z.DeviceTwiddles(F, log_n, z.primitiveRootOfUnity(F, log_n)) as tw:
                for kmax in range(max(2, LOG_TILE[shape] - 4), LOG_TILE[shape] + 1):
                    path.write_text("[\n " + json.dumps({"gpu": name, "field": F.id, "log_n": log_n, "shape": shape,
                                                         "kmax": kmax, "us": 1.0}) + "\n]\n")
                    z.tune_clear()
                    z.tune_load(str(path))
                    try:
                        for mode, want in zip((z.FORWARD, z.INVERSE), wants):
                            y, s, w = torch.zeros_like(x), torch.zeros_like(x), x.clone()
                            torch.cuda.synchronize()
                            z.ntt_device(tw, x.data_ptr(), y.data_ptr(), mode)
                            z.ntt_device(tw, w.data_ptr(), w.data_ptr(), mode, d_scratch=s.data_ptr())
                            torch.cuda.synchronize()
                            what = f"{F.name} 2^{log_n} kmax {kmax} mode {mode}"
                            np.testing.assert_array_equal(_host(y), want, err_msg=what)
                            np.testing.assert_array_equal(_host(w), want, err_msg=what + " in place")
                    finally:
                        z.tune_clear()


@pytest.mark.parametrize("shape", sorted(LOG_TILE))
def test_batches_of_small_sizes(z, shape):
    """One batch over all small sizes, both directions, in place and not."""
    import torch
    for F, fid in _fields(z):
        tabs, jobs, outs, keep = [], [], [], []
        for log_n in range(1, 15):
            _, root = O.primitive_root(fid, log_n)
            _, stages = O.precompute_twiddles(fid, log_n, root)
            tabs.append(z.DeviceTwiddles(F, log_n, z.primitiveRootOfUnity(F, log_n)))
            a = _edge_elements(fid, 1 << log_n, 20 * log_n + shape)
            for mode, inverse in ((z.FORWARD, False), (z.INVERSE, True)):
                want = _want(fid, a, log_n, stages, inverse)
                src, same, dst = _dev(a), _dev(a), torch.zeros(4 << log_n, dtype=torch.int64, device="cuda")
                jobs += [{"kind": z.JOB_NTT, "tw": tabs[-1], "mode": mode, "src": src.data_ptr(), "dst": dst.data_ptr()},
                         {"kind": z.JOB_NTT, "tw": tabs[-1], "mode": mode, "src": same.data_ptr(),
                          "dst": same.data_ptr()}]
                outs += [(dst, want, log_n, mode), (same, want, log_n, mode)]
                keep.append(src)
        torch.cuda.synchronize()
        with z.Batch(F, jobs, shape=shape) as b:
            b.run()
            torch.cuda.synchronize()
            b.status()
        for got, want, log_n, mode in outs:
            np.testing.assert_array_equal(_host(got), want, err_msg=f"{F.name} 2^{log_n} mode {mode}")
        for t in tabs:
            t.close()


@pytest.mark.parametrize("log_n", [17, 18])
def test_extreme_values_and_tables(z, log_n):
    """The widest ranges inside a pass: BN254-Fr's butterflies start from u below 1.07 p, leave
    results below 3.07 p and then 5.07 p; BLS12-381-Fr's stay below 2 p."""
    n = 1 << log_n
    for F, fid in _fields(z):
        p = O.MODULI[fid]
        row = {k: np.array(O.int_to_limbs(v), dtype=np.uint64) for k, v in (("p-1", p - 1), ("1", 1), ("0", 0))}
        row["one"] = O.from_int(fid, 1)
        full = {k: np.ascontiguousarray(np.tile(v, (n, 1))) for k, v in row.items()}
        alternating = np.ascontiguousarray(np.where((np.arange(n) % 2 == 0)[:, None], row["0"], row["p-1"]))
        for data, entry in ((full["p-1"], "p-1"), (alternating, "p-1"), (full["p-1"], "1"), (full["p-1"], "one"),
                            (full["p-1"], "0")):
            table = [np.ascontiguousarray(full[entry][:1 << s]) for s in range(log_n)]
            for inverse in (False, True):
                got = data.copy()
                (z.inttWithTwiddles if inverse else z.nttWithTwiddles)(F, got, log_n, table)
                np.testing.assert_array_equal(got, _want(fid, data, log_n, table, inverse),
                                              err_msg=f"{F.name} entry {entry} inverse {inverse}")


@pytest.mark.parametrize("log_n", [1, 3, 9, 13, 17])
def test_caller_entries_at_or_above_the_modulus(z, log_n):
    """They count as their residues."""
    for F, fid in _fields(z):
        p, rng = O.MODULI[fid], np.random.default_rng(log_n)
        table = [_edge_elements(fid, 1 << s, 30 * log_n + s) for s in range(log_n)]
        above = []
        for t in table:
            t = t.copy()
            for i in rng.permutation(len(t))[:200]:
                v = O.limbs_to_int(t[i])
                t[i] = O.int_to_limbs(v + int(rng.integers(0, ((1 << 256) - 1 - v) // p + 1)) * p)
            t[0] = O.int_to_limbs(O.limbs_to_int(table[len(above)][0]) + p)  # entry 0 is never one
            above.append(t)
        a = _edge_elements(fid, 1 << log_n, 40 + log_n)
        for inverse in (False, True):
            got = a.copy()
            (z.inttWithTwiddles if inverse else z.nttWithTwiddles)(F, got, log_n, above)
            np.testing.assert_array_equal(got, _want(fid, a, log_n, table, inverse), err_msg=f"{F.name} {inverse}")


@pytest.mark.parametrize("log_n", [1, 7, 8, 9, 15, 16, 17, 20])
def test_captured_transforms_of_the_other_field(z, log_n):
    import torch
    F, n = z.BLS12_381_FR, 1 << log_n
    stream = torch.cuda.Stream()
    with z.DeviceTwiddles(F, log_n, z.primitiveRootOfUnity(F, log_n)) as tw, torch.cuda.stream(stream):
        src, mid, dst = (torch.zeros(4 * n, dtype=torch.int64, device="cuda") for _ in range(3))
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            z.ntt_device(tw, src.data_ptr(), mid.data_ptr(), z.FORWARD, stream=stream.cuda_stream)
            z.ntt_device(tw, mid.data_ptr(), dst.data_ptr(), z.INVERSE, stream=stream.cuda_stream)
        for seed in (1, 2):
            z.random_elements(F, seed, src.data_ptr(), n, stream=stream.cuda_stream)
            z.ntt_device(tw, src.data_ptr(), mid.data_ptr(), z.FORWARD, stream=stream.cuda_stream)
            want = mid.clone()
            mid.zero_()
            dst.zero_()
            graph.replay()
            stream.synchronize()
            assert torch.equal(mid, want) and torch.equal(dst, src)

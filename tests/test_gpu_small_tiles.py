"""The small fields' whole-tile passes (needs a B200): every stage count per pass the planner
uses (sizes 2^12 to 2^22), data and caller tables at the ends of the fields' ranges, and the
scaling by shift powers in an extension's inverse.  Bit-exact against the oracle."""
from __future__ import annotations

import os

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

WORKERS = min(os.cpu_count() or 1, 64)


@pytest.fixture(scope="module")
def z(zntt):
    zntt.init(0)
    return zntt


def _fields(z):
    return [(z.GOLDILOCKS, O.GOLDILOCKS), (z.BABYBEAR, O.BABYBEAR)]


def _slots(fid, values):
    s = O.elems(len(values))
    s[:, 0] = np.asarray(values, dtype=np.uint64)
    return O.to_mont(fid, s)


def _canon(fid, slots):
    return np.ascontiguousarray(O.from_mont(fid, np.ascontiguousarray(slots))[:, 0])


def _edge(F, n, seed):
    """Values at both ends of [0, p) and around words of ones, among random ones."""
    p = F.modulus
    r = np.random.default_rng(seed)
    x = np.array([int(v) % p for v in r.integers(0, 1 << 64, n, dtype=np.uint64)], dtype=np.uint64) if n <= 1 << 14 \
        else r.integers(0, p, n, dtype=np.uint64)
    ends = np.array([p - 1, 0, 1, p - 2, 0xFFFFFFFF % p, (p - 1) // 2, (p + 1) // 2, (p - (1 << 16)) % p], dtype=np.uint64)
    pos = r.permutation(n)[: n // 2]
    x[pos] = ends[np.arange(len(pos)) % len(ends)]
    return x


def _device(a):
    import torch
    return torch.from_numpy(a.view(np.int64).copy()).cuda()


def _host(t):
    return t.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("log_n", range(12, 23))
def test_every_pass_length(z, log_n):
    import torch
    n = 1 << log_n
    for F, fid in _fields(z):
        x = _edge(F, n, log_n)
        root = z.primitiveRootOfUnity(F, log_n)
        _, stages = O.precompute_twiddles(fid, log_n, _slots(fid, [int(root[0])])[0])
        with z.DeviceTwiddles(F, log_n, root) as tw:
            for mode, inverse in ((z.FORWARD, False), (z.INVERSE, True)):
                data = _slots(fid, x)
                O.ntt_with_twiddles(fid, data, log_n, stages, inverse=inverse, workers=WORKERS)
                want = _canon(fid, data)
                src, dst = _device(x), torch.zeros(n, dtype=torch.int64, device="cuda")
                torch.cuda.synchronize()
                z.ntt_device(tw, src.data_ptr(), dst.data_ptr(), mode)
                z.ntt_device(tw, src.data_ptr(), src.data_ptr(), mode)  # in place
                torch.cuda.synchronize()
                np.testing.assert_array_equal(_host(dst), want, err_msg=f"{F.name} 2^{log_n} {mode}")
                np.testing.assert_array_equal(_host(src), want, err_msg=f"{F.name} 2^{log_n} {mode} in place")


@pytest.mark.parametrize("log_n", [12, 15, 19])
def test_caller_tables_with_unit_first_entries(z, log_n):
    """Tables that are no root's powers: entries 0 are one, the others anything."""
    for F, fid in _fields(z):
        table = []
        for s in range(log_n):
            t = _edge(F, 1 << s, 31 * log_n + s) if s else np.ones(1, dtype=np.uint64)
            t[0] = 1
            table.append(t)
        x = _edge(F, 1 << log_n, 5)
        for inverse in (False, True):
            data = _slots(fid, x)
            O.ntt_with_twiddles(fid, data, log_n, [_slots(fid, t) for t in table], inverse=inverse, workers=WORKERS)
            got = x.copy()
            (z.inttWithTwiddles if inverse else z.nttWithTwiddles)(F, got, log_n, table)
            np.testing.assert_array_equal(got, _canon(fid, data), err_msg=f"{F.name} 2^{log_n} inverse={inverse}")


@pytest.mark.parametrize("log_in,log_out", [(11, 12), (12, 13), (14, 14), (16, 19), (17, 18)])
def test_column_extensions(z, log_in, log_out):
    import torch
    m = 3
    for F, fid in _fields(z):
        shift = 31
        cols = [_edge(F, 1 << log_in, 100 * log_in + k) for k in range(m)]
        src = _device(np.concatenate(cols))
        dst = torch.zeros(m << log_out, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        with z.DeviceTwiddles(F, log_in, z.primitiveRootOfUnity(F, log_in)) as ti, \
                z.DeviceTwiddles(F, log_out, z.primitiveRootOfUnity(F, log_out)) as to:
            z.coset_lde_columns(ti, to, np.array([shift, 0, 0, 0], dtype=np.uint64),
                                [src.data_ptr() + k * (8 << log_in) for k in range(m)],
                                [dst.data_ptr() + k * (8 << log_out) for k in range(m)])
        got = _host(dst).reshape(m, -1)
        for k in range(m):
            want = O.coset_lde(fid, _slots(fid, cols[k]), log_in, log_out - log_in, _slots(fid, [shift])[0],
                               workers=WORKERS)
            np.testing.assert_array_equal(got[k], _canon(fid, want), err_msg=f"{F.name} column {k}")

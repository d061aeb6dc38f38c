"""Polynomial products in a batch read the other factor's transform, which other CTAs of the
same launch wrote a moment before: many such jobs of several passes each, run and replayed on
changed inputs, so that a line of an earlier run would show.  Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def z(zntt):
    zntt.init(0)
    return zntt


@pytest.mark.parametrize("shape", [-1, 0, 3])
def test_replayed_products_follow_their_inputs(z, shape):
    import torch
    for F, fid in ((z.BN254_FR, O.BN254_FR), (z.BLS12_381_FR, O.BLS12_381_FR)):
        rng = np.random.default_rng(90 + shape)
        tabs, jobs, bufs = {}, [], []
        for q in range(40):
            L = int(rng.integers(12, 16))
            n = 1 << L
            la = int(rng.integers(n // 4, n // 2 + 1))
            lb = int(rng.integers(n // 4, n + 2 - la))
            if L not in tabs:
                tabs[L] = z.DeviceTwiddles(F, L, z.primitiveRootOfUnity(F, L))
            a, b, got, want = (torch.zeros(4 * k, dtype=torch.int64, device="cuda") for k in (la, lb, la + lb - 1,
                                                                                          la + lb - 1))
            jobs.append({"kind": z.JOB_POLY_MUL, "tw": tabs[L], "src": a.data_ptr(), "len": la, "src2": b.data_ptr(),
                         "len2": lb, "dst": got.data_ptr()})
            bufs.append((L, la, lb, a, b, got, want))
        with z.Batch(F, jobs, shape=shape) as batch:
            assert batch.info()["passes"] >= 6 * len(jobs)
            for run in range(4):
                for q, (L, la, lb, a, b, got, want) in enumerate(bufs):
                    z.random_elements(F, 1000 * run + 2 * q, a.data_ptr(), la)
                    z.random_elements(F, 1000 * run + 2 * q + 1, b.data_ptr(), lb)
                    z.poly_mul_device(tabs[L], a.data_ptr(), la, b.data_ptr(), lb, want.data_ptr())
                    got.zero_()
                torch.cuda.synchronize()
                batch.run(graph=run > 0)
                torch.cuda.synchronize()
                batch.status()
                for q, (*_, got, want) in enumerate(bufs):
                    assert torch.equal(got, want), (F.name, run, q)
        # The plain products that these are compared with, against the schoolbook product.
        L, la, lb, a, b, got, _ = min(bufs, key=lambda x: x[1] * x[2])
        ha, hb, hc = (t.cpu().numpy().view(np.uint64).reshape(-1, 4) for t in (a, b, got))
        xs = O.random_elements(fid, 5, 4)
        np.testing.assert_array_equal(O.poly_eval(fid, hc, xs),
                                      O.elementwise(fid, "mul", O.poly_eval(fid, ha, xs), O.poly_eval(fid, hb, xs)))
        for t in tabs.values():
            t.close()

"""Extensions of a single evaluation, a constant polynomial: every value is that evaluation.
Needs a B200."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def z(zntt):
    zntt.init(0)
    return zntt


@pytest.mark.parametrize("log_out", [0, 1, 2, 9, 17])
def test_extension_of_one_evaluation(z, log_out):
    import torch
    for F in z.FIELDS:
        shift = z.to_montgomery(F, 5)
        with z.DeviceTwiddles(F, 0, z.primitiveRootOfUnity(F, 0)) as ti, \
                z.DeviceTwiddles(F, log_out, z.primitiveRootOfUnity(F, log_out)) as to:
            for seed in (1, 2):  # the second call finds the first one's buffers in the pool
                x = torch.zeros(4, dtype=torch.int64, device="cuda")
                z.random_elements(F, seed, x.data_ptr(), 1)
                y = torch.full((4 << log_out,), 99, dtype=torch.int64, device="cuda")
                torch.cuda.synchronize()
                z.coset_lde_device(ti, to, shift, x.data_ptr(), y.data_ptr())
                torch.cuda.synchronize()
                assert (y.view(-1, 4) == x).all(), (F.name, seed)

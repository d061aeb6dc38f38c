"""Host tables written by precomputeTwiddles (libs/ntt/src/root.zig:112-134) in pieces of 2^22
entries, which stages begin and end inside of.  Needs a B200."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def z(zntt):
    zntt.init(0)
    return zntt


@pytest.mark.parametrize("log_n", [1, 2, 3, 9, 21, 22, 23, 24])
def test_host_tables_match_the_oracle(z, log_n):
    for F, fid in ((z.BN254_FR, O.BN254_FR), (z.BLS12_381_FR, O.BLS12_381_FR)):
        root = z.primitiveRootOfUnity(F, log_n)
        tab = z.precomputeTwiddles(F, log_n, root)
        st, want = O.precompute_twiddles(fid, log_n, root)
        assert st == O.OK and len(tab) == len(want) == log_n
        for s in range(log_n):
            np.testing.assert_array_equal(np.asarray(tab[s]), want[s], err_msg=f"{F.name} stage {s}")
        z.freeTwiddles(F, tab)

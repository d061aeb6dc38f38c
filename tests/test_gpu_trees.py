"""Commitments whose caller waits for the root (one launch for the whole tree) against the same
commitment only enqueued (a launch per few levels) and the oracle (needs a B200)."""
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


def _layer(z, F, n, seed):
    import torch
    if F.limbs == 4:
        t = torch.empty(4 * n, dtype=torch.int64, device="cuda")
        z.random_elements(F, seed, t.data_ptr(), n)
    else:
        v = np.random.default_rng(seed).integers(0, F.modulus, n, dtype=np.uint64)
        t = torch.from_numpy(v.view(np.int64)).cuda()
    torch.cuda.synchronize()
    return t


@pytest.mark.parametrize("log_n", [1, 2, 8, 9, 10, 13, 14, 15, 17, 18, 19])
def test_waited_and_enqueued_trees_agree(z, log_n):
    import torch
    for F in (*z.FIELDS, *z.SMALL_FIELDS):
        layer = _layer(z, F, 1 << log_n, 40 + log_n)
        # Garbage in the node arrays: every node, node 0 included, is written.
        waited, enqueued = (torch.full((4 << log_n,), -1, dtype=torch.int64, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        for _ in range(2):  # the second time on the counters that the first one left
            root = z.fri_commit_layer(F, layer.data_ptr(), log_n, waited.data_ptr())
        assert z.lib().zntt_fri_commit_layer(F.id, layer.data_ptr(), log_n, enqueued.data_ptr(), None, None) == 0
        torch.cuda.synchronize()
        assert torch.equal(waited, enqueued), (F.name, log_n)
        assert root == waited[4:8].cpu().numpy().tobytes()


@pytest.mark.parametrize("log_n", [9, 10, 16])
def test_roots_on_alternating_streams(z, log_n):
    """Calls on different streams share the counters and the root's place, one at a time."""
    import torch
    streams = [torch.cuda.Stream() for _ in range(3)]
    for F, fid in ((z.BN254_FR, O.BN254_FR), (z.GOLDILOCKS, O.GOLDILOCKS)):
        nodes = torch.zeros(4 << log_n, dtype=torch.int64, device="cuda")
        layers = [_layer(z, F, 1 << log_n, 70 + k) for k in range(3)]
        torch.cuda.synchronize()
        roots = [z.fri_commit_layer(F, layers[k % 3].data_ptr(), log_n, nodes.data_ptr(),
                                    stream=streams[k % 3].cuda_stream) for k in range(9)]
        assert roots[:3] == roots[3:6] == roots[6:] and len(set(roots)) == 3
        host = layers[0].cpu().numpy().view(np.uint64)
        if F.limbs == 4:
            slots = host.reshape(-1, 4).copy()
        else:
            slots = O.elems(len(host))
            slots[:, 0] = host
            slots = O.to_mont(fid, slots)
        want = np.asarray(O.fri_commit_layer(fid, slots, log_n, workers=WORKERS))
        assert want.tobytes()[32:64] == roots[0]

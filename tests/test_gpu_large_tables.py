"""Twiddle tables of 2^29 elements and more are strided, and extension tables of that size hold
32-byte factors: transforms of these sizes against values computed on the host, in as much
memory as they are meant to take.  Needs a B200 with about 135 GB free (each test says so when
it has less)."""
from __future__ import annotations

import gc

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
GIB = 1 << 30
FID = O.BLS12_381_FR
P = O.MODULI[FID]


@pytest.fixture
def fresh(zntt):
    """The library with nothing cached, before and after."""
    import torch
    zntt.init(0)
    zntt.shutdown()
    zntt.init(0)
    gc.collect()
    torch.cuda.empty_cache()
    yield zntt
    zntt.shutdown()
    zntt.init(0)
    gc.collect()
    torch.cuda.empty_cache()


def _need(gib):
    import torch
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    if free < gib * GIB:
        pytest.skip(f"{free / GIB:.0f} GiB free, {gib} needed")


def _root(log_n):
    st, r = O.primitive_root(FID, log_n)
    assert st == O.OK
    return O.to_ints(O.from_mont(FID, r.reshape(1, 4)))[0]


def _mont(values):
    return O.to_mont(FID, O.from_ints([v % P for v in values]))


def _put(t, index, values):
    """Canonical values at elements `index` of a device vector, in Montgomery form."""
    import torch
    rows = torch.from_numpy(_mont(values).view(np.int64)).cuda()
    t.view(-1, 4)[torch.tensor(index, device="cuda")] = rows


def _get(t, index):
    import torch
    rows = t.view(-1, 4)[torch.tensor(index, device="cuda")].cpu().numpy().view(np.uint64).copy()
    return O.to_ints(O.from_mont(FID, rows))


def _samples(n, seed):
    rng = np.random.default_rng(seed)
    return [0, 1, 2, 3, n // 2 - 1, n // 2, n // 2 + 1, n - 2, n - 1] + [int(v) for v in rng.integers(0, n, 55)]


def test_transforms_on_a_strided_table(fresh):
    """Five nonzero inputs spread over the vector make every stage's factors count: output k is
    sum x_i w^(ik), and the inverse's the same with w^-1 over n; then back to the input."""
    import torch
    z, log_n = fresh, 29
    F, n = z.BLS12_381_FR, 1 << log_n
    _need(72)
    at = [1, 3, (1 << 28) + 12345, (1 << 20) + 77, n - 1]
    xs = [5, P - 2, 1 << 200, 7 << 100, 123456789]
    w = _root(log_n)
    x = torch.zeros(4 * n, dtype=torch.int64, device="cuda")
    y = torch.empty_like(x)
    _put(x, at, xs)
    ks = _samples(n, 1)
    with z.DeviceTwiddles(F, log_n, z.primitiveRootOfUnity(F, log_n)) as tw:
        for mode, base, scale in ((z.FORWARD, w, 1), (z.INVERSE, pow(w, -1, P), pow(n, -1, P))):
            torch.cuda.synchronize()
            z.ntt_device(tw, x.data_ptr(), y.data_ptr(), mode)
            torch.cuda.synchronize()
            want = [scale * sum(v * pow(base, i * k % n, P) for i, v in zip(at, xs)) % P for k in ks]
            assert _get(y, ks) == want, mode
        # A batch takes the same table.
        y.zero_()
        torch.cuda.synchronize()
        with z.Batch(F, [{"kind": z.JOB_NTT, "tw": tw, "mode": z.INVERSE, "src": x.data_ptr(),
                          "dst": y.data_ptr()}]) as b:
            b.run()
            torch.cuda.synchronize()
            b.status()
        assert _get(y, ks) == want
        z.ntt_device(tw, y.data_ptr(), y.data_ptr(), z.FORWARD, d_scratch=0)
        torch.cuda.synchronize()
        assert torch.equal(x, y)


def test_an_extension_of_2p29_fits(fresh):
    """2^29 evaluations extended to 2^30 on a coset: evaluations 16 GiB, output 32, and 82 of the
    library's, where flat tables and 64-byte factors would take it to 192."""
    import torch
    z, li, lo = fresh, 29, 30
    F, n, m = z.BLS12_381_FR, 1 << li, 1 << lo
    _need(134)
    at = [2, (1 << 27) + 5, n - 3]
    es = [9, P - 1, 1 << 150]
    wi, wo, g = _root(li), _root(lo), 5
    ev = torch.zeros(4 * n, dtype=torch.int64, device="cuda")
    out = torch.empty(4 * m, dtype=torch.int64, device="cuda")
    _put(ev, at, es)
    torch.cuda.synchronize()
    with z.DeviceTwiddles(F, li, z.primitiveRootOfUnity(F, li)) as ti, \
            z.DeviceTwiddles(F, lo, z.primitiveRootOfUnity(F, lo)) as to:
        z.coset_lde_device(ti, to, z.to_montgomery(F, g), ev.data_ptr(), out.data_ptr())
    torch.cuda.synchronize()
    # The polynomial through the evaluations e_i at wi^i, at x = g wo^k (no point of the domain):
    # (x^n - 1) / n * sum e_i wi^i / (x - wi^i).
    ks = _samples(m, 2)
    want = []
    for k in ks:
        x = g * pow(wo, k, P) % P
        s = sum(e * pow(wi, i, P) * pow(x - pow(wi, i, P), -1, P) for i, e in zip(at, es))
        want.append((pow(x, n, P) - 1) * pow(n, -1, P) * s % P)
    assert _get(out, ks) == want


def _fold_inputs(log_n):
    layer = O.random_elements(FID, 300 + log_n, 1 << log_n)
    return layer, O.random_elements(FID, 400 + log_n, 1)[0]


@pytest.mark.parametrize("log_n", [1, 2, 5, 9, 13])
def test_folds_with_a_large_table(fresh, log_n):
    """Folds (alone, and with the commitment of their result) by the table of a 2^30 domain, which
    takes 16 GiB: 32 bytes an entry."""
    import torch
    z, log_table = fresh, 30
    F, half = z.BLS12_381_FR, 1 << (log_n - 1)
    _need(20)
    layer, alpha = _fold_inputs(log_n)
    want = O.fri_fold(FID, layer, log_n, alpha)
    x = torch.from_numpy(layer.view(np.int64).reshape(-1).copy()).cuda()
    y = torch.zeros(4 * half, dtype=torch.int64, device="cuda")
    nodes = torch.zeros(32 * half, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    z.fri_fold(F, x.data_ptr(), log_n, alpha, y.data_ptr(), log_table=log_table)
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < 17 * GIB
    assert np.array_equal(y.cpu().numpy().view(np.uint64).reshape(-1, 4), want)
    if log_n < 2:
        return
    y.zero_()
    torch.cuda.synchronize()
    root = z.fri_fold_commit(F, x.data_ptr(), log_n, alpha, y.data_ptr(), nodes.data_ptr(), log_table=log_table)
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy().view(np.uint64).reshape(-1, 4), want)
    tree = O.fri_commit_layer(FID, want, log_n - 1)
    assert root == bytes(bytearray(np.asarray(tree[1]).view(np.uint8)))
    assert np.array_equal(nodes.cpu().numpy(), np.asarray(tree).view(np.uint8).reshape(-1))


def test_a_fold_and_commitment_of_2p31_fits(fresh):
    """A layer of 2^31 folded and committed: 64 GiB in, 32 out, 32 of nodes and 32 of factors."""
    import torch
    z, log_n = fresh, 31
    F, n = z.BLS12_381_FR, 1 << log_n
    _need(163)
    half = n // 2
    at = _samples(half, 7)
    lo, hi = [3 * i + 1 for i in range(len(at))], [P - 5 * i for i in range(len(at))]
    x = torch.zeros(4 * n, dtype=torch.int64, device="cuda")
    y = torch.empty(4 * half, dtype=torch.int64, device="cuda")
    nodes = torch.empty(32 * half, dtype=torch.uint8, device="cuda")
    _put(x, at, lo)
    _put(x, [j + half for j in at], hi)
    alpha = 1 << 77
    torch.cuda.synchronize()
    root = z.fri_fold_commit(F, x.data_ptr(), log_n, z.to_montgomery(F, alpha), y.data_ptr(), nodes.data_ptr())
    torch.cuda.synchronize()
    g = pow(_root(32), 2, P)
    got = dict(zip(at, _get(y, at)))
    for j, a, b in zip(at, lo, hi):
        assert got[j] == ((a + b) + alpha * (a - b) * pow(g, -j, P)) * pow(2, -1, P) % P, j
    assert root == bytes(bytearray(nodes[32:64].cpu().numpy()))
    # Leaf j hashes values j and j + half / 2; a parent its two children.
    quarter = half // 2
    pair = _get(y, [1, 1 + quarter])
    leaf = O.blake3(b"".join(v.to_bytes(32, "little") for v in pair))
    assert leaf == bytes(bytearray(nodes[32 * (quarter + 1):32 * (quarter + 2)].cpu().numpy()))
    kids = bytes(bytearray(nodes[64:128].cpu().numpy()))
    assert O.blake3(kids) == root

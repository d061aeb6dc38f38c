"""The transforms' fixed-factor products and element moves at their edges (needs a B200):
vectors on 16-byte boundaries only, whole transforms of values at the ends of the range, and
caller tables whose entries sit there too.  Bit-exact against the oracle."""
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


def _edge_elements(fid, n, seed):
    """Values at the ends of the range and with saturated low words, among random ones."""
    p = O.MODULI[fid]
    top = p >> 224
    vals = [p - 1, 0, 1, p - 2, (top << 224) - 1, (p >> 1), (p >> 1) + 1, (1 << 224) - 1, (top - 1 << 224) | ((1 << 224) - 1)]
    a = O.random_elements(fid, seed, n)
    edge = O.from_ints(vals)
    pos = np.random.default_rng(seed).permutation(n)[: max(1, n // 2)]
    a[pos] = edge[np.arange(len(pos)) % len(vals)]
    return a


@pytest.mark.parametrize("log_n", [1, 2, 3, 4, 7, 8, 9, 10, 11, 13, 17, 18, 19])
def test_vectors_on_16_byte_boundaries(z, log_n):
    import torch
    n = 1 << log_n
    for F, fid in _fields(z):
        a = _edge_elements(fid, n, 100 + log_n)
        _, root = O.primitive_root(fid, log_n)
        _, stages = O.precompute_twiddles(fid, log_n, root)
        with z.DeviceTwiddles(F, log_n, z.primitiveRootOfUnity(F, log_n)) as tw:
            for mode, inverse in ((z.FORWARD, False), (z.INVERSE, True)):
                want = a.copy()
                O.ntt_with_twiddles(fid, want, log_n, stages, inverse=inverse)
                for so, do in ((2, 2), (2, 0), (0, 2)):  # offsets in u64 words: 16 bytes past a 256-byte boundary
                    src = torch.zeros(4 * n + 4, dtype=torch.int64, device="cuda")
                    dst = torch.zeros(4 * n + 4, dtype=torch.int64, device="cuda")
                    src[so:so + 4 * n] = torch.from_numpy(a.view(np.int64).reshape(-1)).cuda()
                    torch.cuda.synchronize()
                    z.ntt_device(tw, src.data_ptr() + 8 * so, dst.data_ptr() + 8 * do, mode)
                    torch.cuda.synchronize()
                    got = dst[do:do + 4 * n].cpu().numpy().view(np.uint64).reshape(-1, 4)
                    assert np.array_equal(got, want), (F.name, log_n, mode, so, do)
                    assert not dst[:do].any() and not dst[do + 4 * n:].any()


@pytest.mark.parametrize("log_n", [2, 5, 9, 12])
def test_caller_tables_at_the_ends_of_the_range(z, log_n):
    n = 1 << log_n
    for F, fid in _fields(z):
        table = [_edge_elements(fid, 1 << s, 7 * log_n + s) for s in range(log_n)]
        a = _edge_elements(fid, n, log_n)
        for inverse in (False, True):
            want, got = a.copy(), a.copy()
            O.ntt_with_twiddles(fid, want, log_n, table, inverse=inverse)
            (z.inttWithTwiddles if inverse else z.nttWithTwiddles)(F, got, log_n, table)
            assert np.array_equal(got, want), (F.name, log_n, inverse)


def test_extension_between_misaligned_vectors(z):
    import torch
    F, fid = z.BLS12_381_FR, O.BLS12_381_FR
    li, lo = 9, 11
    a = _edge_elements(fid, 1 << li, 5)
    shift = z.to_montgomery(F, 5)
    want = O.coset_lde(fid, a, li, lo - li, shift)
    src = torch.zeros(4 * (1 << li) + 2, dtype=torch.int64, device="cuda")
    dst = torch.zeros(4 * (1 << lo) + 2, dtype=torch.int64, device="cuda")
    src[2:] = torch.from_numpy(a.view(np.int64).reshape(-1)).cuda()
    torch.cuda.synchronize()
    with z.DeviceTwiddles(F, li, z.primitiveRootOfUnity(F, li)) as ti, \
            z.DeviceTwiddles(F, lo, z.primitiveRootOfUnity(F, lo)) as to:
        job = {"kind": z.JOB_COSET_LDE, "tw": to, "tw_in": ti, "shift": shift, "src": src.data_ptr() + 16,
               "dst": dst.data_ptr() + 16}
        with z.Batch(F, [job]) as b:
            b.run()
            torch.cuda.synchronize()
            b.status()
        assert np.array_equal(dst[2:].cpu().numpy().view(np.uint64).reshape(-1, 4), want.reshape(-1, 4))


@pytest.mark.parametrize("log_n", [1, 7, 8, 9, 15, 16, 17, 20])
def test_captured_transforms_replay(z, log_n):
    """Transforms captured by the caller's CUDA graph (their passes' launches overlap) replay on
    new data with the results of direct calls."""
    import torch
    F, n = z.BN254_FR, 1 << log_n
    stream = torch.cuda.Stream()
    with z.DeviceTwiddles(F, log_n, z.primitiveRootOfUnity(F, log_n)) as tw, torch.cuda.stream(stream):
        src, mid, dst = (torch.zeros(4 * n, dtype=torch.int64, device="cuda") for _ in range(3))

        def both():
            z.ntt_device(tw, src.data_ptr(), mid.data_ptr(), z.FORWARD, stream=stream.cuda_stream)
            z.ntt_device(tw, mid.data_ptr(), dst.data_ptr(), z.INVERSE, stream=stream.cuda_stream)

        both()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            both()
        for seed in (1, 2):
            z.random_elements(F, seed, src.data_ptr(), n, stream=stream.cuda_stream)
            both()
            want = mid.clone()
            mid.zero_()
            dst.zero_()
            graph.replay()
            stream.synchronize()
            assert torch.equal(mid, want) and torch.equal(dst, src)


@pytest.mark.parametrize("log_n", [8, 9, 11])
def test_in_place_without_scratch_can_be_captured(z, log_n):
    """Up to the untuned plan's tile (2^11; 2^12 for the small fields) an in-place transform needs
    no scratch: it neither waits nor allocates, so a caller's graph can hold it."""
    import torch
    z.tune_clear()
    stream = torch.cuda.Stream()
    for F, L in ((z.BN254_FR, log_n), (z.BLS12_381_FR, log_n), (z.GOLDILOCKS, log_n + 1), (z.BABYBEAR, log_n + 1)):
        words = F.limbs << L
        with z.DeviceTwiddles(F, L, z.primitiveRootOfUnity(F, L)) as tw, torch.cuda.stream(stream):
            data = torch.zeros(words, dtype=torch.int64, device="cuda")
            if F.limbs == 4:
                z.random_elements(F, L, data.data_ptr(), 1 << L, stream=stream.cuda_stream)
            else:
                data += torch.randint(0, F.modulus if F.name == "babybear" else 1 << 62, (words,), device="cuda")
            orig, want = data.clone(), torch.zeros_like(data)
            z.ntt_device(tw, data.data_ptr(), want.data_ptr(), z.FORWARD, stream=stream.cuda_stream)
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                z.ntt_device(tw, data.data_ptr(), data.data_ptr(), z.FORWARD, stream=stream.cuda_stream)
            graph.replay()
            stream.synchronize()
            assert torch.equal(data, want), F.name
            z.ntt_device(tw, data.data_ptr(), data.data_ptr(), z.INVERSE, stream=stream.cuda_stream)
            stream.synchronize()
            assert torch.equal(data, orig), F.name

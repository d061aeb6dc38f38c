"""The transform library's workloads as measurable cases.

Each case is one call (or one short sequence of calls) that a program using the
library makes through its Python binding, on inputs drawn from a seed:

  ntt     one transform of device elements: forward, inverse, or both in turn
          (ntt_device), over each field;
  host    one zig-ntt drop-in call on a host array with a precomputed table
          (nttWithTwiddles / inttWithTwiddles), copies included;
  batch   many transforms of uneven sizes and mixed directions in one
          persistent launch (Batch, replayed as a CUDA graph);
  lde     coset extensions of many columns in one persistent launch;
  poly    the product of two device polynomials of any lengths;
  trace   a STARK prover's trace step over a small field: extend every column
          to the coset, then commit the rows of the result;
  fri     a FRI prover's commit phase: per round commit the layer, take the
          challenge from its root, fold.

`listed` holds the sizes of the repository's own benchmark and tests; `draw`
spreads over the ranges that they stand for.
"""
from __future__ import annotations

import hashlib
import importlib.util
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    name = "zig_algebra_b200"
    if name not in sys.modules:
        pkg = os.path.join(ROOT, "zig-algebra_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


z = _package()
FIELD = {F.name: F for F in (*z.FIELDS, *z.SMALL_FIELDS)}
# The coset shift: a multiplicative generator (the first quadratic non-residue
# the reference's root derivation finds for the 256-bit fields).
SHIFT = {"bn254_fr": 5, "bls12_381_fr": 5, "goldilocks": 7, "babybear": 31}

_kept: dict = {}  # what a program keeps for its lifetime: the stream, the tables, the tuned plans


def _stream():
    """The program's CUDA stream; the tuned plans shipped with the library are loaded once."""
    if "stream" not in _kept:
        z.init(torch.cuda.current_device())
        z.tune_load(os.path.join(ROOT, "zig-algebra_b200", "tune", "b200.json"))
        _kept["stream"] = torch.cuda.Stream()
    return _kept["stream"]


def _table(F, log_n):
    key = ("device", F.name, log_n)
    if key not in _kept:
        _kept[key] = z.DeviceTwiddles(F, log_n, z.primitiveRootOfUnity(F, log_n))
    return _kept[key]


def _host_table(F, log_n):
    key = ("host", F.name, log_n)
    if key not in _kept:
        _kept[key] = z.precomputeTwiddles(F, log_n, z.primitiveRootOfUnity(F, log_n))
    return _kept[key]


def _scalar(F, x):
    return z.to_montgomery(F, x) if F.limbs == 4 else np.array([x, 0, 0, 0], dtype=np.uint64)


def _elements(F, count, gen):
    """`count` field elements in the library's layout, uniform below the modulus (for the
    256-bit fields up to the top limb's last value)."""
    dev = gen.device
    if F.limbs == 4:
        x = torch.randint(-(1 << 63), (1 << 63) - 1, (count, 4), dtype=torch.int64, device=dev, generator=gen)
        x[:, 3] = torch.randint(0, F.modulus >> 192, (count,), dtype=torch.int64, device=dev, generator=gen)
        return x.reshape(-1)
    if F.name == "goldilocks":
        hi = torch.randint(0, (1 << 32) - 1, (count,), dtype=torch.int64, device=dev, generator=gen)
        lo = torch.randint(0, 1 << 32, (count,), dtype=torch.int64, device=dev, generator=gen)
        return (hi << 32) | lo
    return torch.randint(0, F.modulus, (count,), dtype=torch.int64, device=dev, generator=gen)


def _buffer(F, count):
    return torch.empty(count * F.limbs, dtype=torch.int64, device="cuda")


# --- the cases -------------------------------------------------------------------------


def listed():
    return [
        # The smallest device call of the benchmark: forward and back, two launches' latency.
        {"name": "bn254_roundtrip_2p12", "op": "ntt", "field": "bn254_fr", "log_n": 12, "mode": "both"},
        # The zig-ntt drop-in call of a host program with a precomputed table.
        {"name": "bn254_host_2p14", "op": "host", "field": "bn254_fr", "log_n": 14, "mode": "inverse"},
        # One large transform with the vector inside L2: a prover's usual circuit size.
        {"name": "bn254_ntt_2p20", "op": "ntt", "field": "bn254_fr", "log_n": 20, "mode": "forward"},
        # The headline: one transform larger than L2.
        {"name": "bn254_ntt_2p24", "op": "ntt", "field": "bn254_fr", "log_n": 24, "mode": "forward"},
        # Interpolation over the other 256-bit field.
        {"name": "bls_intt_2p22", "op": "ntt", "field": "bls12_381_fr", "log_n": 22, "mode": "inverse"},
        # 512 polynomials of 2^10..2^16 and 8 of 2^20, directions mixed, one launch.
        {"name": "bn254_batch_520", "op": "batch", "field": "bn254_fr", "small": 512, "lo": 10, "hi": 16, "large": 8,
         "log_large": 20, "mix": 33},
        # 64 columns extended to four times their length on a coset, one launch.
        {"name": "bls_lde_64x2p18", "op": "lde", "field": "bls12_381_fr", "log_in": 18, "log_out": 20, "columns": 64},
        # A product of two polynomials whose lengths are no power of two.
        {"name": "bn254_poly_ragged", "op": "poly", "field": "bn254_fr", "len_a": 1000003, "len_b": 700001},
        # A trace of 64 columns over a 64-bit field: extension, then the row commitment.
        {"name": "goldilocks_trace_64x2p18", "op": "trace", "field": "goldilocks", "log_in": 18, "log_out": 20,
         "columns": 64},
        # One large transform over a 32-bit field.
        {"name": "babybear_ntt_2p22", "op": "ntt", "field": "babybear", "log_n": 22, "mode": "both"},
        # The commit phase of a FRI proof over a 256-bit field.
        {"name": "bn254_fri_2p22", "op": "fri", "field": "bn254_fr", "log_n": 22, "log_final": 10},
        # The same over a 64-bit field at a small domain: rounds dominated by latency.
        {"name": "goldilocks_fri_2p18", "op": "fri", "field": "goldilocks", "log_n": 18, "log_final": 8},
    ]


def _log_uniform(rng: random.Random, lo, hi):
    """An integer of [lo, hi], uniform over its logarithm."""
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def draw(rng: random.Random):
    op = rng.choice(["ntt", "ntt", "ntt", "host", "batch", "lde", "poly", "trace", "fri"])
    wide = rng.choice(["bn254_fr", "bls12_381_fr"])
    small = rng.choice(["goldilocks", "babybear"])
    either = rng.choice([wide, wide, small])
    mode = rng.choice(["forward", "inverse"])
    if op == "ntt":
        return {"op": op, "field": either, "log_n": rng.randint(10, 24), "mode": mode}
    if op == "host":
        return {"op": op, "field": either, "log_n": rng.randint(8, 17), "mode": mode}
    if op == "batch":
        lo = rng.randint(10, 13)
        return {"op": op, "field": wide, "small": _log_uniform(rng, 8, 512), "lo": lo, "hi": rng.randint(lo, 16),
                "large": rng.randint(0, 8), "log_large": rng.randint(17, 20), "mix": rng.randrange(1 << 16)}
    if op == "lde":
        log_in = rng.randint(10, 18)
        return {"op": op, "field": wide, "log_in": log_in, "log_out": log_in + rng.randint(1, 2),
                "columns": _log_uniform(rng, 1, 48)}
    if op == "poly":
        return {"op": op, "field": wide, "len_a": _log_uniform(rng, 16, 1 << 21), "len_b": _log_uniform(rng, 16, 1 << 21)}
    if op == "trace":
        log_in = rng.randint(10, 18)
        return {"op": op, "field": small, "log_in": log_in, "log_out": log_in + rng.randint(1, 3),
                "columns": rng.randint(1, 64)}
    log_n = rng.randint(12, 22)
    return {"op": op, "field": rng.choice([wide, small]), "log_n": log_n, "log_final": rng.randint(3, 10)}


def _batch_jobs(case):
    """(log2 size, mode) of each job of a batch case, from its own number."""
    r = np.random.default_rng(case["mix"])
    logs = [int(v) for v in r.integers(case["lo"], case["hi"] + 1, case["small"])] + [case["log_large"]] * case["large"]
    return [(L, z.INVERSE if v < 0.5 else z.FORWARD) for L, v in zip(logs, r.random(len(logs)))]


class _BatchOwner:
    """Closes a batch with the state that holds it."""

    def __init__(self, batch):
        self.batch = batch

    def __del__(self):
        torch.cuda.synchronize()
        self.batch.close()


def prepare(case, seed):
    F = FIELD[case["field"]]
    stream = _stream()
    with torch.cuda.stream(stream):
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        state = _PREPARE[case["op"]](case, F, gen)
    stream.synchronize()
    state["op"], state["field"], state["stream"] = case["op"], F, stream.cuda_stream
    return state


def _prepare_ntt(case, F, gen):
    n = 1 << case["log_n"]
    state = {"mode": case["mode"], "tw": _table(F, case["log_n"]), "src": _elements(F, n, gen), "dst": _buffer(F, n)}
    if case["mode"] == "both":
        state["back"] = _buffer(F, n)
    return state


def _prepare_host(case, F, gen):
    x = _elements(F, 1 << case["log_n"], gen).cpu().numpy().view(np.uint64)
    return {"mode": case["mode"], "log_n": case["log_n"], "tw": _host_table(F, case["log_n"]),
            "data": x.reshape(-1, 4) if F.limbs == 4 else x}


def _prepare_batch(case, F, gen):
    plan = _batch_jobs(case)
    total = sum(1 << L for L, _ in plan)
    src, dst = _elements(F, total, gen), _buffer(F, total)
    jobs, off = [], 0
    for L, mode in plan:
        jobs.append({"kind": z.JOB_NTT, "tw": _table(F, L), "mode": mode, "src": src.data_ptr() + off,
                     "dst": dst.data_ptr() + off})
        off += 32 << L
    return {"src": src, "dst": dst, "batch": _BatchOwner(z.Batch(F, jobs))}


def _prepare_lde(case, F, gen):
    m, li, lo = case["columns"], case["log_in"], case["log_out"]
    src, dst = _elements(F, m << li, gen), _buffer(F, m << lo)
    shift = _scalar(F, SHIFT[F.name])
    jobs = [{"kind": z.JOB_COSET_LDE, "tw": _table(F, lo), "tw_in": _table(F, li), "shift": shift,
             "src": src.data_ptr() + i * (32 << li), "dst": dst.data_ptr() + i * (32 << lo)} for i in range(m)]
    return {"src": src, "dst": dst, "batch": _BatchOwner(z.Batch(F, jobs))}


def _prepare_poly(case, F, gen):
    la, lb = case["len_a"], case["len_b"]
    return {"tw": _table(F, (la + lb - 2).bit_length()), "a": _elements(F, la, gen), "len_a": la,
            "b": _elements(F, lb, gen), "len_b": lb, "dst": _buffer(F, la + lb - 1)}


def _prepare_trace(case, F, gen):
    m, li, lo = case["columns"], case["log_in"], case["log_out"]
    src, dst = _elements(F, m << li, gen), _buffer(F, m << lo)
    return {"tw_in": _table(F, li), "tw_out": _table(F, lo), "shift": _scalar(F, SHIFT[F.name]), "log_out": lo,
            "src": src, "dst": dst, "nodes": torch.zeros(8 << lo, dtype=torch.int64, device="cuda"),
            "ins": [src.data_ptr() + i * (8 << li) for i in range(m)],
            "outs": [dst.data_ptr() + i * (8 << lo) for i in range(m)]}


def _prepare_fri(case, F, gen):
    log_n, log_final = case["log_n"], case["log_final"]
    rounds = log_n - log_final
    layers = [_elements(F, 1 << log_n, gen)] + [_buffer(F, 1 << (log_n - r)) for r in range(1, rounds + 1)]
    nodes = [torch.zeros(4 << (log_n - r), dtype=torch.int64, device="cuda") for r in range(rounds)]
    return {"log_n": log_n, "log_final": log_final, "layers": layers, "nodes": nodes}


_PREPARE = {"ntt": _prepare_ntt, "host": _prepare_host, "batch": _prepare_batch, "lde": _prepare_lde,
            "poly": _prepare_poly, "trace": _prepare_trace, "fri": _prepare_fri}


def _digest(root: bytes):
    return np.frombuffer(root, dtype=np.uint8)


def run(state):
    F, st, op = state["field"], state["stream"], state["op"]
    if op == "ntt":
        src, dst = state["src"], state["dst"]
        if state["mode"] == "both":
            z.ntt_device(state["tw"], src.data_ptr(), dst.data_ptr(), z.FORWARD, stream=st)
            z.ntt_device(state["tw"], dst.data_ptr(), state["back"].data_ptr(), z.INVERSE, stream=st)
            return {"forward": dst, "back": state["back"]}
        z.ntt_device(state["tw"], src.data_ptr(), dst.data_ptr(),
                     z.INVERSE if state["mode"] == "inverse" else z.FORWARD, stream=st)
        return dst
    if op == "host":
        data = state["data"].copy()  # the call works in place; the program keeps its input
        (z.inttWithTwiddles if state["mode"] == "inverse" else z.nttWithTwiddles)(F, data, state["log_n"], state["tw"])
        return data.view(np.int64)
    if op in ("batch", "lde"):
        state["batch"].batch.run(stream=st, graph=True)
        return state["dst"]
    if op == "poly":
        z.poly_mul_device(state["tw"], state["a"].data_ptr(), state["len_a"], state["b"].data_ptr(), state["len_b"],
                          state["dst"].data_ptr(), stream=st)
        return state["dst"]
    if op == "trace":
        z.coset_lde_columns(state["tw_in"], state["tw_out"], state["shift"], state["ins"], state["outs"], stream=st)
        root = z.merkle_commit_rows(F, state["outs"], state["log_out"], state["nodes"].data_ptr(), stream=st)
        return {"columns": state["dst"], "nodes": state["nodes"], "root": _digest(root)}

    def challenge(_round, root):  # the caller's transcript, reduced to one hash
        return _scalar(F, int.from_bytes(hashlib.blake2s(root).digest(), "little") % F.modulus)

    roots = z.fri_commit_phase(F, state["log_n"], state["log_final"], [t.data_ptr() for t in state["layers"]],
                               [t.data_ptr() for t in state["nodes"]], challenge, stream=st)
    return {"layers": state["layers"][1:], "nodes": state["nodes"], "roots": _digest(b"".join(roots))}


# --- what a pass cannot do without --------------------------------------------------------


def work(case):
    """Bytes: every input read once and every output written once.  Flops: field operations
    (a butterfly is one product and two sums) and hash compressions, one each."""
    F = FIELD[case["field"]]
    size, op = 8 * F.limbs, case["op"]
    ntt = lambda L: 3 * L << L >> 1  # noqa: E731 -- field operations of one transform
    if op in ("ntt", "host"):
        times = 2 if case["mode"] == "both" else 1
        return {"bytes": (times + 1 if op == "ntt" else 2) * size << case["log_n"], "flops": times * ntt(case["log_n"])}
    if op == "batch":
        jobs = _batch_jobs(case)
        return {"bytes": sum(2 * size << L for L, _ in jobs), "flops": sum(ntt(L) for L, _ in jobs)}
    if op in ("lde", "trace"):
        m, li, lo = case["columns"], case["log_in"], case["log_out"]
        flops = m * (ntt(li) + ntt(lo) + (2 << li))
        moved = m * size * ((1 << li) + (1 << lo))
        if op == "trace":
            blocks = -(-m * z._num_bytes(F) // 64)
            flops += (blocks + 1) << lo
            moved += 64 << lo
        return {"bytes": moved, "flops": flops}
    if op == "poly":
        n = case["len_a"] + case["len_b"] - 1
        L = (n - 1).bit_length()
        return {"bytes": size * 2 * n, "flops": 3 * ntt(L) + (2 << L)}
    rounds = case["log_n"] - case["log_final"]
    halves = sum(1 << (case["log_n"] - r - 1) for r in range(rounds))  # folded values, and leaves, of all rounds
    return {"bytes": (size << case["log_n"]) + size * halves + 64 * halves, "flops": 7 * halves}


# --- the same results from plain integers ---------------------------------------------------


def _root_of_unity(p, two_adicity, log_n):
    """z^((p-1)/2^log_n) with z the first quadratic non-residue from 2 on."""
    q = 2
    while pow(q, (p - 1) // 2, p) != p - 1:
        q += 1
    return pow(q, (p - 1) >> log_n, p)


def _transform(values, p, root):
    """sum_j x_j root^(jk) by radix-2 decimation in time on an array of Python integers."""
    n = len(values)
    if n == 1:
        return values
    even, odd = _transform(values[0::2], p, root * root % p), _transform(values[1::2], p, root * root % p)
    w = np.empty(n // 2, dtype=object)
    acc = 1
    for i in range(n // 2):
        w[i] = acc
        acc = acc * root % p
    t = odd * w % p
    return np.concatenate([(even + t) % p, (even - t) % p])


def _ints(F, words):
    w = words.reshape(-1, F.limbs).astype(object)
    return sum(w[:, k] << (64 * k) for k in range(F.limbs))


def _words(F, values):
    out = np.empty((len(values), F.limbs), dtype=np.uint64)
    for k in range(F.limbs):
        out[:, k] = np.array([int(v) >> (64 * k) & 0xFFFFFFFFFFFFFFFF for v in values], dtype=np.uint64)
    return torch.from_numpy(out.reshape(-1).view(np.int64))


def exact(case, seed):
    """The transforms and the polynomial products of up to 2^14 points in integers.  Elements of
    the 256-bit fields are Montgomery limbs, and a transform is linear: it acts on the limbs'
    value as on the element.  The other cases are whole numbers through and through."""
    F = FIELD[case["field"]]
    p = F.modulus
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["op"] in ("ntt", "host") and case["log_n"] <= 14:
        n = 1 << case["log_n"]
        x = _ints(F, _elements(F, n, gen).cpu().numpy().view(np.uint64))
        w = _root_of_unity(p, F.two_adicity, case["log_n"])
        if case["mode"] == "both":
            return {"forward": _words(F, _transform(x, p, w)), "back": _words(F, x)}
        if case["mode"] == "forward":
            y = _transform(x, p, w)
        else:
            y = _transform(x, p, pow(w, -1, p)) * pow(n, -1, p) % p
        y = _words(F, y)
        return y.reshape(-1, 4) if case["op"] == "host" and F.limbs == 4 else y
    if case["op"] == "poly" and case["len_a"] + case["len_b"] <= 1 << 14:
        a = _ints(F, _elements(F, case["len_a"], gen).cpu().numpy().view(np.uint64))
        b = _ints(F, _elements(F, case["len_b"], gen).cpu().numpy().view(np.uint64))
        # Kronecker substitution: coefficient sums stay below 2^(2*256 + 14).
        width = 72
        pack = lambda v: int.from_bytes(b"".join(int(c).to_bytes(width, "little") for c in v), "little")  # noqa: E731
        n = len(a) + len(b) - 1
        prod = (pack(a) * pack(b)).to_bytes(width * (n + 1), "little")
        rinv = pow(1 << 256, -1, p)  # two factors in Montgomery form carry one factor 2^256 too many
        return _words(F, [int.from_bytes(prod[width * i:width * (i + 1)], "little") * rinv % p for i in range(n)])
    return None

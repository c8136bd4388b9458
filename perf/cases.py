"""Performance cases of the squaring engine: what users of the package run, through its public API.

A PRP or LL test is a long run of squarings mod 2^E - 1 (Plan.squareLoop, one Gerbicz block of up to
1,000 at a time), with a modMul per block, expMul for proofs, word buffers written and read at
savefile points, and batches of small exponents side by side. Sizes follow the repository's own
workloads: 256K words (E about 5 million), 8M (E = 136,181,029), 20M (E = 331,480,451), batches of
exponents in [1M, 20M], and the FFT lengths in between that double checks fall on.

Residues are uniform E-bit values, as they are after the first few dozen squarings of any test.
"""
import math

import numpy as np
import torch

import gpuowl_b200 as owl

# exponent range that the FFT lengths 64K to 20M words serve
E_MIN, E_MAX = 1_000_003, 335_000_001
# squarings of one call: a Gerbicz block
N_MAX = 1000
# the most floating-point work of one pass (below that of the largest listed case)
FLOPS_MAX = 2.0e11


def listed():
    return [
        # one product of two residues at the 256K length: the Gerbicz update of a small test
        {"name": "modmul_256k", "kind": "modmul", "E": 4_989_349},
        # a savefile point of a wavefront test: words to the device and back, host buffers
        {"name": "checkpoint_8m", "kind": "checkpoint", "E": 136_181_029},
        # the PRP driver from the start through its first blocks and Gerbicz check, plan included
        {"name": "prp_driver_64k", "kind": "prp", "E": 1_257_787, "n": 10_000},
        # a Gerbicz block at the 256K length
        {"name": "square_256k", "kind": "square", "E": 4_989_349, "n": 1000, "ll": False, "roe": False, "split": 0},
        # LL at the 1M length
        {"name": "ll_1m", "kind": "square", "E": 19_100_017, "n": 500, "ll": True, "roe": False, "split": 0},
        # 5 * 2^19 words, round-off measured (the sampled squarings of a run)
        {"name": "square_2560k", "kind": "square", "E": 45_600_013, "n": 400, "ll": False, "roe": True, "split": 0},
        # LL double check at the 4M length
        {"name": "ll_4m", "kind": "square", "E": 73_900_031, "n": 250, "ll": True, "roe": False, "split": 0},
        # a wavefront PRP test at the 8M length
        {"name": "square_8m", "kind": "square", "E": 136_181_029, "n": 200, "ll": False, "roe": False, "split": 0},
        # the same test in the split-precision (tensor-core) form of the column pass
        {"name": "split_8m", "kind": "square", "E": 136_181_029, "n": 100, "ll": False, "roe": False, "split": 1},
        # a 100-million-digit PRP test at the 20M length
        {"name": "square_20m", "kind": "square", "E": 331_480_451, "n": 60, "ll": False, "roe": False, "split": 0},
        # a proof step: a 64-bit power times a second residue
        {"name": "expmul_5m", "kind": "expmul", "E": 89_300_021, "h_seed": 11},
        # many small exponents of uneven lengths as one batch
        {"name": "batch_24", "kind": "batch", "count": 24, "E_lo": 1_000_003, "E_hi": 20_000_003, "spread": 3, "n": 150},
    ]


def _log_odd(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | 1


def draw(rng):
    kind = rng.choice(["square"] * 6 + ["split", "modmul", "expmul", "checkpoint", "batch", "prp"])
    if kind == "prp":
        return {"kind": "prp", "E": _log_odd(rng, E_MIN, 4_000_000), "n": 1000 * rng.randint(2, 8)}
    if kind == "batch":
        lo = _log_odd(rng, E_MIN, 4_000_000)
        return {"kind": "batch", "count": rng.randint(5, 24), "E_lo": lo, "E_hi": _log_odd(rng, 4 * lo, 20_000_003),
                "spread": rng.randint(0, 1 << 20), "n": rng.randint(20, 130)}
    if kind == "split":
        # the FFT lengths whose columns have a split-precision form: 2^22 to 2^23 and 5 * 2^21, 5 * 2^22 words
        lo, hi = rng.choice([(60_000_001, 75_000_001), (100_000_001, 147_000_001), (310_000_001, 335_000_001)])
        c = {"kind": "square", "E": _log_odd(rng, lo, hi), "n": rng.randint(10, 40), "ll": rng.random() < 0.3,
             "roe": rng.random() < 0.3, "split": 1}
        return c
    E = _log_odd(rng, E_MIN, E_MAX)
    if kind in ("modmul", "checkpoint"):
        return {"kind": kind, "E": E}
    if kind == "expmul":
        return {"kind": "expmul", "E": _log_odd(rng, E_MIN, 100_000_001), "h_seed": rng.randint(0, 1 << 20)}
    words = owl.fft_choose(E)[0]
    most = max(2, min(N_MAX, int(FLOPS_MAX / _square_flops(words))))
    n = most if rng.random() < 0.6 else max(1, int(math.exp(rng.uniform(0.0, math.log(most)))))
    return {"kind": "square", "E": E, "n": n, "ll": rng.random() < 0.3, "roe": rng.random() < 0.3, "split": 0}


def _words(E, seed, salt):
    """A uniform E-bit residue as compact 32-bit words."""
    g = np.random.Generator(np.random.PCG64([int(seed) & 0xFFFFFFFF, salt, E]))
    w = g.integers(0, 1 << 32, size=owl.n_words(E), dtype=np.uint32)
    w[-1] &= np.uint32((1 << (E % 32)) - 1)
    return w


def _power(case):
    g = np.random.Generator(np.random.PCG64([case["h_seed"], 64]))
    return int(g.integers(0, 1 << 63)) | (1 << 63)


def _batch_exponents(case):
    """The batch's exponents: log-uniform in [E_lo, E_hi], fixed by the case."""
    g = np.random.Generator(np.random.PCG64([case["spread"], case["count"]]))
    u = g.uniform(math.log(case["E_lo"]), math.log(case["E_hi"]), size=case["count"])
    return [int(math.exp(x)) | 1 for x in u]


class _Digits:
    """A plan's word buffer as a torch tensor (no copy); keeps the plan alive."""

    def __init__(self, plan, buf):
        self.plan = plan
        self.__cuda_array_interface__ = {"shape": (plan.N,), "typestr": "<i4", "data": (buf, False), "version": 3}

    def tensor(self):
        return torch.as_tensor(self, device="cuda")


def _buffer(plan, words=None):
    buf = plan.alloc()
    if words is not None:
        plan.writeIn(buf, words)
    return buf


def prepare(case, seed):
    kind = case["kind"]
    if kind == "prp":
        # the driver makes its own plan; the seed moves the exponent within its FFT length
        g = np.random.Generator(np.random.PCG64([int(seed) & 0xFFFFFFFF, case["E"]]))
        return {"kind": kind, "E": case["E"] + 2 * int(g.integers(0, 1000)), "n": case["n"]}
    if kind == "batch":
        plans = [owl.Plan(E) for E in _batch_exponents(case)]
        bufs = [_buffer(p, _words(p.E, seed, i)) for i, p in enumerate(plans)]
        return {"kind": kind, "n": case["n"], "plans": plans, "bufs": bufs, "batch": owl.Batch(plans),
                "out": [_Digits(p, b).tensor() for p, b in zip(plans, bufs)]}
    E = case["E"]
    plan = owl.Plan(E, split=case.get("split", 0))
    s = {"kind": kind, "plan": plan}
    if kind == "checkpoint":
        s["words"] = _words(E, seed, 0)
        s["buf"] = _buffer(plan)
        s["out"] = _Digits(plan, s["buf"]).tensor()
        return s
    s["a"] = _buffer(plan, _words(E, seed, 0))
    s["work"] = _buffer(plan)
    s["out"] = _Digits(plan, s["work"]).tensor()
    if kind == "square":
        s["args"] = {"n": case["n"], "ll": case["ll"], "roe": case["roe"]}
    else:
        s["b"] = _buffer(plan, _words(E, seed, 1))
        s["h"] = _power(case) if kind == "expmul" else 0
    return s


def run(state):
    kind = state["kind"]
    if kind == "prp":
        r = owl.prp_run(state["E"], block=1000, log_step=5000, stop_after=state["n"])
        # the residues that the driver logs, with their iterations
        return {"checkpoints": np.array(r["checkpoints"], dtype=np.uint64).view(np.uint32), "n_errors": r["n_errors"]}
    if kind == "batch":
        # in place: each pass goes on from the last one
        state["batch"].square(state["bufs"], state["n"], roe=False)
        return state["out"]
    plan = state["plan"]
    if kind == "square":
        plan.squareLoop(state["work"], state["a"], **state["args"])
        return state["out"]
    if kind == "checkpoint":
        plan.writeIn(state["buf"], state["words"])
        return {"digits": state["out"], "words": plan.readOut(state["buf"])}
    plan.copy(state["work"], state["a"])
    if kind == "modmul":
        plan.modMul(state["work"], state["b"])
    else:
        plan.expMul(state["work"], state["h"], state["b"])
    return state["out"]


def _square_flops(n):
    """One squaring of n words: a complex FFT of n/2 points each way, and about 20 operations a word
    for the two weightings, the pair squaring, the rounding and the carry."""
    return 5.0 * n * math.log2(n / 2) + 20.0 * n


def work(case):
    """Bytes: the n 32-bit words of each residue read once and written once per call. Flops: the FFTs'."""
    kind = case["kind"]
    if kind == "batch":
        sizes = [owl.fft_choose(E)[0] for E in _batch_exponents(case)]
        return {"bytes": sum(8.0 * n for n in sizes), "flops": sum(_square_flops(n) for n in sizes) * case["n"]}
    n = owl.fft_choose(case["E"])[0]
    if kind == "prp":
        # from 3 to a 64-bit residue
        return {"bytes": 16.0, "flops": _square_flops(n) * case["n"]}
    if kind == "checkpoint":
        # compact words in and out, digits written and read
        return {"bytes": 2 * case["E"] / 8.0 + 8.0 * n, "flops": 0.0}
    if kind == "modmul":
        return {"bytes": 12.0 * n, "flops": 1.5 * _square_flops(n)}
    if kind == "expmul":
        h = _power(case)
        return {"bytes": 12.0 * n, "flops": _square_flops(n) * (h.bit_length() + bin(h).count("1"))}
    return {"bytes": 8.0 * n, "flops": _square_flops(n) * case["n"]}


def _balanced(value, E):
    """The balanced digits of value mod 2^E - 1 at the default FFT length: word k holds bits
    [ceil(k E / n), ceil((k + 1) E / n)) and lies in [-2^(b-1), 2^(b-1))."""
    n = owl.fft_choose(E)[0]
    at = (np.arange(n + 1, dtype=np.int64) * E + n - 1) // n
    raw = np.frombuffer(value.to_bytes(E // 8 + 9, "little"), dtype=np.uint8).astype(np.int64)
    first = at[:-1] // 8
    v = sum(raw[np.minimum(first + i, raw.size - 1)] << (8 * i) for i in range(5)) >> (at[:-1] % 8)
    bits = np.diff(at)
    d = (v & ((1 << bits) - 1)).tolist()
    half = (1 << (bits - 1)).tolist()
    c = 0
    for k in list(range(n)) + list(range(n)):  # the second round takes the carry out of the top word
        x = d[k] + c
        c = 0
        if x >= half[k]:
            x -= 2 * half[k]
            c = 1
        d[k] = x
    return np.array(d, dtype=np.int32)


def exact(case, seed):
    """Whole numbers: the product by Python's integers where that is quick."""
    if case["kind"] == "checkpoint":
        return {"digits": None, "words": _words(case["E"], seed, 0)}
    if case["kind"] != "modmul" or case["E"] > 6_000_000:
        return None
    E = case["E"]
    a, b = (int.from_bytes(_words(E, seed, i).tobytes(), "little") for i in (0, 1))
    m = (1 << E) - 1
    p = a * b
    p = (p & m) + (p >> E)
    p = (p & m) + (p >> E)
    return _balanced(p, E)

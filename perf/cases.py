"""The work this library is measured on: what programs have it do, through its
public entry points.

Transforms of one size (the reference programs' sizes 2^4..2^10 and the large
ones of the batch workloads), one call at a time and in uniform batches; the
mixed-size batch of the persistent kernel, forward and inverse; a polynomial
product; the vector ops; a modulus without the pseudo-Mersenne form; and the
host-buffer call of a drop-in user.  Buffers are device tensors unless the
case says otherwise, elements are 16-byte residues.
"""
from __future__ import annotations

import numpy as np
import torch

import benchntt_b200 as bn

DEVICE = 0
KIND_FORWARD, KIND_INVERSE, KIND_POLYMUL = "forward", "inverse", "polymul"
KIND_BATCH, KIND_BATCH_INVERSE = "batch", "batch_inverse"
KIND_BLAS, KIND_HOST = "blas", "host_forward"

# A 124-bit prime that is not 2^124 - k for a small k: takes the general
# multiply (whose reference Barrett reduction is exact for it).
Q_GENERAL = 0xB504F333F9DE6484597D89B3754ABE9
AXPY_X = (208488538572646751 << 64) | 12808410693871070164   # the reference drivers' scalar

MAX_BUTTERFLIES = 1024 * (1 << 15) * 16      # the largest listed case
MAX_VECTOR = 1 << 24

_CTX = None


def context() -> bn.Context:
    """One context (device, stream) for the program, as a user keeps it."""
    global _CTX
    if _CTX is None:
        _CTX = bn.Context(DEVICE)
    return _CTX


def listed() -> list[dict]:
    return [
        # one transform per call, the reference programs' unit of work: launch latency
        {"name": "ntt_1024_x1", "kind": KIND_FORWARD, "log2n": 10, "count": 1, "prime": "reference", "layout": 0},
        # a uniform batch of the smallest reference size: little work per element
        {"name": "ntt_16_x65536", "kind": KIND_FORWARD, "log2n": 4, "count": 65536, "prime": "reference", "layout": 0},
        # a uniform batch of the largest reference size
        {"name": "ntt_1024_x65536", "kind": KIND_FORWARD, "log2n": 10, "count": 65536, "prime": "reference", "layout": 0},
        # transforms above one tile, a few at a time: two passes that do not fill the device evenly
        {"name": "ntt_8192_x37", "kind": KIND_FORWARD, "log2n": 13, "count": 37, "prime": "friendly", "layout": 0},
        # the largest uniform batch: 2^26 elements through two passes over HBM
        {"name": "ntt_65536_x1024", "kind": KIND_FORWARD, "log2n": 16, "count": 1024, "prime": "reference", "layout": 0},
        # a * b mod (x^N + 1) for RLWE-sized rings: forward, fused forward-and-multiply, inverse (native u128 layout)
        {"name": "polymul_4096_x2048", "kind": KIND_POLYMUL, "log2n": 12, "count": 2048, "prime": "friendly", "layout": 1},
        # the mixed-size batch: 100,000 of 2^4..2^10 with 64 of 2^16 and 4 of 2^20 among them, one launch
        {"name": "batch_uneven", "kind": KIND_BATCH, "small": 100000, "lo": 4, "hi": 10, "large_16": 64, "large_20": 4,
         "prime": "reference", "layout": 0, "shape_seed": 4},
        # the inverse of a ragged list over the whole range of small sizes, with a few large ones
        {"name": "batch_inverse_ragged", "kind": KIND_BATCH_INVERSE, "small": 30001, "lo": 1, "hi": 12, "large_16": 7,
         "large_20": 1, "prime": "friendly", "layout": 0, "shape_seed": 9},
        # the vector op with the most arithmetic at the benchmark's length
        {"name": "axpy_16777216", "kind": KIND_BLAS, "op": "axpy", "length": 1 << 24, "layout": 0},
        # a short vector of odd length, cache-resident
        {"name": "vvmul_100003", "kind": KIND_BLAS, "op": "vvmul", "length": 100003, "layout": 1},
        # ntt() takes its modulus at run time: a prime with no special form
        {"name": "general_1024_x8192", "kind": KIND_FORWARD, "log2n": 10, "count": 8192, "prime": "general", "layout": 0},
        # the drop-in call shape: host arrays in, host arrays out
        {"name": "host_1024_x4096", "kind": KIND_HOST, "log2n": 10, "count": 4096, "prime": "reference", "layout": 0},
    ]


def _log_uniform(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng) -> dict:
    kind = rng.choice([KIND_FORWARD] * 4 + [KIND_INVERSE] * 2 + [KIND_POLYMUL, KIND_BATCH, KIND_BATCH_INVERSE, KIND_BLAS,
                                                                KIND_BLAS, KIND_HOST])
    layout = rng.choice([0, 0, 1])
    if kind == KIND_BLAS:
        return {"kind": kind, "op": rng.choice(["vvadd", "vvsub", "vvmul", "axpy"]),
                "length": _log_uniform(rng, 1000, MAX_VECTOR), "layout": layout}
    if kind in (KIND_BATCH, KIND_BATCH_INVERSE):
        lo = rng.randint(1, 4)
        return {"kind": kind, "small": _log_uniform(rng, 300, 100000), "lo": lo, "hi": rng.randint(lo + 3, 10),
                "large_16": rng.randint(0, 64), "large_20": rng.randint(0, 4),
                "prime": rng.choice(["reference", "friendly"]), "layout": layout, "shape_seed": rng.randint(1, 1 << 30)}
    prime = rng.choice(["reference", "friendly"])
    if kind == KIND_FORWARD and rng.random() < 0.2:
        prime = "general"
    log2n = rng.randint(3, 20) if kind in (KIND_FORWARD, KIND_INVERSE) else rng.randint(8, 16)
    per = (1 << (log2n - 1)) * log2n
    limit = MAX_BUTTERFLIES // per
    if prime == "general" or kind == KIND_POLYMUL:
        limit //= 8
    if kind == KIND_HOST:
        limit //= 16
    limit = min(limit, (1 << 26) >> log2n)
    return {"kind": kind, "log2n": log2n, "count": _log_uniform(rng, 1, max(1, limit)),
            "prime": "friendly" if kind == KIND_POLYMUL else prime, "layout": layout}


# ------------------------------------------------------------------ helpers
_FRIENDLY = None


def _modulus(prime: str) -> tuple[int, int]:
    global _FRIENDLY
    if prime == "reference":
        return bn.Q_NTT, bn.MU_NTT
    if prime == "general":
        return Q_GENERAL, (1 << 251) // Q_GENERAL
    if _FRIENDLY is None:
        _FRIENDLY = bn.ntt_prime(21)
    return _FRIENDLY


def _residues(count: int, q: int, layout: int, gen: torch.Generator) -> torch.Tensor:
    """Uniform residues: the high word below q's, the low word any."""
    dev = gen.device
    hi = torch.randint(0, q >> 64, (count,), dtype=torch.int64, device=dev, generator=gen)
    lo = torch.randint(-(1 << 63), (1 << 63) - 1, (count,), dtype=torch.int64, device=dev, generator=gen)
    return torch.stack((hi, lo) if layout == bn.LAYOUT_HILO else (lo, hi), dim=1)


def _gen(seed: int, device: str = "cuda") -> torch.Generator:
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return g


def _psi(q: int, mu: int, log2n: int) -> int:
    """A primitive 2N-th root of unity."""
    return bn.powmod(q, mu, bn.root_of_unity(q, mu, 21), 1 << (21 - log2n - 1))


def _table(case: dict, log2n: int, seed: int) -> np.ndarray:
    """Twiddles as the caller has them: the root powers of the friendly prime,
    else table data without structure (the reference's data files)."""
    q, mu = _modulus(case["prime"])
    if case["prime"] == "friendly":
        return bn.twiddles_negacyclic(q, mu, log2n, _psi(q, mu, log2n), case["layout"])
    t = _residues(1 << log2n, q, case["layout"], _gen(seed * 64 + log2n, "cpu"))
    return t.numpy().view(np.uint64)


def _plan(case: dict, log2n: int, seed: int) -> bn.Plan:
    q, mu = _modulus(case["prime"])
    if case["prime"] == "friendly":
        return bn.Plan.negacyclic(context(), log2n, q, mu, _psi(q, mu, log2n), case["layout"])
    return bn.Plan(context(), log2n, q, mu, _table(case, log2n, seed), case["layout"])


def _batch_logns(case: dict) -> np.ndarray:
    rng = np.random.default_rng(case["shape_seed"])
    small = rng.integers(case["lo"], case["hi"] + 1, size=case["small"])
    logns = np.concatenate([small, np.full(case["large_16"], 16), np.full(case["large_20"], 20)]).astype(np.int64)
    rng.shuffle(logns)
    return logns


# ------------------------------------------------------------ the interface
def prepare(case: dict, seed: int) -> dict:
    kind, layout = case["kind"], case["layout"]
    gen = _gen(seed)
    if kind == KIND_BLAS:
        n = case["length"]
        a, b = (_residues(n, bn.Q_BLAS, layout, gen) for _ in range(2))
        state = {"a": a, "b": b, "c": torch.empty_like(a)}
    elif kind in (KIND_BATCH, KIND_BATCH_INVERSE):
        logns = _batch_logns(case)
        lens = np.left_shift(1, logns)
        offs = (np.cumsum(lens) - lens) * 16
        sizes = sorted(set(int(v) for v in logns))
        plan_of = {n: i for i, n in enumerate(sizes)}
        x = _residues(int(lens.sum()), _modulus(case["prime"])[0], layout, gen)
        y = torch.empty_like(x)
        engine = bn.Batch(context(), [_plan(case, n, seed) for n in sizes])
        jobs = bn.Batch.jobs((x.data_ptr() + offs).tolist(), (y.data_ptr() + offs).tolist(),
                             [plan_of[int(n)] for n in logns])
        state = {"x": x, "y": y, "engine": engine, "jobs": jobs}
    else:
        log2n, count = case["log2n"], case["count"]
        q = _modulus(case["prime"])[0]
        plan = _plan(case, log2n, seed)
        x = _residues(count << log2n, q, layout, gen)
        state = {"plan": plan, "x": x, "y": torch.empty_like(x), "count": count}
        if kind == KIND_POLYMUL:
            state["b"] = _residues(count << log2n, q, layout, gen)
            state["bh"] = torch.empty_like(x)
        if kind == KIND_HOST:
            state["x"] = x.cpu().pin_memory().numpy().view(np.uint64)
            state["y"] = torch.empty(x.shape, dtype=torch.int64, pin_memory=True).numpy().view(np.uint64)
    state["case"] = case
    torch.cuda.synchronize()
    return state


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == KIND_BLAS:
        bn.blas(context(), case["op"], state["c"], state["a"], state["b"], bn.Q_BLAS, bn.MU_BLAS, AXPY_X, case["layout"])
        return state["c"]
    if kind == KIND_BATCH:
        state["engine"].run_dev(state["jobs"])
        return state["y"]
    if kind == KIND_BATCH_INVERSE:
        state["engine"].run_inverse_dev(state["jobs"])
        return state["y"]
    plan, x, y, count = state["plan"], state["x"], state["y"], state["count"]
    if kind == KIND_INVERSE:
        plan.inverse(y, x, count)
    elif kind == KIND_POLYMUL:
        plan.forward(state["bh"], state["b"], count)
        plan.forward_mul(y, x, state["bh"], True, count)
        plan.inverse(y, y, count)
    else:
        plan.forward(y, x, count)
    return y.view(np.int64) if kind == KIND_HOST else y


def work(case: dict) -> dict:
    """Each input and output element once (16 bytes; tables once), and the
    multiply-adds of the arithmetic: 21 32-bit ones for a product reduced mod
    a pseudo-Mersenne q (16 + 4 + 1), 48 for a general one (three 128-bit
    products); an addition or subtraction mod q as 4."""
    kind = case["kind"]
    if kind == KIND_BLAS:
        n = case["length"]
        per = {"vvadd": 4, "vvsub": 4, "vvmul": 2 * 21, "axpy": 2 * 21 + 4}[case["op"]]
        return {"bytes": 48 * n, "flops": per * n}
    if kind in (KIND_BATCH, KIND_BATCH_INVERSE):
        logns = _batch_logns(case)
        elems = int(np.left_shift(1, logns).sum())
        tables = sum(1 << int(n) for n in set(logns.tolist()))
        bfly = int((np.left_shift(1, logns) // 2 * logns).sum())
    else:
        elems, tables = case["count"] << case["log2n"], 1 << case["log2n"]
        bfly = elems // 2 * case["log2n"]
    if kind == KIND_POLYMUL:
        return {"bytes": 48 * elems + 32 * tables, "flops": (3 * bfly + elems) * 50}
    mul = 2 * (48 if case["prime"] == "general" else 21)
    return {"bytes": 32 * elems + 16 * tables, "flops": bfly * (mul + 8)}


def _ints(t, layout: int) -> np.ndarray:
    """Elements as exact Python integers."""
    a = np.ascontiguousarray(t.cpu().numpy() if isinstance(t, torch.Tensor) else t).view(np.uint64).reshape(-1, 2)
    hi, lo = (a[:, 0], a[:, 1]) if layout == bn.LAYOUT_HILO else (a[:, 1], a[:, 0])
    return hi.astype(object) * (1 << 64) + lo.astype(object)


def _elements(v: np.ndarray, layout: int) -> torch.Tensor:
    hi = (v >> 64).astype(np.uint64).view(np.int64)
    lo = (v & ((1 << 64) - 1)).astype(np.uint64).view(np.int64)
    return torch.from_numpy(np.stack((hi, lo) if layout == bn.LAYOUT_HILO else (lo, hi), axis=1))


def exact(case: dict, seed: int):
    """The outputs in Python integers, for the cases small enough for that."""
    kind, layout = case["kind"], case["layout"]
    if kind == KIND_BLAS:
        if case["length"] > 1 << 20:
            return None
        s = prepare(case, seed)
        a, b, q = _ints(s["a"], layout), _ints(s["b"], layout), bn.Q_BLAS
        c = {"vvadd": lambda: a + b, "vvsub": lambda: a - b, "vvmul": lambda: a * b,
             "axpy": lambda: a + AXPY_X * b}[case["op"]]() % q
        return _elements(c, layout)
    if kind not in (KIND_FORWARD, KIND_HOST) or (case["count"] << case["log2n"]) * case["log2n"] > 1 << 23:
        return None
    n, count, q = case["log2n"], case["count"], _modulus(case["prime"])[0]
    tw = _ints(_table(case, n, seed), layout)
    v = _ints(prepare(case, seed)["x"], layout)
    for s in range(n):   # stage s pairs indices that differ in bit n-1-s; block u takes entry 2^s + u
        v = v.reshape(count, 1 << s, 2, 1 << (n - 1 - s))
        p = v[:, :, 1] * tw[1 << s:2 << s].reshape(1, -1, 1) % q
        v = np.stack(((v[:, :, 0] + p) % q, (v[:, :, 0] - p) % q), axis=2)
    return _elements(v.reshape(-1), layout)

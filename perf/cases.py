"""The workloads whose speed counts: multi-double GEMMs as programs call them.

``listed()`` names twelve calls over the whole range of the library: the
BF16 slice-digit form (the default of ``gemm``) from a 64^3 double-double
product to the quad-double 8192^3 one, the batched plan, the host-buffer
entry, a plan with its own workspace, transposed operands with odd sizes, and
the two FP64 forms that stay as drop-ins of the reference.  ``draw(rng)``
gives one more call of the same families with other sizes.
"""
import importlib
import math

import numpy as np

PKG = "multiple-double-arithmetic-matrix-matrix-multiplication_gb300"
api = importlib.import_module(PKG + ".api")

# digits per operand of the BF16 form, by limb count
DIGITS = {2: 14, 4: 28, 8: 55, 16: 110}
# FP64 operations of one multi-double multiply-add in the plain form
PLAIN_FLOPS = {2: 43, 4: 425, 8: 2011}
EXACT_LIMIT = 22_000_000  # m n k up to which exact() takes seconds


def _gemm(name, entry, form, p, m, n, k, dist="uniform", spread=False):
    case = {"entry": entry, "form": form, "p": p, "m": m, "n": n, "k": k, "dist": dist,
            "spread": spread}
    return {"name": name, **case} if name else case


def _batch(name, count, shapes_seed):
    case = {"entry": "batch", "form": "slice_bf16", "count": count, "shapes_seed": shapes_seed}
    return {"name": name, **case} if name else case


def listed():
    return [
        # smallest call: one 64^3 double-double product, all launches and latency
        _gemm("dd64", "gemm", "slice_bf16", 2, 64, 64, 64),
        # a program's inner product of moderate size through a plan it keeps
        _gemm("qd256_plan", "plan", "slice_bf16", 4, 256, 256, 256),
        # the ordinary quad-double product
        _gemm("qd1024", "gemm", "slice_bf16", 4, 1024, 1024, 1024),
        # octo-double with badly scaled rows and columns (2^-32 .. 2^32)
        _gemm("od2048_spread", "gemm", "slice_bf16", 8, 2048, 2048, 2048, spread=True),
        # hexa-double, the widest type
        _gemm("hd1024", "gemm", "slice_bf16", 16, 1024, 1024, 512),
        # odd sizes, B given transposed, rows padded: a caller with its own layout
        _gemm("qd_ragged_ex", "gemm_ex", "slice_bf16", 4, 1000, 777, 1531),
        # tall and narrow (a block of vectors): operand traffic rather than products
        _gemm("dd_tall", "gemm", "slice_bf16", 2, 16001, 96, 3001, dist="normal"),
        # the largest: the headline quad-double product, normal entries
        _gemm("qd8192", "gemm", "slice_bf16", 4, 8192, 8192, 8192, dist="normal"),
        # many small products of mixed sizes and limb counts in one tuned plan
        _batch("batch64", 64, 3),
        # host arrays in, host array out
        _gemm("qd2048_host", "host", "slice_bf16", 4, 2048, 2048, 2048, dist="normal"),
        # the plain CUDA-core product (matmulTCnt's arithmetic)
        _gemm("plain_qd512", "gemm", "plain", 4, 512, 512, 512),
        # the FP64 tensor-core split form (the method of the reference)
        _gemm("split_qd", "gemm", "fp64split", 4, 251, 300, 277),
    ]


def _size(rng, lo, hi):
    """A size, even over its logarithm; every other one odd, some round."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    kind = rng.random()
    if kind < 0.5:
        return max(lo, min(hi, int(v) | 1))
    step = 64 if kind < 0.8 and v >= 64 else 1
    return max(lo, min(hi, int(v) // step * step))


def draw(rng):
    big = {c["name"]: c for c in listed()}
    while True:
        kind = rng.random()
        if kind < 0.45:
            c = _gemm(None, "gemm", "slice_bf16", rng.choice([2, 4, 4, 8, 16]),
                      _size(rng, 32, 12000), _size(rng, 32, 12000), _size(rng, 32, 8192),
                      rng.choice(["uniform", "normal"]), rng.random() < 0.25)
            limit = big["qd8192"]
        elif kind < 0.6:
            c = _gemm(None, "gemm_ex", "slice_bf16", rng.choice([2, 4, 8]),
                      _size(rng, 64, 2500), _size(rng, 64, 2500), _size(rng, 64, 2500))
            limit = big["od2048_spread"]
        elif kind < 0.7:
            c = _gemm(None, "plan", "slice_bf16", rng.choice([2, 4, 8]),
                      _size(rng, 32, 1024), _size(rng, 32, 1024), _size(rng, 32, 1024))
            limit = big["od2048_spread"]
        elif kind < 0.8:
            return _batch(None, rng.randint(12, 64), rng.randrange(1 << 30))
        elif kind < 0.87:
            c = _gemm(None, "host", "slice_bf16", rng.choice([2, 4]),
                      _size(rng, 128, 3000), _size(rng, 128, 3000), _size(rng, 128, 3000))
            limit = big["qd2048_host"]
        elif kind < 0.94:
            c = _gemm(None, "gemm", "plain", rng.choice([2, 4, 8]),
                      _size(rng, 32, 700), _size(rng, 32, 700), _size(rng, 32, 700))
            limit = big["plain_qd512"]
        else:
            c = _gemm(None, "gemm", "fp64split", rng.choice([2, 4]),
                      _size(rng, 32, 512), _size(rng, 32, 512), _size(rng, 32, 512))
            limit = {**c, "p": 4, "m": 512, "n": 512, "k": 512}
        w, top = work(c), work(limit)
        if w["flops"] <= top["flops"] and w["bytes"] <= top["bytes"]:
            return c


def _batch_shapes(case):
    rng = np.random.default_rng(case["shapes_seed"])
    out = []
    for _ in range(case["count"]):
        m, n, k = (int(v) * 32 for v in rng.integers(1, 17, size=3))
        out.append((int(rng.choice([2, 4, 8])), m, n, k))
    return out


def _operands(case, seed):
    p, m, n, k = case["p"], case["m"], case["n"], case["k"]
    lo, hi = (-32, 32) if case["spread"] else (0, 0)
    A = api.generate(case["dist"], p, m, k, 2 * seed, lo, hi, scale_rows=case["spread"])
    if case["entry"] == "gemm_ex":
        # B as its transpose, in a buffer whose rows are three entries longer
        store = api.generate(case["dist"], p, n, k + 3, 2 * seed + 1, lo, hi)
        return A, store[:, :k, :]
    return A, api.generate("uniform", p, k, n, 2 * seed + 1, lo, hi, scale_cols=case["spread"])


def prepare(case, seed):
    entry = case["entry"]
    if entry == "batch":
        pairs = []
        for i, (p, m, n, k) in enumerate(_batch_shapes(case)):
            s = (seed * 1000 + i) * 2
            pairs.append((api.generate("uniform", p, m, k, s),
                          api.generate("uniform", p, k, n, s + 1)))
        plan = api.BatchPlan(pairs)
        plan.tune()
        return {"entry": entry, "plan": plan}
    A, B = _operands(case, seed)
    state = {"entry": entry, "form": case["form"], "A": A, "B": B}
    if entry == "host":
        for key in ("A", "B"):
            buf = api.HostBuffer(tuple(state[key].shape))
            buf.array[...] = state[key].cpu().numpy()
            state[key + "_buffer"], state[key] = buf, buf.array
    if entry == "plan":
        state["plan"] = api.Plan(case["form"], case["p"], case["m"], case["n"], case["k"])
    return state


def run(state):
    entry = state["entry"]
    if entry == "batch":
        return state["plan"].run()
    A, B = state["A"], state["B"]
    if entry == "plan":
        return state["plan"].run(A, B)
    if entry == "host":
        return api.gemm_host(A, B, state["form"])
    if entry == "gemm_ex":
        return api.gemm_ex(A, B, state["form"], trans_b=True)
    return api.gemm(A, B, state["form"])


def _digit_products(p):
    """Digit-plane products of the BF16 form when digits i and j of both
    operands meet once: s squares and floor(s^2 / 4) cross products."""
    s = DIGITS[p]
    return s + s * s // 4


def _work(form, p, m, n, k):
    if form == "plain":
        per = PLAIN_FLOPS[p]
    elif form == "fp64split":
        per = 4 * p * (4 * p + 1)
    else:
        per = 2 * _digit_products(p)
    return 8 * p * (m * k + k * n + m * n), per * m * n * k


def work(case):
    if case["entry"] == "batch":
        shapes = _batch_shapes(case)
    else:
        shapes = [(case["p"], case["m"], case["n"], case["k"])]
    parts = [_work(case["form"], *s) for s in shapes]
    return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}


def _integers(X):
    """Entries of X (rows, cols, P) as Python integers times 2^-shift."""
    frac, e = np.frexp(X)
    shift = 53 - int(e[frac != 0].min(initial=0))
    mant = np.ldexp(frac, 53).astype(np.int64)
    ints = mant.astype(object) << np.maximum(e - 53 + shift, 0).astype(object)
    return ints.sum(axis=2), shift


def _round(v, shift, p):
    """v 2^-shift as p doubles, each the nearest to what is left."""
    out = []
    for _ in range(p):
        x = float(v)
        out.append(math.ldexp(x, -shift))
        v -= int(x)
    return out


def exact(case, seed):
    if case["entry"] == "batch" or case["p"] > 4:
        return None
    m, n, k, p = case["m"], case["n"], case["k"], case["p"]
    if m * n * k > EXACT_LIMIT:
        return None
    A, B = (X.cpu().numpy() for X in _operands(case, seed))
    if case["entry"] == "gemm_ex":
        B = B.transpose(1, 0, 2)
    (a, sa), (b, sb) = _integers(A), _integers(B)
    C = a.dot(b)
    out = np.array([_round(v, sa + sb, p) for v in C.reshape(-1)], dtype=np.float64)
    return out.reshape(m, n, p)

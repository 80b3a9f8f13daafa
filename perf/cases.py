"""Performance cases of the exact multiply and the callers that feed it.

Each case is one call that a program computing constants to many digits makes:
a single product at the sizes the splitting tree, the Newton iteration and the
radix conversion reach, a batch of products (one level of a tree), and the
three whole callers (series, quotient, conversion).  Operands are uniformly
random limbs, as the values of those trees are.  All outputs are integers and
exact.

listed() gives the fixed cases, draw(rng) others of the same ranges.
"""
import ctypes
import math

import numpy as np
import torch

import bluecrunch_b200 as bc
from bluecrunch_b200.bigfloat import Lib, limbs

# Ranges: products from the shortest the FFT multiply is used for (the host
# library multiplies below 100 limbs itself) to 2^26 limbs per operand; batch
# lengths and counts of bench.py's batched workload; series terms, quotient and
# conversion lengths up to what ten million and a few million digits need.
PRODUCT_MIN, PRODUCT_MAX = 128, 1 << 26
HOST_MAX = 1 << 20
BATCH_LO, BATCH_HI = 128, 262144
BATCH_ITEMS = 600
SERIES_MAX = 1_700_000
QUOTIENT_MAX = 300_000
RADIX_MAX = 400_000
SERIES_SHIFT = 1000  # a seed moves a series' first term by less than this


def listed():
    return [
        # the shortest products: a conversion's lowest power-table entries and
        # the first Newton levels; all latency
        {"name": "product_256", "kind": "product", "AL": 256, "BL": 256, "host": False},
        # a Newton level of the host library: operands and result in ordinary
        # host memory, lengths of no round number
        {"name": "product_host_3001", "kind": "product", "AL": 3001, "BL": 2777, "host": True},
        # the smallest product of the size sweep that bench.py prints
        {"name": "product_16k", "kind": "product", "AL": 16384, "BL": 16384, "host": False},
        # the middle of a splitting tree, odd and uneven lengths
        {"name": "product_200k_odd", "kind": "product", "AL": 200_003, "BL": 150_001, "host": False},
        # squaring, as the power table of the conversion does
        {"name": "square_3m_odd", "kind": "square", "AL": 3_000_017, "host": False},
        # a long operand times a short one (1:8), as near a splitting tree's edge
        {"name": "product_8m_1m", "kind": "product", "AL": 1 << 23, "BL": 1 << 20, "host": False},
        # the headline product: the top of e's tree at 10^8 to 10^9 digits
        {"name": "product_16m", "kind": "product", "AL": 1 << 24, "BL": 1 << 24, "host": False},
        # the largest of the range
        {"name": "product_64m", "kind": "product", "AL": 1 << 26, "BL": 1 << 26, "host": False},
        # one level of a tree: independent products of many lengths in one call
        {"name": "batch_600", "kind": "batch", "n": BATCH_ITEMS, "lo": BATCH_LO, "hi": BATCH_HI, "sibling": False},
        # e's series to ten million digits: every level of the tree
        {"name": "series_1700k", "kind": "series", "a": 0, "terms": SERIES_MAX},
        # the division that follows the series
        {"name": "quotient_300k", "kind": "quotient", "n": QUOTIENT_MAX},
        # binary to decimal: power table, product tree, leaves, merges
        {"name": "radix_400k", "kind": "radix", "n": RADIX_MAX},
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], uniform in its logarithm, odd half of the time."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, n | 1 if rng.random() < 0.5 else n))


def draw(rng):
    kind = rng.choice(["product"] * 5 + ["unbalanced", "square", "host", "batch", "series", "quotient", "radix"])
    if kind == "product":  # like neighbours of a tree: lengths within a factor of two
        a = _log(rng, PRODUCT_MIN, PRODUCT_MAX)
        return {"kind": "product", "AL": a, "BL": max(PRODUCT_MIN, int(a * rng.uniform(0.5, 1.0))), "host": False}
    if kind == "unbalanced":
        a = _log(rng, 16 * PRODUCT_MIN, PRODUCT_MAX)
        return {"kind": "product", "AL": a, "BL": _log(rng, PRODUCT_MIN, a // 4), "host": False}
    if kind == "square":
        return {"kind": "square", "AL": _log(rng, PRODUCT_MIN, PRODUCT_MAX), "host": False}
    if kind == "host":
        a = _log(rng, PRODUCT_MIN, HOST_MAX)
        return {"kind": "product", "AL": a, "BL": max(PRODUCT_MIN, int(a * rng.uniform(0.5, 1.0))), "host": True}
    if kind == "batch":
        return {"kind": "batch", "n": _log(rng, 20, BATCH_ITEMS), "lo": BATCH_LO, "hi": _log(rng, 4096, BATCH_HI),
                "sibling": rng.random() < 0.5}
    if kind == "series":
        a = rng.choice([0, 0, rng.randrange(1, 1 << 20)])
        return {"kind": "series", "a": a, "terms": _log(rng, 1000, SERIES_MAX - a if a else SERIES_MAX)}
    if kind == "quotient":
        return {"kind": "quotient", "n": _log(rng, 4000, QUOTIENT_MAX)}
    return {"kind": "radix", "n": _log(rng, 4000, RADIX_MAX)}


# ---------------------------------------------------------------- inputs
def _random_limbs(n, gen):
    """n random limbs in device memory, the top one nonzero."""
    x = torch.randint(-(1 << 31), 1 << 31, (n,), dtype=torch.int64, device="cuda", generator=gen).to(torch.int32)
    x[-1] |= 1
    return x


def _batch_lengths(case, seed):
    rng = np.random.default_rng(seed)
    lo, hi, n = np.log(case["lo"]), np.log(case["hi"]), case["n"]
    al = np.exp(rng.uniform(lo, hi, n)).astype(np.int64)
    if case["sibling"]:  # the two children of a tree node are of nearly one length
        return al, np.maximum(1, (al * rng.uniform(0.875, 1.125, n)).astype(np.int64))
    return al, np.exp(rng.uniform(lo, hi, n)).astype(np.int64)


def _numpy(x):
    return x.cpu().numpy().view(np.uint32)


def _fraction(n, gen):
    """Limbs of a value in [2, 3) with n - 1 limbs below the point."""
    x = _numpy(_random_limbs(n, gen)).copy()
    x[-1] = 2
    return x


def _series_cap(case):
    """Limbs that hold P and Q of a series case whatever the seed."""
    top = case["a"] + SERIES_SHIFT
    return int((math.lgamma(top + case["terms"] + 1) - math.lgamma(top + 1)) / math.log(2) / 32) + 4


def prepare(case, seed):
    bc.init(0)
    kind = case["kind"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if kind in ("product", "square"):
        AL = case["AL"]
        a = _random_limbs(AL, gen)
        b = None if kind == "square" else _random_limbs(case["BL"], gen)
        CL = AL + (AL if b is None else case["BL"])
        if case["host"]:
            state = {"a": _numpy(a).copy(), "b": None if b is None else _numpy(b).copy(),
                     "out": np.zeros(CL, dtype=np.uint32)}
        else:
            state = {"a": a, "b": b, "out": torch.zeros(CL, dtype=torch.int32, device="cuda")}
    elif kind == "batch":
        # the lengths belong to the case, the limbs to the seed
        al, bl = _batch_lengths(case, case["n"])
        off = np.concatenate([[0], np.cumsum(al + bl)])
        pool = _random_limbs(int(off[-1]), gen)
        out = torch.zeros(int(off[-1]), dtype=torch.int32, device="cuda")
        descs = (bc.MulDesc * case["n"])()
        for i in range(case["n"]):
            x, na, nb = int(off[i]), int(al[i]), int(bl[i])
            descs[i] = bc.MulDesc(out.data_ptr() + 4 * x, na + nb, pool.data_ptr() + 4 * x, na,
                                  pool.data_ptr() + 4 * (x + na), nb)
        state = {"pool": pool, "out": out, "descs": descs}
    elif kind == "series":
        dll = ctypes.CDLL(bc.GPU_LIB)
        fn = dll.bc_gpu_e_series
        fn.restype, fn.argtypes = bc.GPU_SYMBOLS["bc_gpu_e_series"]
        libc = ctypes.CDLL(None)
        libc.free.restype, libc.free.argtypes = None, [ctypes.c_void_p]
        # another seed sums another range of (nearly) the same length
        a = case["a"] + seed % SERIES_SHIFT
        state = {"fn": fn, "free": libc.free, "a": a, "b": a + case["terms"], "cap": _series_cap(case)}
    else:
        n = case["n"]
        lib = Lib()
        x = lib.make(_fraction(n, gen), exp=-(n - 1))
        y = lib.make(_fraction(n, gen), exp=-(n - 1))
        state = {"lib": lib, "x": x, "y": y, "n": n}
    state["kind"] = kind
    torch.cuda.synchronize()
    return state


# ---------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind in ("product", "square"):
        return bc.mul(state["a"], state["b"], out=state["out"])
    if kind == "batch":
        bc.mul_batch_desc(state["descs"], len(state["descs"]))
        return state["out"]
    if kind == "series":
        p, q = ctypes.POINTER(ctypes.c_uint32)(), ctypes.POINTER(ctypes.c_uint32)()
        pl, ql = ctypes.c_size_t(), ctypes.c_size_t()
        code = state["fn"](state["a"], state["b"], ctypes.byref(p), ctypes.byref(pl), ctypes.byref(q),
                           ctypes.byref(ql))
        if code != bc.BC_OK:
            raise bc.BcError(code, "bc_gpu_e_series")
        P, Q = (np.zeros(state["cap"], dtype=np.uint32) for _ in range(2))
        P[:pl.value] = np.ctypeslib.as_array(p, (pl.value,))
        Q[:ql.value] = np.ctypeslib.as_array(q, (ql.value,))
        state["free"](p)
        state["free"](q)
        return {"P": P, "Q": Q}
    lib = state["lib"]
    r = lib.make()
    if kind == "quotient":
        lib.div(r, state["y"], state["x"], state["n"])
    else:
        lib.radix(r, state["x"])
    got = {"limbs": limbs(r), "exp": int(r.exp), "sign": int(r.sign)}
    lib.free(r)
    return got


# ---------------------------------------------------------------- necessary work
def _product_work(AL, BL, square):
    """Operands in, product out; the transforms of a real convolution of
    16-bit digits (AL + BL complex points, 5 N log2 N each) and the products."""
    N = AL + BL
    passes = 2 if square else 3
    return 4.0 * ((AL if square else AL + BL) + N), passes * 5.0 * N * math.log2(max(N, 2)) + 6.0 * N


def _series_levels(a, b):
    """(AL, BL) of the two products of every node above leaves of 1024 terms."""
    def length(lo, hi):
        return max(1, int((math.lgamma(hi + 1) - math.lgamma(lo + 1)) / math.log(2) / 32) + 1)
    todo, out = [(a, b)], []
    while todo:
        lo, hi = todo.pop()
        if hi - lo > 1024:
            m = (lo + hi) // 2
            out.append((length(lo, m), length(m, hi)))
            todo += [(lo, m), (m, hi)]
    return out


def work(case):
    kind = case["kind"]
    if kind in ("product", "square"):
        nbytes, flops = _product_work(case["AL"], case.get("BL", case["AL"]), kind == "square")
    elif kind == "batch":
        al, bl = _batch_lengths(case, case["n"])
        each = [_product_work(int(x), int(y), False) for x, y in zip(al, bl)]
        nbytes, flops = sum(e[0] for e in each), sum(e[1] for e in each)
    elif kind == "series":
        a, b = case["a"], case["a"] + case["terms"]
        total = (math.lgamma(b + 1) - math.lgamma(a + 1)) / math.log(2) / 8
        nbytes = 2 * total
        # two products per node, the right Q transformed once for both
        flops = sum(5.0 / 3 * _product_work(x, y, False)[1] for x, y in _series_levels(a, b)) or 2.0 * case["terms"] ** 2 / 32
    elif kind == "quotient":
        # each level two products at its precision, the last the quotient
        n = case["n"]
        nbytes = 12.0 * n
        flops = _product_work(n, n, False)[1]
        while n > 100:
            flops += 2 * _product_work(n, n, False)[1]
            n = n // 2 + 1
    else:
        # a product of the node's length by half of it, at every depth down to leaves of 1000 digits
        n, flops = case["n"], 0.0
        nbytes, nodes, k = 8.0 * n, 1, case["n"]
        while k > 1000:
            flops += nodes * _product_work(k, (k + 1) // 2, False)[1]
            nodes, k = 2 * nodes, (k + 1) // 2
        flops = flops or 2.0 * n * n
    return {"bytes": float(nbytes), "flops": float(flops)}


# ---------------------------------------------------------------- exact values
EXACT_LIMBS = 400_000  # operand limbs of a product that Python's integers take a few seconds for
EXACT_TERMS = 20_000


def _as_int(x):
    return int.from_bytes(np.ascontiguousarray(x).astype("<u4").tobytes(), "little")


def exact(case, seed):
    """The product (or P and Q of the series) by Python's integers."""
    kind = case["kind"]
    if kind in ("product", "square") and case["AL"] + case.get("BL", case["AL"]) <= EXACT_LIMBS:
        s = prepare(case, seed)
        a = s["a"] if case["host"] else _numpy(s["a"])
        b = a if s["b"] is None else (s["b"] if case["host"] else _numpy(s["b"]))
        c = np.frombuffer((_as_int(a) * _as_int(b)).to_bytes(4 * (a.size + b.size), "little"), dtype="<u4")
        return c.copy() if case["host"] else torch.from_numpy(c.view(np.int32).copy())
    if kind == "series" and case["terms"] <= EXACT_TERMS:
        a = case["a"] + seed % SERIES_SHIFT
        P, Q = 1, a + 1
        for k in range(a + 2, a + case["terms"] + 1):
            P, Q = P * k + 1, Q * k
        cap = _series_cap(case)
        return {n: np.frombuffer(v.to_bytes(4 * cap, "little"), dtype="<u4").copy() for n, v in (("P", P), ("Q", Q))}
    return None

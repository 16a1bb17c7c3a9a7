"""The work this library does for its users, as measurable cases.

A case is one call of a public entry point (multifloats_b200.api) on inputs of
the sizes and value distributions that the benchmark configurations name, or on
odd sizes between them.  `listed` gives the fixed cases, `draw` another one of
the same ranges, `prepare` what a program holds before the call, `run` the call,
`work` the bytes and operations it cannot do without, `exact` the result in
binary64 arithmetic from plain torch.

Results are double-double: every entry is a pair (hi, lo) whose sum is the
value.  `exact` puts the binary64 value in hi and zero in lo.
"""
import math

import numpy as np
import torch

from multifloats_b200 import api

UNARY = ("exp", "log", "sin", "cos", "sqrt", "exp2", "log2", "log10")
REDUCE = {"sum": api.sum_dd, "dot": api.dot_product, "norm2": api.norm2,
          "csum": api.csum_dd, "cdot": api.cdot_product, "cnorm2": api.cnorm2}


def listed():
    return [
        # the smallest call: a dot product inside an iterative solver
        {"name": "dot_1000", "kind": "reduce", "op": "dot", "n": 1000},
        # a map over an ordinary array
        {"name": "exp_100003", "kind": "unary", "op": "exp", "n": 100003},
        # a map over a large array, the heaviest function
        {"name": "sin_2e24", "kind": "unary", "op": "sin", "n": 1 << 24},
        # the reduction of the benchmark configuration (2^26 elements)
        {"name": "dot_2e26", "kind": "reduce", "op": "dot", "n": 1 << 26},
        # a matrix-vector product of a solver, odd sizes
        {"name": "mv_4099x3001", "kind": "mv", "m": 4099, "k": 3001},
        # the smallest GEMM configuration
        {"name": "gemm_256", "kind": "gemm", "form": "plain", "complex": False, "m": 256, "k": 256, "n": 256},
        # a rectangular product with no round size
        {"name": "gemm_1531x977x1203", "kind": "gemm", "form": "plain", "complex": False,
         "m": 1531, "k": 977, "n": 1203},
        # the reference-identical product at the headline size
        {"name": "gemm_4096", "kind": "gemm", "form": "plain", "complex": False, "m": 4096, "k": 4096, "n": 4096},
        # the headline: the split form of the same product, row / column exponents in [-16, 16]
        {"name": "crt_4096", "kind": "gemm", "form": "crt", "complex": False, "m": 4096, "k": 4096, "n": 4096},
        # a complex product of ordinary odd size in the split form
        {"name": "ccrt_1009x1100x907", "kind": "gemm", "form": "crt", "complex": True,
         "m": 1009, "k": 1100, "n": 907},
        # the batch configuration: 2000 products, sizes log-uniform in [16, 1024]
        {"name": "batch_2000", "kind": "batch", "form": "split", "complex": False, "count": 2000, "hi": 1024,
         "shapes": 5},
        # a caller of the drop-in symbol: host arrays in and out
        {"name": "host_gemm_500x400x600", "kind": "host_gemm", "m": 500, "k": 400, "n": 600},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("reduce", "unary", "mv", "vm", "plain", "plain", "split_forms", "split_forms", "batch",
                       "host_gemm"))
    if kind == "reduce":
        op = rng.choice(sorted(REDUCE))
        return {"kind": kind, "op": op, "n": _log(rng, 1000, 1 << (24 if op[0] == "c" else 26))}
    if kind == "unary":
        return {"kind": kind, "op": rng.choice(UNARY), "n": _log(rng, 1000, 1 << 24)}
    if kind in ("mv", "vm"):
        return {"kind": kind, "m": _log(rng, 200, 6000), "k": _log(rng, 200, 6000)}
    if kind == "batch":
        return {"kind": kind, "form": rng.choice(("plain", "split", "crt")), "complex": rng.random() < 0.3,
                "count": _log(rng, 20, 500), "hi": _log(rng, 64, 700), "shapes": rng.randrange(1 << 30)}
    if kind == "host_gemm":
        return {"kind": kind, "m": _log(rng, 50, 900), "k": _log(rng, 50, 900), "n": _log(rng, 50, 900)}
    cplx = rng.random() < 0.35
    if kind == "plain":
        form, lo, hi = "plain", 64, 1000 if cplx else 1800
    else:
        form, lo, hi = rng.choice(("split", "crt", "crt")), 200, 1500 if cplx else 3000
    return {"kind": "gemm", "form": form, "complex": cplx, "m": _log(rng, lo, hi), "k": _log(rng, lo, hi),
            "n": _log(rng, lo, hi)}


# ---- inputs ---------------------------------------------------------------------
def _rand(g, shape, lo, hi):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _dd(g, hi):
    """hi with a low limb hi 2^-53 U[-1, 1), renormalised; limbs interleaved on the last axis, flattened."""
    lo = hi * _rand(g, hi.shape, -1.0, 1.0) * 2.0 ** -53
    s = hi + lo
    bb = s - hi
    return torch.stack((s, (hi - (s - bb)) + (lo - bb)), -1).reshape(-1)


def _matrix(g, rows, cols, cplx, R=0, per="row"):
    """Column-major rows x cols: U[-1, 1), or with R > 0 +-U[1, 2) 2^e, e ~ U{-R..R} per row or per column."""
    shape = (cols, rows, 2) if cplx else (cols, rows)
    if R:
        u = _rand(g, shape, 1.0, 2.0)
        u = torch.where(_rand(g, shape, 0.0, 1.0) < 0.5, -u, u)
        e = torch.randint(-R, R + 1, (rows if per == "row" else cols,), generator=g, device="cuda").double()
        e = torch.exp2(e).reshape((1, -1) if per == "row" else (-1, 1))
        u = u * (e[..., None] if cplx else e)
    else:
        u = _rand(g, shape, -1.0, 1.0)
    return _dd(g, u)


def _unary_input(g, op, n):
    if op == "exp":
        return _dd(g, _rand(g, n, -300.0, 300.0))
    if op == "exp2":
        return _dd(g, _rand(g, n, -400.0, 400.0))
    if op in ("sin", "cos"):  # a tenth of them next to multiples of pi/2
        x = _rand(g, n, -1e6, 1e6)
        near = torch.round(x / (math.pi / 2)) * (math.pi / 2) + _rand(g, n, -1e-12, 1e-12)
        return _dd(g, torch.where(_rand(g, n, 0.0, 1.0) < 0.1, near, x))
    return _dd(g, torch.exp2(_rand(g, n, -400.0, 400.0)))


def _batch_shapes(case):
    """Sizes log-uniform in [16, hi], from the case's own seed `shapes`."""
    r = np.random.default_rng(case["shapes"])
    return np.rint(np.exp(r.uniform(math.log(16), math.log(case["hi"]), (case["count"], 3)))).astype(int).tolist()


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "reduce":
        w = 2 if case["op"][0] == "c" else 1
        x = [_dd(g, _rand(g, case["n"] * w, -1.0, 1.0)) for _ in range(2 if "dot" in case["op"] else 1)]
        return {"case": case, "x": x}
    if kind == "unary":
        return {"case": case, "x": [_unary_input(g, case["op"], case["n"])]}
    if kind in ("mv", "vm"):
        return {"case": case, "a": _matrix(g, case["m"], case["k"], False),
                "v": _matrix(g, case["k"] if kind == "mv" else case["m"], 1, False)}
    if kind == "host_gemm":
        m, k, n = case["m"], case["k"], case["n"]
        return {"case": case, "a": _matrix(g, m, k, False).cpu().numpy(), "b": _matrix(g, k, n, False).cpu().numpy()}
    if kind == "gemm":
        m, k, n = case["m"], case["k"], case["n"]
        R = 0 if case["form"] == "plain" else 16
        return {"case": case, "a": _matrix(g, m, k, case["complex"], R, "row"),
                "b": _matrix(g, k, n, case["complex"], R, "col")}
    # batch: all operands in three buffers, a plan over their parts
    w = 4 if case["complex"] else 2
    shapes = _batch_shapes(case)
    size = [sum(w * m * k for m, k, n in shapes), sum(w * k * n for m, k, n in shapes),
            sum(w * m * n for m, k, n in shapes)]
    a, b = (_dd(g, _rand(g, s // 2, -1.0, 1.0)) for s in size[:2])
    c = torch.empty(size[2], dtype=torch.float64, device="cuda")
    problems, i, j, l = [], 0, 0, 0
    for m, k, n in shapes:
        problems.append((a[i:i + w * m * k], b[j:j + w * k * n], c[l:l + w * m * n], m, k, n))
        i, j, l = i + w * m * k, j + w * k * n, l + w * m * n
    plan = api.GemmBatch(problems, form=case["form"], complex_=case["complex"])
    return {"case": case, "plan": plan, "c": c, "problems": problems}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "reduce":
        return REDUCE[case["op"]](*state["x"])
    if kind == "unary":
        return api.unary(case["op"], state["x"][0])
    if kind == "mv":
        return api.matmuldd_mv(state["a"], state["v"], case["m"], case["k"])
    if kind == "vm":
        return api.matmuldd_vm(state["v"], state["a"], case["m"], case["k"])
    if kind == "batch":
        state["plan"].run()
        return state["c"]
    if kind == "host_gemm":
        return api.matmuldd_mm(state["a"], state["b"], case["m"], case["k"], case["n"])
    args = (state["a"], state["b"], case["m"], case["k"], case["n"])
    if case["form"] == "plain":
        return (api.cmatmuldd_mm if case["complex"] else api.matmuldd_mm)(*args)
    name = ("c" if case["complex"] else "") + "matmuldd_mm_" + case["form"]
    return getattr(api, name)(*args)[0]


def work(case):
    """Bytes: each operand read once, each result written once (16 bytes per
    double-double).  Flops: one double-double multiply and one add per product
    term (a complex term is four of them); per element of a map, one."""
    kind = case["kind"]
    if kind == "reduce":
        w = 16 * (2 if case["op"][0] == "c" else 1)
        return {"bytes": w * case["n"] * (2 if "dot" in case["op"] else 1) + w, "flops": 2 * case["n"]}
    if kind == "unary":
        return {"bytes": 32 * case["n"], "flops": case["n"]}
    if kind in ("mv", "vm"):
        m, k = case["m"], case["k"]
        return {"bytes": 16 * (m * k + m + k), "flops": 2 * m * k}
    if kind == "batch":
        shapes = _batch_shapes(case)
    else:
        shapes = [(case["m"], case["k"], case["n"])]
    w = 2 if case.get("complex") else 1
    return {"bytes": sum(16 * w * (m * k + k * n + m * n) for m, k, n in shapes),
            "flops": sum(2 * w * w * m * k * n for m, k, n in shapes)}


# ---- the same results in binary64 ---------------------------------------------------
def _value(x):
    """A double-double array in binary64 (hi + lo rounds to hi)."""
    v = x.reshape(-1, 2)
    return v[:, 0] + v[:, 1]


def _pairs(v):
    return torch.stack((v, torch.zeros_like(v)), -1).reshape(-1)


def _product(a, b, m, k, n, cplx):
    a, b = _value(a), _value(b)
    if cplx:
        a, b = torch.view_as_complex(a.reshape(-1, 2)), torch.view_as_complex(b.reshape(-1, 2))
    c = b.reshape(n, k) @ a.reshape(k, m)  # column-major operands: C^T = B^T A^T
    return _pairs((torch.view_as_real(c) if cplx else c).reshape(-1))


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "unary":
        op = case["op"]
        hi, lo = s["x"][0].reshape(-1, 2).unbind(-1)
        f = getattr(torch, op)(hi)
        slope = {"exp": f, "exp2": f * math.log(2), "log": 1 / hi, "log2": 1 / (hi * math.log(2)),
                 "log10": 1 / (hi * math.log(10)), "sqrt": 0.5 / f,
                 "sin": torch.cos(hi), "cos": -torch.sin(hi)}[op]
        return _pairs(f + lo * slope)
    if kind == "reduce":
        op, x = case["op"], [_value(v) for v in s["x"]]
        if op[0] == "c" and op != "cnorm2":
            z = [torch.view_as_complex(v.reshape(-1, 2)) for v in x]
            r = z[0].sum() if op == "csum" else torch.vdot(z[0], z[1])
            return _pairs(torch.view_as_real(r).reshape(-1))
        r = {"sum": lambda: x[0].sum(), "dot": lambda: torch.dot(x[0], x[1])}.get(op, lambda: x[0].square().sum().sqrt())
        return _pairs(r().reshape(1))
    if kind == "mv":
        return _pairs(_value(s["v"]) @ _value(s["a"]).reshape(case["k"], case["m"]))
    if kind == "vm":
        return _pairs(_value(s["a"]).reshape(case["k"], case["m"]) @ _value(s["v"]))
    if kind == "batch":
        return torch.cat([_product(a, b, m, k, n, case["complex"]) for a, b, c, m, k, n in s["problems"]])
    if kind == "host_gemm":
        a, b = torch.from_numpy(s["a"]).cuda(), torch.from_numpy(s["b"]).cuda()
        return _product(a, b, case["m"], case["k"], case["n"], False).cpu().numpy()
    return _product(s["a"], s["b"], case["m"], case["k"], case["n"], case["complex"])

"""Workloads of the compute entry points, for timing and for comparing outputs.

A case is a dict of plain values.  Its "op" is one of
  saxpy    n elements, z = alpha x + y
  matvec   m x n, y = alpha A x + beta y (A stored column-major when trans_a)
  matmul   m x n x k, device operands, every engine; "workspace": the caller
           keeps a workspace of the queried size, else the library's own
  grouped  count uneven products in one plan, packed and contracted by its graph
  host     matmul on pinned host buffers: upload, contraction and download
Operands are uniform[-1, 1), the distribution of the benchmark and the tests.
"""
import math
import random

import torch

import gatlas_b200 as g

# BF16 (or FP8) products per multiply-add of each tensor-core engine
PRODUCTS = {"buffer": 1, "image": 1, "tc_bf16": 1, "tc_split3": 3, "tc_split6": 6, "tc_fp8": 1}
# most multiply-add work of a drawn case: tensor cores (the 8192^3 split product), SIMT float, SIMT double
MAX_TC_FLOPS, MAX_F32_FLOPS, MAX_F64_FLOPS = 3 * 2 * 8192 ** 3, 4e10, 1.5e10


def _matmul(name, m, n, k, engine, **more):
    case = {"op": "matmul", "m": m, "n": n, "k": k, "engine": engine, "dtype": "float32",
            "trans_a": False, "trans_b": False, "alpha": 1.0, "beta": 0.0, "batch": 1, "workspace": False}
    case.update(more)
    return dict(case, name=name) if name else case


def _matvec(name, m, n, engine, **more):
    case = {"op": "matvec", "m": m, "n": n, "engine": engine, "dtype": "float32", "trans_a": False,
            "alpha": 1.0, "beta": 0.0}
    case.update(more)
    return dict(case, name=name) if name else case


def listed():
    return [
        # the smallest vector update of the serving mix: launch and call latency
        {"name": "saxpy_64k", "op": "saxpy", "n": 65536, "dtype": "float32", "engine": "buffer", "alpha": 0.5},
        # the smallest matrix-vector product of the serving mix, accumulating into y
        _matvec("gemv_1k", 1024, 1024, "buffer", alpha=0.75, beta=0.5),
        # y = A^T x for a matrix whose sides are odd, so that no row starts on a vector boundary
        _matvec("gemv_ragged_t", 3001, 7013, "buffer", trans_a=True),
        # the benchmark's memory-bound matrix-vector product, TMA engine
        _matvec("gemv_image_16k", 16384, 16384, "image"),
        # the benchmark's plain SGEMM at the default parameter point
        _matmul("sgemm_1k", 1024, 1024, 1024, "buffer"),
        # a large FP32 product with fused multiply-add accuracy, TMA engine, B stored transposed
        _matmul("sgemm_image_3k", 3072, 2560, 2048, "image", trans_b=True),
        # a double-precision update with odd sides
        _matmul("dgemm_ragged", 1531, 1277, 1021, "buffer", dtype="float64", alpha=0.5, beta=0.5),
        # a few rows of activations against a wide weight matrix
        _matmul("bf16_skinny", 64, 4096, 8192, "tc_bf16"),
        # an FP32-accurate update of ordinary, ragged size with both operands stored transposed
        _matmul("split3_ragged", 1000, 777, 1100, "tc_split3", trans_a=True, trans_b=True, alpha=0.5, beta=0.5),
        # the headline: FP32-accurate SGEMM, 8192^3, workspace kept by the caller
        _matmul("split3_8k", 8192, 8192, 8192, "tc_split3", workspace=True),
        # block-scaled FP8 from FP32 operands, quantised on each call
        _matmul("fp8_4k", 4096, 4096, 4096, "tc_fp8", workspace=True),
        # many uneven products at once, as the serving loop batches them
        {"name": "grouped_256", "op": "grouped", "count": 256, "mix": 1, "largest": 2048, "engine": "tc_split3"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["saxpy", "matvec", "matvec", "simt", "simt", "tc", "tc", "tc", "tc", "grouped", "host"])
    if op == "saxpy":
        dtype = rng.choice(["float32", "float32", "float64"])
        n = _log(rng, 1 << 16, 1 << (26 if dtype == "float32" else 25))
        return {"op": "saxpy", "n": n, "dtype": dtype, "engine": rng.choice(["buffer", "image"]), "alpha": 0.5}
    if op == "matvec":
        dtype = rng.choice(["float32", "float32", "float64"])
        engine = rng.choice(["buffer", "image"])
        while True:
            m, n = _log(rng, 1024, 32768), _log(rng, 1024, 32768)
            if m * n <= 1 << 27:
                break
        if engine == "image":  # TMA operands have 16-byte rows
            m, n = m // 4 * 4, n // 4 * 4
        beta = rng.choice([0.0, 0.5])
        return _matvec("", m, n, engine, dtype=dtype, trans_a=rng.random() < 0.5, beta=beta)
    if op == "simt":
        dtype = rng.choice(["float32", "float32", "float64"])
        engine = rng.choice(["buffer", "buffer", "image"])
        most = MAX_F32_FLOPS if dtype == "float32" else MAX_F64_FLOPS
        while True:
            m, n, k = (_log(rng, 64, 4096) for _ in range(3))
            if 2.0 * m * n * k <= most:
                break
        if engine == "image":
            m, n, k = m // 4 * 4, n // 4 * 4, k // 4 * 4
        return _matmul("", m, n, k, engine, dtype=dtype, trans_a=rng.random() < 0.5, trans_b=rng.random() < 0.5,
                       alpha=0.5, beta=rng.choice([0.0, 0.5]))
    if op == "tc":
        engine = rng.choice(["tc_bf16", "tc_split3", "tc_split3", "tc_split6", "tc_fp8"])
        while True:
            m, n, k = (_log(rng, 64, 8192) for _ in range(3))
            batch = rng.choice([1, 1, 1, 8]) if max(m, n, k) <= 1024 else 1
            if 2.0 * m * n * k * batch * PRODUCTS[engine] <= MAX_TC_FLOPS:
                break
        return _matmul("", m, n, k, engine, trans_a=rng.random() < 0.5, trans_b=rng.random() < 0.5, batch=batch,
                       alpha=0.5, beta=rng.choice([0.0, 0.5]), workspace=rng.random() < 0.5)
    if op == "grouped":
        return {"op": "grouped", "count": _log(rng, 32, 256), "mix": rng.randrange(1 << 20),
                "largest": rng.choice([512, 1024, 2048]), "engine": rng.choice(["tc_bf16", "tc_split3"])}
    return {"op": "host", "m": _log(rng, 512, 4096), "n": _log(rng, 512, 4096), "k": _log(rng, 512, 4096),
            "engine": rng.choice(["tc_split3", "tc_bf16"])}


def _uniform(n, dtype, gen):
    return torch.empty(n, dtype=getattr(torch, dtype), device="cuda").uniform_(-1.0, 1.0, generator=gen)


def _shapes(case):
    """The products of a grouped case: sides log-uniform, multiples of 16; layouts, alpha and beta random."""
    rng = random.Random(case["mix"])
    side = lambda: max(16, _log(rng, 16, case["largest"]) // 16 * 16)  # noqa: E731
    return [{"m": side(), "n": side(), "k": side(), "trans_a": rng.random() < 0.5, "trans_b": rng.random() < 0.5,
             "alpha": rng.uniform(0.5, 2.0), "beta": float(rng.randrange(2))} for _ in range(case["count"])]


def _operands(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    op = case["op"]
    if op == "saxpy":
        return {v: _uniform(case["n"], case["dtype"], gen) for v in ("x", "y")}
    if op == "matvec":
        return {"A": _uniform(case["m"] * case["n"], case["dtype"], gen), "x": _uniform(case["n"], case["dtype"], gen),
                "y": _uniform(case["m"], case["dtype"], gen)}
    if op == "matmul":
        m, n, k, b = case["m"], case["n"], case["k"], case["batch"]
        return {"A": _uniform(b * m * k, case["dtype"], gen), "B": _uniform(b * k * n, case["dtype"], gen),
                "C": _uniform(b * m * n, case["dtype"], gen)}
    if op == "host":
        m, n, k = case["m"], case["n"], case["k"]
        return {"A": _uniform(m * k, "float32", gen), "B": _uniform(k * n, "float32", gen)}
    # grouped: each operand kind in one pool, sides are multiples of 16, so every product starts 256-byte aligned
    shapes = _shapes(case)
    pools = {}
    for name, (i, j) in {"A": ("m", "k"), "B": ("k", "n"), "C": ("m", "n")}.items():
        sizes = [s[i] * s[j] for s in shapes]
        pools[name] = (_uniform(sum(sizes), "float32", gen), sizes)
    return {"shapes": shapes, "pools": pools}


def prepare(case, seed):
    s = _operands(case, seed)
    s["case"] = case
    op = case["op"]
    if op == "saxpy":
        s["z"] = torch.empty_like(s["y"])
    elif op == "matmul" and case["workspace"]:
        size = g.matmul_workspace_size(case["m"], case["n"], case["k"], case["engine"], case["trans_a"],
                                       case["trans_b"], case["batch"])
        s["workspace"] = torch.empty(size, dtype=torch.uint8, device="cuda")
    elif op == "host":
        for v in ("A", "B"):
            s[v] = torch.empty(s[v].numel(), pin_memory=True).copy_(s[v])
        s["C"] = torch.empty(case["m"] * case["n"], pin_memory=True)
    elif op == "grouped":
        parts = {v: torch.split(pool, sizes) for v, (pool, sizes) in s["pools"].items()}
        instances = [dict(q, gemm=1, A=parts["A"][i], B=parts["B"][i], C=parts["C"][i])
                     for i, q in enumerate(s["shapes"])]
        s["plan"] = g.Grouped(instances, engine=case["engine"])
    return s


def run(state):
    c = state["case"]
    if c["op"] == "saxpy":
        return g.saxpy(c["alpha"], state["x"], state["y"], out=state["z"], engine=c["engine"])
    if c["op"] == "matvec":
        return g.matvec(state["A"], state["x"], c["m"], c["n"], y=state["y"], trans_a=c["trans_a"], gemv=True,
                        alpha=c["alpha"], beta=c["beta"], engine=c["engine"])
    if c["op"] == "matmul":
        return g.matmul(state["A"], state["B"], c["m"], c["n"], c["k"], C=state["C"], trans_a=c["trans_a"],
                        trans_b=c["trans_b"], gemm=True, alpha=c["alpha"], beta=c["beta"], engine=c["engine"],
                        batch=c["batch"], workspace=state.get("workspace"))
    if c["op"] == "host":
        return g.matmul_host(state["A"], state["B"], c["m"], c["n"], c["k"], state["C"], engine=c["engine"])
    state["plan"].launch_graph()
    return state["pools"]["C"][0]


def work(case):
    """Each operand read once and each result written once (read too where beta is used); one multiply-add is two
    operations, and a split engine runs three or six products for one."""
    op = case["op"]
    size = 8 if case.get("dtype") == "float64" else 4
    if op == "saxpy":
        return {"bytes": 3 * size * case["n"], "flops": 2 * case["n"]}
    if op == "matvec":
        m, n = case["m"], case["n"]
        return {"bytes": size * (m * n + n + m * (2 if case["beta"] else 1)), "flops": 2 * m * n}
    if op == "grouped":
        shapes = _shapes(case)
        return {"bytes": sum(4 * (q["m"] * q["k"] + q["k"] * q["n"] + q["m"] * q["n"] * (2 if q["beta"] else 1))
                             for q in shapes),
                "flops": PRODUCTS[case["engine"]] * sum(2 * q["m"] * q["n"] * q["k"] for q in shapes)}
    m, n, k, b = case["m"], case["n"], case["k"], case.get("batch", 1)
    return {"bytes": b * size * (m * k + k * n + m * n * (2 if case.get("beta") else 1)),
            "flops": b * PRODUCTS[case["engine"]] * 2 * m * n * k}


def _product(A, B, m, n, k, trans_a, trans_b):
    a = A.double().view(k, m).t() if trans_a else A.double().view(m, k)
    b = B.double().view(n, k).t() if trans_b else B.double().view(k, n)
    return (a @ b).reshape(-1)


def exact(case, seed):
    s = _operands(case, seed)
    op = case["op"]
    if op == "saxpy":
        return case["alpha"] * s["x"].double() + s["y"].double()
    if op == "matvec":
        m, n = case["m"], case["n"]
        a = s["A"].double().view(n, m).t() if case["trans_a"] else s["A"].double().view(m, n)
        return case["alpha"] * (a @ s["x"].double()) + case["beta"] * s["y"].double()
    if op == "host":
        return _product(s["A"], s["B"], case["m"], case["n"], case["k"], False, False)
    if op == "matmul":
        m, n, k, b = case["m"], case["n"], case["k"], case["batch"]
        p = [_product(s["A"][i * m * k:(i + 1) * m * k], s["B"][i * k * n:(i + 1) * k * n], m, n, k, case["trans_a"],
                      case["trans_b"]) for i in range(b)]
        return case["alpha"] * torch.cat(p) + case["beta"] * s["C"].double()
    parts = {v: torch.split(pool, sizes) for v, (pool, sizes) in s["pools"].items()}
    return torch.cat([q["alpha"] * _product(parts["A"][i], parts["B"][i], q["m"], q["n"], q["k"], q["trans_a"],
                                            q["trans_b"]) + q["beta"] * parts["C"][i].double()
                      for i, q in enumerate(s["shapes"])])

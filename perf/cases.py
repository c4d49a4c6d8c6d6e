"""The work a user of this library has it do, as measurable cases.

Every case goes through a public entry point of ``tensilelite_gb300``:

* ``gemm``     ``Handle.gemm`` on column-major buffers: every input type, layout, alpha/beta, padded
               leading dimensions, batches, and the FP32-accurate split kernels;
* ``linear``   ``linear``: the fused bias / activation layer of an inference program;
* ``train``    ``matmul`` and its gradients: one forward and backward of a projection;
* ``grouped``  one persistent launch over many independent problems (the plan is kept);
* ``quantize`` ``Handle.quantize_fp8``: per-tensor scaling of a tensor ahead of an FP8 GEMM.

``prepare`` makes what such a program has in hand (operands on the GPU, the problem description, the
output buffer, the plan); ``run`` is one pass.  ``exact`` is the same result in 64 bits from plain
torch.
"""
import math

import numpy as np
import torch

import tensilelite_gb300 as tl

TORCH = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16, "fp8": torch.float8_e4m3fn}
BYTES = {"fp32": 4, "fp16": 2, "bf16": 2, "fp8": 1}


def _gemm(name, dtype, layout, m, n, k, *, beta=0.0, alpha=1.0, batch=1, pad=0, kernel="auto", dist="normal"):
    return {"name": name, "kind": "gemm", "dtype": dtype, "layout": layout, "m": m, "n": n, "k": k, "alpha": alpha,
            "beta": beta, "batch": batch, "pad": pad, "kernel": kernel, "dist": dist}


def listed():
    return [
        # the plain FP32 call of the original benchmark: a small GEMM, where latency counts
        _gemm("fp32_480x512x512_nn", "fp32", "NN", 480, 512, 512, dist="uniform"),
        # FP32 as the command line runs it: TN, every dimension padded by 64, alpha and beta set
        _gemm("fp32_4096_tn_padded", "fp32", "TN", 4096, 4096, 4096, alpha=0.314, beta=0.2718, pad=64),
        # an inference layer on a few rows (a decode step): the weights are read once, bias and GELU fused
        {"name": "linear_bf16_32x1024x4096", "kind": "linear", "dtype": "bf16", "rows": 32, "k": 1024, "n": 4096,
         "activation": "gelu"},
        # a small half-precision GEMM with a long sum and few output tiles
        _gemm("bf16_480x1024x4096_nn", "bf16", "NN", 480, 1024, 4096, beta=0.5),
        # the ordinary large half-precision GEMM, with a C operand
        _gemm("bf16_4096_nn", "bf16", "NN", 4096, 4096, 4096, beta=0.5),
        # ragged matrices in a strided batch (per-head or per-expert products), neither side a multiple of a tile
        _gemm("fp16_1000x600x520_nt_batch24", "fp16", "NT", 1000, 600, 520, batch=24),
        # the FP8 GEMM on quantised operands in the layout of a linear layer, bf16 result
        _gemm("fp8_8192_tn", "fp8", "TN", 8192, 8192, 8192),
        # per-tensor quantisation of a layer's activations ahead of an FP8 GEMM
        {"name": "quantize_bf16_4096x4096", "kind": "quantize", "dtype": "bf16", "count": 4096 * 4096},
        # FP32-accurate GEMM on the tensor cores, two bf16 pieces per operand, large
        _gemm("bf16x3_8192_nn", "fp32", "NN", 8192, 8192, 8192, kernel="bf16x3", dist="uniform"),
        # the same with three pieces (full FP32 accuracy) at an ordinary, ragged size
        _gemm("bf16x6_3000x2000x2600_tn", "fp32", "TN", 3000, 2000, 2600, kernel="bf16x6", dist="uniform"),
        # many independent problems of uneven sizes in one launch
        {"name": "grouped_bf16_256", "kind": "grouped", "dtype": "bf16", "layout": "NN", "count": 256, "most": 2048,
         "most_k": 4096, "shape_seed": 3},
        # training step of a projection: forward, input gradient and weight gradient
        {"name": "train_bf16_4096x1024x4096", "kind": "train", "dtype": "bf16", "rows": 4096, "k": 1024, "n": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sizes(rng, lo, hi, most):
    """m, n, k spread over the logarithm of the range, with at most `most` multiply-adds."""
    while True:
        s = [_log(rng, lo, hi) for _ in range(3)]
        if s[0] * s[1] * s[2] <= most:
            return s


def _up(x, to):
    return (x + to - 1) // to * to


def draw(rng):
    kind = rng.choice(["half", "half", "half", "batch", "fp32", "split", "fp8", "linear", "train", "grouped", "quantize"])
    layout = rng.choice(["NN", "NT", "TN", "TT"])
    beta = rng.choice([0.0, 0.0, 0.5])
    half = rng.choice(["bf16", "fp16"])
    if kind == "fp32":
        m, n, k = _sizes(rng, 64, 6144, 4096 ** 3)
        c = _gemm("", "fp32", layout, m, n, k, beta=beta, pad=rng.choice([0, 0, 64]))
    elif kind == "half":
        m, n, k = _sizes(rng, 64, 8192, 6144 ** 3)
        if rng.random() < 0.85:      # most programs keep rows on 16-byte boundaries; some do not
            m, n, k = _up(m, 8), _up(n, 8), _up(k, 8)
        elif m * n * k > 2048 ** 3:
            m, n, k = m // 4 + 1, n // 4 + 1, k // 4 + 1
        c = _gemm("", half, layout, m, n, k, beta=beta)
    elif kind == "batch":
        m, n, k = (_up(x, 8) for x in _sizes(rng, 64, 2048, 1024 ** 3))
        c = _gemm("", half, layout, m, n, k, beta=beta, batch=rng.randint(2, 32))
    elif kind == "split":
        m, n, k = (_up(x, 8) for x in _sizes(rng, 256, 8192, 4096 ** 3))
        c = _gemm("", "fp32", layout, m, n, k, beta=beta, kernel=rng.choice(["bf16x3", "bf16x6"]), dist="uniform")
    elif kind == "fp8":
        m, n, k = (_up(x, 16) for x in _sizes(rng, 128, 8192, 8192 ** 3))
        c = _gemm("", "fp8", "TN", m, n, k)
    elif kind == "linear":
        c = {"kind": "linear", "dtype": half, "rows": _log(rng, 1, 4096), "k": _up(_log(rng, 128, 8192), 8),
             "n": _up(_log(rng, 128, 8192), 8), "activation": rng.choice(["none", "relu", "gelu", "silu"])}
    elif kind == "train":
        c = {"kind": "train", "dtype": half, "rows": _up(_log(rng, 64, 8192), 8), "k": _up(_log(rng, 128, 4096), 8),
             "n": _up(_log(rng, 128, 4096), 8)}
    elif kind == "grouped":
        c = {"kind": "grouped", "dtype": half, "layout": rng.choice(["NN", "TN"]), "count": rng.randint(4, 256),
             "most": 16 * rng.randint(16, 128), "most_k": 64 * rng.randint(8, 64), "shape_seed": rng.randrange(1 << 20)}
    else:
        c = {"kind": "quantize", "dtype": rng.choice(["bf16", "fp16", "fp32"]), "count": _log(rng, 4096, 1 << 26)}
    c.pop("name", None)
    return c


def _shapes(case):
    """(rows, columns) in storage order and leading dimensions of A, B and C/D, column-major."""
    m, n, k, pad = case["m"], case["n"], case["k"], case["pad"]
    ta, tb = case["layout"][0] == "T", case["layout"][1] == "T"
    ra, ca = (k, m) if ta else (m, k)
    rb, cb = (n, k) if tb else (k, n)
    return ta, tb, (ra, ca, ra + pad), (rb, cb, rb + pad), m + pad


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _values(g, count, dist):
    if dist == "uniform":
        return torch.rand(count, device="cuda", generator=g).mul_(2).sub_(1)
    return torch.randn(count, device="cuda", generator=g)


def _fp8(x):
    """Per-tensor E4M3 quantisation in plain torch: (values, scale)."""
    amax = float(x.abs().max())
    return (x * (448.0 / amax)).clamp_(-448, 448).to(torch.float8_e4m3fn), amax / 448.0


def _operands(case, seed):
    """A, B (flat, storage type), C or None, and the FP8 scales."""
    g = _gen(seed)
    _, _, (_, ca, lda), (_, cb, ldb), ldc = _shapes(case)
    batch, dt = case["batch"], case["dtype"]
    sa = sb = 1.0
    if dt == "fp8":
        A, sa = _fp8(_values(g, batch * lda * ca, case["dist"]))
        B, sb = _fp8(_values(g, batch * ldb * cb, case["dist"]))
    else:
        A = _values(g, batch * lda * ca, case["dist"]).to(TORCH[dt])
        B = _values(g, batch * ldb * cb, case["dist"]).to(TORCH[dt])
    C = None
    if case["beta"] != 0.0:
        C = torch.randn(batch * ldc * case["n"], device="cuda", generator=g).to(_out(case))
    return A, B, C, sa, sb


def _out(case):
    return torch.bfloat16 if case["dtype"] == "fp8" else TORCH[case["dtype"]]


def _group_sizes(case):
    r = np.random.default_rng(case["shape_seed"])
    count, top, top_k = case["count"], case["most"] // 16, case["most_k"] // 64
    M = 16 * r.integers(4, top + 1, count)
    N = 16 * r.integers(4, top + 1, count)
    K = 64 * r.integers(1, top_k + 1, count)
    return [(int(a), int(b), int(c)) for a, b, c in zip(M, N, K)]


def _group_operands(case, seed):
    sizes = _group_sizes(case)
    g = _gen(seed)
    dt = TORCH[case["dtype"]]
    A = torch.randn(sum(m * k for m, _, k in sizes), device="cuda", generator=g).to(dt)
    B = torch.randn(sum(n * k for _, n, k in sizes), device="cuda", generator=g).to(dt)
    return (sizes, A.split([m * k for m, _, k in sizes]), B.split([n * k for _, n, k in sizes]))


def _rows(case, seed, scale):
    """X (rows, k), W (k, n) and a third generator draw's source."""
    g = _gen(seed)
    dt = TORCH[case["dtype"]]
    X = (torch.randn(case["rows"], case["k"], device="cuda", generator=g) * scale).to(dt)
    W = (torch.randn(case["k"], case["n"], device="cuda", generator=g) * scale).to(dt)
    return X, W, g, dt


def _linear_inputs(case, seed):
    X, W, g, dt = _rows(case, seed, 1.0)
    W = (W.float() / math.sqrt(case["k"])).to(dt)
    return X, W, torch.randn(case["n"], device="cuda", generator=g).to(dt)


def _train_inputs(case, seed):
    X, W, g, dt = _rows(case, seed, 0.02)
    return X, W, torch.randn(case["rows"], case["n"], device="cuda", generator=g).to(dt)


def prepare(case, seed):
    h = tl.default_handle()
    kind = case["kind"]
    if kind == "gemm":
        ta, tb, (_, _, lda), (_, _, ldb), ldc = _shapes(case)
        A, B, C, sa, sb = _operands(case, seed)
        od = _out(case)
        p = tl.Problem.make(case["m"], case["n"], case["k"], dtype=case["dtype"], out_dtype=tl.torch_dtype_code(od),
                            trans_a=ta, trans_b=tb, alpha=case["alpha"], beta=case["beta"], lda=lda, ldb=ldb, ldc=ldc,
                            ldd=ldc, batch=case["batch"], kernel=case["kernel"], scale_a=sa, scale_b=sb)
        D = torch.zeros(case["batch"] * ldc * case["n"], dtype=od, device="cuda")
        return {"kind": kind, "h": h, "p": p, "A": A, "B": B, "C": C, "D": D}
    if kind == "linear":
        X, W, b = _linear_inputs(case, seed)
        return {"kind": kind, "X": X, "W": W, "b": b, "activation": case["activation"]}
    if kind == "train":
        X, W, dY = _train_inputs(case, seed)
        return {"kind": kind, "X": X.requires_grad_(), "W": W.requires_grad_(), "dY": dY}
    if kind == "grouped":
        sizes, A, B = _group_operands(case, seed)
        ta = case["layout"] == "TN"
        D = torch.zeros(sum(m * n for m, n, _ in sizes), dtype=TORCH[case["dtype"]], device="cuda")
        probs = [tl.Problem.make(m, n, k, dtype=case["dtype"], trans_a=ta, kernel="tcgen05") for m, n, k in sizes]
        plan = h.grouped_plan(probs, list(D.split([m * n for m, n, _ in sizes])), None, list(A), list(B))
        return {"kind": kind, "plan": plan, "D": D}
    src = (torch.randn(case["count"], device="cuda", generator=_gen(seed))).to(TORCH[case["dtype"]])
    return {"kind": kind, "h": h, "src": src, "code": tl.torch_dtype_code(src.dtype), "n": case["count"],
            "dst": torch.zeros(case["count"], dtype=torch.uint8, device="cuda"),
            "scale": torch.zeros(1, device="cuda"), "amax": torch.zeros(1, device="cuda")}


def run(state):
    kind = state["kind"]
    if kind == "gemm":
        state["h"].gemm(state["p"], state["D"], state["C"], state["A"], state["B"])
        return state["D"]
    if kind == "linear":
        return tl.linear(state["X"], state["W"], state["b"], activation=state["activation"])
    if kind == "train":
        Y = tl.matmul(state["X"], state["W"])
        dX, dW = torch.autograd.grad(Y, (state["X"], state["W"]), state["dY"])
        return {"Y": Y, "dX": dX, "dW": dW}
    if kind == "grouped":
        state["plan"].launch()
        return state["D"]
    state["h"].quantize_fp8(state["src"], state["n"], state["dst"], state["scale"], state["amax"],
                            src_dtype=state["code"])
    return {"fp8": state["dst"], "scale": state["scale"], "amax": state["amax"]}


def work(case):
    kind = case["kind"]
    es = BYTES[case["dtype"]]
    if kind == "gemm":
        m, n, k, b = case["m"], case["n"], case["k"], case["batch"]
        od = 2 if case["dtype"] == "fp8" else es
        return {"bytes": b * ((m * k + k * n) * es + m * n * od * (2 if case["beta"] != 0.0 else 1)),
                "flops": 2.0 * m * n * k * b}
    if kind == "linear":
        r, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": es * (r * k + k * n + n + r * n), "flops": 2.0 * r * k * n}
    if kind == "train":
        r, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": es * (2 * r * k + 2 * k * n + 2 * r * n), "flops": 6.0 * r * k * n}
    if kind == "grouped":
        s = _group_sizes(case)
        return {"bytes": es * sum(m * k + k * n + m * n for m, n, k in s), "flops": 2.0 * sum(m * n * k for m, n, k in s)}
    return {"bytes": (es + 1) * case["count"], "flops": 2.0 * case["count"]}


def _matrix(flat, rows, cols, ld, batch):
    """A column-major batch as (batch, rows, cols) in 64 bits."""
    return flat.view(batch, cols, ld)[:, :, :rows].transpose(1, 2).double()


def exact(case, seed):
    kind = case["kind"]
    if kind == "gemm":
        ta, tb, (ra, ca, lda), (rb, cb, ldb), ldc = _shapes(case)
        A, B, C, sa, sb = _operands(case, seed)
        m, n, batch = case["m"], case["n"], case["batch"]
        a, b = _matrix(A, ra, ca, lda, batch), _matrix(B, rb, cb, ldb, batch)
        a, b = (a.transpose(1, 2) if ta else a), (b.transpose(1, 2) if tb else b)
        d = float(np.float32(case["alpha"])) * sa * sb * (a @ b)
        if C is not None:
            d += float(np.float32(case["beta"])) * _matrix(C, m, n, ldc, batch)
        out = torch.zeros(batch, n, ldc, dtype=torch.float64, device="cuda")
        out[:, :, :m] = d.transpose(1, 2)
        return out.view(-1)
    if kind == "linear":
        X, W, b = _linear_inputs(case, seed)
        y = X.double() @ W.double() + b.double()
        act = case["activation"]
        if act == "relu":
            y = y.clamp(min=0)
        elif act == "gelu":
            y = torch.nn.functional.gelu(y, approximate="tanh")
        elif act == "silu":
            y = torch.nn.functional.silu(y)
        return y
    if kind == "train":
        X, W, dY = (t.double() for t in _train_inputs(case, seed))
        return {"Y": X @ W, "dX": dY @ W.T, "dW": X.T @ dY}
    if kind == "grouped":
        sizes, A, B = _group_operands(case, seed)
        outs = []
        for (m, n, k), a, b in zip(sizes, A, B):
            at = a.view(m, k).double() if case["layout"] == "TN" else a.view(k, m).t().double()
            outs.append((at @ b.view(n, k).t().double()).t().reshape(-1))
        return torch.cat(outs)
    src = (torch.randn(case["count"], device="cuda", generator=_gen(seed))).to(TORCH[case["dtype"]])
    amax = src.double().abs().max().reshape(1)
    return {"fp8": None, "scale": amax / 448.0, "amax": amax}

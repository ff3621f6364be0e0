"""Performance cases: what programs that use this library have it compute.

Each case is one pass through a public entry point of ``maxmulsk_b200`` with
everything a program holds between calls (operands, a plan, a workspace, a
grouped handle, training state) prepared before. The kinds are

* ``matmul``   C = A @ B on CUDA tensors, plan picked by the library;
* ``plan``     the same with the picked plan and workspace kept by the caller;
* ``host``     the drop-in call of the reference's C API on host buffers;
* ``grouped``  a batch of uneven GEMMs, planned once and replayed;
* ``train``    one training step of the learned plan picker.

Inputs are uniform in [-1, 1); ``dist = "normal"`` draws N(0, 1/K), the
activations-times-weights shapes with few rows.

First-call plan searches are off (MAXMULSK_AUTOTUNE=0, a documented switch): a
serving process cannot afford one on a request, and without it the same shape
runs the same plan in every process.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

os.environ.setdefault("MAXMULSK_AUTOTUNE", "0")

import maxmulsk_b200 as mm  # noqa: E402
from maxmulsk_b200 import workloads  # noqa: E402
from maxmulsk_b200.picker import F, H, NPARAM, O  # noqa: E402

PRECISION = {"fp32": mm.Precision.FP32, "tf32x3": mm.Precision.TF32X3, "bf16x6": mm.Precision.BF16X6,
             "bf16x9": mm.Precision.BF16X9, "split_auto": mm.Precision.SPLIT_AUTO}
PAD = 64            # floats between the operands of a grouped batch (256 bytes)
LR, BETA1, BETA2, EPS = 1e-3, 0.9, 0.999, 1e-8
STEP0 = 100         # Adam step at which a training state starts


def _gemm(name, kind, precision, M, K, N, dist="uniform"):
    case = {"kind": kind, "precision": precision, "M": M, "K": K, "N": N, "dist": dist}
    return case | {"name": name} if name else case


def listed():
    return [
        # The smallest product of the square sweep: call and launch latency.
        _gemm("f32_256", "matmul", "fp32", 256, 256, 256),
        # An ordinary FP32 product whose every size is odd.
        _gemm("f32_ragged", "matmul", "fp32", 777, 1531, 901),
        # The largest product of the square sweep on the FP32 path.
        _gemm("f32_4096", "matmul", "fp32", 4096, 4096, 4096),
        # The reference's own call: pageable host arrays in and out.
        _gemm("host_f32_1024", "host", "fp32", 1024, 1024, 1024),
        # Few rows times a weight matrix (decode): the smallest and the
        # largest of the narrow-M benchmark shapes.
        _gemm("x6_narrow_64x8192", "matmul", "bf16x6", 64, 8192, 512, "normal"),
        _gemm("x6_narrow_128x32768", "matmul", "bf16x6", 128, 32768, 512, "normal"),
        # The default split mode on an ordinary square.
        _gemm("tf32_2048", "matmul", "tf32x3", 2048, 2048, 2048),
        # The most exact split mode on sizes that fit no tile and no TMA row.
        _gemm("x9_ragged", "matmul", "bf16x9", 1500, 2049, 1999),
        # The headline product, plan and workspace kept by the caller.
        _gemm("auto_4096", "plan", "split_auto", 4096, 4096, 4096),
        # Batches of uneven GEMMs (the grouped benchmark's distribution).
        {"name": "grouped_f32_128", "kind": "grouped", "precision": "fp32", "count": 128, "shapes": 2026},
        {"name": "grouped_x6_256", "kind": "grouped", "precision": "bf16x6", "count": 256, "shapes": 2026},
        # One step of the picker's training on its 2000 training shapes, both
        # plan classes: forward, backward, Adam.
        {"name": "picker_train", "kind": "train", "rows": 4000},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def _size(rng, lo, hi):
    """Log-uniform; half of the sizes are rounded to a multiple of 64 (of 4
    below 128), the rest left as they fall, odd ones among them."""
    v = _log(rng, lo, hi)
    if rng.random() < 0.5:
        q = 64 if v >= 128 else 4
        v = max(q, v // q * q)
    return max(lo, min(hi, v))


def draw(rng):
    r = rng.random()
    if r < 0.30:        # FP32 products
        return _gemm(None, "matmul", "fp32", *(_size(rng, 32, 4096) for _ in range(3)))
    if r < 0.55:        # split-precision products
        prec = rng.choice(["tf32x3", "bf16x6", "bf16x9", "split_auto"])
        kind = rng.choice(["matmul", "plan"])
        return _gemm(None, kind, prec, _size(rng, 256, 4096), _size(rng, 256, 4096), _size(rng, 256, 4096))
    if r < 0.75:        # few rows, long K
        prec = rng.choice(["bf16x6", "bf16x6", "bf16x9", "fp32"])
        return _gemm(None, "matmul", prec, _log(rng, 1, 128), _size(rng, 2048, 32768), 64 * rng.randint(4, 32), "normal")
    if r < 0.83:
        return _gemm(None, "host", "fp32", _size(rng, 128, 1536), _size(rng, 128, 1536), _size(rng, 128, 1536))
    if r < 0.92:
        return {"kind": "grouped", "precision": rng.choice(["fp32", "bf16x6"]),
                "count": rng.randint(96, 128), "shapes": rng.randint(1, 1 << 20)}
    return {"kind": "train", "rows": _log(rng, 256, 8192)}


# --------------------------------------------------------------------------- inputs
def _fill(n, seed, dist, K, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    if dist == "normal":
        return torch.randn(n, generator=g, device=device, dtype=torch.float32) * (1.0 / math.sqrt(K))
    return torch.rand(n, generator=g, device=device, dtype=torch.float32) * 2.0 - 1.0


def _operands(case, seed, device="cuda"):
    M, K, N = case["M"], case["K"], case["N"]
    a = _fill(M * K, 2 * seed + 1, case["dist"], K, device).view(M, K)
    b = _fill(K * N, 2 * seed + 2, case["dist"], K, device).view(K, N)
    return a, b


def _offsets(sizes):
    out, at = [], 0
    for n in sizes:
        out.append(at)
        at += -(-n // PAD) * PAD
    return out, at


def _group(case, seed):
    """Shapes, the operand and result buffers, and where each problem's parts begin."""
    shapes = workloads.grouped_problems(case["count"], case["shapes"])
    ao, na = _offsets([m * k for m, k, n in shapes])
    bo, nb = _offsets([k * n for m, k, n in shapes])
    co, nc = _offsets([m * n for m, k, n in shapes])
    return shapes, _fill(na, 2 * seed + 1, "uniform", 1), _fill(nb, 2 * seed + 2, "uniform", 1), ao, bo, co, nc


def _train_state(case, seed):
    """A picker training state part of the way through: shapes' features, ln
    times, the candidates that ran, weights scaled by fan-in, Adam moments."""
    B = case["rows"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def u(*shape):
        return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float32)

    x = u(B, F)
    x[:, 3:6] = torch.floor(x[:, 3:6] * 16.0) / 16.0
    x[:, 6] = (torch.arange(B, device="cuda") >= B // 2).float()
    t = 4.0 + 2.5 * (x[:, :1] + x[:, 1:2] + x[:, 2:3] - 1.5) * 2.0 + 0.3 * torch.randn(B, O, generator=g, device="cuda")
    mask = (u(B, O) < 0.9).float()
    mask[: B // 2, 24:] = 0.0            # 24 candidates in the FP32 class, 48 in the other
    parts = []
    for fin, fout, bias in ((F, H, 0.0), (H, H, 0.0), (H, O, 4.0)):
        parts.append(torch.randn(fin * fout, generator=g, device="cuda") / math.sqrt(fin))
        parts.append(torch.full((fout,), bias, device="cuda"))
    params = torch.cat(parts)
    m = 1e-3 * torch.randn(NPARAM, generator=g, device="cuda")
    v = 1e-5 * (0.5 + u(NPARAM))
    return {"x": x.reshape(-1).contiguous(), "t": t.reshape(-1).contiguous(), "mask": mask.reshape(-1).contiguous(),
            "params": params, "m": m, "v": v, "count": float(mask.sum().item())}


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "train":
        s |= _train_state(case, seed)
        B = case["rows"]
        for name, n in (("z1", B * H), ("h1", B * H), ("z2", B * H), ("h2", B * H), ("y", B * O),
                        ("work", B * (O + 2 * H)), ("rowloss", B), ("grads", NPARAM)):
            s[name] = torch.empty(n, device="cuda", dtype=torch.float32)
        s["step"] = STEP0
        return s
    precision = PRECISION[case["precision"]]
    s["precision"] = precision
    if kind == "grouped":
        shapes, a, b, ao, bo, co, nc = _group(case, seed)
        s["a"], s["b"], s["c"] = a, b, torch.zeros(nc, device="cuda", dtype=torch.float32)
        problems = [(a[i:i + m * k], b[j:j + k * n], s["c"][o:o + m * n], m, k, n)
                    for (m, k, n), i, j, o in zip(shapes, ao, bo, co)]
        torch.cuda.synchronize()         # the group is planned with its buffers idle
        plan = None if precision == mm.Precision.FP32 else mm.make_plan(precision, 128, 128, 0)
        s["group"] = mm.Grouped(problems, plan)
        return s
    M, K, N = case["M"], case["K"], case["N"]
    if kind == "host":
        a, b = _operands(case, seed, "cpu")
        s["a"], s["b"], s["c"] = a.numpy(), b.numpy(), np.zeros((M, N), np.float32)
        return s
    s["a"], s["b"] = _operands(case, seed)
    if kind == "plan":
        s["plan"] = mm.choose(M, K, N, precision)
        nb = mm.workspace_bytes(M, K, N, s["plan"])
        s["ws"] = torch.empty(max(1, nb), device="cuda", dtype=torch.uint8)
        s["ws_bytes"] = nb
        s["c"] = torch.empty(M, N, device="cuda", dtype=torch.float32)
    return s


# --------------------------------------------------------------------------- one pass
def _train_step(s):
    L = mm.lib()
    B = s["case"]["rows"]
    st = torch.cuda.current_stream().cuda_stream
    p = {k: s[k].data_ptr() for k in ("x", "t", "mask", "params", "m", "v", "z1", "h1", "z2", "h2", "y", "work",
                                      "rowloss", "grads")}
    mm.check(L.maxmulsk_mlp_forward_dev(p["params"], p["x"], B, p["z1"], p["h1"], p["z2"], p["h2"], p["y"], st),
             "forward")
    mm.check(L.maxmulsk_mlp_backward_dev(p["params"], p["x"], p["z1"], p["h1"], p["z2"], p["h2"], p["y"], p["t"],
                                         p["mask"], B, s["count"], p["grads"], p["work"], p["rowloss"], st),
             "backward")
    s["step"] += 1
    mm.check(L.maxmulsk_mlp_adam_dev(p["params"], p["grads"], p["m"], p["v"], LR, BETA1, BETA2, EPS, s["step"], st),
             "adam")
    return {"y": s["y"], "rowloss": s["rowloss"], "grads": s["grads"], "params": s["params"], "m": s["m"],
            "v": s["v"]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "matmul":
        return mm.matmul(state["a"], state["b"], state["precision"])
    if kind == "train":
        return _train_step(state)
    if kind == "grouped":
        mm.check(state["group"].launch(), "grouped launch")
        return state["c"]
    M, K, N = case["M"], case["K"], case["N"]
    if kind == "plan":
        mm.check(mm.sgemm_plan_dev(state["a"], state["b"], state["c"], M, K, N, state["plan"], state["ws"],
                                   state["ws_bytes"]), "plan")
        return state["c"]
    mm.check(mm.sgemm_v3(state["a"], state["b"], state["c"], M, K, N), "v3")
    return state["c"]


# --------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    if case["kind"] == "train":
        B, weights = case["rows"], F * H + H * H + H * O
        # features, targets and mask in; predictions and losses out; weights
        # and both moments read and written, gradients written
        return {"bytes": 4 * (B * (F + 3 * O + 1) + 7 * NPARAM), "flops": 2 * B * (3 * weights - F * H)}
    if case["kind"] == "grouped":
        shapes = workloads.grouped_problems(case["count"], case["shapes"])
    else:
        shapes = [(case["M"], case["K"], case["N"])]
    return {"bytes": sum(4 * (m * k + k * n + m * n) for m, k, n in shapes),
            "flops": sum(2 * m * k * n for m, k, n in shapes)}


# --------------------------------------------------------------------------- the same in 64 bits
def _exact_train(case, seed):
    s = _train_state(case, seed)
    B = case["rows"]
    x, t, mask = (s[k].double().view(B, -1) for k in ("x", "t", "mask"))
    p = s["params"].double().requires_grad_(True)
    cuts, at = [], 0
    for n in (F * H, H, H * H, H, H * O, O):
        cuts.append(p[at:at + n])
        at += n
    w1, b1, w2, b2, w3, b3 = cuts
    gelu = torch.nn.functional.gelu
    h1 = gelu(x @ w1.view(F, H) + b1)
    h2 = gelu(h1 @ w2.view(H, H) + b2)
    y = h2 @ w3.view(H, O) + b3
    d = torch.where(mask != 0, y - t, torch.zeros_like(y))
    rowloss = (d * d).sum(1)
    (rowloss.sum() / s["count"]).backward()
    g, step = p.grad, STEP0 + 1
    with torch.no_grad():
        m = BETA1 * s["m"].double() + (1 - BETA1) * g
        v = BETA2 * s["v"].double() + (1 - BETA2) * g * g
        new = p - LR * (m / (1 - BETA1 ** step)) / ((v / (1 - BETA2 ** step)).sqrt() + EPS)
    return {"y": y.detach().reshape(-1), "rowloss": rowloss.detach(), "grads": g, "params": new.detach(), "m": m,
            "v": v}


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "grouped":
        shapes, a, b, ao, bo, co, nc = _group(case, seed)
        c = torch.zeros(nc, device="cuda", dtype=torch.float64)
        for (m, k, n), i, j, o in zip(shapes, ao, bo, co):
            c[o:o + m * n] = (a[i:i + m * k].double().view(m, k) @ b[j:j + k * n].double().view(k, n)).reshape(-1)
        return c
    if case["kind"] == "host":
        a, b = _operands(case, seed, "cpu")
        return a.double().numpy() @ b.double().numpy()
    a, b = _operands(case, seed)
    return a.double() @ b.double()

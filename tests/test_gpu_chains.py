"""Calls that follow one another with nothing between them: each reads what the
call before it wrote and reuses its workspace, and gives what the same calls give
with the device waited for after each."""
import ctypes

import pytest

import maxmulsk_b200 as mm
from maxmulsk_b200 import picker

pytestmark = pytest.mark.gpu

# Sequences of plans, each call's C the next call's A.
PLANS = {
    "fused_simt": [(2, 128, 128, 0, 2), (0, 64, 64, 4, 0), (3, 128, 128, 1, 2), (0, 128, 64, 1, 0)],
    "pair_prepass": [(2, 256, 256, 1, 0), (1, 128, 256, 4, 0), (3, 256, 128, 2, 0), (1, 128, 128, 1, 0)],
    "gemm_fused": [(2, 128, 256, 2, 0), (2, 128, 128, 4, 2), (1, 256, 256, 1, 0), (2, 128, 128, 1, 2)],
    "simt_reduce": [(0, 128, 128, 2, 0), (0, 64, 64, 8, 0), (0, 128, 64, 16, 1), (1, 128, 64, 4, 0)],
}


def _run_and_compare(torch, calls, reset, results, graph=False):
    """calls: a list of functions that issue one call each."""
    reset()
    torch.cuda.synchronize()
    for c in calls:
        c()
        torch.cuda.synchronize()
    want = [r.clone() for r in results]
    s = torch.cuda.Stream()
    reset()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        if graph:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                for c in calls:
                    c()
            g.replay()
        else:
            for c in calls:
                c()
    torch.cuda.synchronize()
    assert mm.stream_status() == 0
    for w, r in zip(want, results):
        assert torch.isfinite(w).all()
        assert torch.equal(w, r)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("M", [33, 64, 200, 1300])
@pytest.mark.parametrize("name", sorted(PLANS))
def test_dependent_calls_on_one_workspace(cuda, name, M, graph):
    torch = cuda
    K = 768
    plans = [mm.make_plan(*p) for p in PLANS[name]] * 3
    nb = max(mm.workspace_bytes(M, K, K, p) for p in plans)
    ws = torch.empty(nb + 256, dtype=torch.uint8, device="cuda")
    wp = ws.data_ptr() + (-ws.data_ptr()) % 256
    src = torch.randn(M, K, device="cuda")
    W = torch.randn(2, K, K, device="cuda") / K ** 0.5
    buf = [torch.empty(M, K, device="cuda") for _ in range(len(plans) + 1)]

    def reset():
        ws.fill_(255)                       # NaN partials, busy-looking counters
        for b in buf:
            b.fill_(float("nan"))
        buf[0].copy_(src)

    def call(i):
        assert mm.sgemm_plan_dev(buf[i], W[i % 2], buf[i + 1], M, K, K, plans[i], wp, nb) == 0, mm.last_error_message()

    _run_and_compare(torch, [lambda i=i: call(i) for i in range(len(plans))], reset, buf, graph)


@pytest.mark.parametrize("plan", [None, (0, 64, 64, 3, 0), (2, 128, 128, 0, 0), (3, 128, 128, 3, 0)])
def test_dependent_grouped_launches(cuda, plan):
    # Two groups that read each other's results: wide, slim, repacked-A (K not a
    # multiple of 4) and FP32 (N not a multiple of 4) problems in each.
    torch = cuda
    sizes = [(200, 768), (33, 768), (64, 2048), (9, 2048), (300, 514), (40, 513), (7, 1000), (513, 256), (16, 256)]
    x, y = ([torch.empty(m, k, device="cuda") for m, k in sizes] for _ in range(2))
    src = [torch.randn(m, k, device="cuda") for m, k in sizes]
    W = [[torch.randn(k, k, device="cuda") / k ** 0.5 for _, k in sizes] for _ in range(2)]
    p = mm.make_plan(*plan) if plan else None
    groups = []
    for a, b, w in ((x, y, W[0]), (y, x, W[1])):
        for t, s in zip(a, src):
            t.copy_(s)
        torch.cuda.synchronize()
        groups.append(mm.Grouped([(a[i], w[i], b[i], m, k, k) for i, (m, k) in enumerate(sizes)], p))

    def reset():
        for t, u, s in zip(x, y, src):
            t.copy_(s)
            u.fill_(float("nan"))

    def call(i):
        assert groups[i % 2].launch() == 0

    try:
        _run_and_compare(torch, [lambda i=i: call(i) for i in range(6)], reset, x + y)
    finally:
        for g in groups:
            g.close()


@pytest.mark.parametrize("B", [5, 300, 4000])
def test_training_steps_back_to_back(cuda, B):
    # Adam reads a step's gradients, and the next step's forward pass the weights
    # that Adam wrote.
    torch = cuda
    F, H, O, P = picker.F, picker.H, picker.O, picker.NPARAM
    X, T = torch.rand(B * F, device="cuda"), torch.rand(B * O, device="cuda") + 3
    mask = (torch.rand(B * O, device="cuda") < 0.9).float()
    p0 = torch.randn(P, device="cuda") * 0.2
    params, m, v, grads = (torch.empty(P, device="cuda") for _ in range(4))
    z1, h1, z2, h2 = (torch.empty(B * H, device="cuda") for _ in range(4))
    y, work, loss = torch.empty(B * O, device="cuda"), torch.empty(B * (O + 2 * H), device="cuda"), torch.empty(B, device="cuda")
    count = float(mask.sum().item())
    L = mm.lib()

    def reset():
        params.copy_(p0)
        m.zero_()
        v.zero_()

    def step(i):
        st = torch.cuda.current_stream().cuda_stream
        a = lambda *t: [ctypes.c_void_p(q.data_ptr()) for q in t]                         # noqa: E731
        assert L.maxmulsk_mlp_forward_dev(*a(params, X), B, *a(z1, h1, z2, h2, y), st) == 0
        assert L.maxmulsk_mlp_backward_dev(*a(params, X, z1, h1, z2, h2, y, T, mask), B, count, *a(grads, work, loss), st) == 0
        assert L.maxmulsk_mlp_adam_dev(*a(params, grads, m, v), 1e-3, 0.9, 0.999, 1e-8, i + 1, st) == 0

    _run_and_compare(torch, [lambda i=i: step(i) for i in range(8)], reset, [params, m, v, grads, y, loss])

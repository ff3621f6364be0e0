"""Kernels that start beside their predecessor's tail still follow the stream's
order: operands rewritten by other kernels just before a call and results read
just after, call after call with one workspace, on a stream of its own and in a
graph, give what the same calls give one at a time."""
import pytest

import maxmulsk_b200 as mm

pytestmark = pytest.mark.gpu

# One kernel; kernel and reduction; pre-pass, GEMM and reduction on one CTA and
# on pairs; the fused kernels; tail-wave splits with arrival counters.
CASES = [((512, 512, 512), (0, 64, 64, 1, 0)), ((300, 700, 260), (0, 128, 64, 4, 0)),
         ((512, 1024, 512), (1, 128, 256, 4, 0)), ((512, 1024, 512), (2, 256, 256, 2, 0)),
         ((512, 1024, 512), (3, 128, 128, 1, 0)), ((128, 4096, 512), (2, 128, 128, 0, 2)),
         ((33, 4096, 512), (2, 128, 128, 0, 2)), ((2560, 512, 2048), (2, 128, 128, 1, 0))]


@pytest.mark.parametrize("shape,plan", CASES)
@pytest.mark.parametrize("graph", [False, True])
def test_calls_follow_the_stream_order(cuda, shape, plan, graph):
    torch = cuda
    M, K, N = shape
    p = mm.make_plan(*plan)
    srcA = torch.randn(6, M, K, device="cuda")
    srcB = torch.randn(6, K, N, device="cuda")
    nb = mm.workspace_bytes(M, K, N, p)
    ws = torch.empty(nb + 256, dtype=torch.uint8, device="cuda")
    wp = ws.data_ptr() + (-ws.data_ptr()) % 256
    want = []
    for a, b in zip(srcA, srcB):
        c = torch.empty(M, N, device="cuda")
        assert mm.sgemm_plan_dev(a, b, c, M, K, N, p, wp, nb) == 0, mm.last_error_message()
        torch.cuda.synchronize()
        want.append(c)
    A, B, C = torch.empty(M, K, device="cuda"), torch.empty(K, N, device="cuda"), torch.empty(M, N, device="cuda")
    got = torch.zeros(18, M, N, device="cuda")

    def calls():
        for i in range(18):
            A.copy_(srcA[i % 6])
            B.copy_(srcB[i % 6])
            assert mm.sgemm_plan_dev(A, B, C, M, K, N, p, wp, nb) == 0
            got[i].copy_(C)
            C.fill_(float("nan"))

    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        if graph:
            calls()
            s.synchronize()
            got.zero_()
            s.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                calls()
            g.replay()
        else:
            calls()
    torch.cuda.synchronize()
    assert mm.stream_status() == 0
    for i in range(18):
        assert torch.equal(got[i], want[i % 6]), i

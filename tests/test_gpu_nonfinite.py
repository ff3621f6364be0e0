"""Infinities and NaN stay in the rows and columns that hold them: the zeros that
kernels multiply past a matrix's edge, or past a K slice, reach no other output."""
import numpy as np
import pytest

import maxmulsk_b200 as mm

pytestmark = pytest.mark.gpu

INF, NAN = float("inf"), float("nan")
# Rows that fill no tile, K past no stage or slice border, N past no tile.
SHAPES = [(5, 132, 260), (17, 1028, 132), (64, 516, 388), (65, 132, 132), (130, 260, 260)]
FP32 = [(0, m, n, s, v) for m, n in ((64, 64), (128, 64), (128, 128)) for s in (1, 3) for v in (0, 1)]
SPLIT = [(2, 128, 128, 1, 2), (2, 128, 128, 4, 2), (3, 128, 128, 0, 2), (1, 128, 128, 1, 0), (2, 256, 256, 1, 0),
         (3, 128, 64, 3, 0)]


def _operands(torch, M, K, N, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    A = torch.randn(M, K, generator=g, device="cuda")
    B = torch.randn(K, N, generator=g, device="cuda")
    # Rows of A and columns of B that get non-finite values, at K's first, last and
    # middle steps.
    return A, B, [(M - 1, K - 1, NAN), (1, 0, INF)], [(K - 1, N - 1, -INF), (K // 2, 2, NAN)]


def _run(torch, A, B, p):
    (M, K), N = A.shape, B.shape[1]
    nb = mm.workspace_bytes(M, K, N, p)
    ws = torch.full((nb + 256,), 255, dtype=torch.uint8, device="cuda")     # NaN where it is read
    C = torch.full((M, N), 3.75, device="cuda")
    wp = ws.data_ptr() + (-ws.data_ptr()) % 256
    assert mm.sgemm_plan_dev(A, B, C, M, K, N, p, wp, nb) == 0, mm.last_error_message()
    assert mm.stream_status() == 0
    return C


@pytest.mark.parametrize("shape", SHAPES + [(33, 37, 71), (130, 259, 201)])
@pytest.mark.parametrize("plan", FP32)
def test_fp32_outputs_are_finite_infinite_or_nan_as_in_fp64(cuda, shape, plan):
    torch = cuda
    A, B, at_a, at_b = _operands(torch, *shape, 7)
    for r, k, v in at_a:
        A[r, k] = v
    for k, c, v in at_b:
        B[k, c] = v
    C = _run(torch, A, B, mm.make_plan(*plan)).cpu().numpy().astype(np.float64)
    with np.errstate(all="ignore"):
        a, b = A.cpu().numpy().astype(np.float64), B.cpu().numpy().astype(np.float64)
        want = (a[:, :, None] * b[None]).sum(1)
    assert np.array_equal(np.isnan(C), np.isnan(want))
    assert np.array_equal(np.where(np.isinf(C), np.sign(C), 0), np.where(np.isinf(want), np.sign(want), 0))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("plan", SPLIT)
def test_split_modes_keep_non_finite_values_in_their_rows_and_columns(cuda, shape, plan):
    torch = cuda
    p = mm.make_plan(*plan)
    A, B, at_a, at_b = _operands(torch, *shape, 8)
    clean = _run(torch, A, B, p)
    bad = torch.zeros(clean.shape, dtype=torch.bool, device="cuda")
    for r, k, v in at_a:
        A[r, k] = v
        bad[r] = True
    for k, c, v in at_b:
        B[k, c] = v
        bad[:, c] = True
    C = _run(torch, A, B, p)
    assert not torch.isfinite(C[bad]).any()
    assert torch.equal(C[~bad], clean[~bad]) and torch.isfinite(clean).all()


def test_grouped_launches_keep_non_finite_values_in_their_rows_and_columns(cuda):
    torch = cuda
    for plan in (None, mm.make_plan(2, 128, 128, 3), mm.make_plan(0, 64, 64, 2)):
        ops = [_operands(torch, *s, 9) for s in SHAPES + [(3, 300, 513)]]
        C = [torch.empty(A.shape[0], B.shape[1], device="cuda") for A, B, _, _ in ops]
        g = mm.Grouped([(A, B, c, A.shape[0], A.shape[1], B.shape[1]) for (A, B, _, _), c in zip(ops, C)], plan)
        try:
            torch.cuda.synchronize()
            assert g.launch() == 0
            torch.cuda.synchronize()
            clean = [c.clone() for c in C]
            for A, B, at_a, at_b in ops:
                for r, k, v in at_a:
                    A[r, k] = v
                for k, c, v in at_b:
                    B[k, c] = v
            torch.cuda.synchronize()
            assert g.launch() == 0
            torch.cuda.synchronize()
            for (A, B, at_a, at_b), c, w in zip(ops, C, clean):
                bad = torch.zeros(c.shape, dtype=torch.bool, device="cuda")
                for r, _, _ in at_a:
                    bad[r] = True
                for _, n, _ in at_b:
                    bad[:, n] = True
                assert not torch.isfinite(c[bad]).any()
                assert torch.equal(c[~bad], w[~bad])
        finally:
            g.close()

"""The split-K reduction kernels at the edges of their dispatch (batch of
slices in flight, outputs per thread, columns per block), bit for bit: the
slices' partial products summed in slice order with FP32 adds."""
import numpy as np
import pytest

import maxmulsk_b200 as mm
from gpu_util import bits, run_plan

pytestmark = pytest.mark.gpu


# Slice counts around the batch sizes; C of a size that is summed one output
# per thread (small, odd, misaligned) and four per thread (552 x 552).
@pytest.mark.parametrize("splits", [3, 4, 5, 8, 9, 16, 17, 64])
@pytest.mark.parametrize("M,N,offset", [(65, 67, 0), (552, 552, 0), (552, 552, 1), (553, 555, 0)])
def test_simt_reduction_sums_slices_in_order(cuda, oracle_mod, splits, M, N, offset):
    K = 32 * splits
    A, B = oracle_mod.fill_uniform(M * K, 5), oracle_mod.fill_uniform(K * N, 6)
    st, C, bands = run_plan(cuda, A, B, M, K, N, mm.make_plan(mm.Precision.FP32, 64, 64, splits), offset=offset)
    assert st == 0 and bands, mm.last_error_message()
    assert np.array_equal(bits(C), bits(oracle_mod.sgemm_panels(A, B, M, K, N, kc=32, fma=True)))


# One or 32 columns per block by the number of tiles; 64 to 256 columns a tile,
# one- and two-CTA tiles; C edges inside a block.
@pytest.mark.parametrize("splits", [3, 5, 9, 17])
@pytest.mark.parametrize("tile", [(128, 64), (128, 128), (128, 256), (256, 128), (256, 256)])
@pytest.mark.parametrize("M,N", [(67, 45), (650, 1283)])
def test_tc_reduction_sums_slices_in_order(cuda, oracle_mod, splits, tile, M, N):
    K = 32 * splits
    A = oracle_mod.fill_uniform(M * K, 7)
    B = oracle_mod.fill_uniform(K * N, 8)
    plan = mm.make_plan(mm.Precision.BF16X6, tile[0], tile[1], splits, chunk=32)
    st, C, bands = run_plan(cuda, A, B, M, K, N, plan)
    assert st == 0 and bands, mm.last_error_message()
    whole = mm.make_plan(mm.Precision.BF16X6, tile[0], tile[1], 1, chunk=32)
    ref = None
    for z in range(splits):
        a = np.ascontiguousarray(A.reshape(M, K)[:, 32 * z:32 * z + 32])
        b = np.ascontiguousarray(B.reshape(K, N)[32 * z:32 * z + 32])
        st, part, _ = run_plan(cuda, a, b, M, 32, N, whole)
        assert st == 0
        ref = part if ref is None else ref + part
    assert np.array_equal(bits(C), bits(ref))

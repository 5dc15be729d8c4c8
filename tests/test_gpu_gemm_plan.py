"""GPU parity of the tensor-core trellis GEMM (decoded weights as the M operand of tcgen05.mma) against the CPU
oracle, with the k split and the tile height forced so that every path runs at its edges: one token in the last
tile, two accumulators, more CTAs in a cluster than tokens, slices of k of unequal length, several passes of the
epilogue. Tolerance 1e-2 of the largest value, as for the other linears."""
import numpy as np
import pytest

from conftest import make_linear
from test_gpu_parity import check_close, gemm_status, run_gemm

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def amp():
    import ampstein_b200
    return ampstein_b200


@pytest.mark.parametrize("m,k,n,K,cb,split,tile", [
    (17, 128, 128, 4, 0, 1, 0), (17, 128, 128, 1, 1, 2, 0), (33, 640, 256, 3, 2, 3, 32), (18, 512, 384, 5, 0, 8, 0),
    (129, 896, 128, 6, 1, 5, 128), (256, 256, 128, 8, 2, 4, 256), (257, 384, 256, 2, 0, 1, 272), (500, 1024, 128, 7, 0, 4, 512),
    (300, 256, 640, 4, 1, 2, 304), (512, 512, 128, 3, 0, 8, 512), (97, 1152, 128, 5, 1, 7, 16), (1030, 256, 128, 4, 2, 1, 0)])
def test_forced_plans(amp, oracle, m, k, n, K, cb, split, tile):
    from ampstein_b200 import _lib
    trellis, suh, svh, x = make_linear(k, n, K, seed=8300 + m + K, m=m)
    svh = (svh.astype(np.float32) / (1.2437 * np.sqrt(k))).astype(np.float16)
    ref = oracle.linear(x, trellis, suh, svh, cb, fp32_out=True)
    _lib.lib().amp_exl3_set_gemm_plan(split, tile)
    try:
        for fp32 in (False, True):
            got = run_gemm(amp, trellis, suh, svh, x, cb, fp32=fp32)
            assert gemm_status() == 0
            check_close(got, ref)
        again = run_gemm(amp, trellis, suh, svh, x, cb, fp32=True)
        assert np.array_equal(got, again)                # fixed order of the partial sums
    finally:
        _lib.lib().amp_exl3_set_gemm_plan(0, 0)

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
    (300, 256, 640, 4, 1, 2, 304), (512, 512, 128, 3, 0, 8, 512), (97, 1152, 128, 5, 1, 7, 16), (1030, 256, 128, 4, 2, 1, 0),
    (65, 384, 256, 2, 2, 3, 0), (130, 640, 128, 2, 1, 2, 0)])
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


# Pairs with k split over two to four of them: few rows, two accumulators, slices of unequal length, several passes of the
# epilogue, several tiles, more than one pair of column blocks
@pytest.mark.parametrize("m,k,n,K,cb,split,tile", [
    (17, 256, 256, 4, 0, 2, 32), (33, 640, 512, 3, 2, 3, 48), (300, 1152, 256, 5, 1, 4, 304), (512, 512, 256, 2, 0, 2, 512),
    (500, 896, 768, 6, 0, 4, 256), (1030, 256, 256, 4, 2, 4, 512), (47, 1024, 1280, 8, 1, 3, 16)])
def test_forced_pair_splits(amp, oracle, m, k, n, K, cb, split, tile):
    from ampstein_b200 import _lib
    trellis, suh, svh, x = make_linear(k, n, K, seed=9100 + m + K, m=m)
    svh = (svh.astype(np.float32) / (1.2437 * np.sqrt(k))).astype(np.float16)
    ref = oracle.linear(x, trellis, suh, svh, cb, fp32_out=True)
    old = _lib.lib().amp_exl3_set_gemm_pair(2)
    _lib.lib().amp_exl3_set_gemm_plan(split, tile)
    try:
        for fp32 in (False, True):
            got = run_gemm(amp, trellis, suh, svh, x, cb, fp32=fp32)
            assert gemm_status() == 0
            check_close(got, ref)
        assert np.array_equal(got, run_gemm(amp, trellis, suh, svh, x, cb, fp32=True))
    finally:
        _lib.lib().amp_exl3_set_gemm_plan(0, 0)
        _lib.lib().amp_exl3_set_gemm_pair(old)


# Either form of the rotation kernel in front of the GEMM (one warp per chunk; eight rows per warp from 6400 chunks on, walking all
# sources from 2560 tasks on), read back from the caller's scratch: bit-exact against the stand-alone Hadamard. Row counts around
# multiples of eight; an input that is only 8-byte aligned.
@pytest.mark.parametrize("m,k,sources,bf16,offset", [
    (17, 4096, 1, False, 0), (199, 4096, 1, False, 0), (201, 4096, 1, True, 0), (207, 4096, 1, False, 4), (81, 4096, 3, False, 0),
    (70, 4096, 3, True, 0), (641, 4096, 3, False, 0), (639, 4096, 2, True, 0), (1025, 1024, 1, True, 4), (6401, 128, 1, False, 0)])
def test_rotation_forms(amp, m, k, sources, bf16, offset):
    dt = torch.bfloat16 if bf16 else torch.float16
    x = torch.randn(m * k + offset, device="cuda").to(dt)[offset:].view(1, m, k)
    n, K = 128, 4
    tr = torch.randint(-32768, 32768, (sources, k // 16, n // 16, 16 * K), dtype=torch.int16, device="cuda")
    suh = torch.randn(sources, k, device="cuda").to(torch.float16)
    svh = torch.ones(sources, n, dtype=torch.float16, device="cuda")
    had = torch.empty(sources, m, k, dtype=torch.float16, device="cuda")
    out = torch.empty(sources, m, n, dtype=torch.float16, device="cuda")
    tables = [amp.ptr_array([t[i].data_ptr() for i in range(sources)]) for t in (tr, suh, svh)]
    amp.mgemm(x, tables[0], out, tables[1], had, tables[2], K, False, False)
    assert gemm_status() == 0
    row, piece = torch.arange(m, device="cuda").view(1, m, 1), torch.arange(8, device="cuda")
    for i in range(sources):
        ref = torch.empty(m, k, dtype=torch.float16, device="cuda")
        amp.had_r_128(x[0].float() if bf16 else x[0], ref, pre_scale=suh[i])      # (bf16 rows: scaled and rotated in fp32)
        got = had[i].view(k // 64, m, 8, 8)                  # (k step, row, 16-byte piece, value); piece p lies at p ^ (row & 7)
        got = got.gather(2, (piece ^ (row & 7)).view(1, m, 8, 1).expand(k // 64, m, 8, 8))
        assert torch.equal(got.permute(1, 0, 2, 3).reshape(m, k).view(torch.int16), ref.view(torch.int16))


# The rotation kernel moves in under the GEMM in front of it: a chain of linears that read each other's output through ONE
# scratch for the rotated input gives the bits of the same chain without dependent launches. Either rotation form (6400 chunks),
# every GEMM form, and decode launches (8 rows) in between.
@pytest.mark.parametrize("rows", [(17, 17, 17), (77, 8, 77), (300, 600, 300), (900, 900, 900)])
def test_dependent_rotations(amp, rows):
    from ampstein_b200 import _lib
    k, K = 1024, 4
    g = torch.Generator(device="cuda").manual_seed(5)
    tr = torch.randint(-32768, 32768, (3, k // 16, k // 16, 16 * K), dtype=torch.int16, device="cuda", generator=g)
    suh = torch.randint(0, 2, (3, k), device="cuda", generator=g).to(torch.float16) * 2 - 1
    svh = torch.full((3, k), 1.0 / (1.2437 * k ** 0.5), dtype=torch.float16, device="cuda")
    x = torch.randn(1000, k, device="cuda", generator=g).to(torch.float16)
    had = torch.empty_like(x)

    def chain():
        a, b = x.clone(), torch.zeros_like(x)
        for _ in range(8):
            for i, m in enumerate(rows):
                _lib.call("amp_exl3_gemm", a.data_ptr(), tr[i].data_ptr(), b.data_ptr(), suh[i].data_ptr(), had.data_ptr(), svh[i].data_ptr(),
                          m, k, k, K, 0, 0, torch.cuda.current_stream().cuda_stream)
                a, b = b, a
        return a, b

    got = chain()
    _lib.lib().amp_exl3_set_pdl(0)
    try:
        ref = chain()
    finally:
        _lib.lib().amp_exl3_set_pdl(1)
    assert gemm_status() == 0
    assert all(torch.equal(p.view(torch.int16), q.view(torch.int16)) for p, q in zip(got, ref))


# Splits whose clusters of three or five fill the device: behind a rotation kernel that is still leaving, the last ones start late
# (410 x 16256 x 1664: 57 us against 41). The plan is not one of them: the result has the bits of the plan named, not of that one.
@pytest.mark.parametrize("m,k,n,K,late,plan", [(410, 16256, 1664, 4, (5, 208), (4, 208)), (736, 10496, 1408, 6, (3, 192), (4, 256)),
                                               (716, 8320, 640, 4, (5, 144), (6, 192))])
def test_clusters_that_start_late_are_not_planned(amp, m, k, n, K, late, plan):
    from ampstein_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(7)
    tr = torch.randint(-32768, 32768, (k // 16, n // 16, 16 * K), dtype=torch.int16, device="cuda", generator=g)
    suh, svh = torch.ones(k, dtype=torch.float16, device="cuda"), torch.ones(n, dtype=torch.float16, device="cuda")
    x = torch.randn(m, k, device="cuda", generator=g).to(torch.float16)
    had = torch.empty_like(x)

    def run(split, tile):
        y = torch.empty(m, n, dtype=torch.float32, device="cuda")
        _lib.lib().amp_exl3_set_gemm_plan(split, tile)
        try:
            _lib.call("amp_exl3_gemm", x.data_ptr(), tr.data_ptr(), y.data_ptr(), suh.data_ptr(), had.data_ptr(), svh.data_ptr(), m, k, n, K, 0, 1,
                      torch.cuda.current_stream().cuda_stream)
        finally:
            _lib.lib().amp_exl3_set_gemm_plan(0, 0)
        return y

    got = run(0, 0)
    assert torch.equal(got, run(*plan)) and not torch.equal(got, run(*late))
    assert gemm_status() == 0

"""What a barrier wait that runs out leaves behind in the tensor-core GEMM: nothing stored by any block that depends on it
(the blocks of a k split, the other block of a pair), the status word set, and the next launch in order. The waits are
made to run out with a limit of two polls (8 us) for the last block of every cluster or pair, while the weights come from
pinned host memory, where a 64-row step of all blocks takes tens of microseconds; the other blocks wait patiently."""
import ctypes

import numpy as np
import pytest

from conftest import make_linear

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# (the last three: pairs with a k split, where a pair that gave up tells the others of its cluster; longer slices of k, so that
# each runs over several fetches from the host)
@pytest.mark.parametrize("m,n,pair,split,tile,k", [(64, 18944, 0, 1, 0, 1024), (64, 9472, 0, 2, 0, 1024), (40, 4608, 0, 4, 0, 1024), (512, 2304, 0, 8, 512, 1024),
                                                   (64, 18944, 2, 0, 0, 1024), (300, 9472, 3, 0, 0, 1024),
                                                   (64, 9472, 2, 2, 64, 2048), (200, 4608, 2, 4, 208, 8192), (512, 9472, 2, 2, 512, 4096)])
def test_nothing_is_stored_after_a_lost_wait(m, n, pair, split, tile, k):
    from ampstein_b200 import _lib
    L = _lib.lib()
    K = 8
    trellis, suh, svh, x = make_linear(k, n, K, seed=8800 + m + split, m=m)
    svh = (svh.astype(np.float32) / (1.2437 * np.sqrt(k))).astype(np.float16)
    host = torch.from_numpy(trellis.view(np.int16)).pin_memory()
    t, s, v, xx = host.cuda(), torch.from_numpy(suh).cuda(), torch.from_numpy(svh).cuda(), torch.from_numpy(x).cuda()
    had = torch.empty_like(xx)

    def run(weight):
        y = torch.full((m, n), -7.0, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        _lib.call("amp_exl3_gemm", xx.data_ptr(), weight.data_ptr(), y.data_ptr(), s.data_ptr(), had.data_ptr(), v.data_ptr(), m, k, n, K, 0, 1,
                  torch.cuda.current_stream().cuda_stream)
        st = ctypes.c_int(-1)
        _lib.call("amp_exl3_gemm_status", ctypes.byref(st))
        return y, st.value

    old = L.amp_exl3_set_gemm_pair(pair)
    L.amp_exl3_set_gemm_plan(split, tile)
    try:
        want, status = run(t)
        assert status == 0 and not bool((want == -7.0).any())
        L.amp_exl3_set_gemm_wait_limit(1 << 14, 1)
        y, status = run(host)
        assert status == 1
        # a block is left alone, or (weights that came in time) holds what it should: nothing in between
        left = y == -7.0
        assert bool((left | (y == want)).all()) and bool(left.any())
        left = left.view(m, n // 128, 128)
        assert torch.equal(left.any(2), left.all(2))
        L.amp_exl3_set_gemm_wait_limit(0, 0)
        y, status = run(host)
        assert status == 0 and torch.equal(y, want)
    finally:
        L.amp_exl3_set_gemm_wait_limit(0, 0)
        L.amp_exl3_set_gemm_plan(0, 0)
        L.amp_exl3_set_gemm_pair(old)

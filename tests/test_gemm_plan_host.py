"""LinearEXL3's per-token path (exl3.GemmPlan): what it hands to the library follows the weight as it is at the call. Host
only: the tensors claim to live on device 0 and the library call is recorded."""
import gc
import weakref

import pytest

torch = pytest.importorskip("torch")


class OnDevice(torch.Tensor):
    """A host tensor that says it is on device 0."""
    is_cuda = property(lambda self: True)

    def get_device(self):
        return 0


def on_device(t):
    return t.as_subclass(OnDevice)


@pytest.fixture
def calls(monkeypatch):
    from ampstein_b200 import _lib, exl3
    out = []
    monkeypatch.setattr(_lib, "call", lambda name, *a: out.append((name, a)))
    monkeypatch.setattr(exl3, "_get_device", lambda: 0)
    monkeypatch.setattr(exl3, "_raw_stream", lambda dev: 0)
    return out


def weight(k=256, n=384, K=4, **kw):
    from ampstein_b200.models import LinearEXL3
    w = int(16 * K)
    return LinearEXL3(on_device(torch.zeros((k // 16, n // 16, w), dtype=torch.int16)), on_device(torch.ones(k, dtype=torch.float16)),
                      on_device(torch.ones(n, dtype=torch.float16)), **kw)


def rows(m, k=256):
    return on_device(torch.zeros((m, k), dtype=torch.float16))


def last(calls):
    """trellis address, m, k, n, K, codebook of the last launch"""
    name, a = calls[-1]
    assert name == "amp_exl3_gemm"
    return (a[1],) + tuple(a[6:11])


def test_codebook_flags_are_read_at_every_call(calls):
    lin = weight()
    lin.forward(rows(2))
    assert last(calls) == (lin.trellis.data_ptr(), 2, 256, 384, 4, 0)
    lin.mul1 = True
    lin.forward(rows(2))
    assert last(calls)[-1] == 2
    lin.mul1, lin.mcg = False, True
    lin.forward(rows(2))
    assert last(calls)[-1] == 1
    lin.mul1 = True
    with pytest.raises(ValueError):
        lin.forward(rows(2))                                 # both flags


def test_a_weight_changed_in_place_is_checked_again(calls):
    lin = weight()
    lin.forward(rows(1))
    smaller = torch.zeros((16, 8, 64), dtype=torch.int16)
    lin.trellis.set_(smaller)                                # same object, other storage: n = 128
    with pytest.raises(ValueError):
        lin.forward(rows(1))                                 # svh still has 384 values
    lin.svh.resize_(128)
    y = lin.forward(rows(1))
    assert tuple(y.shape) == (1, 128) and last(calls) == (smaller.data_ptr(), 1, 256, 128, 4, 0)
    lin.trellis.resize_(16, 8, 48)                           # another bitrate
    lin.forward(rows(1))
    assert last(calls)[4] == 3
    n = len(calls)
    lin.trellis.resize_(8, 8, 48)                            # k = 128: neither the activations nor suh fit
    with pytest.raises(ValueError):
        lin.forward(rows(1))
    lin.trellis.resize_(16, 8, 48)
    lin.suh.resize_(128)
    with pytest.raises(ValueError):
        lin.forward(rows(1))
    lin.suh = on_device(torch.ones((256, 2), dtype=torch.float16)[:, 0])
    with pytest.raises(ValueError):
        lin.forward(rows(1))                                 # not contiguous
    lin.suh = on_device(torch.ones(256))
    with pytest.raises(TypeError):
        lin.forward(rows(1))
    lin.suh = None
    with pytest.raises(TypeError):
        lin.forward(rows(1))
    assert len(calls) == n                                   # nothing was launched


def test_replacing_tensors_and_half_integer_rates(calls):
    lin = weight(mul1=True)
    lin.forward(rows(3))
    lin.trellis = on_device(torch.zeros((16, 24, 40), dtype=torch.int16))       # 2.5 bits
    lin.forward(rows(3))
    assert last(calls) == (lin.trellis.data_ptr(), 3, 256, 384, 256 + 2, 2)
    lin.mul1 = False
    with pytest.raises(ValueError):
        lin.forward(rows(3))                                 # half-integer rates are mul1
    lin.trellis = on_device(torch.zeros((16, 24, 64), dtype=torch.int16))
    lin.forward(rows(3))
    assert last(calls) == (lin.trellis.data_ptr(), 3, 256, 384, 4, 0)


def test_a_replaced_weight_is_not_kept_alive(calls):
    lin = weight()
    lin.forward(rows(1))
    old = weakref.ref(lin.trellis)
    lin.trellis = None
    gc.collect()
    assert old() is None

"""CPU-only: the C-ABI library loads and exports exactly what include/ampstein_b200.h declares,
and the ctypes table binds the same set. No compute call is made."""
import ctypes
import os
import re

import pytest

from conftest import ROOT


def _declared():
    text = open(os.path.join(ROOT, "include", "ampstein_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(amp_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_are_exported_and_bound():
    from ampstein_b200 import _lib
    names = _declared()
    assert "amp_exl3_gemm" in names and "amp_exl3_reconstruct" in names
    L = ctypes.CDLL(_lib.LIB_PATH)
    for n in names:
        assert hasattr(L, n), "library does not export " + n
    bound = set(_lib.SIGNATURES) | {"amp_b200_last_error"}
    assert set(names) == bound, (sorted(set(names) - bound), sorted(bound - set(names)))
    assert _lib.lib().amp_b200_version() >= 1


def test_bad_arguments_return_codes_without_a_gpu():
    """Argument validation happens before any CUDA call, so it can be exercised here."""
    from ampstein_b200 import _lib
    L = _lib.lib()
    buf = ctypes.create_string_buffer(4096)
    p = ctypes.addressof(buf)
    p += (-p) % 16
    # K out of range
    assert L.amp_exl3_reconstruct(p, p, 16, 128, 9, 0, 0, 128, None) < 0
    assert "bitrate" in _lib.last_error()
    # n_out not a multiple of 128
    assert L.amp_exl3_reconstruct(p, p, 16, 128, 4, 0, 0, 64, None) < 0
    # slice out of bounds
    assert L.amp_exl3_reconstruct(p, p, 16, 128, 4, 0, 128, 128, None) < 0
    # gemv: m out of range, k not a multiple of 128, missing scale vectors
    assert L.amp_exl3_gemv(p, p, p, p, p, 17, 128, 128, 4, 0, 0, None) < 0
    assert L.amp_exl3_gemv(p, p, p, p, p, 1, 64, 128, 4, 0, 0, None) < 0
    assert L.amp_exl3_gemv(p, p, p, None, p, 1, 128, 128, 4, 0, 0, None) < 0
    # Hadamard: bad dtype / columns
    assert L.amp_had_r_128(p, p, None, None, 1, 128, 4, 1.0, None) < 0
    assert L.amp_had_r_128(p, p, None, None, 1, 100, 0, 1.0, None) < 0
    # empty problems are a no-op
    assert L.amp_exl3_reconstruct(p, p, 0, 128, 4, 0, 0, 128, None) == 0
    assert L.amp_had_r_128(p, p, None, None, 0, 128, 0, 1.0, None) == 0


@pytest.mark.parametrize("K", [0, 9, 16, 17, 18, 19, 20, -1, 256, 260])
def test_no_entry_takes_an_internal_bitrate_code(K):
    """The decode kernel's instances for half-integer rates have codes of their own (17..19); a caller's K of that value
    is not a bitrate, at any row count and with any entry (amp_exl3_gemv_static asks for the device first and is left out).
    The refusal comes before any CUDA call."""
    from ampstein_b200 import _lib
    L = _lib.lib()
    buf = ctypes.create_string_buffer(4096)
    p = ctypes.addressof(buf)
    p += (-p) % 16
    q = p + 1024                                             # (outputs that must not alias an input)
    bufs = (ctypes.c_void_p * 2)(p, p)
    k = n = 128
    calls = [("amp_exl3_gemv", (p, p, q, p, p, 1, k, n, K, 2, 0, None)),
             ("amp_exl3_gemv_cfg", (p, p, q, p, p, 1, k, n, K, 2, 0, 0, 0, None)),
             ("amp_exl3_gemv_allreduce", (p, p, q, p, p, 1, k, n, K, 2, bufs, bufs, 0, 2, 4096, None)),
             ("amp_exl3_gemv_allreduce_rot", (p, p, q, p, p, 1, k, n, K, 2, bufs, bufs, 0, 2, 4096, p, None)),
             ("amp_exl3_gemv_push", (p, p, p, p, 1, k, n, K, 2, bufs, bufs, 0, 2, 4096, None)),
             ("amp_exl3_gemv_gathered", (p, q, p, p, 1, k, n, K, 2, 0, p, p, 2, 4096, None)),
             ("amp_exl3_gemv_silu_mul", (p, p, p, q, p, p, 1, k, n, K, 2, 0, None)),
             ("amp_exl3_gemv_rms_norm_res", (p, p, p, 1e-5, q, p, q, p, p, 1, k, n, K, 2, 0, None)),
             ("amp_exl3_gemv_add_res", (p, p, p, p, p, q, q, 1, k, n, K, 2, None)),
             ("amp_exl3_gemv_normed", (p, p, p, 1e-5, p, q, p, p, 1, k, n, K, 2, 0, None)),
             ("amp_exl3_mgemm_normed", (p, p, p, 1e-5, p, q, p, p, 1, 1, k, n, K, 2, 0, None, None, None, None))]
    for m in (1, 8, 9, 16, 17, 600):
        calls += [("amp_exl3_gemm", (p, p, q, p, p, p, m, k, n, K, 2, 0, None)),
                  ("amp_exl3_mgemm", (p, p, q, p, p, p, 1, m, k, n, K, 2, 0, None, None, None, 0, None))]
    for name, args in calls:
        if name == "amp_exl3_gemm" and K > 256:
            continue                                         # AMP_EXL3_HALF_RATE is this entry's own; its range: below
        assert getattr(L, name)(*args) < 0, name
        assert "bitrate" in _lib.last_error(), (name, _lib.last_error())
    assert L.amp_exl3_gemm(p, p, q, p, p, p, 1, k, n, 260, 2, 0, None) < 0 and "half-integer" in _lib.last_error()


def test_python_front_end_rejects_cpu_tensors():
    import torch
    import ampstein_b200 as amp
    t = torch.zeros((8, 8, 64), dtype=torch.int16)
    w = torch.zeros((128, 128), dtype=torch.float16)
    with pytest.raises(RuntimeError):
        amp.exl3_reconstruct(w, t, 4)
    with pytest.raises(TypeError):
        amp.exl3_gemm(w, t, w, None, None)


def test_package_imports_on_a_torch_without_cuda():
    """torch's private CUDA functions do not exist in a CPU build; the package imports there, and its operators refuse
    host tensors as they do everywhere."""
    import subprocess
    import sys
    code = ("import torch\n"
            "for n in [n for n in dir(torch._C) if n.startswith('_cuda_')]: delattr(torch._C, n)\n"
            "import ampstein_b200 as amp, ampstein_b200.models\n"
            "try: amp.exl3_reconstruct(torch.zeros((128, 128), dtype=torch.float16), torch.zeros((8, 8, 64), dtype=torch.int16), 4)\n"
            "except RuntimeError as e: print('refused', e)\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("refused"), r.stderr[-2000:]

"""The C-ABI library loads without a GPU and exports every symbol include/eps_b200.h declares."""
import ctypes
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared():
    text = open(os.path.join(ROOT, "include", "eps_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(epsb_[a-z0-9_]+)\s*\(", text)))


def test_library_builds_and_exports_all_symbols():
    from eps_b200 import build
    from eps_b200._lib import SIGNATURES

    path = build.build()
    lib = ctypes.CDLL(path)
    names = _declared()
    assert len(names) >= 20
    for n in names:
        assert hasattr(lib, n), f"{n} is declared in include/eps_b200.h but not exported"
    # the Python binding covers every compute entry point of the header
    assert set(SIGNATURES) == set(names) - {"epsb_last_error", "epsb_version"}
    lib.epsb_version.restype = ctypes.c_int
    assert lib.epsb_version() >= 1


def test_argument_validation_needs_no_gpu():
    """Shape errors are raised on the host before any CUDA call (reference: std::runtime_error)."""
    import pytest

    from eps_b200._lib import EpsError, call

    with pytest.raises(EpsError, match="not divisible by group_size"):
        call("epsb_quant_1x128", None, 4, 100, None, None, 0, None)
    with pytest.raises(EpsError, match="Invalid num_stages"):
        call("epsb_source_plans", None, None, 8, 2, 12, 2, 4, None, None, None, None, None, 0, None)
    with pytest.raises(EpsError, match="K: 100 is not divisible by 128"):
        call("epsb_grouped_gemm_fp8", 0, None, None, None, None, None, 4, 16, 128, 100, None, None, None, None, 0, None)


def test_fastep_reduce_refuses_misaligned_rows():
    """Its rows may be a caller's view into a larger tensor; 16-byte loads from an odd address would fault on the device, so
    the host refuses it (the addresses here are made up: nothing is launched)."""
    import pytest

    from eps_b200._lib import EpsError, call

    a = 1 << 20
    for rows, raw, shared, out in [(a + 2, a, None, a), (a, a + 8, None, a), (a, a, a + 4, a), (a, a, a, a + 14)]:
        with pytest.raises(EpsError, match="row buffers must be 16-byte aligned"):
            call("epsb_fastep_reduce", rows, raw, shared, a, a, 4, 2, 256, out, None)


def test_gemm_kernels_have_no_static_shared_memory():
    """The GEMM kernels use their dynamic shared memory from its first byte, which is 1024-byte aligned as long as no static
    array lies before it (the host refuses the launch otherwise): what ptxas said when they were built."""
    from eps_b200 import build

    names = ("grouped_gemm", "grouped_gemm_bf16")
    logs = [os.path.join(build.OBJ_DIR, n + ".ptxas.log") for n in names]
    build.build(force=not all(os.path.exists(p) for p in logs))
    for p in logs:
        used = [line for line in open(p) if "Used" in line and "registers" in line]
        assert len(used) >= 2 and not any("smem" in line for line in used), (p, used)


def test_missing_library_fails_loudly(monkeypatch):
    import pytest

    from eps_b200 import _lib

    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", "/nonexistent/libeps_b200.so")
    with pytest.raises(_lib.EpsError, match="no CPU or PyTorch fallback"):
        _lib.lib()

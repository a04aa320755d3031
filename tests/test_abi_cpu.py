"""The C-ABI library loads without a GPU and exports every symbol include/glow_b200.h declares."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared():
    text = open(os.path.join(ROOT, "include", "glow_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(glowb200_[a-z0-9_]+)\s*\(", text)))


@pytest.fixture(scope="module")
def built():
    from glow_b200 import build
    return build.build()


def test_library_exports_every_declared_symbol(built):
    lib = ctypes.CDLL(built)
    names = _declared()
    assert len(names) >= 6
    missing = [n for n in names if not hasattr(lib, n)]
    assert not missing, missing


def test_binding_table_matches_header(built):
    from glow_b200 import _lib
    assert sorted(_lib.SIGNATURES) == _declared()
    assert _lib.lib().glowb200_version().startswith(b"glow_b200")


def test_binding_is_of_this_interpreter_and_torch(built, monkeypatch):
    """The CPython module is compiled against both: another torch in the same tree finds none, and builds its own."""
    import torch
    from glow_b200 import _lib
    path = _lib.binding_path()
    assert os.path.exists(path) and torch.__version__ in path and os.path.dirname(path) == os.path.dirname(built)
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    monkeypatch.setattr(_lib, "_binding", None)
    assert _lib.binding_path() != path
    with pytest.raises(ImportError, match="0.0.1.*build it"):
        _lib.binding(None)


def test_host_side_argument_errors_need_no_gpu(built):
    from glow_b200 import _lib
    l = _lib.lib()
    assert l.glowb200_slws_workspace_bytes(1024, 1) >= 1025 * 8
    assert l.glowb200_slws_workspace_bytes(1024, 4) == 4 * l.glowb200_slws_workspace_bytes(1024, 1)
    # in_line that does not match the column count of the kind
    rc = l.glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum(
        None, None, 0, 10, None, None, 1, None, 0, 0, 70, 64, 0, 0, None, 0, None, None)
    assert rc == 1 and b"in_line_size" in l.glowb200_last_error()
    rc = l.glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum(
        None, None, 7, 10, None, None, 1, None, 0, 0, 72, 64, 0, 0, None, 0, None, None)
    assert rc == 1
    # zero segments is a no-op that needs no device
    rc = l.glowb200_fused_rowwise_quantized_sparse_lengths_weighted_sum(
        None, None, 0, 10, None, None, 1, None, 0, 0, 72, 64, 0, 0, None, 0, None, None)
    assert rc == 0
    # Quantize + Transpose: the shuffle is checked on the host; an empty tensor is a no-op
    import ctypes as C
    dims, bad, good = (C.c_int64 * 4)(2, 3, 0, 5), (C.c_int32 * 4)(0, 2, 2, 1), (C.c_int32 * 4)(0, 2, 3, 1)
    rc = l.glowb200_quantize_transpose_i8(None, None, dims, bad, 4, C.c_float(0.1), 0, None)
    assert rc == 1 and b"permutation" in l.glowb200_last_error()
    assert l.glowb200_quantize_transpose_i8(None, None, dims, good, 4, C.c_float(0.1), 0, None) == 0
    assert l.glowb200_transpose(None, None, dims, good, 5, 1, None) == 1
    # the programmatic-launch switch is host state: set, read back, restore
    before = l.glowb200_set_programmatic_launch(0)
    assert l.glowb200_set_programmatic_launch(1) == 0
    assert l.glowb200_set_programmatic_launch(-1) == 1
    assert l.glowb200_set_programmatic_launch(before) in (0, 1)
    l.glowb200_set_programmatic_launch(-1)


@pytest.mark.parametrize("M,K,N", [(8, 64, 32), (300, 64, 32), (300, 33, 40), (300, 0, 40)])
def test_a_right_hand_side_to_turn_round_needs_its_room(built, M, K, N):
    """[K, N] products refuse a workspace without room for the N * K bytes, on the host; the size that the library names
    holds a copy of both operands, wherever they lie."""
    from glow_b200 import _lib
    l, fake, up = _lib.lib(), ctypes.c_void_p(4096), lambda v, a: (v + a - 1) // a * a
    least = up(N * 4, 256) + up(M * 4, 256) + up(N * K, 256)
    named = l.glowb200_i8_gemm_workspace_bytes(M, K, N)
    assert named >= least + up(M * up(K, 16), 256)
    for ws, size in ((None, 0), (None, named), (fake, least - 1)):
        rc = l.glowb200_matmul_i8(fake, fake, fake, M, K, N, 0, 0, 0, 0, 0, 1, 0, ws, size, None, None)
        assert rc == 3 and b"needed" in l.glowb200_last_error()
        rc = l.glowb200_fc_i8_i32(fake, fake, fake, fake, M, K, N, 0, 0, 0, 0, 0, 0, 1, 0, 0, 1, None, 0, ws, size, None, None)
        assert rc == 3

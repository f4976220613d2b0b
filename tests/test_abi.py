"""The C-ABI library loads, exports what include/jq.h declares, and rejects
bad arguments on the host before anything is launched (no GPU needed)."""
import ctypes
import os
import re

import numpy as np

from if_i_could_turn_back_time_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_functions():
    text = open(os.path.join(ROOT, "include", "jq.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(jq_[a-z0-9_]+)\s*\(", text)))


def test_every_declared_symbol_is_exported_and_bound():
    names = _declared_functions()
    assert "jq_gemv_e2m1" in names and "jq_gemv_gf4" in names and "jq_gemv_grouped" in names
    lib = ctypes.CDLL(_lib.lib_path())
    for n in names:
        assert hasattr(lib, n), f"{n} declared in jq.h but not exported"
    assert sorted(_lib.exported_symbols()) == names, "ctypes table and jq.h disagree"


def test_version_and_error_text():
    lib = _lib.load()
    assert lib.jq_version() == 100
    assert _lib.strerror(0) == "ok"
    for code in range(-8, 0):
        assert _lib.strerror(code) not in ("", "unknown status")
    assert "unknown" in _lib.strerror(-999)


def test_host_side_validation_needs_no_gpu():
    lib = _lib.load()
    buf = np.zeros(4096, dtype=np.uint8)
    p = buf.ctypes.data  # 64-byte aligned host address: only used for argument checks
    assert p % 16 == 0
    # null pointers
    assert lib.jq_gemv_e2m1(None, p, p, None, p, 8, 64, 1, 32, 0, 0, 0, None, 0, None) == -1
    assert lib.jq_gemv_gf4(p, p, None, p, None, p, 8, 128, 1, 128, 0, 0, 0, None, 0, None) == -1
    # shapes: K not a multiple of g, g not a multiple of 32, e2m1 without groups
    assert lib.jq_gemv_e2m1(p, p, p, None, p, 8, 100, 1, 32, 0, 0, 0, None, 0, None) == -2
    assert lib.jq_gemv_e2m1(p, p, p, None, p, 8, 64, 1, 16, 0, 0, 0, None, 0, None) == -2
    assert lib.jq_gemv_e2m1(p, p, p, None, p, 8, 64, 1, 0, 0, 0, 0, None, 0, None) == -2
    assert lib.jq_gemv_e2m1(p, p, p, None, p, 0, 64, 1, 32, 0, 0, 0, None, 0, None) == -2
    assert lib.jq_gemv_e2m1(p, p, p, None, p, 8, 64, 0, 32, 0, 0, 0, None, 0, None) == -2
    # rotation block other than 128, or K not a multiple of it
    assert lib.jq_gemv_e2m1(p, p, p, None, p, 8, 64, 1, 32, 64, 0, 0, None, 0, None) == -5
    assert lib.jq_gemv_e2m1(p, p, p, None, p, 8, 64, 1, 32, 128, 0, 0, None, 0, None) == -2
    # misaligned packed weights
    assert lib.jq_gemv_e2m1(p + 4, p, p, None, p, 8, 64, 1, 32, 0, 0, 0, None, 0, None) == -3
    # element types
    assert lib.jq_gemv_e2m1(p, p, p, None, p, 8, 64, 1, 32, 0, 7, 0, None, 0, None) == -4
    # dequant / fwht
    assert lib.jq_dequant_e2m1(None, p, p, 8, 64, 32, None) == -1
    assert lib.jq_dequant_gf4(p, None, p, p, 8, 64, 32, None) == -1
    assert lib.jq_fwht_block(p, p, 1, 100, 128, 0, None) == -2
    assert lib.jq_fwht_block(p, p, 1, 128, 64, 0, None) == -5


def test_host_packer_argument_checks():
    lib = _lib.load()
    W = np.zeros((2, 64), dtype=np.float32)
    q = np.zeros((2, 32), dtype=np.uint8)
    s = np.zeros((2, 2), dtype=np.uint16)
    assert lib.jq_pack_e2m1_host(None, 2, 64, 32, q.ctypes.data, s.ctypes.data, 1) == -1
    assert lib.jq_pack_e2m1_host(W.ctypes.data, 2, 64, 48, q.ctypes.data, s.ctypes.data, 1) == -2
    assert lib.jq_pack_gf4_host(W.ctypes.data, 2, 64, 32, q.ctypes.data, None, s.ctypes.data, 1) == -1
    assert lib.jq_rotate_weights_host(W.ctypes.data, 2, 64, 128, 1) == -2


def test_convolution_geometry_has_to_match_the_packed_matrix():
    """jq_conv_rows takes the row length of the packed matrix and the rows of y; an image that does not give them is
    refused before anything is launched."""
    lib = _lib.load()
    buf = np.zeros(4096, dtype=np.uint8)
    p = (buf.ctypes.data + 255) // 256 * 256

    def call(channels, K, rows, batch=2, g=0):
        c = _lib.jq_conv(batch, channels, 9, 7, 3, 3, 1, 1, 1, 1, 1, 1, (ctypes.c_int64 * 4)(channels * 63, 63, 7, 1))
        return lib.jq_conv_rows(_lib.JQ_FMT_GF4, p, p, p, p, None, p, ctypes.byref(c), 8, K, rows, g, 0, 0, p, 256, p, None)

    assert call(4, 36, 126) == -6                      # the shapes agree: only the scratch is too small
    assert call(3, 36, 126) == -2 and call(5, 36, 126) == -2
    assert call(64, 512, 126, g=64) == -2 and call(32, 576, 126, g=64) == -2
    assert call(4, 36, 125) == -2 and call(4, 36, 63) == -2 and call(4, 36, 126, batch=1) == -2


def test_prepared_activations_are_not_read_through_the_read_only_path():
    """The main kernels start while the kernel that prepares the activation still runs (griddepcontrol.wait orders them);
    read-only loads are for data that nothing writes during the kernel: weights, scales, codebooks, bias."""
    csrc = os.path.join(ROOT, "if_i_could_turn_back_time_b200", "csrc")
    for name in sorted(os.listdir(csrc)):
        text = open(os.path.join(csrc, name)).read()
        if "pdl_wait()" not in text:
            continue
        for load in re.findall(r"__ld(?:g|cg|cs|lu|cv)\s*\(([^;]*)", text):
            assert not re.search(r"\b(?:xscale|xp|xprep)\b", load.split(")")[0]), f"{name}: {load}"
        assert not re.search(r"const\s+\w+\s*\*\s*__restrict__\s+(?:xscale|xp|xprep)\b", text), name

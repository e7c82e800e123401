"""Which tiles the fp32-scale grouped GEMM takes: by the rows that are expected, not by the room in the buffer (host code only)."""
import ctypes

import pytest

from nixl_b200.ops import _lib
from nixl_b200.ops.grouped_gemm import _Params

SINGLE, PAIR = 1, 2


def _mode(**kw):
    p = _Params()
    for k, v in kw.items():
        setattr(p, k, v)
    fn = ctypes.CDLL(_lib.LIB_PATH).nixl_grouped_gemm_fp8_mode
    fn.argtypes, fn.restype = [ctypes.POINTER(_Params)], ctypes.c_int
    return fn(ctypes.byref(p))


@pytest.mark.parametrize("room", [128, 129, 160, 255, 256, 1024])  # tokens the low-latency buffer is sized for
@pytest.mark.parametrize("tokens", [1, 50, 128])
def test_a_decode_step_takes_single_ctas_whatever_the_buffer_holds(room, tokens):
    if tokens <= room:
        assert _mode(groups=32, N=4096, K=4096, a_rows=32 * room, expected_rows=8 * tokens) == SINGLE


@pytest.mark.parametrize("expected", [0, 32 * 200, 10**6])  # unknown; known; more than there is room for
def test_packed_rows_take_pairs_above_128_per_expert(expected):
    assert _mode(groups=32, N=2048, K=7168, a_rows=32 * 200, expected_rows=expected) == PAIR
    assert _mode(groups=32, N=2048, K=7168, a_rows=32 * 128, expected_rows=expected) == SINGLE


def test_what_the_rule_does_not_override():
    few = dict(groups=32, N=4096, K=4096, a_rows=32 * 512, expected_rows=64)
    assert _mode(**few) == SINGLE and _mode(**few, tile_mode=2) == PAIR and _mode(**few, tile_mode=3) == 3
    many = dict(groups=32, N=4096, K=4096, a_rows=32 * 512)
    assert _mode(**many) == PAIR and _mode(**many, tile_mode=1) == SINGLE
    assert _mode(**many, rows_per_expert=512) == SINGLE  # the layout of a dispatch that may still run
    assert _mode(**{**many, "N": 4096 + 128}) == SINGLE
    assert _mode(groups=1, N=4096, K=7168, a_rows=512) == SINGLE  # 32 pair tiles leave SMs idle

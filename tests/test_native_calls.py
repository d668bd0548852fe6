"""The launchers as functions of a CPython module: the same answers as through ctypes, and their arguments' errors."""
import ctypes as C

import pytest

from delta_b200.kernels import lib, native_calls


@pytest.fixture(scope="module")
def both():
    path = lib.build()
    plain = C.CDLL(str(path))
    calls = native_calls.load(plain, path, lib._SIGNATURES)
    if calls is None:
        pytest.skip("no C compiler or no Python.h")
    for name, args in lib._SIGNATURES.items():
        getattr(plain, name).argtypes, getattr(plain, name).restype = args, C.c_int
    return plain, calls


def test_the_same_answers(both):
    """Launchers that look at their numbers only (or return at once because a size is zero): whole numbers of either sign, wrapped ones, truth values."""
    plain, calls = both
    for name, args in [("dk_gemm_small_m_supported", (8, 64, 64, 0)), ("dk_gemm_small_m_supported", (8, -64, 64, True)),
                       ("dk_gemm_tc_supported", (128, 4096, 4096, 1)), ("dk_gemm_tc_supported", ((1 << 32) + 8, 64, 64, 0)),
                       ("dk_gemm_rows_tc_supported", (300, 24, 72, 0)), ("dk_gemm_f32_tc_supported", (1 << 40, 2048, 2048)),
                       ("dk_gemm_f32_tc_supported", ((1 << 40) + 4, 2048, 2048)), ("dk_gemm_f32_tc_supported", (None, 2048, 2048)),
                       ("dk_experts_align", (None, 0, 4, None, 0, None, 0, 64, None)), ("dk_softcap", (None, 0, 2.5, 1, None)),
                       ("dk_decay_attention_tiles_chunk", ())]:
        assert calls[name](*args) == getattr(plain, name)(*args), name


def test_wrong_arguments_are_errors(both):
    _, calls = both
    with pytest.raises(TypeError, match="takes 4 arguments, not 2"):
        calls["dk_gemm_tc_supported"](1, 2)
    with pytest.raises(TypeError):
        calls["dk_gemm_tc_supported"]("8", 64, 64, 0)
    with pytest.raises(TypeError):
        calls["dk_softcap"](None, 0, None, 1.0, None)
    with pytest.raises(TypeError):
        calls["dk_softcap"](1.5, 0, 1.0, 1.0, None)


def test_launchers_with_structures_stay_with_ctypes(both):
    _, calls = both
    assert "dk_attention_plain" not in calls and lib.load().dk_attention_plain.argtypes is not None

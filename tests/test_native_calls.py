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


@pytest.fixture
def apart(tmp_path):
    """The library with a folder of its own for the module."""
    path = tmp_path / "lib.so"
    path.symlink_to(lib.build())
    return C.CDLL(str(path)), path, {k: lib._SIGNATURES[k] for k in ("dk_gemm_tc_supported", "dk_softcap")}


def test_a_compiler_with_arguments(apart, monkeypatch, recwarn):
    monkeypatch.setenv("CC", "gcc -pipe")
    calls = native_calls.load(*apart)
    assert calls is not None and calls["dk_gemm_tc_supported"](128, 4096, 4096, 1) and not recwarn


@pytest.mark.parametrize("cc, why", [("/bin/false -pipe", "false -pipe ended with"), ("/nowhere/cc", "nowhere/cc")])
def test_a_compiler_that_fails_is_told(apart, monkeypatch, cc, why):
    monkeypatch.setenv("CC", cc)
    with pytest.warns(RuntimeWarning, match=f"through ctypes.*{why}"):
        assert native_calls.load(*apart) is None


def test_a_module_that_does_not_load_is_told(apart, tmp_path):
    plain, path, signatures = apart
    assert native_calls.load(plain, path, signatures) is not None
    (so,) = path.parent.glob("dk_calls_*.so")
    other = tmp_path / "other"
    other.mkdir()
    (other / so.name).write_bytes(b"no module")
    with pytest.warns(RuntimeWarning, match="through ctypes"):
        assert native_calls.load(plain, other / "lib.so", signatures) is None


@pytest.mark.parametrize("N, K", [(2048, 2048), (2048, 5504), (2048, 11008), (4096, 11008), (9472, 4096), (11008, 2048), (22016, 4096), (64000, 4096), (128, 1024)])
def test_the_working_memory_of_32_bit_products_is_bounded(N, K):
    """Prompts of any length: 128 MB and no more, and short ones in one pass over the weights."""
    def plan(M):
        kb, launches = C.c_int(), C.c_int()
        assert lib.load().dk_gemm_f32_tc_plan(M, N, K, C.byref(kb), C.byref(launches)) == 0
        return kb.value / 1024, launches.value
    few = plan(1)[1]
    assert plan(256)[1] == few
    for M in (1, 300, 2048, 16384, 1 << 20):
        assert plan(M)[0] <= 128

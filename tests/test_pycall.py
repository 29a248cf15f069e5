"""The CPython entry to the hot C ABI calls (csrc/pycall.c) passes the arguments that ctypes passes: without a device that shows
in the calls that the library refuses, which name the first argument it looks at."""
import pytest

from tensorpencil_b200 import _lib


@pytest.fixture(scope="module")
def calls():
    return _lib.load_calls()


ARGS = {
    "tpb_q8_1_quantize": [None, None, 16, 32, 16],
    "tpb_gguf_gemv_q8n": [None, None, 2, 16, 16, 1.0, 8, 256, 16, 1, 0, 1],
    "tpb_q8_0_gemv_f32": [None, None, 16, 16, 16, 1.0, 8, 256],
    "tpb_convrot_prep": [None, None, 16, 0, 4, 256, 8, 16, 16, None],
    "tpb_convrot_gemm": [None, None, 16, 0, 16, 16, 16, None, 16, 8, 16, 4, 16, 256],
    "tpb_convrot_linear": [None, None, 16, 0, 16, 16, 0, 16, 16, None, 16, 8, 16, 4, 16, 256],
}


@pytest.mark.parametrize("name", sorted(ARGS))
def test_a_null_handle_is_refused_as_by_ctypes(calls, name):
    lib = _lib.load()
    assert len(_lib.SIGNATURES[name][1]) == len(ARGS[name])
    assert getattr(calls, name)(*ARGS[name]) == getattr(lib, name)(*ARGS[name]) == _lib.TPB_ERR_INVALID_ARG


@pytest.mark.parametrize("name", sorted(ARGS) + ["q8_0_linear"])
def test_wrong_arguments_raise(calls, name):
    fn = getattr(calls, name)
    with pytest.raises(TypeError):
        fn(None)
    good = ARGS.get(name, [None, None, 16, 16, 1, 16, 1.0, 8, 256, 16])
    for i, v in enumerate(good):
        bad = list(good)
        bad[i] = "x"
        with pytest.raises(TypeError):
            fn(*bad)

"""The CPython entry to the hot C ABI calls (csrc/pycall.c) passes the arguments that ctypes passes, each in its place: both
are called against a stand-in library that writes down what it is given.  Against the library itself: a null handle is refused, and wrong
numbers and types of arguments raise."""
import ctypes as C
import json
import os
import subprocess
import sys

import pytest

from tensorpencil_b200 import _lib, build


@pytest.fixture(scope="module")
def calls():
    if not os.path.exists(_lib.CALL_PATH):
        pytest.skip("the extension is not built for this interpreter")
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


STUBBED = sorted(ARGS) + ["tpb_q8_0_gemv_q8n"]
C_TYPE = {C.c_void_p: ("void *", "%lld", "(long long)"), C.c_int: ("int", "%d", ""), C.c_int64: ("int64_t", "%lld", "(long long)"),
          C.c_float: ("float", "%.9g", "(double)")}

CHILD = """
import ctypes as C, importlib.machinery, importlib.util, json, sys
stub_path, ext_path, jobs = sys.argv[1], sys.argv[2], json.loads(sys.argv[3])
from tensorpencil_b200 import _lib
stub = C.CDLL(stub_path)
stub.stub_log.restype = C.c_char_p
for name in jobs["stubbed"]:
    getattr(stub, name).restype, getattr(stub, name).argtypes = _lib.SIGNATURES[name]
loader = importlib.machinery.ExtensionFileLoader("_tpbcall", ext_path)
ext = importlib.util.module_from_spec(importlib.util.spec_from_loader("_tpbcall", loader))
loader.exec_module(ext)
out = []
for fail_at, name, args in jobs["calls"]:
    row = []
    for mod in (ext, _lib.CtypesCalls(stub)):
        stub.stub_reset(fail_at)
        rc = getattr(mod, name)(*args)
        row.append([rc, stub.stub_log().decode()])
    out.append(row)
print(json.dumps(out))
"""


@pytest.fixture(scope="module")
def stand_in(tmp_path_factory):
    """A library with the stubbed functions, each of which logs its name and arguments, and the extension linked to it.  stub_reset(i)
    empties the log and lets call i (from 0) report an error."""
    d = tmp_path_factory.mktemp("pycall")
    src = ["#include <stdint.h>", "#include <stdio.h>", "static char log_[1 << 16]; static int len_, n_, fail_ = -1;",
           "const char *stub_log(void) { return log_; }",
           "void stub_reset(int fail_at) { len_ = n_ = 0; log_[0] = 0; fail_ = fail_at; }"]
    for name in STUBBED:
        args = [C_TYPE[t] for t in _lib.SIGNATURES[name][1]]
        params = ", ".join(f"{c} a{i}" for i, (c, _, _) in enumerate(args))
        fmt = " ".join([name] + [f for _, f, _ in args])
        vals = ", ".join(f"{cast}a{i}" for i, (_, _, cast) in enumerate(args))
        src.append(f'int {name}({params}) {{ len_ += snprintf(log_ + len_, sizeof log_ - len_, "{fmt};", {vals}); '
                   f"return n_++ == fail_ ? -2 : 0; }}")
    (d / "stub.c").write_text("\n".join(src))
    subprocess.run([build._nvcc(), "-Xcompiler", "-fPIC", "-shared", "-cudart", "none", str(d / "stub.c"), "-o", str(d / "libtpb200.so")],
                   check=True)
    ext = d / os.path.basename(_lib.CALL_PATH)
    if not build.build_pycall(str(ext), str(d)):
        pytest.skip("Python's headers are not installed")
    return str(d / "libtpb200.so"), str(ext)


def run_both(stand_in, calls):
    jobs = json.dumps({"stubbed": STUBBED, "calls": calls})
    env = dict(os.environ, PYTHONPATH=os.path.dirname(os.path.dirname(os.path.abspath(_lib.__file__))))
    r = subprocess.run([sys.executable, "-c", CHILD, *stand_in, jobs], check=True, capture_output=True, text=True, env=env)
    return json.loads(r.stdout.splitlines()[-1])


def distinct(name):
    """A value of its own for every argument, larger than 32 bits where the type allows it."""
    big = {C.c_void_p: 0x7f0000000000, C.c_int64: 0x500000000, C.c_int: 1000, C.c_float: 0.5}
    return [big[t] + 16 * i if t is not C.c_float else 0.5 + i for i, t in enumerate(_lib.SIGNATURES[name][1])]


def test_every_argument_arrives_in_its_place(stand_in):
    names = sorted(ARGS)
    for name, (ext, ct) in zip(names, run_both(stand_in, [[-1, n, distinct(n)] for n in names])):
        want = " ".join([name] + ["%.9g" % v if isinstance(v, float) else str(v) for v in distinct(name)]) + ";"
        assert ext == ct == [0, want]
    # NULL for None, negative integers, and the status that the function returns
    for name, (ext, ct) in zip(names, run_both(stand_in, [[0, n, ARGS[n][:-1] + [ARGS[n][-1] if ARGS[n][-1] is None else -7]]
                                                          for n in names if _lib.SIGNATURES[n][1][-1] is not C.c_void_p])):
        assert ext == ct and ext[0] == -2


@pytest.mark.parametrize("m", [0, 1, 8, 9, 17])
def test_q8_0_linear_quantises_once_and_runs_groups_of_eight(stand_in, m):
    rows, cols, y, xq = 1000, 4096, 0x7f0000000000, 0x7f3000000000
    args = [0x1000, 0x2000, y, 0x7f1000000000, m, 0x7f2000000000, 0.25, rows, cols, xq]
    groups = [f"tpb_q8_0_gemv_q8n {0x1000} {0x2000} {y + 4 * r * rows} {0x7f2000000000} 0.25 {rows} {cols} {xq} {min(8, m - r)} {r} {m};"
              for r in range(0, m, 8)]
    quant = f"tpb_q8_1_quantize {0x1000} {0x2000} {0x7f1000000000} {m * cols} {xq};"
    (ok_ext, ok_ct), (q_ext, q_ct), (g_ext, g_ct) = run_both(stand_in, [[-1, "q8_0_linear", args], [0, "q8_0_linear", args],
                                                                        [1, "q8_0_linear", args]])
    assert ok_ext == ok_ct == [0, quant + "".join(groups)]
    assert q_ext == q_ct == [-2, quant]                                       # nothing runs behind a call that failed
    assert g_ext == g_ct == [-2 if m else 0, quant + "".join(groups[:1])]


def test_calls_go_through_ctypes_where_the_extension_is_not_built(monkeypatch):
    monkeypatch.setattr(_lib, "CALL_PATH", _lib.CALL_PATH + ".absent")
    monkeypatch.setattr(_lib, "_calls", None)
    calls = _lib.load_calls()
    assert isinstance(calls, _lib.CtypesCalls)
    for name in ARGS:
        assert getattr(calls, name)(*ARGS[name]) == _lib.TPB_ERR_INVALID_ARG
    assert calls.q8_0_linear(None, None, 16, 16, 1, 16, 1.0, 8, 256, 16) == _lib.TPB_ERR_INVALID_ARG


def test_the_extension_is_named_for_this_interpreter():
    import importlib.machinery
    assert any(_lib.CALL_PATH.endswith(sfx) for sfx in importlib.machinery.EXTENSION_SUFFIXES)


def test_nothing_is_built_without_pythons_headers(monkeypatch, tmp_path, capsys):
    monkeypatch.setattr(build.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
    assert build.build_pycall(str(tmp_path / "x.so"), str(tmp_path)) is False
    assert not (tmp_path / "x.so").exists() and "ctypes" in capsys.readouterr().err

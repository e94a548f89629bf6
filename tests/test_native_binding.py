"""The CPython binding: argument errors, its file's ABI tag, and the package without it.  No GPU: every call is refused
before it reaches CUDA."""
import os
import subprocess
import sys
import sysconfig

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ARGUMENTS = (None, None, 4, 8, None)      # of mfar_silu_mul_f16


def test_arguments_are_checked():
    from mustafar_b200 import _lib
    silu = _lib.native().mfar_silu_mul_f16
    assert silu(*ARGUMENTS) == _lib.lib().mfar_silu_mul_f16(*ARGUMENTS) == 1          # null pointers
    for bad in (ARGUMENTS[:4], ARGUMENTS + (0,)):
        with pytest.raises(TypeError):
            silu(*bad)
    for at, value in ((3, 1 << 31), (3, -(1 << 31) - 1), (2, 1 << 63), (0, 1 << 64)):
        with pytest.raises(OverflowError):
            silu(*ARGUMENTS[:at], value, *ARGUMENTS[at + 1:])
    for at, value in ((3, 8.0), (2, None), (0, "x")):
        with pytest.raises(TypeError):
            silu(*ARGUMENTS[:at], value, *ARGUMENTS[at + 1:])


def test_the_file_carries_the_interpreters_tag():
    from mustafar_b200 import _lib, build
    assert os.path.basename(build.NATIVE) == "_native" + sysconfig.get_config_var("EXT_SUFFIX")
    assert _lib.native().__file__ == build.NATIVE


def test_without_headers_the_binding_is_left_out(monkeypatch, tmp_path):
    from mustafar_b200 import build
    monkeypatch.setattr(build.sysconfig, "get_path", lambda name: str(tmp_path))
    assert build.build_native("no compiler is called", 0.0, force=True) is None


def test_without_the_binding_ctypes_serves_the_same_functions():
    code = ("import sys, warnings; sys.modules['mustafar_b200._native'] = None\n"
            "from mustafar_b200 import _lib\n"
            "with warnings.catch_warnings(record=True) as seen:\n"
            "    warnings.simplefilter('always')\n"
            "    assert _lib.native() is _lib.lib() and _lib.native() is _lib.lib()\n"
            "assert len(seen) == 1 and 'ctypes' in str(seen[0].message)\n"
            f"assert _lib.native().mfar_silu_mul_f16(*{ARGUMENTS}) == 1\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

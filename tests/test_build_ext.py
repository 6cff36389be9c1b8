"""The compiled call layer: named for the interpreter, built when it is missing, and optional."""
import os
import subprocess
import sys
import sysconfig

import pytest

from necklace_b200 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.skipif(not os.path.exists(_build.LIB), reason="native library not built")


def test_name_holds_the_interpreter():
    # (a plain _nkpy.so would be imported by any version of Python)
    assert _build.EXT.endswith("_nkpy" + sysconfig.get_config_var("EXT_SUFFIX"))
    assert "cpython-%d%d" % sys.version_info[:2] in os.path.basename(_build.EXT)


def _at(tmp_path, monkeypatch):
    ext = str(tmp_path / os.path.basename(_build.EXT))
    monkeypatch.setattr(_build, "EXT", ext)
    return ext


def test_a_failing_compiler_is_a_warning(tmp_path, monkeypatch):
    ext = _at(tmp_path, monkeypatch)
    for cxx in ("false", "/no/such/compiler"):
        open(ext, "w").close()               # what an earlier build left
        monkeypatch.setenv("CXX", cxx)
        with pytest.warns(UserWarning, match="ctypes"):
            assert not _build.build_ext(force=True)
        assert not os.listdir(tmp_path)      # nothing stale stays to be imported


def test_built_when_missing(tmp_path):
    """A checkout with the library but without the extension."""
    pkg = tmp_path / "necklace_b200"
    for d, _, files in os.walk(os.path.join(ROOT, "necklace_b200")):
        out = os.path.join(str(pkg), os.path.relpath(d, os.path.join(ROOT, "necklace_b200")))
        os.makedirs(out, exist_ok=True)
        for f in files:
            if not f.startswith("_nkpy") and not f.endswith(("_dbg.so", ".pyc")):
                os.symlink(os.path.join(d, f), os.path.join(out, f))
    code = ("from necklace_b200 import _lib; _lib.load(); assert _lib._fast; "
            "assert _lib.value('nkb_gemm_slices', 64, 64, 64, 64, 0) == 1")
    r = subprocess.run([sys.executable, "-c", code], cwd=tmp_path, capture_output=True, text=True,
                       env=dict(os.environ, PYTHONPATH=str(tmp_path)), timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]

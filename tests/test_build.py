"""What the build step needs and when it takes an extension module as up to date (no compiler is run)."""
import importlib.metadata
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def built():
    from cswap_b200 import build
    build.build()
    return build


def test_extension_is_rebuilt_for_another_torch_or_python(built, monkeypatch):
    """The module is tied to the libtorch and the interpreter it was compiled against; when loading it fails
    codec.py sends the user to this build, which must not find it up to date by its file time."""
    ran = []
    monkeypatch.setattr(built.subprocess, "check_call", lambda cmd, **kw: ran.append(cmd))
    monkeypatch.setattr(built, "EXT_STAMP", built.EXT_STAMP + ".test", raising=False)
    if os.path.exists(built.EXT_STAMP[:-len(".test")]):
        shutil.copy(built.EXT_STAMP[:-len(".test")], built.EXT_STAMP)
    try:
        assert built.build_ext() == built.EXT and not ran
        version = importlib.metadata.version
        monkeypatch.setattr(importlib.metadata, "version", lambda n: "9.9.9" if n == "torch" else version(n))
        assert built.build_ext() == built.EXT and len(ran) == 1 and built.EXT in ran[0]
        assert built.build_ext() == built.EXT and len(ran) == 1  # now it is the one for that torch
        var = built.sysconfig.get_config_var
        monkeypatch.setattr(built.sysconfig, "get_config_var", lambda n: "cpython-399" if n == "SOABI" else var(n))
        assert built.build_ext() == built.EXT and len(ran) == 2
    finally:
        if os.path.exists(built.EXT_STAMP):
            os.remove(built.EXT_STAMP)


def test_the_library_is_built_without_torch(built, tmp_path):
    """A program that wants only the C ABI builds it with nvcc alone; the extension is left out."""
    pkg = tmp_path / "cswap_b200"
    pkg.mkdir()
    shutil.copy(os.path.join(ROOT, "cswap_b200", "build.py"), pkg)
    os.symlink(os.path.join(ROOT, "cswap_b200", "csrc"), pkg / "csrc")
    os.symlink(os.path.join(ROOT, "include"), tmp_path / "include")
    shutil.copyfile(built.LIB, pkg / "libcswap_b200.so")  # newer than its sources: nothing to compile
    code = f"import sys, runpy; sys.modules['torch'] = None; sys.argv = ['build.py']; runpy.run_path({str(pkg / 'build.py')!r}, run_name='__main__')"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip() == str(pkg / "libcswap_b200.so") and "extension" in r.stderr
    assert not (pkg / "_codec_ext.so").exists()

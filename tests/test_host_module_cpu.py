"""The extension module belongs to one torch: another one does not get it loaded, and the build makes one for it."""
import importlib.util
import os
import subprocess
import sys

import torch

from starrygl import _C

PKG = os.path.dirname(os.path.dirname(os.path.abspath(_C.__file__)))


def test_build_and_package_agree_on_the_file(monkeypatch):
    spec = importlib.util.spec_from_file_location("sgl_build_names", os.path.join(PKG, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    assert build.host_path() == _C.HOST_PATH and torch.__version__ in os.path.basename(_C.HOST_PATH)
    monkeypatch.setattr(torch, "__version__", "9.9.9")
    assert build._stale(build.host_path(), [])


def test_another_torch_does_not_load_it():
    code = (f"import sys, torch; torch.__version__ = '9.9.9'; sys.path.insert(0, {PKG!r})\n"
            "from starrygl import _C\n"
            "try:\n    _C.host()\nexcept RuntimeError as e:\n    print('refused', 'for this torch' in str(e))\n")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.stdout.strip() == "refused True", r.stdout + r.stderr

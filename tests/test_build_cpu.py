"""A library of torch operators that does not load with the present torch leaves the package importable (the first call says
what to do), and the build replaces it."""
import os
import shutil
import subprocess
import sys

import pytest
import torch

import rwkv_ops_b200
from rwkv_ops_b200 import _lib, _ops, build

PKG = os.path.dirname(rwkv_ops_b200.__file__)


@pytest.mark.parametrize("broken", ["librwkv_ops_b200_torch.so", "librwkv_ops_b200.so"])
def test_package_with_a_library_that_does_not_load(broken, tmp_path):
    build.build()
    copy = tmp_path / "rwkv_ops_b200"
    shutil.copytree(PKG, copy, ignore=shutil.ignore_patterns("csrc", "__pycache__", "*_dev.so"))
    with open(copy / broken, "wb") as f:      # no shared object at all, as good as one with symbols that torch lacks
        f.write(b"not a library")
    code = ("import torch, rwkv_ops_b200 as ro; from rwkv_ops_b200.workloads import rwkv7_inputs; from rwkv_ops_b200 import _lib\n"
            "d = rwkv7_inputs(1, 4, 1)\n"
            "try:\n    ro._ops.load()\nexcept _lib.RwkvB200Error as e:\n    print('said:', e)\n")
    p = subprocess.run([sys.executable, "-c", code], cwd=tmp_path, capture_output=True, text=True,
                       env={**os.environ, "PYTHONPATH": str(tmp_path)})
    assert p.returncode == 0, p.stderr
    assert "said:" in p.stdout and broken in p.stdout and "does not load" in p.stdout


def test_another_torch_needs_another_build(tmp_path, monkeypatch):
    """Which torch the operators were built against decides, not only the times of the files."""
    calls = []
    monkeypatch.setattr(build, "BUILD", str(tmp_path))
    monkeypatch.setattr(build, "TORCH_LIB", str(tmp_path / "lib.so"))

    class Done:
        returncode = 0
        stdout = stderr = ""

    def compiled(cmd, **kw):
        calls.append(cmd)
        (tmp_path / "lib.so").write_bytes(b"")
        return Done

    monkeypatch.setattr(build.subprocess, "run", compiled)
    build.build_torch()
    build.build_torch()
    assert len(calls) == 1
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    build.build_torch()
    build.build_torch()
    assert len(calls) == 2

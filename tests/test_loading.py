"""Loading of the shared libraries: the reason of a failure reaches the caller, a build made later in the
process is picked up, and a host layer built for another torch is not taken for a current one."""

import os
import subprocess
import sys

import pytest
import torch

from conftest import ROOT
from delta_feedback_experiment_b200 import _lib, build

PACKAGE = "delta_feedback_experiment_b200"

SCRIPT = """
import os, sys, torch
import delta_feedback_experiment_b200 as pkg
here, built = os.path.dirname(pkg.__file__), sys.argv[1]
x, w = torch.empty(1, 5, 48, device="meta"), torch.empty(48, 4, device="meta")

def attempt():
    try:
        return [tuple(t.shape) for t in pkg.pkda_qkv_conv(x, w, 16, 32, 1e-6)]
    except RuntimeError as exc:
        return str(exc)

def put(name, data=None):
    path = os.path.join(here, name)
    if os.path.lexists(path):
        os.unlink(path)
    if data is None:
        os.symlink(os.path.join(built, name), path)
    else:
        open(path, "wb").write(data)

from delta_feedback_experiment_b200 import ops
print(ops.LAUNCHES, pkg.pkda_cuda_available(), attempt())
put("libpkda_b200.so", b"not a library")
print(attempt())
put("libpkda_b200.so")
print(attempt())
put("_native.so", b"pkda host layer built for torch 0.1" + bytes(1))
print(attempt())
put("_native.so")
print(attempt(), pkg.pkda_cuda_available())
"""


def test_a_failure_names_its_reason_and_a_later_build_is_seen(tmp_path):
    build.build()
    source, copy = os.path.join(ROOT, PACKAGE), tmp_path / PACKAGE
    copy.mkdir()
    for name in os.listdir(source):
        if name.endswith(".py"):
            (copy / name).write_bytes(open(os.path.join(source, name), "rb").read())
    run = subprocess.run([sys.executable, "-c", SCRIPT, source], capture_output=True, text=True, timeout=600,
                         cwd=tmp_path, env={**os.environ, "PYTHONPATH": str(tmp_path)})
    assert run.returncode == 0, run.stderr
    nothing, broken, half, foreign, good = run.stdout.strip().splitlines()
    assert nothing.startswith("0 False") and "libpkda_b200.so has not been built" in nothing
    assert "has not been built" not in broken and "libpkda_b200.so" in broken   # the loader's own words
    assert "_native.so has not been built" in half
    assert f"not built for torch {torch.__version__}" in foreign
    assert good == f"{[(1, 5, 16)] * 3} True"


def test_a_host_layer_for_another_torch_is_rebuilt(monkeypatch):
    build.build()
    assert not build.needs_build()
    monkeypatch.setattr(torch, "__version__", torch.__version__ + ".1")
    assert not _lib.native_is_current() and build.needs_build()
    monkeypatch.setattr(_lib, "_native", None)
    with pytest.raises(RuntimeError, match="not built for torch"):
        _lib.native()

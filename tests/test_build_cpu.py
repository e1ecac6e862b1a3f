"""The build without a torch, and an extension that does not fit the interpreter."""
import pathlib
import shutil
import subprocess
import sys

import pytest
import torch

from dscuda_b200 import build, library

ROOT = pathlib.Path(__file__).resolve().parents[1]


def test_configures_without_torch(tmp_path):
    """The two libraries and the launchers need neither Python nor torch."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    bare = tmp_path / "python"
    bare.write_text(f"#!/bin/sh\nexec {sys.executable} -I -S \"$@\"\n")          # no site-packages
    bare.chmod(0o755)
    assert subprocess.run([bare, "-c", "import torch"], capture_output=True).returncode != 0
    for interpreter in (str(bare), str(tmp_path / "absent")):
        tree = tmp_path / f"build_{pathlib.Path(interpreter).name}"
        done = subprocess.run([build._tool("cmake"), "-S", str(ROOT), "-B", str(tree), f"-DCMAKE_CUDA_COMPILER={nvcc}", f"-DDSCUDA_PYTHON={interpreter}"],
                              capture_output=True, text=True)
        assert done.returncode == 0, done.stderr[-1000:]
        targets = subprocess.run([build._tool("cmake"), "--build", str(tree), "--target", "help"], capture_output=True, text=True).stdout
        assert "dscuda_mla_bench" in targets and "benchmark_mla_decode" in targets and "dscuda_torch" not in targets


def test_extension_that_does_not_load(tmp_path, monkeypatch):
    monkeypatch.setattr(library, "build_directory", lambda: tmp_path)
    monkeypatch.setattr(library, "library", lambda name: None)
    with pytest.raises(RuntimeError, match="is missing"):
        library.extension.__wrapped__()
    (tmp_path / "_dscuda_torch.so").write_bytes(b"not a library")
    with pytest.raises(RuntimeError, match="does not load into torch .* run `python -m dscuda_b200.build`"):
        library.extension.__wrapped__()


def test_extension_of_another_torch(monkeypatch):
    monkeypatch.setattr(torch, "__version__", "1.0.0+other")
    with pytest.raises(RuntimeError, match="was built for torch"):
        library.extension.__wrapped__()

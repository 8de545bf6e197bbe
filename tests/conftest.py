"""Test configuration: the ``gpu`` marker, import paths and shared helpers."""
from __future__ import annotations

import sys
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent
PKG = ROOT / "vllm-triton-fixed-point-reductions_b200"
for p in (str(ROOT), str(PKG)):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on the B200 box)")


def pytest_collection_modifyitems(config, items):
    if torch.cuda.is_available():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)


@pytest.fixture(scope="session", autouse=True)
def _built_library():
    """Every test may assume that the C-ABI and the operator library exist (they are built in-tree)."""
    import importlib.util

    lib = PKG / "lib" / "libfxpr_b200.so"
    if not (lib.exists() and lib.with_name("libfxpr_torch.so").exists()):
        spec = importlib.util.spec_from_file_location("fxpr_build", PKG / "build.py")
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        mod.build()
    return lib

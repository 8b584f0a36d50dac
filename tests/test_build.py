"""When the operator module is compiled again."""
import os
import sys

import pytest
import torch

from matgptq_b200 import build


@pytest.fixture
def built(tmp_path, monkeypatch):
    """A module that has just been built, as far as build() can tell."""
    module, stamp = tmp_path / "_torch_ops.so", tmp_path / "_torch_ops.txt"
    monkeypatch.setattr(build, "TORCH_OPS_PATH", str(module))
    monkeypatch.setattr(build, "TORCH_OPS_STAMP", str(stamp))
    module.write_bytes(b"")
    stamp.write_text(build._torch_ops_built_with())
    return module, stamp


def test_module_is_current_after_a_build(built):
    assert not build._torch_ops_stale()


@pytest.mark.parametrize("what", ["torch", "python", "source", "module gone", "never recorded"])
def test_module_is_stale(built, monkeypatch, what):
    module, stamp = built
    if what == "torch":
        monkeypatch.setattr(torch, "__version__", "0.0.0")
    elif what == "python":
        monkeypatch.setattr(sys, "version", "0.0.0")
    elif what == "source":
        os.utime(module, (0, 0))
    else:
        (module if what == "module gone" else stamp).unlink()
    assert build._torch_ops_stale()

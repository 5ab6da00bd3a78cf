"""The native call path of the Python layer without a GPU: where it cannot be had the package works without it."""
import os
import subprocess
import sys

import pytest
import torch

from lithos_metal_b200 import _lib, build

CALLS = ("sample", "stochastic", "argmax", "draft_q", "verify", "lm_head")


def test_the_extension_is_named_for_the_python_and_the_torch_it_was_compiled_for():
    name = os.path.basename(build.HOST_OUT)
    assert sys.implementation.cache_tag in name and torch.__version__ in name


@pytest.mark.parametrize("how", ["no compiler", "missing", "does not load"])
def test_every_call_is_left_to_the_python_layer_without_it(monkeypatch, tmp_path, how):
    monkeypatch.setattr(_lib, "_host", None)
    if how == "no compiler":
        def fail(*a, **k):
            raise RuntimeError("g++: not found")
        monkeypatch.setattr(build, "build_host", fail)
        monkeypatch.delenv("LITHOS_B200_NO_BUILD", raising=False)
    else:
        path = tmp_path / "lithos_host.so"
        if how == "does not load":
            path.write_bytes(b"of another torch")
        monkeypatch.setattr(build, "HOST_OUT", str(path))
        monkeypatch.setenv("LITHOS_B200_NO_BUILD", "1")
    with pytest.warns(RuntimeWarning, match="no native call path"):
        h = _lib.host()
    assert all(getattr(h, n)(1, 2, 3) is None for n in CALLS)
    assert _lib.host() is h                                                 # (said once)


def test_the_extension_loads_and_leaves_what_is_not_its_case():
    """Tensors on the CPU are not: the Python layer raises for them."""
    code = "import torch, lithos_metal_b200._lib as L\nh = L.host()\nassert type(h).__name__ == 'module', h\nassert h.argmax(torch.zeros(2, 8), None, False) is None\n"
    subprocess.run([sys.executable, "-c", code], check=True, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

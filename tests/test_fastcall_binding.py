"""The operator call's CPython function: built for one interpreter, and only a faster way of what ctypes does."""
import ctypes
import os
import shutil
import subprocess
import sys
import sysconfig
import types

import numpy as np
import pytest
import torch

import pim_dl_asplos_b200 as P
from pim_dl_asplos_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_the_file_carries_the_interpreters_tag():
    """Another Python does not find it, and binds through ctypes."""
    assert build.FASTCALL.endswith("_fastcall" + sysconfig.get_config_var("EXT_SUFFIX"))
    if P._fast is not None:
        assert P._fast.__file__ == build.FASTCALL


@pytest.mark.parametrize("content", [b"", b"not a shared library"])
def test_a_file_that_does_not_load_leaves_ctypes(tmp_path, content):
    tree = tmp_path / "tree"
    shutil.copytree(os.path.join(ROOT, "pim-dl-asplos_b200"), tree / "pim-dl-asplos_b200",
                    ignore=shutil.ignore_patterns("csrc", "bin", "*.so", "__pycache__"))
    shutil.copy(os.path.join(ROOT, "pim_dl_asplos_b200.py"), tree)
    (tree / "pim-dl-asplos_b200" / os.path.basename(build.FASTCALL)).write_bytes(content)
    r = subprocess.run([sys.executable, "-c", "import pim_dl_asplos_b200 as P; print(P.__file__, P._fast)"], cwd=tree, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    assert str(tree) in r.stdout and r.stdout.strip().endswith("None")


@pytest.mark.skipif(P._fast is None, reason="not built for this interpreter")
@pytest.mark.parametrize("n_tokens", [3, 3.0, 2.9, "3", np.int64(3), np.float32(3), True, 0, -1, 2**32 + 3, None])
def test_arguments_as_through_ctypes(monkeypatch, n_tokens):
    """Both ways of the call hand the library the same numbers."""
    seen = []
    entry = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32, ctypes.c_uint32)(
        lambda *a: seen.append(a) or P.OK)
    ctx = object.__new__(P.LutAmmContext)
    ctx._h, ctx._amm_address = ctypes.c_void_p(0x1000), ctypes.cast(entry, ctypes.c_void_p).value
    ctx._L = types.SimpleNamespace(lutamm_amm=entry, lutamm_destroy=lambda h: None)
    x, y = torch.zeros(5, 4), torch.zeros(5, 8)
    ctx.amm_host(7, x, y, n_tokens=n_tokens, flags=P.FLAG_ASYNC)
    monkeypatch.setattr(P, "_fast", None)
    ctx.amm_host(7, x, y, n_tokens=n_tokens, flags=P.FLAG_ASYNC)
    assert len(seen) == 2 and seen[0] == seen[1] == (0x1000, 7, x.data_ptr(), y.data_ptr(), seen[0][4], P.FLAG_ASYNC)

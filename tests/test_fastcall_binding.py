"""The operator call's CPython function: built for one interpreter, and only a faster way of what ctypes does."""
import os
import shutil
import subprocess
import sys
import sysconfig

import pytest

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

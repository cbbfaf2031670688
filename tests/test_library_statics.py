"""Two copies of the library in one process (two versions, or a program and a
plugin that carry it) do not share their state: a kernel set up in one copy is
not set up in the other."""
import re
import shutil
import subprocess

import pytest


def test_no_writable_symbol_is_shared_between_copies():
    from new_repo_b200 import capi

    if not capi.LIB_PATH.exists() or not shutil.which("nm"):
        pytest.skip("library not built")
    out = subprocess.run(["nm", "-C", str(capi.LIB_PATH)], capture_output=True, text=True, check=True).stdout
    # unique symbols (one per process): the read-only table of the x passes' inputs is the same in every copy
    shared = re.findall(r"^\S+ u (les::.*)$", out, re.M)
    assert not [s for s in shared if not s.endswith("::nin_of_op")], shared

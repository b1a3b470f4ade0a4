"""The host part of the engine is ordinary C++ beside x86: what names x86 targets is
left out where the compiler is not one for x86-64 (a Grace-Blackwell node's is not)."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "rfnetwork_b200" / "csrc"


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("name", ["fdtd_compile.cpp", "fdtd_api.cu"])
def test_no_x86_targets_on_other_hosts(name):
    # the file's own lines, preprocessed as on a host that is not x86-64
    text = re.sub(r"^\s*#\s*include.*$", "", (CSRC / name).read_text(), flags=re.M)
    out = subprocess.run(["g++", "-E", "-P", "-U__x86_64__", "-x", "c++", "-"], input=text, text=True, check=True,
                         capture_output=True).stdout
    assert not re.search(r"target_clones|avx|__builtin_ia32|_mm\d*_", out)

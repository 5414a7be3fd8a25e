"""include/fdtd_b200.h by itself is valid C."""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.mark.skipif(shutil.which("gcc") is None, reason="no C compiler")
def test_header_compiles_as_c(tmp_path):
    source = tmp_path / "uses_header.c"
    source.write_text('#include "fdtd_b200.h"\nint main(void) { return fdtd_version() == 0; }\n')
    done = subprocess.run(["gcc", "-std=c99", "-Wall", "-Werror", "-pedantic", f"-I{ROOT / 'include'}", "-c", str(source),
                           "-o", str(tmp_path / "uses_header.o")], capture_output=True, text=True)
    assert done.returncode == 0, done.stderr

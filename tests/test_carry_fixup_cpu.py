"""The carry fix-up kernels stay inside each row: their source, compiled with
g++ and run on host threads (tests/cuda_on_cpu), on rows that end at an
unreadable page (tests/carry_fixup_check.cpp).  No GPU."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "gpupi_b200" / "csrc"


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not installed")
def test_fixup_stays_inside_rows(tmp_path):
    for name in ("common.cuh", "carry_tile.cuh"):
        # launches are not C++: without the launch shape they parse as calls (the check makes none)
        (tmp_path / name).write_text(re.sub(r"<<<.*?>>>", "", (CSRC / name).read_text(), flags=re.S))
    exe = tmp_path / "carry_fixup_check"
    subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", "-w", f"-I{tmp_path}", f"-I{ROOT / 'tests' / 'cuda_on_cpu'}",
                    str(ROOT / "tests" / "carry_fixup_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stderr)
    assert "carry fix-up ok" in r.stdout

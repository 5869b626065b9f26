"""A kernel's shared-memory limit belongs to the current device: it is raised
on every device that launches the kernel (a fake runtime of 70 devices), and no
translation unit keeps a flag of its own for the whole process."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "atmosphericturbulencesimul_gb300" / "csrc"


def test_limit_is_raised_on_every_device(tmp_path):
    cuda_inc = "/usr/local/cuda/include"
    if not Path(cuda_inc).exists() or shutil.which("g++") is None:
        pytest.skip("g++ or CUDA headers unavailable")
    exe = tmp_path / "smem_emul"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{cuda_inc}", f"-I{CSRC}", str(ROOT / "tests" / "emul" / "smem_emul.cpp"),
                    "-o", str(exe)], check=True)
    out = dict(l.split() for l in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines())
    assert out == {"errors": "0", "once": "64", "again": "6"}


@pytest.mark.parametrize("src", sorted(p.name for p in CSRC.glob("*.cu*")))
def test_no_process_wide_flag(src):
    assert not re.search(r"static\s+bool\s+\w+\s*=", (CSRC / src).read_text())

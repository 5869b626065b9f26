"""CPU emulation of the transforms that run with their stages compiled for the
size: the three-stage rows of 2048, 4096 and 8192 points, the propagation at
2048, and the columns of the large transforms in two passes.

Tolerance 5e-7 of the largest value, as the other emulated transforms."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CHECKS = ["fwd_2048", "inv_2048", "prop_2048", "fwd_4096", "inv_4096", "fwd_8192", "inv_8192", "colfwd_4096", "colinv_4096",
          "colfwd_8192", "colinv_8192"]


@pytest.fixture(scope="module")
def stages(tmp_path_factory):
    exe = tmp_path_factory.mktemp("emul") / "stages_emul"
    cuda_inc = "/usr/local/cuda/include"
    if not Path(cuda_inc).exists() or shutil.which("g++") is None:
        pytest.skip("g++ or CUDA headers unavailable")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{cuda_inc}",
                    f"-I{ROOT / 'atmosphericturbulencesimul_gb300' / 'csrc'}", f"-I{ROOT / 'include'}",
                    str(ROOT / "tests" / "emul" / "stages_emul.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    return {l.split()[0]: float(l.split()[1]) for l in out.strip().splitlines()}


@pytest.mark.parametrize("name", CHECKS)
def test_compiled_stages(stages, name):
    assert stages[name] < 5e-7

"""The chromatic zoom's FP32 bilinear value against the reference's double
expressions, on the CPU (same code as the kernel): over the intensities of PSFs
and the whole range of floats, with fractions that make exact sums and ties,
zeros, denormals, infinities and NaN, every value that is not left to the
doubles is the same float."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def chromat(tmp_path_factory):
    exe = tmp_path_factory.mktemp("emul") / "chromat_emul"
    cuda_inc = "/usr/local/cuda/include"
    if not Path(cuda_inc).exists() or shutil.which("g++") is None:
        pytest.skip("g++ or CUDA headers unavailable")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{cuda_inc}",
                    f"-I{ROOT / 'atmosphericturbulencesimul_gb300' / 'csrc'}", f"-I{ROOT / 'include'}",
                    str(ROOT / "tests" / "emul" / "chromat_emul.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    return {l.split()[0]: tuple(map(float, l.split()[1:])) for l in out.strip().splitlines()}


@pytest.mark.parametrize("name", ["psf", "outside", "outside_few", "outside_close", "outside_wide", "psf_tiny_fractions", "psf_few_fractions", "ties", "dark", "dark_few", "zero",
                                  "wide", "wide_tiny", "faint", "nonfinite"])
def test_the_doubles_result(chromat, name):
    count, differ, _ = chromat[name]
    assert count >= 1000 and differ == 0


def test_the_doubles_are_rare_on_psfs(chromat):
    assert chromat["psf"][2] < 1e-4 and chromat["outside"][2] < 1e-4
    assert chromat["zero"][2] == 0

"""The library's memory pools against a fake CUDA runtime of several devices
(release from any device, room made for an allocation that fails, errors that a
later launch does not report), and on a GPU: memory kept by single calls comes
back with atmwfs_release_workspaces."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_pools_on_a_fake_runtime(tmp_path):
    cuda_inc = "/usr/local/cuda/include"
    if not Path(cuda_inc).exists() or shutil.which("g++") is None:
        pytest.skip("g++ or CUDA headers unavailable")
    exe = tmp_path / "workspace_emul"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{cuda_inc}", f"-I{ROOT / 'atmosphericturbulencesimul_gb300' / 'csrc'}",
                    f"-I{ROOT / 'include'}", str(ROOT / "tests" / "emul" / "workspace_emul.cpp"), "-o", str(exe)], check=True)
    out = dict(l.split() for l in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines())
    assert len(out) == 7 and set(out.values()) == {"1"}, out


@pytest.mark.gpu
def test_single_calls_give_their_memory_back(lib):
    torch = pytest.importorskip("torch")
    from atmosphericturbulencesimul_gb300 import fft2d, release_workspaces
    a = np.ones((4096, 4096), np.complex64)
    fft2d(a)                       # tables and module of this size
    release_workspaces()
    free0 = torch.cuda.mem_get_info()[0]
    fft2d(a)                       # 3 x 134 MB
    kept = free0 - torch.cuda.mem_get_info()[0]
    release_workspaces()
    back = free0 - torch.cuda.mem_get_info()[0]
    assert kept > 100 << 20 and abs(back) < 40 << 20, (kept, back)

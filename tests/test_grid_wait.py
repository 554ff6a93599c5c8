"""What the dependently launched kernels read ahead of the wait for the grid before them.
A grid is promised the writes of earlier grids only after its own griddepcontrol.wait, so
ahead of it a kernel may read what no kernel of the sweep writes, and nothing else."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "cdixx_gb300" / "csrc"


def before_wait(path, name):
    """The code of function `name` up to its wait, without comments."""
    text = re.sub(r"//[^\n]*", "", (CSRC / path).read_text())
    body = re.search(r"\b%s\([^)]*\) \{(.*?)pdl_wait_and_release\(\);" % name, text, re.S)
    assert body, name
    return body.group(1)


@pytest.mark.parametrize("name", ["pty_fwd_rk", "pty_col_rk", "pty_upd_rk"])
def test_sweep_kernels_read_nothing_of_the_sweep_early(name):
    # the object, probe, work, counter, scan order, windows and maxima
    assert not re.findall(r"a\.(?:obj|probe|W|iter|order|win|scal|step)\b|pty_stage_\w+", before_wait("cdx_ptycho.cuh", name))


@pytest.mark.gpu
def test_dependent_positions_equal_plain_launches(tmp_path, torch_cuda):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "pty_chain_check"
    subprocess.run([nvcc, "-std=c++17", "-O3", f"-I{CSRC}", f"-I{ROOT / 'include'}", "-gencode",
                    "arch=compute_103a,code=sm_103a", str(ROOT / "tests" / "cpp" / "pty_chain_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "chain ok" in r.stdout, r.stdout

"""The U-Net's error word (tests/cpp/unet_error_check.cu): a wait that ran out fails one call,
and the network computes again in the next."""
import shutil
import subprocess
from pathlib import Path

import pytest

from cdixx_gb300 import build

ROOT = Path(__file__).resolve().parents[1]
PKG = ROOT / "cdixx_gb300"

pytestmark = pytest.mark.gpu


def test_error_word_is_reported_once(cdx, torch_cuda, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    build.build()   # the objects (nothing to do after a build)
    objs = [str(o) for o in sorted((PKG / "_lib" / "obj").glob("*.o")) if o.name != "cdx_unet.cu.o"]
    exe = tmp_path / "unet_error_check"
    subprocess.run([nvcc, "-std=c++17", "-O1", f"-I{PKG / 'csrc'}", f"-I{ROOT / 'include'}", "-gencode",
                    "arch=compute_103a,code=sm_103a", str(ROOT / "tests" / "cpp" / "unet_error_check.cu"), *objs, "-o",
                    str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "error word ok" in r.stdout, r.stdout

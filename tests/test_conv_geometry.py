"""Host check of the patch geometry and shared-memory plans of the tcgen05 convolutions
(tests/cpp/conv_geometry_check.cu, built with nvcc as host code; no GPU)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_patch_geometry(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not found")
    exe = tmp_path / "conv_geometry_check"
    # cdx_dispatch.cu supplies sm_count; the kernel itself is not launched
    (tmp_path / "sm.cu").write_text("namespace cdx { int sm_count() { return 1; } }\n")
    subprocess.run([nvcc, "-std=c++17", f"-I{ROOT / 'cdixx_gb300' / 'csrc'}", f"-I{ROOT / 'include'}",
                    "-gencode", "arch=compute_103a,code=sm_103a", str(ROOT / "tests" / "cpp" / "conv_geometry_check.cu"),
                    str(tmp_path / "sm.cu"), "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and "geometry ok" in r.stdout, r.stdout

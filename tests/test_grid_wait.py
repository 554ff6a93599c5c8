"""What the dependently launched kernels read ahead of the wait for the grid before them.
A grid is promised the writes of earlier grids only after its own griddepcontrol.wait, so
ahead of it a kernel may read what no kernel of the sweep writes, and nothing else."""
import re
import shutil
import subprocess
from pathlib import Path

import numpy as np
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


def test_pass_kernels_read_nothing_of_the_run_early():
    row = before_wait("cdx_rfft.cuh", "row_pass_body")
    # support words, work, and rho but for its prefetch into the L2
    assert not re.findall(r"a\.(?:mask|in|out)\b|stage_rho\(\);", row)
    col = before_wait("cdx_rfft.cuh", "col_pass_rk")
    assert not re.findall(r"a\.(?:in|out|psi_out)\b", col)
    # the pattern arrays are read early where the host had them complete; the call that
    # makes them on its own stream says so
    assert re.search(r"early = iter && !a\.aux_late && ", col)
    assert re.search(r"c\.aux_late = 1;", (CSRC / "cdx_noalloc.cu").read_text())


@pytest.mark.gpu
def test_dependent_positions_equal_plain_launches(tmp_path, torch_cuda):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "pty_chain_check"
    subprocess.run([nvcc, "-std=c++17", "-O3", f"-I{CSRC}", f"-I{ROOT / 'include'}", "-gencode",
                    "arch=compute_103a,code=sm_103a", str(ROOT / "tests" / "cpp" / "pty_chain_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "chain ok" in r.stdout, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols,batch,ccd", [
    (16, 48, 5, 0), (192, 256, 7, 1), (512, 512, 5, 0), (1024, 768, 1, 0), (2048, 1024, 2, 0), (256, 4096, 3, 1)])
def test_dependent_passes_equal_plain_launches(cdx, torch_cuda, tmp_path, rows, cols, batch, ccd):
    """Many short stretches between shrinkwraps, the support new in each: the tuning file
    chooses dependent or plain launches of the same kernels."""
    import json
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    inten = torch.poisson(torch.rand(rows, cols, device="cuda", generator=g) ** 8 * 6, generator=g)
    torch.cuda.synchronize()   # the contexts read it on streams of their own
    kw = dict(sim_ccd_bit=1, noise_level=4, exposure=0.1) if ccd else {}
    p = cdx.default_params(rows, cols, batch=batch, beta=0.9, shrink_threshold=0.1, autotune=1, **kw)
    out = []
    for pdl in (1, 0):
        f = tmp_path / "tune.json"
        f.write_text(json.dumps({"cdx_tuning": 1, "entries": [
            {"device": torch.cuda.get_device_name(), "rows": rows, "cols": cols, "batch": batch, "pdl_col": pdl,
             "pdl_row": pdl, "row_chunk_bits": 0, "us": 1.0}]}))
        cdx.tuning_load(f)
        with cdx.Context(p) as ctx:
            for k in range(batch):
                ctx.set_pattern(k, inten)
            ctx.random_start(5)
            ctx.run("+".join(["1*shrinkWrap+3*RAAR+2*HIO+1*ER"] * 12))
            assert ctx.tuning()[0] == (3 if pdl else 0)
            out.append([(ctx.get_object(k), ctx.get_support(k)) for k in range(batch)])
    for (a, s), (b, t) in zip(*out):
        assert np.array_equal(a, b) and np.array_equal(s, t) and np.isfinite(a).all()

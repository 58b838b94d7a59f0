"""Host arithmetic of the step kernel's shared memory (propagate.cuh,
stepRoom): no shape asks for more than a CTA may use, whatever the field's
degree.  Compiled for the host with nvcc (no GPU needed)."""
import json
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not Path(NVCC).exists(), reason="nvcc not available")
def test_every_shape_fits_at_every_degree(tmp_path):
    exe = tmp_path / "step_room_check"
    subprocess.run([NVCC, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I", str(ROOT / "parahpop_b200" / "csrc"),
                    str(ROOT / "tests" / "step_room_check.cu"), "-o", str(exe)], check=True)
    out = json.loads(subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout)
    assert out["shapes"] > 8000 and out["over"] == 0 and out["no_warp"] == 0, out

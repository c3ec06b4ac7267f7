"""Length of a batch's step graphs, without a GPU: tests/host_batch_graph.cu is
compiled against the engine's headers.  A graph holds at most 2048 kernels, or
one step's where a step of all scenes has more, counted from the scenes' real
launches (records, dispersive passes and movies among them)."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_graph_length(tmp_path):
    from xfdtd_cuda_b200 import build
    try:
        nvcc = build.nvcc()
    except RuntimeError as e:
        pytest.skip(str(e))
    exe = tmp_path / "host_batch_graph"
    subprocess.run([nvcc, "-std=c++17", "-O2", *build.ARCH, "-I", str(ROOT), "-I", str(ROOT / "include"),
                    "-o", str(exe), str(ROOT / "tests" / "host_batch_graph.cu")], check=True, timeout=600)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout

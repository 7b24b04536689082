"""Host-side rules that send a call to a kernel, compiled from the kernels' own files and checked without a GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = next((c for c in ("/usr/local/cuda/bin/nvcc", shutil.which("nvcc")) if c and os.path.exists(c)), None)


def _run(tmp_path, name):
    exe = str(tmp_path / name)
    src = os.path.join(ROOT, "tests", "native", name + ".cu")
    build = subprocess.run([NVCC, "-O1", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr", "-o", exe, src],
                           stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert build.returncode == 0, build.stdout
    run = subprocess.run([exe], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    return run.returncode, run.stdout


@pytest.mark.skipif(NVCC is None, reason="needs nvcc")
def test_row_matmuls_stay_inside_32_bit_indexes(tmp_path):
    rc, out = _run(tmp_path, "matmul_rows_check")
    assert rc == 0 and "wrong=0" in out, out


@pytest.mark.skipif(NVCC is None, reason="needs nvcc")
def test_depthwise_pieces_are_found_in_few_steps(tmp_path):
    rc, out = _run(tmp_path, "depthwise_pieces_check")
    assert rc == 0 and "wrong=0" in out, out


@pytest.mark.skipif(NVCC is None, reason="needs nvcc")
def test_channel_row_layouts(tmp_path):
    rc, out = _run(tmp_path, "conv_chan_check")
    assert rc == 0 and "wrong=0" in out, out

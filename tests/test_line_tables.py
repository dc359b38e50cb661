"""The [line][k] twiddle tables a domain builds on first use, on a fake CUDA
runtime (line_table_model.cu): no pass reads one before its copy has ended, a
pass whose table finds no memory goes on without it, and a capture under way
on another stream is left alone."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ENGINE = os.path.join(os.path.dirname(HERE), "omr-ntt_gb300")


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    import importlib.util

    spec = importlib.util.spec_from_file_location("engine_build", os.path.join(ENGINE, "build.py"))
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    try:
        nvcc = b.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    exe = str(tmp_path_factory.mktemp("tables") / "model")
    subprocess.run([nvcc, *b.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", b.CSRC,
                    os.path.join(HERE, "line_table_model.cu"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("limit", [1 << 30, 1 << 20, 0], ids=["enough-memory", "too-little", "none"])
def test_table(model, limit):
    r = subprocess.run([model, str(limit)], capture_output=True, text=True, timeout=120)
    assert (r.returncode, r.stdout) == (0, "")

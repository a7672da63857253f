"""mtg_surrogate_loss_grad's results on success and after a timeout, by the engine's own
host code with the GPU calls replaced (tests/surrogate_host/grad_check.cu)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def test_gradient_is_left_alone_after_a_timeout(tmp_path):
    if not os.path.exists(NVCC):
        pytest.skip("nvcc not available")
    out = str(tmp_path / "grad_check")
    r = subprocess.run([NVCC, "-std=c++17", "--expt-relaxed-constexpr", "-Xlinker", "--unresolved-symbols=ignore-all",
                        "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "mt_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "surrogate_host", "grad_check.cu"), "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([out], capture_output=True, text=True, timeout=60)
    from mt_gb300 import _abi, engine
    lines = r.stdout.splitlines()
    assert r.returncode == 0 and lines == [f"timeout: rc {_abi.MTG_E_TIMEOUT} touched 0 loss -1 err 0",
                                           f"success: rc 0 written {engine.SURROGATE_PARAMS} loss 0.6"], r.stdout

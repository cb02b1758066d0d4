"""The surrogate's training kernel when a wait runs out (tests/cpp/test_train_wait.cu)."""
from __future__ import annotations

import os
import subprocess

import pytest

from bbrcit_kde_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EXE = os.path.join(ROOT, "tests", "cpp", "_build", "test_train_wait")


def _compile() -> str:
    try:
        build.nvcc()
    except RuntimeError:
        pytest.skip("needs nvcc")
    os.makedirs(os.path.dirname(EXE), exist_ok=True)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-I", build.CSRC, "-I",
                    build.INCLUDE, os.path.join(ROOT, "tests", "cpp", "test_train_wait.cu"),
                    "-o", EXE], check=True, capture_output=True, text=True)
    return EXE


@pytest.mark.gpu
def test_expired_wait_sets_the_status_and_leaves_nothing_in_flight():
    r = subprocess.run([_compile()], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "ALL PASSED" in r.stdout, r.stdout + r.stderr

"""The pool of device blocks, streams and pinned words on CPU: its host code
against a counting stand-in of the CUDA runtime (tests/native/pool_probe.cpp)."""
from __future__ import annotations

import os
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    cxx = shutil.which("g++")
    cuda = next((p for p in (os.environ.get("CUDA_HOME"), "/usr/local/cuda")
                 if p and (Path(p) / "include" / "cuda_runtime.h").exists()), None)
    if cxx is None or cuda is None:
        pytest.skip("no C++ compiler or CUDA headers")
    exe = tmp_path_factory.mktemp("pool") / "pool_probe"
    env = {k: v for k, v in os.environ.items() if k != "LD_PRELOAD"}
    csrc = ROOT / "hpr-qp-c_b200" / "csrc"
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", f"-I{csrc}", f"-I{cuda}/include", "-o", str(exe),
                    str(ROOT / "tests" / "native" / "pool_probe.cpp"), str(csrc / "context_id.cpp"), str(csrc / "pool.cpp")],
                   check=True, env=env)
    return lambda case: subprocess.run([str(exe), case], capture_output=True, text=True, timeout=60, env=env)


@pytest.mark.parametrize("case", ["first_use", "unknown_context", "release"])
def test_probe(probe, case):
    r = probe(case)
    assert r.returncode == 0, r.stdout + r.stderr

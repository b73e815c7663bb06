"""Asynchronous uploads read their sources when a stream gets to them, not when
the call returns: the host code runs on a stand-in for the CUDA runtime that
reads them as late as it may (tests/cpp/fake_cudart.cpp), through searches,
batches and failures in the middle of them."""

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_sources_outlive_their_uploads(rpg, tmp_path):
    import build

    exe = tmp_path / "upload_lifetime_check"
    objects = [str(build.BUILD / (s + ".o")) for s in build.CUDA_SOURCES + build.CXX_SOURCES]
    compiled = subprocess.run(
        ["g++", "-O1", "-std=c++17", f"-I{ROOT / 'ratpoints-gpu_gb300' / 'csrc'}",
         f"-I{build.cuda_home() / 'include'}", str(ROOT / "tests" / "cpp" / "upload_lifetime_check.cpp"),
         str(ROOT / "tests" / "cpp" / "fake_cudart.cpp"), *objects, "-o", str(exe), "-pthread"],
        capture_output=True, text=True)
    assert compiled.returncode == 0, compiled.stderr
    done = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr
    assert "all sources kept" in done.stdout

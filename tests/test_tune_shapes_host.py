"""A shape of the fast plan selects the primes that a search tests; shapes that
select the same ones run the same kernel, and the tuner times one of them."""

import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
RECORD = "247747600 -985905640 567207969 2396040466 52485681 -470135160 82342800".split()


@pytest.fixture(scope="module")
def check(rpg, tmp_path_factory):
    import build

    exe = tmp_path_factory.mktemp("tune") / "tune_shapes_check"
    objects = [str(build.BUILD / (s + ".o")) for s in build.CUDA_SOURCES + build.CXX_SOURCES]
    compiled = subprocess.run(
        ["g++", "-O1", "-std=c++17", f"-I{ROOT / 'ratpoints-gpu_gb300' / 'csrc'}",
         f"-I{build.cuda_home() / 'include'}", str(ROOT / "tests" / "cpp" / "tune_shapes_check.cpp"),
         str(ROOT / "tests" / "cpp" / "fake_cudart.cpp"), *objects, "-o", str(exe), "-pthread"],
        capture_output=True, text=True)
    assert compiled.returncode == 0, compiled.stderr
    return lambda bound, coefficients: subprocess.run([str(exe), str(bound), *coefficients], capture_output=True,
                                                      text=True, timeout=120)


@pytest.mark.parametrize("bound", [20_000, 400_000, 5_000_000])
@pytest.mark.parametrize("curve", ["c2", "record", "quintic"])
def test_each_set_of_primes_is_timed_once(check, monkeypatch, curve, bound):
    import bench

    monkeypatch.delenv("RPG_TUNE_CACHE", raising=False)
    coefficients = {"c2": bench.c2_curve(), "record": RECORD, "quintic": ["9", "1", "-7", "0", "3", "2"]}[curve]
    done = check(bound, [str(c) for c in coefficients])
    assert done.returncode == 0, done.stdout + done.stderr

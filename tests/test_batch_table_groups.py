"""Curves of a batch with launches of their own whose tables do not fit the
device together: they are swept in groups, the tables of one at a time.  On the
host through a stand-in for the CUDA runtime; on the GPU with groups made small
by RPG_BATCH_TABLE_BYTES, against the batch in one group."""

import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
SEXTIC = ["-533746463", "2318474698", "1819918790", "-3268433658", "1978982371", "1087269120", "-559365050"]
DENSE = "247747600 -985905640 567207969 2396040466 52485681 -470135160 82342800".split()


def test_batches_that_do_not_fit_run_in_groups(rpg, tmp_path):
    import build

    exe = tmp_path / "batch_memory_check"
    objects = [str(build.BUILD / (s + ".o")) for s in build.CUDA_SOURCES + build.CXX_SOURCES]
    compiled = subprocess.run(
        ["g++", "-O1", "-std=c++17", f"-I{ROOT / 'ratpoints-gpu_gb300' / 'csrc'}",
         f"-I{build.cuda_home() / 'include'}", str(ROOT / "tests" / "cpp" / "batch_memory_check.cpp"),
         str(ROOT / "tests" / "cpp" / "fake_cudart.cpp"), *objects, "-o", str(exe), "-pthread"],
        capture_output=True, text=True)
    assert compiled.returncode == 0, compiled.stderr
    done = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("table_bytes", ["1", "4000000", "40000000"])
def test_groups_find_what_one_group_finds(rpg, monkeypatch, table_bytes):
    curves = [{"coefficients": coeffs, "bound": bound, "first": 1, "last": last, "intervals": intervals}
              for coeffs in (SEXTIC, DENSE, ["9", "1", "-7", "0", "3", "2"])
              for bound, last, intervals in ((70_000, 300, ()), (300_000, 90, ()), (20_011, 36_000, ()),
                                             (900, 40, ()), (80_000, 2_000, [("-0.5", "2")]))]
    expected = rpg.batch_search(curves)[:3]
    assert not any(expected[1])
    monkeypatch.setenv("RPG_BATCH_TABLE_BYTES", table_bytes)
    for graph in (True, False):
        assert rpg.batch_search(curves, graph=graph)[:3] == expected
    # run again with room for all survivors: the groups' tables once more
    monkeypatch.setenv("RPG_BATCH_CAPACITY", "16")
    assert rpg.batch_search(curves)[:3] == expected
    monkeypatch.delenv("RPG_BATCH_TABLE_BYTES")
    assert rpg.batch_search(curves)[:3] == expected

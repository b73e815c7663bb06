"""The single-curve kernel's plans on the host: what they say of the curve's
primes, through a small C++ program linked with the library
(tests/cpp/sweep_plan_check.cpp)."""

import math
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
RECORD = "247747600 -985905640 567207969 2396040466 52485681 -470135160 82342800".split()


def primes(lo, hi):
    return [p for p in range(lo, hi) if p > 1 and all(p % f for f in range(2, math.isqrt(p) + 1))]


@pytest.fixture(scope="module")
def check(rpg, tmp_path_factory):
    import build

    exe = tmp_path_factory.mktemp("sweep") / "sweep_plan_check"
    lib_dir = Path(rpg.LIBRARY).parent
    compiled = subprocess.run(
        ["g++", "-O1", "-std=c++17", f"-I{ROOT / 'ratpoints-gpu_gb300' / 'csrc'}", f"-I{ROOT / 'include'}",
         f"-I{build.cuda_home() / 'include'}", str(ROOT / "tests" / "cpp" / "sweep_plan_check.cpp"), "-o", str(exe),
         f"-L{lib_dir}", "-lrpgpu", f"-Wl,-rpath,{lib_dir}", "-pthread"], capture_output=True, text=True)
    assert compiled.returncode == 0, compiled.stderr

    def run(what, bound, coefficients):
        done = subprocess.run([str(exe), what, str(bound), *map(str, coefficients)], capture_output=True, text=True,
                              timeout=120)
        assert done.returncode == 0, done.stderr
        return done.stdout

    return run


def one_residue_curve(q, r):
    """f = A (x - r)^2 + q^2: a square at every x mod the odd primes below 257
    (A is divisible by them), at x = r alone mod q (A is no square mod q), with
    the point (r, q, 1)."""
    a = math.prod(primes(3, 257))
    while pow(a, (q - 1) // 2, q) == 1:
        a += math.prod(primes(3, 257))
    assert a % q
    return [a * r * r + q * q, -2 * a * r, a]


@pytest.mark.parametrize("q", [257, 331, 509])
def test_a_prime_with_one_admitted_residue_is_not_one_without(check, q):
    # more than eight bits of filtering, but not a divisor that d needs
    out = check("admitted", 100_000, one_residue_curve(q, 5)).split()
    assert str(q) in out[:-2]
    assert int(out[-1]) > 0


@pytest.mark.parametrize("coefficients", [RECORD, ["2", "3", "-6", "9"], ["5", "3", "-6", "9", "2"],
                                          ["-9876543210", "1234567", "0", "1"]])
def test_plans_carry_their_primes_residue_counts(check, coefficients):
    for bound in (1_000, 100_000, 10 ** 7):
        check("admitted", bound, coefficients)


# a square at every x modulo every odd prime below 512: no row filters
EVERYTHING = [1, math.prod(primes(3, 512))]


@pytest.mark.parametrize("bound", [1_000, 100_000, 10 ** 8])
def test_a_curve_that_nothing_filters_has_a_cost(check, bound):
    # launches are cut by it, and a batch's ordered: not less than a curve
    # whose words mostly end in the rows
    for everything, sparse in zip(check("cost", bound, EVERYTHING).split(), check("cost", bound, [2, -3, 0, 5]).split()):
        assert float(everything) >= float(sparse) > 0


@pytest.mark.parametrize("bound", [10_400, 12_000, 16_383, 60_000, 65_503, 65_504, 300_000, 1_000_000, 4_000_000])
@pytest.mark.parametrize("coefficients", [RECORD, [2, -3, 0, 5], [-533746463, 2318474698, 1819918790, -3268433658,
                                                                  1978982371, 1087269120, -559365050], EVERYTHING])
def test_a_batch_admits_what_its_curves_take(check, coefficients, bound):
    # curves with launches of their own: not less than their tables, nor much more
    # than the largest
    rows = [list(map(int, line.split())) for line in check("memory", bound, coefficients).splitlines()]
    assert rows
    for last, tables, *estimates in rows:
        assert all(tables <= estimate <= 64 << 20 for estimate in estimates), (last, tables, estimates)


@pytest.mark.gpu
def test_survivors_of_a_curve_that_nothing_filters(rpg):
    # reference plan: every site; fast plan: those that are squares mod 64
    a, d, _ = rpg.sieve(EVERYTHING, 70_000, 11, 12)
    assert sorted(zip(d.tolist(), a.tolist())) == [(k, x) for k in (11, 12) for x in range(-70_000, 70_001)]
    # and not multiples of a row prime (5 and 7) that divides d: F(a, d) = d (d + P a)
    squares = {v * v % 64 for v in range(64)}
    expected = [(k, x) for k in (11, 12) for x in range(-70_000, 70_001)
                if (k % 2 or x % 2) and k * (k + EVERYTHING[1] * x) % 64 in squares]
    a, d, _ = rpg.sieve(EVERYTHING, 70_000, 11, 12, plan="fast")
    assert sorted(zip(d.tolist(), a.tolist())) == expected
    points, status, survivors, _ = rpg.batch_search([{"coefficients": EVERYTHING, "bound": 70_000, "first": 11, "last": 12}])
    assert status == [0] and survivors == [len(expected)]
    assert points[0] == rpg.point_search(EVERYTHING, 70_000, 11, 12)[0]


@pytest.mark.gpu
@pytest.mark.parametrize("q", [257, 331, 509])
def test_the_point_of_a_curve_with_one_admitted_residue(rpg, q):
    curve = one_residue_curve(q, 5)
    points, _ = rpg.point_search(curve, 100_000, 1, 256)
    assert (5, q, 1) in points
    batch, status, _, _ = rpg.batch_search([{"coefficients": curve, "bound": 100_000, "first": 1, "last": 256}])
    assert status == [0] and batch[0] == points


@pytest.mark.gpu
@pytest.mark.parametrize("last", [1, 2, 50, 3_000])
@pytest.mark.parametrize("bound", [70_000, 1_000_003, 4_000_000])
@pytest.mark.parametrize("coefficients", [RECORD, ["2", "-3", "0", "5"]])
def test_launches_count_the_words_they_sweep(rpg, check, coefficients, bound, last):
    # also those of a denominator with fewer sweep items than it has shares
    _, status, _, stats = rpg.batch_search([{"coefficients": coefficients, "bound": bound, "first": 1, "last": last}])
    expected = int(check("swept", bound, [last, *coefficients]))
    assert status == [0] and stats["swept_words"] == expected > 0

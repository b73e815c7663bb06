"""The sieve kernel over the ways it splits a plan's tests (class primes, rows,
late primes, shares of a denominator, ranges of numerators): its survivors are
the oracle's for the reference plan, and those of them that pass the fast
plan's filters for the fast plan."""

import pytest

from test_fast_plan_gpu import check
from test_sieve_gpu import assert_same_set

pytestmark = pytest.mark.gpu

DENSE = "247747600 -985905640 567207969 2396040466 52485681 -470135160 82342800".split()
CURVES = {"sextic": ["-533746463", "2318474698", "1819918790", "-3268433658", "1978982371", "1087269120", "-559365050"],
          "quintic": ["9", "1", "-7", "0", "3", "2"], "dense": DENSE}

# around classes of 16 words of 64 sites (a class prime more or less), of one
# word, and long enough for several class primes
BOUNDS = [31, 32_767, 32_768, 98_303, 163_841, 360_449, 2_500_001]


@pytest.mark.parametrize("bound", BOUNDS)
@pytest.mark.parametrize("curve", CURVES)
def test_survivors(rpg, oracle, curve, bound):
    # the second range has multiples of likely class primes and of candidates
    for first, last in ((1, 12), (3 * 5 * 7 * 11 * 13, 3 * 5 * 7 * 11 * 13 + 2), (349 * 509, 349 * 509 + 1)):
        assert_same_set(rpg, oracle, CURVES[curve], bound, first, last)
        check(rpg, oracle, CURVES[curve], bound, first, last)


def test_square_denominators_with_long_classes(rpg, oracle):
    # few denominators of many words: each is shared out over several CTAs
    check(rpg, oracle, ["7", "-10", "0", "1"], 20_000_003, 14, 19, square=True)
    assert_same_set(rpg, oracle, ["7", "-10", "0", "1"], 20_000_003, 21, 22, square=True)


@pytest.mark.parametrize("plan", ["reference", "fast"])
def test_numerator_ranges(rpg, monkeypatch, plan):
    # a buffer of 64 survivors: denominators are split into ranges of
    # numerators, down to 64, at every position of a class word
    coeffs = ["4", "0", "1", "0", "1"] if plan == "fast" else DENSE
    bound, first, last = (40_009, 1, 3) if plan == "fast" else (400_009, 1, 2)
    expected = sorted(zip(*(v.tolist() for v in rpg.sieve(coeffs, bound, first, last, plan=plan)[:2])))
    monkeypatch.setenv("RPG_SURVIVOR_CAPACITY", "64")
    got = sorted(zip(*(v.tolist() for v in rpg.sieve(coeffs, bound, first, last, plan=plan)[:2])))
    assert got == expected and len(expected) > 0


def test_primes_without_squares(rpg, oracle):
    # 2 + 3 (..) is no square mod 3: only denominators divisible by 3 keep
    # survivors (odd degree), or none at all (even degree, leading coefficient
    # not a square mod 3)
    for coeffs in (["2", "3", "-6", "9"], ["5", "3", "-6", "9", "2"], ["2", "15", "-30", "45", "4"]):
        for first, last in ((1, 40), (13 * 15, 13 * 15 + 3)):
            assert_same_set(rpg, oracle, coeffs, 50_003, first, last)
            check(rpg, oracle, coeffs, 50_003, first, last)
    # modulo a candidate of the reference plan
    coeffs = ["2", "509", "0", "-1018"]  # 2 is not a square mod 509
    assert_same_set(rpg, oracle, coeffs, 20_011, 500, 520)
    check(rpg, oracle, coeffs, 20_011, 500, 520)


def test_batched_curves_with_launches_of_their_own(rpg):
    # either side of the batch's rule: wide rows whatever the denominators,
    # shorter ones only with many; such a curve's points and survivors are
    # those of its own search
    curves = [{"coefficients": CURVES[name], "bound": bound, "first": first, "last": last}
              for name in CURVES
              for bound, first, last in ((65_503, 1, 50), (65_504, 1, 50), (300_000, 7, 7), (20_011, 1, 36_000),
                                         (20_011, 5, 30_000), (9_001, 1, 60_000))]
    points, status, survivors, stats = rpg.batch_search(curves)
    assert status == [0] * len(curves)
    alone = 0
    for c, got, n in zip(curves, points, survivors):
        expected, st = rpg.point_search(c["coefficients"], c["bound"], c["first"], c["last"])
        assert got == expected, c
        alone += n == st["survivor_count"]
        if c["bound"] >= 65_504 or c["last"] == 36_000:
            assert n == st["survivor_count"], c
    assert alone >= 9 and stats["wide_curves"] == 6


@pytest.mark.parametrize("last", [1, 7, 33, 700])
def test_narrow_rows(rpg, last):
    # rows and x ranges either side of the one-word-per-lane steps (32 and 96
    # words), a word's first and last bit, overlapping, empty and many
    # intervals, with few and many denominators per work item
    several = [(f"{i - 3.5:.2f}", f"{i - 3.5 + 0.3 * i:.2f}") for i in range(8)]
    curves = []
    for bound in (1, 31, 32, 1_023, 1_024, 3_071, 3_103, 9_000):
        for intervals in ((), [("-0.5", "0.5")], [("0", "0"), ("-2", "1.75"), ("1.5", "3"), ("5", "4")], several):
            for coeffs, square in ((["1", "0", "0", "1"], False), (["4", "-3", "0", "0", "1"], False),
                                   (["1", "-1", "0", "1"], True)):
                curves.append({"coefficients": coeffs, "bound": bound, "first": 1, "last": last,
                               "intervals": intervals, "square": square})
    points, status, _, stats = rpg.batch_search(curves)
    assert status == [0] * len(curves) and stats["wide_curves"] == 0
    for c, got in zip(curves, points):
        expected, _ = rpg.point_search(c["coefficients"], c["bound"], 1, last, intervals=c["intervals"],
                                       square=c["square"])
        assert got == expected, c

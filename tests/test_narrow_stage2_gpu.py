"""Stage 2 of the batch's narrow kernel: words of one site and words full of
them take different ways through it, and words with several sites go round
again.  The survivors of a curve are the reference plan's that are also squares
modulo 64 and the small primes that filter."""

import math

import pytest

pytestmark = pytest.mark.gpu

PRIMES = [p for p in range(3, 34) if all(p % q for q in range(2, p))]


def everything():
    # 1 + P x, P the product of the 32 largest primes below 512: each site
    # passes every candidate
    largest = [p for p in range(2, 512) if all(p % q for q in range(2, int(p ** 0.5) + 1))][-32:]
    return [1, math.prod(largest)]


CURVES = {"everything": everything(),
          "dense": [247747600, -985905640, 567207969, 2396040466, 52485681, -470135160, 82342800],
          "conic": [1, 0, 1], "quintic": [9, 1, -7, 0, 3, 2], "quartic": [4, 0, 1, 0, 1]}


def plan_primes(coeffs):
    """The primes of the narrow plan: the strongest first, packed into eight
    moduli of at most 34 while m (m + 3) words of each fit."""
    bits = []
    for p in PRIMES:
        squares = {v * v % p for v in range(p)}
        rate = sum(sum(c * x ** i for i, c in enumerate(coeffs)) % p in squares for x in range(p)) / p
        if rate == 0 or -math.log2(rate) >= 0.15:
            bits.append((math.log2(rate) if rate else -8.0, p))
    moduli, primes = [], []
    for _, p in sorted(bits):
        joins = [m for m in moduli if m * p <= 34]
        trial = sorted(moduli)
        if joins:
            trial[trial.index(min(joins))] *= p
        else:
            trial.append(p)
        if len(trial) <= 8 and sum(m * (m + 3) for m in trial) + 4 * (8 - len(trial)) <= 7679:
            moduli = trial
            primes.append(p)
    return primes


def survives(coeffs, primes, a, d):
    n = len(coeffs) - 1
    f = sum(c * a ** i * d ** (n - i) for i, c in enumerate(coeffs)) * (d if n % 2 else 1)
    if a % 2 == 0 and d % 2 == 0 or f % 64 not in {v * v % 64 for v in range(64)}:
        return False
    for p in primes:
        if a % p == 0 and d % p == 0 or f % p not in {v * v % p for v in range(p)}:
            return False
    # denominator primes: an even degree whose leading coefficient is no square mod p | d
    return n % 2 == 1 or all(d % p or coeffs[-1] % p == 0 or
                             pow(coeffs[-1], (p - 1) // 2, p) == 1 for p in range(3, min(d, 511) + 1, 2)
                             if all(p % q for q in range(3, int(p ** 0.5) + 1, 2)))


@pytest.mark.parametrize("bound,last", [(40, 7), (700, 90), (3_200, 33)])
@pytest.mark.parametrize("name", CURVES)
def test_survivors(rpg, name, bound, last):
    coeffs = CURVES[name]
    text = [str(c) for c in coeffs]
    primes = plan_primes(coeffs)
    a, d, _ = rpg.sieve(text, bound, 1, last)
    expected = sum(survives(coeffs, primes, x, y) for x, y in zip(a.tolist(), d.tolist()))
    points, status, survivors, _ = rpg.batch_search([{"coefficients": text, "bound": bound, "first": 1, "last": last}])
    assert status == [0] and survivors == [expected] and expected > 0
    assert points[0] == rpg.point_search(text, bound, 1, last)[0]

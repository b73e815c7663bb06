"""rpg_session_sieve_noalloc takes every numerator bound up to its limits, also
for curves that few primes filter: their classes are few and long, and a row
takes several launches."""

import math

import pytest

from test_zz_no_alloc import _entry

pytestmark = pytest.mark.gpu

PRIMES = [p for p in range(3, 512) if all(p % q for q in range(2, int(p ** 0.5) + 1))]


def count(rpg, coefficients, plan, bound, d):
    import torch

    session = rpg.Session([str(c) for c in coefficients], bound, plan=plan)
    a = torch.full((8,), -1, dtype=torch.int64, device="cuda")
    dd = torch.full((8,), -1, dtype=torch.int32, device="cuda")
    total = torch.zeros(1, dtype=torch.int64, device="cuda")
    try:
        status = _entry(rpg)(session._handle, d, d, a.data_ptr(), dd.data_ptr(), 8, total.data_ptr(), None)
        assert status == 0, rpg.load().rpg_last_error().decode()
        torch.cuda.synchronize()
        assert all(-bound <= x <= bound for x in a.tolist()) and set(dd.tolist()) == {d}
        return int(total.item())
    finally:
        session.close()


def test_reference_plan(rpg):
    pytest.importorskip("torch")
    # every site is a square modulo every candidate: a row of 2^29 words
    bound = (1 << 34) + 12_345
    assert count(rpg, [1, math.prod(PRIMES)], "reference", bound, 1) == 2 * bound + 1


def test_fast_plan(rpg):
    pytest.importorskip("torch")
    # 2 mod 3 (no square: class prime 3, only multiples of 3 as denominators),
    # 1 modulo the other primes
    others = math.prod(PRIMES[1:])
    c = next(v for v in (1 + others * k for k in range(3)) if v % 3 == 2)
    coefficients = [c, 3 * others]
    bound, d = (1 << 34) + 12_345, 3
    squares = {v * v % 64 for v in range(64)}
    residues = {r for r in range(192) if r % 3 and d * (c * d + 3 * others * r) % 64 in squares}
    # numerators a = r mod 192 in [-bound, bound]
    expected = sum((bound - r) // 192 - (-bound - 1 - r) // 192 for r in residues)
    assert count(rpg, coefficients, "fast", bound, d) == expected

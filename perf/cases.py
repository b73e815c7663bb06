"""Cases that measure the rational-point search through its public entry points.

Kinds of case (what a user of the framework runs):

  search  rpg.point_search: one curve, verified points (the fast plan), with the
          options in earnest use: x intervals, square denominators, a first
          denominator above 1, a dense curve
  sieve   rpg.sieve: the modular survivors of the reference plan (the
          run_modular_sieve boundary)
  batch   rpg.batch_search: many curves in one call
  serve   rpg.Server: a burst of requests through a server that stays up

Sizes follow the benchmark configurations (workloads.py), the tests and the
campaign callers.  Curves are random with one known point planted (a user
searches a curve for more points than the ones in hand), so that the outputs
hold points to compare.  All outputs are whole numbers: numerators,
denominators, and the ordinates in 62-bit limbs.
"""

import math
import os
import random
import sys

import numpy as np

_PACKAGE = os.path.join(os.getcwd(), "ratpoints-gpu_gb300")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import ratpoints_gb300 as rpg  # noqa: E402

# the genus-2 curve with the most known points, c0 .. c6 (workloads.RECORD_CURVE)
_DENSE = (247747600, -985905640, 567207969, 2396040466, 52485681, -470135160, 82342800)


def _search(name, degree, bits, bound, last, first=1, intervals=0, square=False, dense=False):
    return {"name": name, "kind": "search", "degree": degree, "bits": bits, "bound": bound, "first": first,
            "last": last, "intervals": intervals, "square": square, "dense": dense}


def _batch(name, curves, degree_lo, degree_hi, bits_lo, bits_hi, bound_lo, bound_hi, last_lo, last_hi,
           intervals=0):
    return {"name": name, "kind": "batch", "curves": curves, "degree_lo": degree_lo, "degree_hi": degree_hi,
            "bits_lo": bits_lo, "bits_hi": bits_hi, "bound_lo": bound_lo, "bound_hi": bound_hi,
            "last_lo": last_lo, "last_hi": last_hi, "intervals": intervals}


def listed():
    return [
        # the smallest call: a first look at a curve, all latency and launches
        _search("search_tiny", 6, 6, 2_000, 2_000),
        # an ordinary look at one curve: the box of the reference's CPU comparison
        _search("search_plain", 6, 32, 300_000, 300_000),
        # the headline search: degree 6, 5e13 sites
        _search("search_large", 6, 32, 5_000_000, 5_000_000),
        # a curve with hundreds of points: square modulo most small primes, so
        # that the rows are of large primes and filter weakly
        _search("search_dense", 6, 32, 10_000_000, 100_000, dense=True),
        # an integral Weierstrass cubic: square denominators, huge rows
        _search("search_square", 3, 40, 1_000_000_000, 4_001, square=True),
        # odd degree, ragged sizes, a continued search (first above 1), two intervals
        _search("search_ranges", 5, 64, 1_234_567, 400_003, first=1_001, intervals=2),
        # many curves of uneven degree, coefficient size, height and depth
        _batch("batch_mixed", 512, 3, 10, 8, 64, 1_000, 1_000_000, 1_000, 1_000_000),
        # a campaign's screen: many quartics and cubics to a small height
        _batch("batch_screen", 384, 3, 4, 16, 48, 2_000, 30_000, 500, 10_000),
        # high degree, coefficients of several words, three intervals each
        _batch("batch_highdegree", 96, 12, 40, 100, 256, 100_000, 100_000, 100_000, 100_000, intervals=3),
        # a burst of requests of mixed height, three in ten for the first point only
        {"name": "serve_burst", "kind": "serve", "requests": 128, "degree_lo": 2, "degree_hi": 12,
         "bits_lo": 16, "bits_hi": 128, "bound_lo": 100, "bound_hi": 300_000, "first_share": 0.3},
        # the sieve alone behind the reference's boundary: exactly its survivor set
        {"name": "sieve_reference", "kind": "sieve", "degree": 6, "bits": 32, "bound": 5_000_000, "first": 1,
         "last": 40_009, "square": False, "dense": False},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("search", "search", "search", "search_dense", "search_square", "batch", "batch_high",
                       "batch_small", "serve", "sieve"))
    if kind == "search":
        bound = _log_uniform(rng, 1_000, 6_000_000)
        last = _log_uniform(rng, 500, 4_000_000)
        first = 1 if rng.random() < 0.6 else rng.randint(1, last // 2)
        return _drawn(_search("", rng.randint(3, 12), rng.randint(8, 64), bound, last, first,
                              rng.choice((0, 0, 0, 1, 3))))
    if kind == "search_dense":
        return _drawn(_search("", 6, 32, _log_uniform(rng, 30_000, 10_000_000), _log_uniform(rng, 1_000, 100_000),
                              dense=True))
    if kind == "search_square":
        return _drawn(_search("", rng.choice((3, 3, 5)), rng.randint(8, 40),
                              _log_uniform(rng, 100_000, 1_000_000_000), _log_uniform(rng, 100, 4_000), square=True))
    if kind == "batch":
        lo, hi = _log_uniform(rng, 200, 10_000), _log_uniform(rng, 20_000, 1_000_000)
        return _drawn(_batch("", _log_uniform(rng, 2, 400), 3, rng.randint(4, 10), 8, 64, lo, hi, 300,
                             _log_uniform(rng, 2_000, 600_000)))
    if kind == "batch_high":
        bound = _log_uniform(rng, 5_000, 150_000)
        return _drawn(_batch("", _log_uniform(rng, 4, 96), rng.randint(8, 14), 40, 64, 256, bound, bound, 1_000,
                             bound, intervals=rng.randint(1, 4)))
    if kind == "batch_small":
        return _drawn(_batch("", _log_uniform(rng, 8, 600), 3, rng.randint(3, 6), 8, 48, 200,
                             _log_uniform(rng, 1_000, 40_000), 100, _log_uniform(rng, 500, 12_000)))
    if kind == "serve":
        return {"kind": "serve", "requests": _log_uniform(rng, 4, 128), "degree_lo": 2, "degree_hi": 12,
                "bits_lo": 16, "bits_hi": 128, "bound_lo": 100, "bound_hi": _log_uniform(rng, 3_000, 250_000),
                "first_share": 0.3}
    return {"kind": "sieve", "degree": rng.randint(3, 8), "bits": rng.randint(8, 64),
            "bound": _log_uniform(rng, 2_000, 5_000_000), "first": 1, "last": _log_uniform(rng, 500, 40_000),
            "square": False, "dense": rng.random() < 0.3}


def _drawn(case):
    del case["name"]
    return case


# ---------------------------------------------------------------------------
# Inputs


def _convolve(p, q):
    out = [0] * (len(p) + len(q) - 1)
    for i, x in enumerate(p):
        for j, y in enumerate(q):
            out[i + j] += x * y
    return out


def _signed(rng, bits):
    """A nonzero integer of at most `bits` bits."""
    while True:
        v = rng.randrange(-(1 << bits), 1 << bits)
        if v:
            return v


def _random_curve(rng, degree, bits, bound, first, last):
    """Coefficients c0 .. cn of about `bits` bits of a squarefree polynomial
    f = g^2 + (v x - u) h, which has the point x = u / v (and is otherwise
    random), and that x."""
    while True:
        v = rng.randint(first, min(last, first + min(1 << max(3, bits // 3), 1000)))
        u = rng.randint(-min(bound, 4 * v), min(bound, 4 * v))
        size = max(1, max(abs(u), v).bit_length())
        g = [_signed(rng, max(1, bits // 2 - 1)) for _ in range((degree - 1) // 2 + 1)]
        h = [_signed(rng, max(2, bits - size)) for _ in range(degree)]
        f = _convolve([-u, v], h)
        for i, x in enumerate(_convolve(g, g)):
            f[i] += x
        coeffs = [str(c) for c in f]
        if f[-1] and rpg.is_squarefree(coeffs):
            return coeffs, u / v


def _monic_curve(rng, degree, bits):
    """c0 .. cn = 1 of a squarefree x^n + c_(n-2) x^(n-2) + .. + c0 through an integral point."""
    while True:
        f = [0] + [_signed(rng, bits) for _ in range(degree - 2)] + [0, 1]
        u, y = rng.randint(-1000, 1000), rng.getrandbits(bits // 2)
        f[0] = y * y - sum(c * u ** i for i, c in enumerate(f))
        coeffs = [str(c) for c in f]
        if rpg.is_squarefree(coeffs):
            return coeffs


def _dense_curve(rng):
    """A translate x -> x + k of the dense curve, reversed or reflected at
    random: the same local behaviour, other coefficients."""
    k = rng.randint(-40, 40)
    shifted = [0]
    for c in reversed(_DENSE):  # Horner in (x + k)
        shifted = _convolve(shifted, [k, 1])
        shifted[0] += c
    shifted = shifted[:len(_DENSE)]
    if rng.random() < 0.5 and shifted[0]:
        shifted.reverse()
    if rng.random() < 0.5:
        shifted = [c if i % 2 == 0 else -c for i, c in enumerate(shifted)]
    return [str(c) for c in shifted]


def _intervals(rng, count, x):
    """`count` intervals, the first around the known point."""
    out = []
    for i in range(count):
        width = rng.uniform(0.05, 1)
        lo = x - width * rng.uniform(0.2, 0.8) if i == 0 else rng.uniform(-4, 4)
        out.append((f"{lo:.4f}", f"{lo + width:.4f}"))
    return out


def _curve(rng, degree, bits, bound, first, last, intervals=0):
    coeffs, x = _random_curve(rng, degree, bits, bound, first, last)
    return {"coefficients": coeffs, "bound": bound, "first": first, "last": last,
            "intervals": _intervals(rng, intervals, x)}


def _single_curve(rng, case):
    """(coefficients, intervals) of a search or sieve case."""
    if case["dense"]:
        return _dense_curve(rng), []
    if case["square"]:
        return _monic_curve(rng, case["degree"], case["bits"]), []
    curve = _curve(rng, case["degree"], case["bits"], case["bound"], case["first"], case["last"],
                   case.get("intervals", 0))
    return curve["coefficients"], curve["intervals"]


def prepare(case, seed):
    rng = random.Random(int(seed) * 1_000_003 + 17)
    kind = case["kind"]
    state = {"case": case, "kind": kind}
    if kind in ("search", "sieve"):
        state["coefficients"], state["intervals"] = _single_curve(rng, case)
        return state
    if kind == "batch":
        state["curves"] = [
            _curve(rng, rng.randint(case["degree_lo"], case["degree_hi"]), rng.randint(case["bits_lo"], case["bits_hi"]),
                   _log_uniform(rng, case["bound_lo"], case["bound_hi"]), 1,
                   _log_uniform(rng, case["last_lo"], case["last_hi"]), case["intervals"])
            for _ in range(case["curves"])]
        return state
    requests = []
    for _ in range(case["requests"]):
        bound = _log_uniform(rng, case["bound_lo"], case["bound_hi"])
        curve = _curve(rng, rng.randint(case["degree_lo"], case["degree_hi"]),
                       rng.randint(case["bits_lo"], case["bits_hi"]), bound, 1, bound)
        requests.append((curve, rng.random() < case["first_share"]))
    state["requests"] = requests
    state["server"] = rpg.Server()  # a serving program keeps it
    return state


# ---------------------------------------------------------------------------
# One pass


_ROWS = 4096        # points of a pass (hundreds at most on the curves searched)
_LIMBS = 8          # 62-bit limbs of an ordinate (the largest here has about 470 bits)
_LOW = (1 << 62) - 1


def _points(answers):
    """Point lists [(a, y, d)] of one or many curves as one array of fixed
    size: rows of curve + 1, a, d and the limbs of y, zeros after the last."""
    out = np.zeros((_ROWS, 3 + _LIMBS), dtype=np.int64)
    at = 0
    for i, points in enumerate(answers):
        for a, y, d in points:
            row = out[at]  # past the last row: an IndexError
            row[0], row[1], row[2] = i + 1, a, d
            for k in range(_LIMBS):
                if not y:
                    break
                row[3 + k] = y & _LOW
                y >>= 62
            at += 1
    return out


def _sites(a, d, rows):
    """Modular survivors in (d, a) order (a batch's sites arrive in no order),
    zeros after the last."""
    order = np.lexsort((a, d))
    out = np.zeros((2, rows), dtype=np.int64)
    out[0, :a.size] = a[order]
    out[1, :d.size] = d[order]
    return out


def run(state):
    case, kind = state["case"], state["kind"]
    if kind == "search":
        points, _ = rpg.point_search(state["coefficients"], case["bound"], case["first"], case["last"],
                                     intervals=state["intervals"], square=case["square"])
        return _points([points])
    if kind == "sieve":
        a, d, _ = rpg.sieve(state["coefficients"], case["bound"], case["first"], case["last"], square=case["square"])
        return _sites(a, d, 1 << 20 if case["dense"] else 1 << 18)
    if kind == "batch":
        points, status, _, _ = rpg.batch_search(state["curves"])
        return {"points": _points(points), "status": np.array(status, dtype=np.int64)}
    server = state["server"]
    ids = [server.submit(curve, first) for curve, first in state["requests"]]
    answers = [server.wait(i) for i in ids]
    return {"points": _points([points for _, points, _ in answers]),
            "status": np.array([status for status, _, _ in answers], dtype=np.int64)}


# ---------------------------------------------------------------------------
# What a pass cannot do without


def _boxes(case):
    """(count, numerator bound, denominators) of the boxes a pass decides; the
    expected box where sizes are drawn per curve."""
    if case["kind"] in ("search", "sieve"):
        return [(1, case["bound"], case["last"] - case["first"] + 1)]

    def mean(lo, hi):  # of a log-uniform draw
        return (hi - lo) / math.log(hi / lo) if hi > lo else lo

    if case["kind"] == "batch":
        return [(case["curves"], mean(case["bound_lo"], case["bound_hi"]), mean(case["last_lo"], case["last_hi"]))]
    lo, hi = case["bound_lo"], case["bound_hi"]
    square = (hi * hi - lo * lo) / (2 * math.log(hi / lo))  # mean of H^2
    return [(case["requests"], math.sqrt(square), math.sqrt(square))]


def work(case):
    """bytes: the coefficients in and one point per curve out.  flops: one
    64-bit word operation per 64 sites of the box (every site is decided)."""
    total_bytes = flops = 0.0
    for count, bound, denominators in _boxes(case):
        degree = case.get("degree", 0.5 * (case.get("degree_lo", 0) + case.get("degree_hi", 0)))
        bits = case.get("bits", 0.5 * (case.get("bits_lo", 0) + case.get("bits_hi", 0)))
        total_bytes += count * ((degree + 1) * bits / 8 + 32)
        flops += count * (2 * bound + 1) * denominators / 64
    return {"bytes": total_bytes, "flops": flops}


# ---------------------------------------------------------------------------
# The same answers by exact integer arithmetic, for boxes small enough


def exact(case, seed):
    """The points of a small search: sites filtered by residues of F(a, d)
    modulo primes (numpy, 64 bits), then an exact integer square root."""
    if case["kind"] != "search" or case["square"] or (2 * case["bound"] + 1) * (case["last"] - case["first"] + 1) > 2e7:
        return None
    rng = random.Random(int(seed) * 1_000_003 + 17)
    coeffs, intervals = _single_curve(rng, case)
    c = [int(v) for v in coeffs]
    n = len(c) - 1
    even = n + n % 2  # F(a, d) = d^even f(a / d)

    def value(a, d):
        return sum(ci * a ** i * d ** (even - i) for i, ci in enumerate(c))

    points = []
    root = math.isqrt(c[-1]) if n % 2 == 0 and c[-1] >= 0 else 0
    if n % 2 == 1 or root * root == c[-1]:
        points.append((1, root, 0))
    a = np.arange(-case["bound"], case["bound"] + 1, dtype=np.int64)
    primes = (101, 103, 107, 109, 113, 127, 131, 137, 139, 149, 151, 157)
    squares = {}
    for p in primes:
        squares[p] = np.zeros(p, dtype=bool)
        squares[p][np.arange(p, dtype=np.int64) ** 2 % p] = True
    for d in range(case["first"], case["last"] + 1):
        left = a
        for p in primes:
            v = np.zeros(p, dtype=np.int64)
            x = np.arange(p, dtype=np.int64)
            for i in range(n, -1, -1):  # Horner in a with powers of d
                v = (v * x + c[i] * pow(d, even - i, p)) % p
            left = left[squares[p][v][left % p]]
        for x in left.tolist():
            if math.gcd(x, d) != 1:
                continue
            f = value(x, d)
            y = math.isqrt(f) if f >= 0 else -1
            if y >= 0 and y * y == f and (not intervals or any(
                    _at_most(lo, x, d) and not _below(hi, x, d) for lo, hi in intervals)):
                points.append((x, y, d))
    return _points([points])


def _scaled(text):
    """A bound with four decimals, in ten-thousandths."""
    return round(float(text) * 10_000)


def _at_most(bound, a, d):
    return _scaled(bound) * d <= a * 10_000


def _below(bound, a, d):
    return _scaled(bound) * d < a * 10_000

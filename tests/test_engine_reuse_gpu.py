"""What searches leave for the next one in the process (batch engines, table
memory, host threads) must not change its results: batches of other sizes and
kinds before, several threads at a time, capacities fixed small by
RPG_BATCH_CAPACITY, a release in between, and a session whose last launch was
on the caller's own stream."""

import threading

import pytest

pytestmark = pytest.mark.gpu

CURVES = [["1", "0", "1"], ["4", "0", "1", "0", "1"], ["9", "1", "-7", "0", "3", "2"], ["0", "-4", "0", "1"],
          ["1", "1", "-7", "0", "3", "2", "25"]]


def batch(shift, bounds, last, intervals=()):
    return [{"coefficients": CURVES[(i + shift) % len(CURVES)], "bound": bound, "first": 1, "last": last,
             "intervals": list(intervals)} for i, bound in enumerate(bounds)]


# narrow rows; curves with launches of their own; interval curves with wide
# rows; one curve; none
BATCHES = [batch(0, [500] * 40, 60), batch(1, [70_000, 900, 200_000], 400),
           batch(2, [70_000] * 3, 50, [("-0.5", "2")]), batch(3, [1_000], 10), []]


def answers(rpg, curves):
    points, status, survivors, _ = rpg.batch_search(curves)
    return points, status, survivors


def test_batches_after_one_another_and_at_once(rpg, monkeypatch):
    expected = []
    for curves in BATCHES:
        rpg.release_cached_resources()
        expected.append(answers(rpg, curves))
    for curves, (points, status, _) in zip(BATCHES, expected):
        single = [rpg.point_search(c["coefficients"], c["bound"], c["first"], c["last"], intervals=c["intervals"])[0]
                  for c in curves]
        assert points == single and not any(status)
    for order in ([0, 1, 2, 3, 4], [1, 0, 4, 2, 0, 3, 1]):
        for i in order:
            assert answers(rpg, BATCHES[i]) == expected[i], (order, i)
    # overflows the first survivor buffers, on engines that have larger ones
    monkeypatch.setenv("RPG_BATCH_CAPACITY", "16")
    for i in (0, 1):
        assert answers(rpg, BATCHES[i]) == expected[i]
    monkeypatch.delenv("RPG_BATCH_CAPACITY")
    # more threads than engines are kept
    wrong = []

    def work(k):
        for i in range(len(BATCHES)):
            at = (i + k) % len(BATCHES)
            if answers(rpg, BATCHES[at]) != expected[at]:
                wrong.append((k, at))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_search_after_a_session_on_another_stream(rpg):
    # the session's tables are in use on the caller's stream when it is
    # destroyed; the next search must not build its own in their place
    torch = pytest.importorskip("torch")
    import ctypes

    curve, other = CURVES[4], CURVES[2]
    expected = rpg.sieve(curve, 200_003, 1, 3_000, plan="fast")
    want_other = rpg.point_search(other, 100_000, 1, 500)[0]
    lib = rpg.load()
    session = ctypes.c_void_p()
    array = (ctypes.c_char_p * len(curve))(*[c.encode() for c in curve])
    assert lib.rpg_session_create(array, len(curve), 200_003, rpg.RPG_SIEVE_FAST_PLAN, -1, ctypes.byref(session)) == 0
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        a = torch.zeros(1 << 20, dtype=torch.int64, device="cuda")
        d = torch.zeros(1 << 20, dtype=torch.int32, device="cuda")
        count = torch.zeros(1, dtype=torch.int64, device="cuda")
    fn = lib.rpg_session_sieve_noalloc
    fn.restype = ctypes.c_int32
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int32, ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p,
                   ctypes.c_uint64, ctypes.c_void_p, ctypes.c_void_p]
    assert fn(session, 1, 3_000, a.data_ptr(), d.data_ptr(), 1 << 20, count.data_ptr(), stream.cuda_stream) == 0
    lib.rpg_session_destroy(session)
    assert rpg.point_search(other, 100_000, 1, 500)[0] == want_other
    stream.synchronize()
    n = int(count.item())
    assert n == len(expected[0])
    got = sorted(zip(a[:n].tolist(), d[:n].tolist()))
    assert got == sorted(zip(expected[0].tolist(), expected[1].tolist()))

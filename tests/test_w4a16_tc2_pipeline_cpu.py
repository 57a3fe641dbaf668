"""CPU model of the pipeline of the 4-bit GEMM over pairs of SMs: two threads that issue the weights' copies in turn, four conversion groups, an MMA
issuer, and barriers by parity that are looked at ahead of time.  Whatever order the copies land in, a group must read the weights it means to, and no
copy may go where weights are still to be read."""
import ctypes
import random

import pytest

from tests.test_w4a16_tc_pipeline_cpu import _Barrier

GROUPS, ISSUERS = 4, 2


def _issuer(me, slots, raw, stages, m):
    st = me
    free = False
    while st < stages:
        s = st % raw
        while not free and not m["raw_empty"][s].passes(st // raw % 2 ^ 1):
            yield False
        assert m["unread"][s] is None, "copy %d goes over %s" % (st, m["unread"][s])
        nxt = st + ISSUERS
        free = m["raw_empty"][nxt % raw].passes(nxt // raw % 2 ^ 1)
        m["unread"][s] = st
        m["raw_full"][s].arrive(1)
        m["flying"].append((m["now"] + m["rng"].choice([3, 3, 3, 40, 400]), s, st))
        st = nxt
        yield True


def _group(me, slots, raw, stages, m, look_behind):
    ready = False
    for st in range(me, stages, GROUPS):
        s, a = st % raw, st % slots
        while not ready and not m["raw_full"][s].passes(st // raw % 2):
            yield False
        assert m["content"][s] == st, "group %d read %s for %d" % (me, m["content"][s], st)
        nxt = st + GROUPS
        look = lambda: m["raw_full"][nxt % raw].passes(nxt // raw % 2)  # noqa: E731
        yield True
        free = m["a_empty"][a].passes(st // slots % 2 ^ 1)
        if not look_behind:
            ready = look()
        yield True
        while not free and not m["a_empty"][a].passes(st // slots % 2 ^ 1):
            yield False
        assert st < slots or m["mma"] > st - slots, "group %d took the slot of %d before it was multiplied" % (me, st - slots)
        if look_behind:
            ready = look()
        yield True
        m["unread"][s] = None
        m["raw_empty"][s].arrive()
        yield True
        m["a_full"][a].arrive()
        yield True


def _multiply(slots, stages, m):
    for st in range(stages):
        while not m["a_full"][st % slots].passes(st // slots % 2):
            yield False
        m["mma"] = st + 1
        m["a_empty"][st % slots].arrive()
        yield True


def _run(slots, raw, stages, seed, look_behind=True):
    """Steps the roles in a random order, some of them slower for a while; raises on a wrong read, a wrong copy or a standstill."""
    rng = random.Random(seed)
    m = {"rng": rng, "now": 0, "mma": 0, "flying": [], "content": [None] * raw, "unread": [None] * raw}
    for name, n in (("raw_full", raw), ("raw_empty", raw), ("a_full", slots), ("a_empty", slots)):
        m[name] = [_Barrier(1) for _ in range(n)]
    roles = [_issuer(i, slots, raw, stages, m) for i in range(ISSUERS)] + [_group(g, slots, raw, stages, m, look_behind) for g in range(GROUPS)]
    roles.append(_multiply(slots, stages, m))
    idle = 0
    while m["mma"] < stages:
        m["now"] += 1
        for x in [f for f in m["flying"] if f[0] <= m["now"]]:
            m["flying"].remove(x)
            m["content"][x[1]] = x[2]
            m["raw_full"][x[1]].land()
        if m["now"] % 50 == 1:
            weights = [rng.choice([1, 1, 1, 20]) for _ in roles]
        done = next(rng.choices(roles, weights)[0], False)
        idle = 0 if done or m["flying"] else idle + 1
        assert idle < 4000, "standstill at %d of %d" % (m["mma"], stages)


@pytest.mark.parametrize("ntok", range(32, 257, 32))
def test_every_group_reads_its_weights(lib, ntok):
    slots, raw = ctypes.c_int(), ctypes.c_int()
    assert lib.zl_w4_pairs_rings(ntok, ctypes.byref(slots), ctypes.byref(raw)) == 0
    for seed in range(80):
        _run(slots.value, raw.value, stages=64, seed=seed)


def test_a_look_ahead_of_the_wait_for_its_slot_would_not_do(lib):
    """What the model is for: at 256 tokens a group that looks before it knows its slot of A to be free takes the phase before last for its own."""
    slots, raw = ctypes.c_int(), ctypes.c_int()
    assert lib.zl_w4_pairs_rings(256, ctypes.byref(slots), ctypes.byref(raw)) == 0
    with pytest.raises(AssertionError):
        for seed in range(80):
            _run(slots.value, raw.value, stages=64, seed=seed, look_behind=False)


@pytest.mark.parametrize("ntok", [0, 16, 48, 288])
def test_tiles_that_do_not_exist(lib, ntok):
    slots, raw = ctypes.c_int(), ctypes.c_int()
    assert lib.zl_w4_pairs_rings(ntok, ctypes.byref(slots), ctypes.byref(raw)) != 0

"""CPU model of the 4-bit stream-k kernel's pipeline: a weight producer, conversion groups that take the stages in turn, an MMA issuer, and
barriers that are waited for by parity.  Whatever order the copies land in, a group must read the stage it means to."""
import ctypes
import random

import pytest


class _Barrier:
    """mbarrier: a phase ends with `count` arrivals and all announced bytes; a wait names the parity of the phase it wants ended and is
    let through whenever the phase that runs has the other one."""

    def __init__(self, count):
        self.count, self.arrived, self.bytes, self.phase = count, 0, 0, 0

    def _end(self):
        if self.arrived == self.count and self.bytes == 0:
            self.arrived, self.phase = 0, self.phase + 1

    def arrive(self, bytes_=0):
        if self.arrived == self.count:
            raise AssertionError("one arrival too many")
        self.arrived += 1
        self.bytes += bytes_
        self._end()

    def land(self):
        self.bytes -= 1
        self._end()

    def passes(self, parity):
        return self.phase % 2 != parity


def _run(groups, a_stages, raw_stages, stages, seed):
    """Steps the roles in a random order, copies landing late now and then; raises on a wrong read, a wrong arrival or a standstill."""
    rng = random.Random(seed)
    raw_full, raw_empty = ([_Barrier(1) for _ in range(raw_stages)] for _ in range(2))
    a_full, a_empty = ([_Barrier(1) for _ in range(a_stages)] for _ in range(2))
    content = [None] * raw_stages                       # stage whose weights lie in the slot
    flying = []                                         # (time of landing, slot, stage)
    issued, mma, now = 0, 0, 0
    at = list(range(groups))                            # stage each group is about to read, or has read (then: reading[g])
    reading = [False] * groups
    idle = 0
    while mma < stages:
        now += 1
        done = False
        for x in [f for f in flying if f[0] <= now]:
            flying.remove(x)
            content[x[1]] = x[2]
            raw_full[x[1]].land()
            done = True
        role = rng.randrange(groups + 2)
        if role == groups and issued < stages:
            s = issued % raw_stages
            if raw_empty[s].passes(issued // raw_stages % 2 ^ 1):
                raw_full[s].arrive(1)
                flying.append((now + rng.choice([3, 3, 3, 200]), s, issued))
                issued, done = issued + 1, True
        elif role == groups + 1:
            a = mma % a_stages
            if a_full[a].passes(mma // a_stages % 2):
                a_empty[a].arrive()
                mma, done = mma + 1, True
        elif role < groups and at[role] < stages:
            st = at[role]
            s, a = st % raw_stages, st % a_stages
            if not reading[role]:
                if raw_full[s].passes(st // raw_stages % 2):
                    assert content[s] == st, "group %d read stage %s for %d" % (role, content[s], st)
                    raw_empty[s].arrive()
                    reading[role], done = True, True
            elif a_empty[a].passes(st // a_stages % 2 ^ 1):
                a_full[a].arrive()
                at[role], reading[role], done = st + groups, False, True
        idle = 0 if done or flying else idle + 1
        assert idle < 2000, "standstill at %d of %d" % (mma, stages)


@pytest.mark.parametrize("ntok", [32, 64, 128, 256])
def test_every_group_reads_its_stage(lib, ntok):
    out = (ctypes.c_int * 3)()
    assert lib.zl_w4_tc_pipeline(ntok, out) == 0
    for seed in range(60):
        _run(*out, stages=60, seed=seed)


@pytest.mark.parametrize("a_stages", [2, 3])
def test_three_slots_for_two_groups_would_not_do(a_stages):
    """What the model is for: a group a stage ahead takes a slot whose bytes for the other group are on their way."""
    with pytest.raises(AssertionError):
        for seed in range(60):
            _run(2, a_stages, 3, stages=60, seed=seed)

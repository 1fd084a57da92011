"""The end of a pair of CTAs in which a wait ran out (csrc/pair_drain.h), against a model of the leader's barriers."""
import ctypes
import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "enterprise-inference_b200", "csrc")
STAGES = 6


class Owed(ctypes.Structure):
    _fields_ = [("parity", ctypes.c_int), ("fill", ctypes.c_int), ("announce", ctypes.c_int)]


@pytest.fixture(scope="module")
def owed(tmp_path_factory):
    d = tmp_path_factory.mktemp("pair")
    src, so = d / "owed.cpp", d / "owed.so"
    src.write_text('#include "pair_drain.h"\nextern "C" b200::PairOwed owed(int s, int n, int l, int p) { return b200::pair_owed(s, n, l, p); }\n')
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    fn = ctypes.CDLL(str(so)).owed
    fn.restype = Owed
    return fn


class Barrier:
    """One arrival a phase, bytes announced and landed."""
    def __init__(self):
        self.phase, self.pending, self.tx = 0, 1, 0

    def _step(self):
        if self.pending == 0 and self.tx == 0:
            self.phase, self.pending = self.phase + 1, 1

    def expect(self, n):
        assert self.pending == 1, "a second arrival in one phase"
        self.tx += n
        self.pending = 0
        self._step()

    def land(self, n):
        self.tx -= n
        assert abs(self.tx) < 1 << 20
        self._step()


@pytest.mark.parametrize("seed", range(200))
def test_everything_that_was_issued_has_landed_before_the_end(owed, seed):
    r = random.Random(seed)
    total = r.choice([1, 3, 6, 7, 40])
    half = [r.choice([18432, 20480, 32768]) for _ in range(total)]
    bars = [Barrier() for _ in range(STAGES)]
    done, count, running = 0, [0, 0], [True, True]     # fills whose MMAs are committed; fills of leader and peer; who still issues
    flight = []                                        # (stage, bytes) not landed yet
    mma, steps, stop_at, lost = True, 0, r.randint(0, 4 * total), r.random() < 0.5   # lost: bytes that come only at the very end
    while any(running) or mma:
        steps += 1
        who = r.choice(["lead", "peer", "mma", "land"])
        marked = steps > stop_at
        if who in ("lead", "peer"):
            c = who == "peer"
            if running[c]:
                i = count[c]
                if i == total or (marked and r.random() < 0.3):     # the mark is seen some time after it was set
                    running[c] = False
                elif i < STAGES or done > i - STAGES:
                    if not c:
                        bars[i % STAGES].expect(2 * half[i])
                    flight.append((i % STAGES, half[i]))
                    count[c] += 1
                elif marked:
                    running[c] = False
        elif who == "mma" and mma:
            if done < total and bars[done % STAGES].phase > done // STAGES:
                done += 1
            elif done == total or marked:
                mma = False
        elif who == "land" and flight and not (lost and marked):
            stage, n = flight.pop(r.randrange(len(flight)))
            bars[stage].land(n)
    for s in range(STAGES):
        o = owed(s, STAGES, *count)
        n = [len(range(s, c, STAGES)) for c in count]
        assert abs(n[0] - n[1]) <= 1
        if o.parity < 0:
            assert n == [0, 0]
            continue
        if o.announce > 0:
            bars[s].expect(half[o.fill])
        elif o.announce < 0:
            bars[s].land(half[o.fill])
        mine = [b for t, b in flight if t == s]
        for b in mine:
            assert bars[s].phase == max(n) - 1, "the wait would end before the last bytes are there"
            bars[s].land(b)
        assert bars[s].phase == max(n) and (max(n) - 1) & 1 == o.parity and bars[s].tx == 0


@pytest.mark.parametrize("stages", [5, 7])
@pytest.mark.parametrize("seed", range(60))
def test_rings_of_other_depths(owed, seed, stages, monkeypatch):
    monkeypatch.setitem(globals(), "STAGES", stages)
    test_everything_that_was_issued_has_landed_before_the_end(owed, seed)

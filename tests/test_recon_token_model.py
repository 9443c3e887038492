"""The reconstruction epilogue's hand-offs (csrc/crt.cu, k_crt_recon), replayed on the
CPU: four parts per lane quadrant, a token that goes round them once per N tile, and part
0's fixed-point results in two alternating slots.  Barriers have mbarrier semantics (one
arrival completes a phase; a waiter sees only the parity of the current phase), so a
barrier that runs a phase ahead of its reader shows up as a wait that never ends, and a
slot written before its last reader as a stale or early value."""
import random

import pytest


class Bar:
    def __init__(self):
        self.phase = 0  # completed phases

    def arrive(self):
        self.phase += 1

    def done(self, parity):  # the phase with this parity has completed and the next one not
        return (self.phase & 1) != parity


def run(nts, seed, parity_slots=True):
    rng = random.Random(seed)
    tok = [None] * 4
    tokbar = [Bar() for _ in range(4)]
    q = [None, None]
    qready = [Bar(), Bar()]
    log = []

    def part(p):
        ntok, first = 0, True
        for et, nt in enumerate(nts):
            for j in range(nt):
                yield None
                if j == 0:
                    b = (et & 1) if parity_slots else 0
                    par = ((et >> 1) & 1) if parity_slots else (et & 1)
                    if p == 0:
                        q[b] = et
                        yield None
                        qready[b].arrive()
                    else:
                        while not qready[b].done(par):
                            yield "wait"
                        yield None
                        assert q[b] == et, (p, et, q)
                if p > 0 or not first:
                    while not tokbar[p].done(ntok & 1):
                        yield "wait"
                    ntok += 1
                    yield None
                    if p > 0 or j > 0:
                        assert tok[p] == (et, j, p), (tok[p], et, j, p)
                first = False
                log.append((et, j, p))
                nxt = (p + 1) & 3
                tok[nxt] = (et, j, p + 1) if p < 3 else (et, j + 1, 0)
                yield None
                tokbar[nxt].arrive()

    procs = [part(p) for p in range(4)]
    live, idle = list(range(4)), 0
    while live:
        p = rng.choice(live)
        for _ in range(rng.randint(1, 12)):
            try:
                r = next(procs[p])
            except StopIteration:
                live.remove(p)
                idle = 0
                break
            if r == "wait":
                idle += 1
                break
            idle = 0
        assert idle < 2000, "deadlock"
    assert log == [(et, j, p) for et, nt in enumerate(nts) for j in range(nt) for p in range(4)]


@pytest.mark.parametrize("nts", [[1] * 12, [2] * 8, [5] * 5, [2, 1, 1, 3, 1, 1, 1, 2, 4, 1], [1, 1, 2, 1, 5, 1, 1]])
def test_token_order(nts):
    for seed in range(60):
        run(nts, seed)


def test_one_slot_would_not_do():
    with pytest.raises(AssertionError):
        for seed in range(300):
            run([1] * 12, seed, parity_slots=False)

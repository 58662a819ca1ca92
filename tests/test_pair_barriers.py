"""The barrier protocol of the products by pairs of SMs (k_gemm_pair, vb_gemm_tc.cu) as a model of events on the CPU: two producers, the
warp that issues for both blocks, copies that land and commits that arrive in any order.  No schedule may end in a deadlock, overwrite a
stage that is still read, multiply operands that are not there, or send an arrival to a block that has left."""
import random

import pytest


class Barrier:
    def __init__(self):
        self.pending, self.tx, self.phase = 1, 0, 0

    def _check(self):
        if self.pending == 0 and self.tx == 0:
            self.phase, self.pending = self.phase + 1, 1

    def arrive(self, expect=0):
        assert self.pending > 0
        self.tx += expect
        self.pending -= 1
        self._check()

    def complete(self):
        self.tx -= 1
        self._check()

    def passed(self, parity):
        return (self.phase & 1) != parity


def late_arrivals(rng, stages, nk, copies, drain):
    """One random schedule; how many arrivals are still on their way when a block leaves."""
    full = [Barrier() for _ in range(stages)]
    empty = [[Barrier() for _ in range(stages)] for _ in range(2)]
    accum = [Barrier(), Barrier()]
    loaded, drained, issued, left = [0, 0], [0, 0], 0, [False, False]
    landed = [[(-1, 0)] * stages for _ in range(2)]
    reading, queue, events, late = set(), [], [], 0
    first = max(0, nk - stages)
    while not all(left):
        acts = []
        for r in (0, 1):
            if loaded[r] < nk:
                if empty[r][loaded[r] % stages].passed((loaded[r] // stages & 1) ^ 1):
                    acts.append(("load", r))
            elif drain and first + drained[r] < nk:
                kb = first + drained[r]
                if empty[r][kb % stages].passed(kb // stages & 1):
                    acts.append(("drain", r))
            elif not left[r] and accum[r].passed(0):
                acts.append(("leave", r))
        if issued < nk and full[issued % stages].passed(issued // stages & 1):
            acts.append(("issue",))
        if queue:
            acts.append(("product",))
        acts += [("event", i) for i in range(len(events))]
        assert acts, "deadlock"
        act = rng.choice(acts)
        if act[0] == "load":
            r, kb = act[1], loaded[act[1]]
            assert all(q % stages != kb % stages for q in reading), "a stage is overwritten while products read it"
            landed[r][kb % stages] = (kb, 0)
            if r == 0:
                full[kb % stages].arrive(2 * copies)
            events += [("copy", r, kb)] * copies
            loaded[r] += 1
        elif act[0] == "drain":
            drained[act[1]] += 1
        elif act[0] == "leave":
            r = act[1]
            left[r] = True
            late += sum(e[0] != "copy" and e[1] == r for e in events)
        elif act[0] == "issue":
            assert all(landed[r][issued % stages] == (issued, copies) for r in (0, 1)), "operands are not there"
            reading.add(issued)
            queue += [("product", issued), ("empty", issued % stages)] + ([("accum", 0)] if issued == nk - 1 else [])
            issued += 1
        elif act[0] == "product":
            what, i = queue.pop(0)
            if what == "product":
                reading.remove(i)
            else:
                events += [(what, 0, i), (what, 1, i)]
        else:
            what, r, i = events.pop(act[1])
            if what == "copy":
                landed[r][i % stages] = (i, landed[r][i % stages][1] + 1)
                full[i % stages].complete()
            else:
                (empty[r][i] if what == "empty" else accum[r]).arrive()
    return late


@pytest.mark.parametrize("stages", [2, 4, 8])
def test_no_arrival_reaches_a_block_that_has_left(stages):
    rng = random.Random(stages)
    cases = [(rng.randint(1, 3 * stages), rng.choice((1, 2, 6))) for _ in range(1500)]
    assert all(late_arrivals(rng, stages, nk, copies, True) == 0 for nk, copies in cases)
    assert any(late_arrivals(rng, stages, nk, copies, False) for nk, copies in cases)  # what the wait at the end is for

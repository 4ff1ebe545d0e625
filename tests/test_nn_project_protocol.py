"""The barrier protocol of nn_project_kernel (csrc/nn_spectral.cuh), every order
of its copies, two converting sets, products and completions: no set reads the
accumulators before the last product, no buffer is used before it is full or
written while it is in use, and no order gets stuck.

A barrier is its number of completed phases; a wait for parity p passes while the
phase in progress has the other parity, as mbarrier.try_wait.parity does."""
import collections

import pytest

State = collections.namedtuple("State", "copied landed conv issued done ended")


def explore(n, stages, single_phase_end):
    """Every reachable state of n chunks in a ring of `stages`.  Returns whether
    a set can pass its last wait with products still running."""
    def phases(completed, s):   # of a stage's barrier when these chunks completed it
        return sum(1 for i in completed if i % stages == s)

    def passes(completed, s, parity):
        return (phases(completed, s) & 1) != parity

    early = False
    first = State(0, frozenset(), (0, 1), 0, 0, (False, False))
    seen, todo = {first}, [first]
    while todo:
        x = todo.pop()
        landed, done = x.landed, frozenset(range(x.done))
        # chunks whose h is converted: set p takes p, p + 2, ..
        converted = frozenset(i for p in (0, 1) for i in range(p, x.conv[p], 2))
        nxt = []
        if x.copied < n:   # copies: the stage's last products are over
            c = x.copied
            if c < stages or passes(done, c % stages, (c // stages - 1) & 1):
                assert c < stages or c - stages < x.done, "copied over operands in use"
                nxt.append(x._replace(copied=c + 1))
        for c in range(x.copied):   # a copy lands, in any order
            if c not in landed:
                nxt.append(x._replace(landed=landed | {c}))
        for p in (0, 1):
            i = x.conv[p]
            if i < n and passes(landed, i % stages, (i // stages) & 1):
                assert i in landed, "h read before it landed"
                assert i < stages or i - stages < x.done, "rounded over an operand in use"
                conv = (i + 2, x.conv[1]) if p == 0 else (x.conv[0], i + 2)
                nxt.append(x._replace(conv=conv))
            if i >= n and not x.ended[p]:
                last = n - 1
                if x.done == n if single_phase_end else \
                        passes(done, last % stages, (last // stages) & 1):
                    early = early or x.done < n
                    nxt.append(x._replace(ended=(True, x.ended[1]) if p == 0
                                          else (x.ended[0], True)))
        i = x.issued
        if i < n and passes(landed, i % stages, (i // stages) & 1) and \
                passes(converted, i % stages, (i // stages) & 1):
            assert i in landed and i in converted, "product of operands not yet there"
            nxt.append(x._replace(issued=i + 1))
        if x.done < x.issued:   # products complete in order
            nxt.append(x._replace(done=x.done + 1))
        assert nxt or x.ended == (True, True), f"stuck at {x}"
        for y in nxt:
            if y not in seen:
                seen.add(y)
                todo.append(y)
    return early


@pytest.mark.parametrize("stages", [4, 8])
@pytest.mark.parametrize("over", [-3, 0, 1, 2, 3, 5])
def test_epilogue_waits_for_the_last_product(stages, over):
    assert not explore(stages + over, stages, single_phase_end=True)


def test_the_last_chunks_own_barrier_is_not_enough():
    """What the one-phase barrier is for: a wait for the last chunk's stage by its
    parity lets the other set through a phase early."""
    assert explore(6, 4, single_phase_end=False)
    assert not explore(4, 4, single_phase_end=False)

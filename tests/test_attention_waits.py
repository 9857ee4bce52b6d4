"""The waits of a chain of attention's forward kernel (softmax_chain and the MMA thread in attention_tc.cu), as a model that runs every
order of events: a wait by parity has to end, and must not end before the phase that it is for."""
import pytest


def outcomes(chain, mma):
    """All ways in which the two programs can end: 'done', 'stuck' or 'early' (a wait has passed before its products were complete).
    chain: ("wait", barrier, phase, products that are then complete) or ("arrive", barrier); mma: ("wait", barrier, phase), ("scores",),
    ("product",) or ("commit", barrier).  The tensor cores work in order; a commit arrives at any time after the work issued before it,
    in no order among commits."""
    found, seen, todo = set(), set(), [(0, 0, 0, frozenset())]  # places in both programs, work complete (in places of mma), commits arrived
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        at, at_mma, complete, arrived = state
        barriers = [op[1] for op in chain[:at] if op[0] == "arrive"] + [mma[i][1] for i in arrived]
        passes = lambda op: op[0] != "wait" or barriers.count(op[1]) & 1 != op[2] & 1  # the current phase has the other parity
        following = []
        if at < len(chain) and passes(chain[at]):
            if chain[at][0] == "wait" and mma[:complete].count(("product",)) < chain[at][3]:
                found.add("early")
            following.append((at + 1, at_mma, complete, arrived))
        if at_mma < len(mma) and passes(mma[at_mma]):
            following.append((at, at_mma + 1, complete, arrived))
        if complete < at_mma:
            following.append((at, at_mma, complete + 1, arrived))
        following += [(at, at_mma, complete, arrived | {i}) for i in range(complete) if mma[i][0] == "commit" and i not in arrived]
        if not following:
            found.add("done" if at == len(chain) and at_mma == len(mma) else "stuck")
        todo += following
    return found


def protocol(steps, buffers, own_barrier, rescale=True):
    """A chain's programs.  `own_barrier`: products are counted on a barrier of their own, which is awaited to rescale and for the last two
    products; else they are told by the barrier of the scores that take their buffer."""
    s, p = (lambda n: f"s{n % buffers}"), (lambda n: f"p{n % buffers}")
    chain, mma = [], []
    for n in range(steps):
        chain.append(("wait", s(n), n // buffers, max(n + 1 - buffers, 0)))
        if rescale and n and buffers == 2:
            chain.append(("wait", "o", n - 1, n) if own_barrier else ("wait", s(n + 1), (n + 1) // 2, n))
        chain.append(("arrive", p(n)))
    if own_barrier:
        chain += [("wait", "o", n, n + 1) for n in range(max(steps - 2, 0), steps)]
    else:
        chain.append(("wait", s(steps - 1), (steps - 1) // buffers + 1, steps))
    for n in range(min(steps, buffers)):
        mma += [("scores",), ("commit", s(n))]
    for n in range(steps):
        mma += [("wait", p(n), n // buffers), ("product",)] + [("commit", "o")] * own_barrier
        if n + buffers < steps:
            mma.append(("scores",))
        if n + buffers < steps or not own_barrier:
            mma.append(("commit", s(n + buffers)))
    return chain, mma


@pytest.mark.parametrize("rescale", [False, True])
@pytest.mark.parametrize("buffers", [1, 2])
@pytest.mark.parametrize("steps", range(1, 7))
def test_every_wait_ends_and_none_early(steps, buffers, rescale):
    assert outcomes(*protocol(steps, buffers, False, rescale)) == {"done"}


@pytest.mark.parametrize("steps", range(2, 5))
def test_the_model_finds_a_phase_that_is_missed(steps):
    """Products on a barrier of their own, both last ones awaited at the end: the first of these waits can come when the second phase is over."""
    assert "stuck" in outcomes(*protocol(steps, 2, True, rescale=False))

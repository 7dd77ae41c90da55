"""The hand-off of the two softmax warps that share rows in the prompt attention (csrc/q3_prefill_attn_tc.cu), as a state machine whose
interleavings are all walked: whichever wait gives up, at whatever moment, both warps reach the end."""
import itertools

import pytest

# Where a warp is.  It waits for the scores of its tile (S), leaves its maxima, meets its partner at a barrier, reads the partner's maxima, waits for the
# output of the tile before if a maximum grew (O), hands P over and goes on.
WAIT_S, MEET, BARRIER, READ, WAIT_O, HAND, DONE = range(7)


def stuck_states(tiles, grows, publish, places):
    """Reachable states in which a warp waits at the barrier for a partner that never comes.

    publish: a warp that gave up says so at the next barrier (else it leaves at once); places: how many tiles' maxima are kept apart."""
    start = (((WAIT_S, 0, True),) * 2, ((None,) * 2,) * places, (0, 0), (0, 0))
    seen, todo, stuck = {start}, [start], []
    while todo:
        state = todo.pop()
        following = list(successors(state, tiles, grows, publish, places))
        if not following and any(w[0] != DONE for w in state[0]):
            stuck.append(state)
        for n in following:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return stuck


def successors(state, tiles, grows, publish, places):
    warps, slots, meets, handed = state

    def put(me, warp, slots=slots, meets=meets, handed=handed):
        return (tuple(warp if k == me else w for k, w in enumerate(warps)), slots, meets, handed)

    def bump(pair, me):
        return tuple(v + (k == me) for k, v in enumerate(pair))

    for me in range(2):
        pc, i, ok = warps[me]
        if pc == WAIT_S:
            if i >= tiles:
                yield put(me, (DONE, i, ok))
                continue
            if ok and min(handed) >= i:        # the scores can be there: both have handed the tile before over
                yield put(me, (MEET, i, True))
            # a wait gives up after a while, or because somebody else has (it may have looked at its barrier just before)
            yield put(me, (MEET, i, False) if publish else (DONE, i, False))
        elif pc == MEET:
            now = tuple(tuple(ok if k == me else v for k, v in enumerate(s)) if b == i % places else s for b, s in enumerate(slots))
            yield put(me, (BARRIER, i, ok), slots=now, meets=bump(meets, me))
        elif pc == BARRIER:
            if meets[1 - me] >= meets[me]:
                yield put(me, (READ, i, ok))
        elif pc == READ:
            if not (ok and slots[i % places][1 - me]):
                yield put(me, (DONE, i, False))
            else:
                yield put(me, (WAIT_O if i > 0 and grows[i] else HAND, i, True))
        elif pc == WAIT_O:
            yield put(me, (HAND, i, True))     # (both have handed the tile before over, or this one would not have begun)
            yield put(me, (WAIT_S, i + 1, False) if publish else (DONE, i, False))
        elif pc == HAND:
            yield put(me, (WAIT_S, i + 1, True), handed=bump(handed, me))


@pytest.mark.parametrize("tiles", [1, 2, 3, 4])
def test_softmax_warps_that_give_up_do_not_leave_their_partner_waiting(tiles):
    for grows in itertools.product([False, True], repeat=tiles):
        assert not stuck_states(tiles, grows, publish=True, places=2)


def test_the_model_finds_the_partner_that_waits_for_good():
    """A warp that leaves at once, and one place for the maxima of all tiles, each leave a partner at the barrier."""
    assert stuck_states(2, (False, False), publish=False, places=2)
    assert stuck_states(3, (True, True, True), publish=True, places=1)

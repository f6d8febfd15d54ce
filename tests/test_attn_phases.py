"""The order of the barriers of the prompt attention (attn_flash.cu), every interleaving of its roles: a phase of a barrier that
completes twice before its waiter looks is lost, and the waiter stays behind for good."""
from collections import deque

import pytest


def stuck_states(tiles, places, held):
    """Reachable states in which no role can go on although not all are done.  Roles: the loaders of keys and of values, the MMA
    thread, two softmax groups (group w takes the tiles w, w + 2, ...).  held: a group arrives on p_full only once the product of its
    tile before is done.  Barriers are counts of completed phases, of which a waiter sees the parity."""
    program = [("scores", t) for t in range(min(places, tiles))]
    for t in range(tiles):
        program += [("values", t), ("weights", t), ("product", t)] + [("scores", t + places)] * (t + places < tiles)

    def done(count, phase):
        return (count ^ phase) & 1 == 1

    def plus(counts, i):
        return tuple(c + (j == i) for j, c in enumerate(counts))

    def steps(s):
        k, v, pc, groups, k_full, v_full, s_full, p_full, o_done = s
        if k < tiles and (k < 2 or done(s_full[(k - 2) % places], (k - 2) // places)):
            yield k + 1, v, pc, groups, plus(k_full, k % 2), v_full, s_full, p_full, o_done
        if v < tiles and (v < 2 or done(o_done[v % 2], (v - 2) // 2)):
            yield k, v + 1, pc, groups, k_full, plus(v_full, v % 2), s_full, p_full, o_done
        if pc < len(program):
            op, t = program[pc]
            if op == "product":
                yield k, v, pc + 1, groups, k_full, v_full, s_full, p_full, plus(o_done, t % 2)
            elif op == "scores":
                if done(k_full[t % 2], t // 2):
                    yield k, v, pc + 1, groups, k_full, v_full, plus(s_full, t % places), p_full, o_done
            elif done((v_full if op == "values" else p_full)[t % 2], t // 2):
                yield k, v, pc + 1, groups, k_full, v_full, s_full, p_full, o_done
        for w, t in enumerate(groups):
            if t < tiles and done(s_full[t % places], t // places) and (not held or t < 2 or done(o_done[w], (t - 2) // 2)):
                yield k, v, pc, tuple(g + 2 * (i == w) for i, g in enumerate(groups)), k_full, v_full, s_full, plus(p_full, w), o_done

    first = (0, 0, 0, (0, 1), (0, 0), (0, 0), (0,) * places, (0, 0), (0, 0))
    seen, todo, stuck = {first}, deque([first]), 0
    while todo:
        s = todo.popleft()
        after = list(steps(s))
        stuck += not after and not (s[0] == s[1] == tiles and s[2] == len(program) and min(s[3]) >= tiles)
        todo.extend(a for a in set(after) - seen)
        seen.update(after)
    return stuck


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 5, 8, 16])
def test_no_phase_is_lost(tiles):
    assert stuck_states(tiles, places=2, held=False) == 0
    assert stuck_states(tiles, places=3, held=True) == 0
    if tiles > 2:
        assert stuck_states(tiles, places=3, held=False) > 0  # what the wait is for

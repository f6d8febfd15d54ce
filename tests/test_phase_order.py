"""The order of barriers whose phases are told apart by parity alone, every interleaving of a kernel's roles: a phase that completes
twice before its waiter looks is lost, and one asked for while the phase before it is still open is granted too early."""
from collections import deque

import pytest


def stuck_states(tiles, places, held):
    """Prompt attention (attn_flash.cu): reachable states in which no role can go on although not all are done.  Roles: the loaders of keys and of values, the MMA
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


def early_reads(chunks, stages, buffers, buffer_first):
    """The ternary product of up to 128 rows a tile (gemm_tc.cu): reachable states in which unpack warps read a stage whose copies
    have not landed.  Two sets of warps take the chunks in turn; a chunk lies in stage chunk mod stages and is unpacked into buffer
    chunk mod buffers; copies land in any order.  buffer_first: a set waits for its buffer (the product of `buffers` chunks before)
    and then for the copies, instead of the other way round."""
    def done(count, phase):
        return (count ^ phase) & 1 == 1

    def plus(counts, i):
        return tuple(c + (j == i) for j, c in enumerate(counts))

    def steps(s):
        # issued copies, those that landed, per set (chunk, has it got what it waits for first), completed phases of the stages, unpacked
        # chunks, products done
        issued, landed, sets, full, unpacked, mma = s
        if issued < chunks and (issued < stages or (mma > issued - stages and issued - stages in unpacked)):
            yield issued + 1, landed, sets, full, unpacked, mma
        for c in range(max(0, issued - stages), issued):
            if c not in landed:
                yield issued, landed | {c}, sets, plus(full, c % stages), unpacked, mma
        for w, (g, first) in enumerate(sets):
            if g >= chunks:
                continue
            copies, buffer = done(full[g % stages], g // stages), g < buffers or mma > g - buffers
            if not first and (buffer if buffer_first else copies):
                yield issued, landed, tuple((g, True) if i == w else x for i, x in enumerate(sets)), full, unpacked, mma
            if first and (copies if buffer_first else buffer):
                yield issued, landed, tuple((g + 2, False) if i == w else x for i, x in enumerate(sets)), full, unpacked | {g}, mma
        if mma < chunks and mma in unpacked:
            yield issued, landed, sets, full, unpacked, mma + 1

    def early(s):
        return any(first and not buffer_first and g not in s[1] for g, first in s[2]) or not s[4] <= s[1]

    first = (0, frozenset(), ((0, False), (1, False)), (0,) * stages, frozenset(), 0)
    seen, todo, bad = {first}, deque([first]), 0
    while todo:
        s = todo.popleft()
        if early(s):
            bad += 1
            continue
        after = set(steps(s))
        assert after or s[5] == chunks  # nobody waits for good
        todo.extend(after - seen)
        seen.update(after)
    return bad


@pytest.mark.parametrize("chunks", [1, 4, 5, 6, 8, 11])
def test_no_stage_is_read_early(chunks):
    assert early_reads(chunks, 5, 4, buffer_first=True) == 0
    if chunks > 5:
        assert early_reads(chunks, 5, 4, buffer_first=False) > 0  # what the order is for
    assert early_reads(chunks, 4, 4, buffer_first=False) == 0     # (an even ring: a set meets the same stages again and again)

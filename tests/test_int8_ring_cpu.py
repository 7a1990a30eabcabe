"""The ring of the int8 tensor-core projection (gemm_tc.cu), walked through in every order in which its tiles can land: waits
by parity (passed whenever the open phase has the other parity) must never let a converting group through early."""
import pytest


def rings():
    """(stages, converting groups) of the instances: rows per tile, one or two matrices (TcCfg)."""
    for rows in (32, 128, 256):
        for matrices in (1, 2):
            stages = min(10, 225 * 1024 // (matrices * (16384 + 8192) + rows * 128))
            yield stages, max(1, (4 if rows >= 128 else 2) // matrices)


def walk(stages, groups, blocks, wait_empty):
    """Blocks that some order of events converts before they have landed; "stuck" where nothing can go on."""
    shares = [range(g, blocks, groups) for g in range(groups)]
    wrong, seen = set(), set()
    todo = [(min(stages, blocks), frozenset(), (0,) * groups, frozenset(), 0)]  # requested, landed, per group, converted, multiplied
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        asked, landed, at, converted, used = state
        after = [(asked, landed | {b}, at, converted, used) for b in range(asked) if b not in landed]
        if asked < blocks and used > asked - stages:
            after.append((asked + 1, landed, at, converted, used))
        if used < blocks and used in landed and used in converted:
            after.append((asked, landed, at, converted, used + 1))
        for g, share in enumerate(shares):
            if at[g] == len(share):
                continue
            block = share[at[g]]
            use = block // stages
            freed = len(range(block % stages, used, stages))
            if wait_empty and use > 0 and freed % 2 == (use - 1) % 2:
                continue
            phases = len([b for b in range(block % stages, blocks, stages) if b in landed])
            if phases % 2 == use % 2:
                continue
            if block not in landed or (wait_empty and freed != use):
                wrong.add(block)
                continue
            after.append((asked, landed, at[:g] + (at[g] + 1,) + at[g + 1:], converted | {block}, used))
        if not after and used < blocks:
            wrong.add("stuck")
        todo += after
    return wrong


@pytest.mark.parametrize("stages,groups", sorted(set(rings())))
def test_no_group_passes_a_wait_early(stages, groups):
    blocks = min(2 * stages + 2, stages + 5)
    assert not walk(stages, groups, blocks, wait_empty=stages % groups != 0)
    assert bool(walk(stages, groups, blocks, wait_empty=False)) == (stages % groups != 0)

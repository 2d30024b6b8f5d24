"""The problem list of a window against a plain restatement, at the edges of the pairs' split over warps (1 to 128 rows, 1 to 32
slots), few and the most experts, one rank and two."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,slots,experts", [(1, 1, 4), (3, 9, 128), (32, 32, 64), (33, 31, 40), (126, 9, 128), (128, 32, 1022), (128, 2, 2)])
@pytest.mark.parametrize("world", [1, 2])
def test_problem_list(lib, rows, slots, experts, world):
    from tensorfold_b200 import _lib

    gen = torch.Generator().manual_seed(rows + slots)
    total = experts + 1
    pick = torch.stack([torch.randperm(total, generator=gen)[:slots] if slots <= total else torch.randint(0, total, (slots,), generator=gen)
                        for _ in range(rows)]).to(torch.int32)
    room = _lib.load().tf_moe_max_problems(rows, slots, total)
    members = {}
    for i, e in enumerate(pick.flatten().tolist()):
        members.setdefault(e, []).append(i)
    want_rows, want_expert, want_loc, owned = [], [], {}, []
    rank, per = world - 1, experts // world
    for e in sorted(members):
        for q in range(0, len(members[e]), 8):
            part, p = members[e][q:q + 8], len(want_rows)
            want_rows.append([i // slots * 32 + i % slots for i in part] + [-1] * (8 - len(part)))
            want_expert.append(e if world == 1 else per if e >= experts else e % per)
            want_loc.update({i: p * 8 + j for j, i in enumerate(part)})
            if (q // 8 % world if e >= experts else e // per) == rank:
                owned.append(p)
    new = lambda n: torch.zeros(n, dtype=torch.int32, device="cuda")
    expert, count, prob_rows, loc, sel, sel_count = new(room), new(1), new(room * 8), new(rows * slots), new(room), new(1)
    _lib.check(_lib.load().tf_moe_group(pick.cuda(), rows, slots, total, room, expert, count, prob_rows, loc, experts, rank, world, sel, sel_count,
                                        _lib.stream()), "group")
    n = len(want_rows)
    assert int(count) == n <= room
    assert prob_rows.reshape(-1, 8)[:n].tolist() == want_rows
    assert loc.tolist() == [want_loc[i] for i in range(rows * slots)]
    if world == 1:
        assert expert[:n].tolist() == want_expert
    else:
        assert int(sel_count) == len(owned) and sel[:len(owned)].tolist() == owned
        assert expert[:n][owned].tolist() == [want_expert[p] for p in owned]

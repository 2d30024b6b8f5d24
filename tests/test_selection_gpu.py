"""The slice, merge and draw kernels where their routes change: slices off a 16-byte boundary, short rows, keys that crowd at
the selection bound (the exact route), and the fused draw against the two separate steps."""

import numpy as np
import pytest
import torch

from oracle import lane_oracle as O

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("rows,vocab,k", [(1, 5, 3), (1, 64, 64), (2, 501, 64), (1, 4095, 28), (3, 16377, 28), (9, 16385, 1), (130, 33001, 28), (2, 248319, 64)])
@pytest.mark.parametrize("kind", ["normal", "ties", "ascending", "crowded"])
def test_selection_is_exact(lib, rows, vocab, k, kind):
    from tensorfold_b200 import topk

    gen = torch.Generator().manual_seed(vocab + k)
    x = torch.randn((rows, vocab), generator=gen)
    if kind == "ties":
        x = (x * 2).round() / 2 + 0.0               # + 0.0: no negative zeros, which the oracle ranks as zeros
    elif kind == "ascending":
        x = torch.linspace(-4, 4, vocab).repeat(rows, 1) + torch.arange(rows)[:, None]
    elif kind == "crowded":                         # one value almost everywhere: more keys reach any bound than a slice keeps
        x = torch.where(torch.rand((rows, vocab), generator=gen) < 0.9, torch.full_like(x, 0.5), x)
    x = x.to(BF)
    idx, val = topk.topk_rows(x.cuda(), k)
    widx, wval = O.topk_rows(x.float().numpy(), k)
    assert np.array_equal(idx.cpu().numpy(), widx) and np.array_equal(val.cpu().numpy(), wval)


@pytest.mark.parametrize("vocab,top_k,top_p", [(40, 8, 0.9), (5003, 1, 0.5), (33001, 20, 0.95), (33001, 56, 1.0)])
def test_fused_draw_equals_selection_then_draw(lib, vocab, top_k, top_p):
    from tensorfold_b200 import exact_sampling as S

    gen = torch.Generator().manual_seed(vocab + top_k)
    logits = (3 * torch.randn((37, vocab), generator=gen)).to(BF).cuda()
    positions = torch.arange(100, 137, device="cuda")
    s = S.Sampling(seed=5, temperature=0.7, top_k=top_k, top_p=top_p)
    fused = S.sample_rows(logits, positions, s)
    assert torch.equal(fused, S.sample_rows(logits, positions, s, top=S.top_candidates(logits, s)))
    assert np.array_equal(fused.cpu().numpy(), np.array(O.sample_rows(logits.float().cpu().numpy(), positions.cpu().numpy(), s)))


@pytest.mark.parametrize("vocab,k", [(7, 7), (100, 64), (255, 33), (256, 32), (511, 64), (513, 64), (600, 28), (1025, 28), (1500, 64), (1848, 28), (2055, 64)])
@pytest.mark.parametrize("off", [0, 5])
def test_short_rows(lib, vocab, k, off):
    """Slices whose entries leave some warps empty or partly filled, on and off a 16-byte boundary: random, in rising and falling
    order, and with the largest values side by side at either end."""

    from tensorfold_b200 import topk

    gen = torch.Generator().manual_seed(vocab)
    x = torch.randn((5, vocab + 8), generator=gen)
    x[1], x[2] = x[1].sort().values, x[2].sort(descending=True).values
    x[3, off:off + 9] += 50.0
    x[4, off + vocab - 9:off + vocab] += 50.0
    x = x.to(BF)
    idx, val = topk.topk_rows(x.cuda()[:, off:off + vocab], k)
    widx, wval = O.topk_rows(x[:, off:off + vocab].float().numpy(), k)
    assert np.array_equal(idx.cpu().numpy(), widx) and np.array_equal(val.cpu().numpy(), wval)

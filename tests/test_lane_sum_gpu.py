"""The lane matmul's shared K-segment sum where it can go wrong: fewer schedule items than workers (idle workers between the
segments' holders), as many, a block of more segments than accumulator units, and both passes of the 128-row bucket."""

import pytest
import torch

from oracle import lane_oracle as O
from tests.helpers import assert_close, assert_same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(24, 128), (16, 5120), (64, 9472), (256, 1024), (256, 9536), (520, 512), (1000, 2368), (1024, 5120), (2300, 1088)])
def test_any_split_has_the_bits_of_single_rows(lib, n, k):
    from tensorfold_b200 import _lib, lane_qmm

    gen = torch.Generator().manual_seed(n + k)
    q = O.random_q4(gen, n, k, 64)
    w = lane_qmm.tile_weight(q.words.cuda(), q.scales.cuda(), q.biases.cuda(), 64)
    x = torch.randn((128, k), generator=gen).to(torch.bfloat16).cuda()
    rows = (0, 7, 15, 31, 63, 64, 127)
    one = torch.cat([lane_qmm.lane_matmul(x[i:i + 1], w, f32=True) for i in rows])
    for m in (9, 16, 17, 32, 33, 64, 65, 128):
        for _ in range(3):                                   # the flags of an earlier launch must not count
            y = lane_qmm.lane_matmul(x[:m], w, f32=True)
        at = [i for i in rows if i < m]
        assert_same_bits(y[at], one[:len(at)], f"{m} rows")
    assert_close(y.to(torch.bfloat16), O.qmm(x.cpu(), q.words, q.scales, q.biases, 64), f"{n}x{k}")
    torch.cuda.synchronize()
    _lib.status(y.device).raise_if_set()


@pytest.mark.parametrize("rows", [8, 16, 64, 128])
def test_timeline_stamps_of_cut_blocks(lib, rows):
    """Workers that park a segment stamp it (5), and those that add parked segments stamp the sum's end (6), in every bucket."""

    from tensorfold_b200 import _lib, lane_qmm, synthetic

    gen = torch.Generator(device="cuda").manual_seed(1)
    w = synthetic.random_q4(gen, 5120, 4096, 64, "cuda")
    x = lane_qmm.pack_rows(torch.randn((rows, 4096), generator=gen, device="cuda").to(torch.bfloat16), 64)
    stamps = torch.zeros(148 + 512 * 148 * 16, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    _lib.check(lib.tf_qmm_set_trace(stamps), "trace")
    try:
        lane_qmm.lane_matmul(x, w)
        torch.cuda.synchronize()
    finally:
        _lib.check(lib.tf_qmm_set_trace(None), "trace off")
    s = stamps[148:148 + 148 * 16].reshape(148, 16).cpu()
    done, parked, summed, end = s[:, 4], s[:, 5], s[:, 6], s[:, 9]
    assert bool((done > 0).all()) and bool((end >= done).all())
    assert int((parked > 0).sum()) >= 128 and int((summed > 0).sum()) >= 20      # 20 column blocks, all of them cut
    at = (parked > 0) & (summed > 0)
    if rows > 8:                                             # every worker that parks also adds
        assert bool((summed[at] >= parked[at]).all()) and int(at.sum()) == int((parked > 0).sum())

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

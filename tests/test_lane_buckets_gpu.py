"""The lane matmul's buckets above 8 rows where the sharing of K segments changes: fewer schedule items than workers, a block cut
among eight workers, whole blocks beside cut ones, and both row passes of the 128-row bucket. A row has the bits of that row alone
(the 8-row bucket, whose sums are put together in another way)."""

import pytest
import torch

from oracle import lane_oracle as O
from tests.helpers import assert_close, assert_same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group", [64, 32])
@pytest.mark.parametrize("n,k", [(24, 64), (300, 128), (256, 1024), (260, 4096), (4864, 320), (9000, 704)])
def test_wide_buckets_have_the_bits_of_single_rows(lib, n, k, group):
    from tensorfold_b200 import _lib, lane_qmm

    gen = torch.Generator().manual_seed(n + k)
    q = O.random_q4(gen, n, k, group)
    w = lane_qmm.tile_weight(q.words.cuda(), q.scales.cuda(), q.biases.cuda(), group)
    x = torch.randn((128, k), generator=gen).to(torch.bfloat16)
    rows = (0, 8, 15, 16, 31, 32, 63, 64, 72, 127)
    one = torch.cat([lane_qmm.lane_matmul(x[i:i + 1].cuda(), w) for i in rows])
    for m in (9, 16, 17, 32, 33, 64, 65, 121, 128):
        y = lane_qmm.lane_matmul(x[:m].cuda(), w)
        got = [i for i in rows if i < m]
        assert_same_bits(y[got], one[:len(got)], f"{m} rows")
        assert_same_bits(lane_qmm.lane_matmul(x[:m].cuda(), w, f32=True).to(torch.bfloat16), y, f"{m} rows, fp32 sums")
    assert_close(y, O.qmm(x, q.words, q.scales, q.biases, group), f"{n}x{k} g{group}")
    torch.cuda.synchronize()
    _lib.status(y.device).raise_if_set()

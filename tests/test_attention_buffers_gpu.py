"""Attention with one and with two K and V buffers a block: which one runs depends on the number of (sequence, KV head, query group)
columns and on the capacity the launch is made for, and must not show in a single bit. Chunks of 2 (below 8192 keys), 8 and 32 tiles."""

import pytest
import torch

from oracle import lane_oracle as O
from tests.helpers import assert_close, assert_same_bits

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _cache(lens, hk, d, width, seed):
    from tensorfold_b200 import lane_attention as LA

    gen = torch.Generator(device="cuda").manual_seed(seed)
    pages = [max(1, -(-n // 16)) for n in lens]
    kv = LA.PagedKV(1, len(lens), sum(pages), hk, d, max(pages), "cuda")
    kv.k.normal_(generator=gen)
    kv.v.normal_(generator=gen)
    for s, n in enumerate(lens):
        kv.reserve(s, max(n, 1))
    kv.sync_table()
    return kv, gen


def _attend(kv, lens, q, k_new, v_new, width, capacity):
    from tensorfold_b200 import lane_attention as LA

    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    n = len(lens)
    return LA.lane_attention(q, k_new, v_new, kv.k[0], kv.v[0], kv.table, i32(lens), i32(list(range(0, n * width + 1, width))),
                             i32([m + t + 1 for m in lens for t in range(width)]), scale=q.shape[-1] ** -0.5, max_window=width,
                             max_chunks=LA.chunks_for(max(capacity, max(lens)) + width))


@pytest.mark.parametrize("h,hk,d,n,long", [(16, 1, 256, 16, 20000), (6, 1, 256, 17, 8200), (16, 2, 256, 8, 12000), (24, 4, 256, 4, 9000),
                                           (24, 4, 256, 4, 66000), (24, 4, 256, 5, 130), (16, 2, 128, 40, 9000)])
@pytest.mark.parametrize("width", [1, 8])
def test_alone_among_others_and_at_any_capacity(lib, h, hk, d, n, long, width):
    lens = [long] + [(37 * i * i) % 700 for i in range(1, n)]
    kv, gen = _cache(lens, hk, d, width, h + n)
    rows = n * width
    q = torch.randn((rows, h, d), generator=gen, device="cuda").to(BF)
    k_new, v_new = (torch.randn((rows, hk, d), generator=gen, device="cuda").to(BF) for _ in range(2))
    every = _attend(kv, lens, q, k_new, v_new, width, 0)
    assert_same_bits(_attend(kv, lens, q, k_new, v_new, width, 100000), every, "a larger capacity")
    table = kv.table
    for s in (0, n - 1):
        kv.table = table[s:s + 1].contiguous()
        part = slice(s * width, (s + 1) * width)
        for capacity in (0, 100000):
            alone = _attend(kv, lens[s:s + 1], q[part], k_new[part], v_new[part], width, capacity)
            assert_same_bits(alone, every[part], f"sequence {s} alone, capacity {capacity}")
    pages = table[0, :-(-long // 16)].long()
    flat = lambda t: t[0, pages].permute(0, 2, 1, 3).reshape(-1, hk, d)[:long]
    keys, vals = torch.cat([flat(kv.k), k_new[:width]]).cpu(), torch.cat([flat(kv.v), v_new[:width]]).cpu()
    want = O.attention(q[:width].cpu(), keys, vals, torch.arange(long + 1, long + width + 1), d ** -0.5)
    assert_close(every[:width], want, f"{long} keys")

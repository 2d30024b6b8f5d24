"""A weight that is written on the stream just before a plain-rows matmul is the weight that the matmul reads: the matmul copies its
first weights without waiting for the packing kernel in front of it, so that kernel may let it start only once it has itself
waited for the writer."""

import re
from pathlib import Path

import pytest
import torch

from oracle import lane_oracle as O
from tests.helpers import assert_same_bits

CSRC = Path(__file__).resolve().parent.parent / "tensorfold_b200" / "csrc"


def test_packing_waits_before_it_lets_the_matmul_start():
    pack = re.search(r"__global__ void pack_rows_kernel\(.*?\n}\n", (CSRC / "qmm.cu").read_text(), re.S).group(0)
    assert re.findall(r"pdl_\w+\(\)", re.sub(r"//[^\n]*", "", pack)) == ["pdl_wait()", "pdl_launch_dependents()"]


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 8, 40, 130])
@pytest.mark.parametrize("n,k", [(1024, 5120), (9000, 704)])
def test_a_weight_refilled_in_place_is_the_one_read(lib, rows, n, k):
    from tensorfold_b200 import lane_qmm

    gen = torch.Generator().manual_seed(rows + n)
    a, b = (O.random_q4(gen, n, k, 64) for _ in range(2))
    words = lambda q: (q.words.cuda(), q.scales.cuda(), q.biases.cuda())
    wa, wb = lane_qmm.tile_weight(*words(a), 64), lane_qmm.tile_weight(*words(b), 64)
    x = torch.randn((rows, k), generator=gen).to(torch.bfloat16).cuda()
    want_a, want_b = lane_qmm.lane_matmul(x, wa), lane_qmm.lane_matmul(x, wb)
    buf = lane_qmm.QWeight(wa.tiled.clone(), n, k, 64)
    torch.cuda.synchronize()
    for src, want in ((wb, want_b), (wa, want_a), (wb, want_b)):
        buf.tiled.copy_(src.tiled)
        assert_same_bits(lane_qmm.lane_matmul(x, buf), want, "refilled by a copy")
    raw = words(b)
    fresh = lane_qmm.tile_weight(*raw, 64)                  # the tiling kernel right in front
    assert_same_bits(lane_qmm.lane_matmul(x, fresh), want_b, "just tiled")
    assert_same_bits(lane_qmm.lane_matmul(x, *raw), want_b, "tiled inside the call")


@pytest.mark.gpu
def test_stored_weights_are_read_at_every_call(lib):
    """The call shape with stored words: other values at the same addresses, however they got there, are the ones multiplied."""

    from tensorfold_b200 import lane_qmm

    gen = torch.Generator().manual_seed(3)
    a, b = (O.random_q4(gen, 300, 128, 64) for _ in range(2))
    x = torch.randn((3, 128), generator=gen).to(torch.bfloat16).cuda()
    cuda = lambda q: [t.cuda() for t in (q.words, q.scales, q.biases)]
    want = [lane_qmm.lane_matmul(x, lane_qmm.tile_weight(*cuda(q), 64)) for q in (a, b)]
    held = cuda(a)
    assert_same_bits(lane_qmm.lane_matmul(x, *held), want[0], "first values")
    for t, new in zip(held, cuda(b)):
        t.data.copy_(new)
    assert_same_bits(lane_qmm.lane_matmul(x, *held), want[1], "overwritten in place")
    for i in (0, 1, 0, 1):                                   # freed and allocated again, at the same addresses
        del held
        held = cuda((a, b)[i])
        assert_same_bits(lane_qmm.lane_matmul(x, *held), want[i], "new tensors")

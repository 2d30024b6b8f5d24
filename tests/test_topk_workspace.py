"""One top-k workspace serves every call that is no larger than the one it was made for, although fewer rows are cut into more
slices; the largest vocabulary."""

import pytest
import torch


def test_workspace_grows_with_rows_vocabulary_and_k(lib):
    for vocab in (1, 4095, 4096, 8192, 16000, 16376, 32000, 151936, 248320, 262144, 1048576):
        sizes = [lib.tf_topk_scratch_bytes(r, vocab, 28) for r in range(1, 400)]
        assert all(a <= b for a, b in zip(sizes, sizes[1:])), vocab
        assert all(lib.tf_topk_scratch_bytes(r, vocab, 1) * 28 == sizes[r - 1] for r in (1, 7, 148, 399))
    for rows in (1, 8, 73, 74, 128):
        sizes = [lib.tf_topk_scratch_bytes(rows, v, 8) for v in range(1, 300000, 997)]
        assert all(a <= b for a, b in zip(sizes, sizes[1:])), rows
    assert lib.tf_topk_scratch_bytes(0, 8, 1) == lib.tf_topk_scratch_bytes(1, 8, 65) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("largest", [4, 8, 128])
@pytest.mark.parametrize("vocab", [16000, 248320])
def test_one_workspace_over_row_counts(lib, largest, vocab):
    from tensorfold_b200 import _lib, topk

    k = 28
    size = lib.tf_topk_scratch_bytes(largest, vocab, k)
    room = torch.full((size + 256,), 0x5A, dtype=torch.uint8, device="cuda")      # a margin that no call may write
    x = torch.randn((largest, vocab), generator=torch.Generator().manual_seed(vocab)).to(torch.bfloat16).cuda()
    want = topk.topk_rows(x, k)
    for rows in range(1, largest + 1):
        idx = torch.empty((rows, k), dtype=torch.int32, device="cuda")
        val = torch.empty((rows, k), device="cuda")
        _lib.check(lib.tf_topk_rows(x, vocab, rows, vocab, k, idx, val, room, size, _lib.stream()), f"{rows} rows")
        assert torch.equal(idx, want[0][:rows]) and torch.equal(val, want[1][:rows]), rows
    assert bool((room[size:] == 0x5A).all())


@pytest.mark.gpu
@pytest.mark.parametrize("vocab", [1048063, 1048064, 1048065, 1048570, 1048576])
@pytest.mark.parametrize("off", [0, 3])
def test_the_largest_vocabularies(lib, vocab, off):
    """Up to 64 slices of 16384 entries, on and off a 16-byte boundary (``off`` entries into a row)."""

    from tensorfold_b200 import topk

    rows, k = 2, 28
    wide = torch.randn((rows, vocab + 8), generator=torch.Generator().manual_seed(vocab)).to(torch.bfloat16)
    x = wide.cuda()[:, off:off + vocab]
    idx, val = topk.topk_rows(x, k)
    order = torch.sort(wide[:, off:off + vocab].float(), dim=1, descending=True, stable=True)
    assert torch.equal(idx.cpu().long(), order.indices[:, :k]) and torch.equal(val.cpu(), order.values[:, :k])


def test_a_longer_vocabulary_is_refused(lib):
    from tensorfold_b200 import _lib

    one = 256                                               # an address that a refused call does not read
    assert lib.tf_topk_rows(one, 1048577, 1, 1048577, 1, one, one, one, 1 << 30, None) == _lib.TF_EINVAL

"""The gated-DeltaNet kernels at the edges of their thread blocks: value dims that fill half of a 64-row block, windows of several
8-row passes, and grids on both sides of one block an SM (148), where the mixer changes its register split."""

import pytest
import torch

from oracle import lane_oracle as O
from tests.helpers import assert_same_bits
from tests.test_gdn_attention_gpu import _mixer_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dv", [32, 64, 96, 160])
@pytest.mark.parametrize("width", [1, 8, 9, 33])
def test_chain_and_replay_at_any_value_dim(lib, dv, width):
    from tensorfold_b200 import lane_gdn

    gen = torch.Generator().manual_seed(dv + width)
    kh, vh = 2, 4
    norm = lambda *s: torch.nn.functional.normalize(torch.randn(s, generator=gen), dim=-1)
    q, k = norm(width, kh, 128).to(torch.bfloat16), norm(width, kh, 128).to(torch.bfloat16)
    v = torch.randn((width, vh, dv), generator=gen).to(torch.bfloat16)
    g, beta = torch.rand((width, vh), generator=gen), torch.rand((width, vh), generator=gen)
    state = 0.1 * torch.randn((1, vh, dv, 128), generator=gen)
    starts = torch.tensor([0, width], dtype=torch.int32).cuda()
    dev = [t.cuda() for t in (q, k, v, g, beta)]
    final = torch.empty_like(state).cuda()
    y = lane_gdn.gated_delta_chain(*dev, state.cuda(), starts, state_out=final)
    y_ref, s_ref = O.gdn_recurrence(q, k, v, g, beta, state[0])
    # fp32 sums of up to 128 terms over `width` dependent steps; y has one bf16 rounding
    assert (final[0].cpu() - s_ref).abs().max() < 1e-4 * max(1.0, float(s_ref.abs().max()))
    assert (y.float().cpu() - y_ref.float()).abs().max() <= 2 ** -7 * y_ref.float().abs().max() + 1e-5
    replayed = state.cuda()
    lane_gdn.replay(*dev[1:], replayed, starts, torch.tensor([width], dtype=torch.int32).cuda())
    assert_same_bits(replayed, final)


@pytest.mark.parametrize("widths,nk,nv,group", [([128], 1, 2, 64), ([33, 1, 8, 9], 37, 37, 32), ([33, 1, 8, 9], 38, 38, 32), ([17] * 5, 16, 48, 64)])
def test_mixer_on_both_sides_of_a_block_an_sm(lib, widths, nk, nv, group):
    from tensorfold_b200 import lane_gdn, lane_glue

    d = lambda t: t.cuda()
    proj, conv_state, conv_w, a_log, dt_bias, norm_w, state, starts, row_seq, row_idx = map(d, _mixer_inputs(len(widths), widths, nk, nv))
    c = (2 * nk + nv) * 128
    # a copy with the row stride rounded up to 8 bytes, the kernels' alignment (37 heads leave an odd one)
    wide = torch.zeros((proj.shape[0], -(-proj.shape[1] // 8) * 8), dtype=proj.dtype, device="cuda")
    wide[:, :proj.shape[1]] = proj
    qkv, z, bb, aa = wide[:, :c], wide[:, c:c + nv * 128], wide[:, c + nv * 128:c + nv * 128 + nv], wide[:, c + nv * 128 + nv:c + nv * 128 + 2 * nv]
    q, k, v, g, beta = lane_glue.gdn_pre(qkv, conv_state, conv_w, row_seq, row_idx, aa, bb, a_log, dt_bias, nk=nk, nv=nv)
    y = lane_gdn.gated_delta_chain(q, k, v, g, beta, state, starts)
    want_packed, want_rows = lane_glue.gdn_post(y, z, norm_w, 1e-6, group=group, rows_out=True)
    rec = (torch.empty_like(k), torch.empty_like(v), torch.empty_like(g), torch.empty_like(beta))
    packed, rows = lane_gdn.gdn_mixer(qkv, z, aa, bb, conv_state, conv_w, a_log, dt_bias, norm_w, state, starts,
                                      nk=nk, nv=nv, eps=1e-6, group=group, record=rec, rows_out=True)
    assert_same_bits(rows, want_rows, "mixer rows")
    assert torch.equal(packed.data, want_packed.data)
    for got, want in zip(rec, (k, v, g, beta)):
        assert torch.equal(got, want)


@pytest.mark.parametrize("vh,windows,layers", [(4, 1, 1), (4, 6, 1), (4, 7, 1), (4, 9, 1), (4, 10, 1), (32, 1, 6), (32, 7, 1), (32, 1, 8)])
def test_replay_has_the_chain_state_at_any_grid(lib, vh, windows, layers):
    """Both sides of the lines between one and two value rows a thread, and between three and four blocks an SM."""

    from tensorfold_b200 import lane_gdn

    gen = torch.Generator(device="cuda").manual_seed(vh + windows)
    width, kh = 3, vh // 2
    rows = width * windows
    rnd = lambda *s: torch.randn(s, generator=gen, device="cuda")
    k = torch.nn.functional.normalize(rnd(layers, rows, kh, 128), dim=-1).to(torch.bfloat16)
    v = rnd(layers, rows, vh, 128).to(torch.bfloat16)
    g, beta = (torch.rand((layers, rows, vh), generator=gen, device="cuda") for _ in range(2))
    state = 0.1 * rnd(layers, windows, vh, 128, 128)
    starts = torch.arange(0, rows + 1, width, dtype=torch.int32, device="cuda")
    want = torch.empty_like(state)
    for i in range(layers):
        for s in range(windows):                             # one window a call: the small grid
            part = slice(s * width, (s + 1) * width)
            final = torch.empty_like(state[i, s:s + 1])
            y = lane_gdn.gated_delta_chain(k[i, part], k[i, part], v[i, part], g[i, part], beta[i, part], state[i, s:s + 1],
                                           torch.tensor([0, width], dtype=torch.int32, device="cuda"), state_out=final)
            want[i, s] = final[0]
            if s == 0:
                first = y
        every = lane_gdn.gated_delta_chain(k[i], k[i], v[i], g[i], beta[i], state[i], starts)
        assert_same_bits(every[:width], first, "chain rows")
    keep = torch.full((windows,), width, dtype=torch.int32, device="cuda")
    if layers == 1:
        lane_gdn.replay(k[0], v[0], g[0], beta[0], state[0], starts, keep)
    else:
        lane_gdn.replay(k, v, g, beta, state, starts, keep)
    assert_same_bits(state, want, "replayed states")

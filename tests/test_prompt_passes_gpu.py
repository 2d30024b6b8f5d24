"""Prompts in passes of up to 128 rows: the first token and the committed state of passes of 8 rows, bit for bit, whatever the number
of passes and of rows in the last one, behind a kept prefix, on the wide-row kernel and in any ``prompt_rows``."""

import pytest
import torch

from oracle import lane_oracle as O
from tests.helpers import assert_same_bits

pytestmark = pytest.mark.gpu

DENSE = dict(hidden=256, intermediate=512, layers=4, heads=4, kv_heads=2, head_dim=128, vocab=512, k_heads=2, v_heads=4, dk=128, dv=128)
MOE = dict(hidden=256, intermediate=0, layers=4, heads=4, kv_heads=2, head_dim=128, vocab=512, k_heads=2, v_heads=4, dk=128, dv=128,
           group=32, experts=8, top_k=2, moe_intermediate=128)


@pytest.fixture(scope="module", params=["dense", "moe"])
def weights(lib, request):
    from tensorfold_b200 import forward as F

    return F.load_weights(O.random_model(O.Config(**(DENSE if request.param == "dense" else MOE)), seed=43), "cuda")


def _tokens(n, seed=1):
    return torch.randint(0, 512, (n,), generator=torch.Generator().manual_seed(seed)).tolist()


def _same_state(a, b, lens):
    assert a.lens == b.lens == lens
    assert_same_bits(a.rec, b.rec, "recurrent states")
    assert_same_bits(a.conv, b.conv, "conv tails")
    for s, n in enumerate(lens):
        pages = -(-n // 16)
        for x, y in ((a.kv.k, b.kv.k), (a.kv.v, b.kv.v)):
            rows = lambda st, t: t[:, st.kv.table_host[s, :pages].long().cuda()].permute(0, 1, 3, 2, 4).flatten(1, 2)[:, :n]
            assert_same_bits(rows(a, x), rows(b, y), "keys or values")


@pytest.mark.parametrize("n", [9, 64, 65, 128, 129, 203, 300])
def test_engine_prompt_equals_passes_of_8_rows(weights, n):
    from tensorfold_b200 import decode, forward as F
    from tensorfold_b200.exact_sampling import Sampling

    w, prompt, sampling = weights, _tokens(n), Sampling(seed=n, temperature=0.8, top_k=20, top_p=0.95)
    st = F.State(w, 1, 512)
    pending = decode.prefill(w, st, [prompt], sampling, chunk=8)
    for rows in (128, 100, 8):
        eng = decode.Engine(w, max_context=512, prompt_rows=rows)
        assert eng.generate(prompt, 1, sampling)["tokens"] == pending
        _same_state(eng.state, st, [n])
    # a longer prompt behind the kept one, its tail in one or more passes
    for more in (5, 130):
        longer = prompt + _tokens(more, seed=2)
        eng = decode.Engine(w, max_context=512)
        eng.generate(prompt, 1, sampling)
        before = eng.state
        got = eng.generate(longer, 1, sampling)["tokens"]
        assert eng.state is before, "the prefix was not kept"
        st2 = F.State(w, 1, 512)
        assert got == decode.prefill(w, st2, [longer], sampling, chunk=8)
        _same_state(eng.state, st2, [len(longer)])
    # and what follows the prompt
    want = decode.serial_decode(w, st, pending, 6, sampling).tokens[0]
    assert decode.Engine(w, max_context=512).generate(prompt, 6, sampling)["tokens"] == want


def test_several_prompts_and_the_wide_kernel(lib):
    from tensorfold_b200 import decode, forward as F

    w = F.enable_wide(F.load_weights(O.random_model(O.Config(**DENSE), seed=44), "cuda"))
    prompts = [_tokens(n, seed=n) for n in (150, 3, 70)]
    for wide in (False, True):
        states, firsts = [], []
        for chunk in (8, 31, 128):
            st = F.State(w, 3, 512, wide=wide)
            firsts.append(decode.prefill(w, st, prompts, None, chunk=chunk))
            states.append(st)
        assert firsts[0] == firsts[1] == firsts[2]
        for st in states[1:]:
            _same_state(st, states[0], [150, 3, 70])


def test_prompt_rows_bound_the_memory_of_a_pass(weights):
    from tensorfold_b200 import decode

    peaks = {}
    for rows in (8, 128):
        eng = decode.Engine(weights, max_context=512, prompt_rows=rows)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        held = torch.cuda.memory_allocated()
        eng.generate(_tokens(300), 1)
        peaks[rows] = torch.cuda.max_memory_allocated() - held
    assert peaks[8] < peaks[128] / 2, peaks
    for bad in (0, 129):
        with pytest.raises(ValueError):
            decode.Engine(weights, max_context=512, prompt_rows=bad)


def test_a_replaced_weight_has_no_wide_twin(lib):
    """The wide twins belong to the weights they were made from: another weight in their place is not given one silently."""

    import weakref

    from tensorfold_b200 import forward as F, synthetic

    w = F.enable_wide(F.load_weights(O.random_model(O.Config(**DENSE), seed=45), "cuda"))
    old = weakref.ref(w.head)
    w.head = synthetic.random_q4(torch.Generator(device="cuda").manual_seed(1), w.head.n, w.head.k, w.head.group, "cuda")
    assert old() is not None
    with pytest.raises(KeyError):
        F.tree_forward(w, torch.zeros(1, dtype=torch.int32, device="cuda"), [1], F.State(w, 1, 64, wide=True))

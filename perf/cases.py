"""What is timed: the work a program built on this package has it do, through the package's public entry points.

Kinds of cases:

* ``step``: one decode round of ``runner.LaneRunner`` - ``step`` (host tokens in, chosen tokens out) and ``commit`` of the
  rows that were accepted - over one or many sequences, each with its own window width and context. Dense models on the lane
  kernel or (``wide``) on the wide-row kernel, or the mixture-of-experts model. The models are the package's two
  configurations at their full widths, with fewer layers: layers repeat, so a shallower model has the same
  kernels, launches and proportions, and its weights still exceed the L2 cache many times over.
* ``generate``: ``decode.Engine.generate`` on a new prompt up to its first token: prompt processing.
* ``matmul`` and ``prefill_matmul``: one 4-bit projection on the lane kernel and on the wide-row kernel.
* ``gdn``: the gated-DeltaNet mixer of one layer over many sequences' windows.
* ``sample``: the tokens of a batch of vocabulary rows.

Random weights, states and tokens: every path's cost is independent of their values, except for the
experts that the rows of a mixture-of-experts step choose, which are as many as with a random router.
"""

import random

import torch

from tensorfold_b200 import decode, forward, lane_gdn, lane_qmm, prefill_qmm, runner, synthetic
from tensorfold_b200.exact_sampling import Sampling, sample_rows

BF16 = torch.bfloat16
GROWTH = 256            # tokens a context grows by before a step's sequences start again from their first length
MODELS = {"dense27b": synthetic.DENSE_27B, "moe30b": synthetic.MOE_30B}


def _step(name, model, layers, seqs, width, ctx, sampled=False, wide=False):
    """``width`` and ``ctx``: (smallest, largest) over the sequences."""

    return {"name": name, "kind": "step", "model": model, "layers": layers, "seqs": seqs, "width_lo": width[0], "width_hi": width[1],
            "ctx_lo": ctx[0], "ctx_hi": ctx[1], "sampled": sampled, "wide": wide}


def listed():
    return [
        # one user, no drafts: every token is one pass of one row (the baseline that drafted decoding is compared with)
        _step("step_dense_serial", "dense27b", 16, 1, (1, 1), (1024, 1024)),
        # one user with a drafter: a window of 8 rows, the package's benchmark workload
        _step("step_dense_window8", "dense27b", 16, 1, (8, 8), (4096, 4096)),
        # a few users, ragged windows, long and unequal contexts, sampled tokens
        _step("step_dense_ragged_long", "dense27b", 16, 4, (2, 8), (8192, 32768), sampled=True),
        # a busy server: 16 users x 8 rows fill the 128-row forward, on the wide-row kernel
        _step("step_dense_16_users", "dense27b", 16, 16, (8, 8), (4096, 4096), wide=True),
        # mixture of experts, one user with short drafts: few experts are touched, launches count
        _step("step_moe_window4", "moe30b", 8, 1, (4, 4), (2048, 2048)),
        # mixture of experts, continuous batch of 32 users with ragged windows and contexts of 1k..16k
        _step("step_moe_32_users", "moe30b", 8, 32, (1, 7), (1024, 16384)),
        # a question of a few hundred tokens: what a user waits for before the first token
        {"name": "generate_prompt", "kind": "generate", "layers": 8, "prompt": 203},
        # the smallest projection of a decode step (keys or values of one row)
        {"name": "matmul_small", "kind": "matmul", "rows": 1, "n": 1024, "k": 5120, "group": 64},
        # the package's single-operator workload: 8 rows times one MLP projection
        {"name": "matmul_mlp_8_rows", "kind": "matmul", "rows": 8, "n": 17408, "k": 5120, "group": 64},
        # a long prompt's rows times one MLP projection
        {"name": "prefill_matmul", "kind": "prefill_matmul", "rows": 500, "n": 17408, "k": 5120, "group": 64},
        # the recurrence of one layer over 32 users x 8 rows
        {"name": "gdn_32_users", "kind": "gdn", "seqs": 32, "width": 8},
        # tokens of a full step: 128 rows of the 248320-word vocabulary
        {"name": "sample_128_rows", "kind": "sample", "rows": 128, "vocab": 248320, "top_k": 20},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "generate", "matmul", "matmul", "prefill_matmul", "gdn", "sample"])
    if kind == "step":
        what = rng.choice(["one", "few", "wide", "moe"])
        sampled = rng.random() < 0.5
        if what == "one":
            w, ctx = rng.randint(1, 8), _log(rng, 256, 32768)
            return _nameless(_step("", "dense27b", 8, 1, (w, w), (ctx, ctx), sampled))
        if what == "few":
            lo, ctx = rng.randint(1, 4), _log(rng, 512, 16384)
            return _nameless(_step("", "dense27b", 8, rng.randint(2, 4), (lo, rng.randint(lo, 8)), (ctx, 2 * ctx), sampled))
        if what == "wide":
            lo, ctx = rng.randint(1, 8), _log(rng, 512, 8192)
            return _nameless(_step("", "dense27b", 8, rng.randint(5, 16), (lo, rng.randint(lo, 8)), (ctx // 2, ctx), sampled, wide=True))
        lo, ctx = rng.randint(1, 3), _log(rng, 1024, 16384)
        return _nameless(_step("", "moe30b", 8, _log(rng, 1, 24), (lo, rng.randint(lo, 5)), (ctx // 2, ctx), sampled))
    if kind == "generate":
        return {"kind": "generate", "layers": 8, "prompt": _log(rng, 12, 400)}
    if kind == "matmul":
        return {"kind": "matmul", "rows": _log(rng, 1, 128), "n": _log(rng, 500, 35000), "k": 64 * _log(rng, 8, 270), "group": rng.choice([32, 64])}
    if kind == "prefill_matmul":
        return {"kind": "prefill_matmul", "rows": _log(rng, 30, 700), "n": _log(rng, 1000, 17408), "k": 64 * _log(rng, 16, 100),
                "group": rng.choice([32, 64])}
    if kind == "gdn":
        return {"kind": "gdn", "seqs": _log(rng, 1, 32), "width": rng.randint(1, 8)}
    return {"kind": "sample", "rows": _log(rng, 1, 128), "vocab": _log(rng, 30000, 250000), "top_k": rng.choice([0, 8, 20, 50])}


def _nameless(case):
    del case["name"]
    return case


def _config(case):
    return forward.Config(**dict(MODELS[case.get("model", "dense27b")], layers=case["layers"]))


def _layout(case):
    """Each sequence's window width and context: a fixed function of the case (the same work for every seed)."""

    rng = random.Random(case["seqs"] * 1000 + case["width_hi"])
    widths = [rng.randint(case["width_lo"], case["width_hi"]) for _ in range(case["seqs"])]
    while sum(widths) > lane_qmm.MAX_ROWS:
        widths[widths.index(max(widths))] -= 1
    return widths, [rng.randint(case["ctx_lo"], case["ctx_hi"]) for _ in range(case["seqs"])]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    host = random.Random(seed)
    kind = case["kind"]

    def normal(*shape, scale=1.0, dtype=BF16):
        return (scale * torch.randn(shape, generator=gen, device="cuda")).to(dtype)

    if kind == "step":
        cfg = _config(case)
        w = synthetic.random_weights(cfg, seed=seed)
        if case["wide"]:
            forward.enable_wide(w)
        widths, ctxs = _layout(case)
        room = max(ctxs) + GROWTH
        st = forward.State(w, case["seqs"], room + max(widths), wide=case["wide"])
        sampling = Sampling(seed=seed, temperature=0.8, top_k=20, top_p=0.95) if case["sampled"] else None
        run_ = runner.LaneRunner(w, st, widths, max_context=room, sampling=sampling)
        run_.capture()
        # committed sequences of the given lengths: keys, values, recurrent states and conv tails of ordinary sizes
        st.kv.k.normal_(generator=gen)
        st.kv.v.normal_(generator=gen)
        st.rec.normal_(0.0, 0.1, generator=gen)
        st.conv.normal_(generator=gen)
        st.lens = list(ctxs)
        run_.refresh()
        tokens = torch.tensor([host.randrange(cfg.vocab) for _ in range(sum(widths))], dtype=torch.int32)
        return {"kind": kind, "runner": run_, "state": st, "tokens": tokens, "keep": [host.randint(1, x) for x in widths], "start": ctxs}
    if kind == "generate":
        cfg = _config(case)
        w = synthetic.random_weights(cfg, seed=seed)
        engine = decode.Engine(w, max_context=512)
        return {"kind": kind, "engine": engine, "prompt": [host.randrange(cfg.vocab) for _ in range(case["prompt"])]}
    if kind in ("matmul", "prefill_matmul"):
        n, k, g = case["n"], case["k"], case["group"]
        q = synthetic.random_q4(gen, n, k, g, "cuda")
        if kind == "prefill_matmul":
            q = prefill_qmm.tile_weight(*lane_qmm.untile_weight(q), g)
        return {"kind": kind, "x": normal(case["rows"], k), "weight": q}
    if kind == "gdn":
        nk, nv, seqs, width = 16, 32, case["seqs"], case["width"]
        c = (2 * nk + nv) * 128
        per = max(1, lane_qmm.MAX_ROWS // width)              # sequences a call: a packed buffer holds 128 rows
        conv = normal(seqs, 3, c)
        rec = normal(seqs, nv, 128, 128, scale=0.1, dtype=torch.float32)
        calls = []
        for s0 in range(0, seqs, per):
            s1 = min(seqs, s0 + per)
            r = (s1 - s0) * width
            starts = torch.arange(0, r + 1, width, dtype=torch.int32, device="cuda")
            record = (torch.zeros((r, nk, 128), dtype=BF16, device="cuda"), torch.zeros((r, nv, 128), dtype=BF16, device="cuda"),
                      torch.zeros((r, nv), device="cuda"), torch.zeros((r, nv), device="cuda"))
            calls.append((normal(r, c + nv * 128 + 2 * nv), conv[s0:s1], rec[s0:s1], starts, record))
        return {"kind": kind, "nk": nk, "nv": nv, "c": c, "calls": calls, "conv_w": normal(c, 4, scale=0.3),
                "a_log": normal(nv, scale=0.5, dtype=torch.float32), "dt_bias": normal(nv, scale=0.5, dtype=torch.float32), "norm": 1 + normal(128, scale=0.05)}
    if kind == "sample":
        positions = torch.randint(1, 32768, (case["rows"],), generator=gen, device="cuda")
        sampling = Sampling(seed=seed, temperature=0.8, top_k=case["top_k"], top_p=0.95) if case["top_k"] else None     # 0: greedy
        return {"kind": kind, "logits": normal(case["rows"], case["vocab"], scale=3.0), "positions": positions, "sampling": sampling}
    raise ValueError(kind)


def run(state):
    kind = state["kind"]
    if kind == "step":
        r, st = state["runner"], state["state"]
        if st.lens[0] + state["keep"][0] > state["start"][0] + GROWTH or any(
                n + k > s + GROWTH for n, k, s in zip(st.lens, state["keep"], state["start"])):
            st.lens = list(state["start"])                    # the sequences start again from their first length
            r.refresh()
        r.step(state["tokens"])
        r.commit(state["keep"])
        # the chosen tokens are the logits' largest entries or a draw from them: compared through the logits, whose
        # two largest bf16 values often tie
        return {"logits": r.logits, "rec": st.rec, "conv": st.conv, "k": st.kv.k, "v": st.kv.v}
    if kind == "generate":
        e = state["engine"]
        e.generate(state["prompt"], 1)                        # the first token: as for a step, its state is compared
        return {"rec": e.state.rec, "conv": e.state.conv, "k": e.state.kv.k, "v": e.state.kv.v}
    if kind == "matmul":
        return lane_qmm.lane_matmul(state["x"], state["weight"])
    if kind == "prefill_matmul":
        return prefill_qmm.prefill_matmul(state["x"], state["weight"])
    if kind == "gdn":
        c, nk, nv = state["c"], state["nk"], state["nv"]
        out = []
        for proj, conv, rec, starts, record in state["calls"]:
            z, b, a = proj[:, c:c + nv * 128], proj[:, c + nv * 128:c + nv * 128 + nv], proj[:, c + nv * 128 + nv:]
            _, rows = lane_gdn.gdn_mixer(proj[:, :c], z, a, b, conv, state["conv_w"], state["a_log"], state["dt_bias"], state["norm"], rec, starts,
                                         nk=nk, nv=nv, eps=1e-6, group=64, record=record, rows_out=True)
            out.append((rows, *record))
        return out
    return sample_rows(state["logits"], state["positions"], state["sampling"])


def _weight_bytes(n, k, group):
    return n * k / 2 + n * (k // group) * 4


def _model_work(case, rows, contexts, logit_rows):
    """Bytes and operations of the layers and the head for ``rows`` rows over sequences with ``contexts`` committed keys."""

    c = _config(case)
    kd, vd, g = c.k_heads * 128, c.v_heads * 128, c.group
    att = sum(not c.is_linear(i) for i in range(c.layers))
    gdn = c.layers - att
    dense = gdn * [(2 * kd + 2 * vd + 2 * c.v_heads, c.hidden), (c.hidden, vd)] + \
        att * [((2 * c.heads + 2 * c.kv_heads) * c.head_dim, c.hidden), (c.hidden, c.heads * c.head_dim)] + [(c.vocab, c.hidden)]
    if not c.experts:
        dense += c.layers * [(2 * c.intermediate, c.hidden), (c.hidden, c.intermediate)]
    nbytes = sum(_weight_bytes(n, k, g) for n, k in dense)
    flops = sum(2 * n * k * (logit_rows if n == c.vocab else rows) for n, k in dense)
    if c.experts:
        expert = [(2 * c.moe_intermediate, c.hidden), (c.hidden, c.moe_intermediate)]
        touched = c.experts * (1 - (1 - c.top_k / c.experts) ** rows) + 1
        nbytes += c.layers * (touched * sum(_weight_bytes(n, k, g) for n, k in expert) + (c.experts + 1) * c.hidden * 2)
        flops += c.layers * rows * (c.top_k + 1) * sum(2 * n * k for n, k in expert)
    keys = sum(contexts)
    nbytes += att * keys * 2 * c.kv_heads * c.head_dim * 2                              # keys and values read
    nbytes += 2 * gdn * len(contexts) * c.v_heads * 128 * 128 * 4                       # recurrent states read and, committed, written
    nbytes += rows * (c.hidden // 2 + c.hidden // g * 4) + logit_rows * c.vocab * 2     # embedding rows, logits
    flops += gdn * rows * c.v_heads * 7 * 128 * 128
    return nbytes, flops, att * c.heads * c.head_dim * 4


def work(case):
    kind = case["kind"]
    if kind == "step":
        widths, ctxs = _layout(case)
        nbytes, flops, per_key = _model_work(case, sum(widths), ctxs, sum(widths))
        return {"bytes": nbytes, "flops": flops + per_key * sum(w * c for w, c in zip(widths, ctxs))}
    if kind == "generate":
        n = case["prompt"]
        nbytes, flops, per_key = _model_work(case, n, [n], 1)
        return {"bytes": nbytes, "flops": flops + per_key * n * n / 2}
    if kind in ("matmul", "prefill_matmul"):
        m, n, k = case["rows"], case["n"], case["k"]
        return {"bytes": _weight_bytes(n, k, case["group"]) + m * k * 2 + m * n * 2, "flops": 2 * m * n * k}
    if kind == "gdn":
        r = case["seqs"] * case["width"]
        c = 64 * 128
        return {"bytes": case["seqs"] * (32 * 128 * 128 * 4 + 3 * c * 2) + r * (c + 2 * 32 * 128 + 48 * 128) * 2, "flops": r * 32 * 7 * 128 * 128}
    return {"bytes": case["rows"] * case["vocab"] * 2, "flops": case["rows"] * case["vocab"]}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"                   # tokens of given logits
    if case["kind"] in ("step", "generate"):
        return {"rel": 2e-2}             # bf16 activations rounded some ten times a layer, through 8 to 16 layers
    return {"rel": 1e-2}                 # one bf16 rounding of fp32 sums, or of fp32 arithmetic on bf16 inputs

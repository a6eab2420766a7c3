"""Logits at the layer widths the benchmarks run, through the engine, over every kernel route.

The tiny configurations of the other tests stop at 128-wide layers and a vocabulary of 1,000, so
they never reach the kernels the benchmark numbers come from: the tcgen05 head (5 to 64 rows of a
65,536 x 2,048 matrix) with its cluster split-K reduction, the 16-row variants of the
weight-streaming kernel, the tcgen05 route of the down projection, the fused SwiGLU and conv
epilogues at 2,048 channels, the library route above them. Here three-layer cuts (conv, conv,
full attention) of the 1.2B-, 350M- and 2.6B-size configurations run with random bfloat16
weights: by replay (whole, tail decoded, portions, mixed) against the float64 plain
implementation, and through ``LLM.generate`` with captured graphs at live batches of 1 to 64
with every route counted.

What can be asked of bfloat16 here. With random weights the 65,536 logits of a row are close to
independent normal values whose best two lie about 0.2 sigma apart on average, so a few rows in
a hundred are near ties that 16-bit rounding decides the other way. The reference's bar for its
own engine on a real checkpoint is an argmax agreement of 0.97 and no gap over 0.15 nats
(Tokenomos tests/core/test_engine.py:98-102). Measured on a B200 over 150 rows per width and
way of cutting: agreement 0.96 to 0.98, the worst chosen token 0.03 nats below the best, every
row whose best two oracle logits are further apart than 0.15 nats agreed; errors of 1.1 to 1.7 %
of the largest logit against the oracle (the largest of 65,536 errors of a row), 1.0 to 1.7 %
between two ways of cutting (a step of a few decoded tokens and a prompt portion round at
different places, see tests/test_replay.py). The test holds the gap to 0.08 nats, the agreement
to 0.94 over all rows and to 1.0 over the clear ones, and the 32-bit path to full agreement.
"""

from __future__ import annotations

import pytest
import torch

import plain_lfm3
import trace_util

pytestmark = pytest.mark.gpu

BASE = {
    "architectures": ["Lfm3ForCausalLM"], "num_hidden_layers": 3,
    "layer_types": ["conv", "conv", "full_attention"], "num_key_value_heads": 8, "head_dim": 64,
    "vocab_size": 65536, "rope_theta": 1000000.0, "norm_eps": 1e-5, "conv_L_cache": 3,
    "conv_bias": False, "tie_embedding": True,
}
WIDTHS = {
    # the cut of the 1.2B-size benchmark configuration, with the per-head output gate its folder has
    "1.2B": dict(BASE, hidden_size=2048, num_attention_heads=32, intermediate_size=8192, attention_gate=True),
    "350M": dict(BASE, hidden_size=1024, num_attention_heads=16, intermediate_size=4608),
    "2.6B": dict(BASE, hidden_size=2048, num_attention_heads=32, intermediate_size=10752),
}
PAGE = 16
# relative to the largest |logit| of the request; measured on a B200: 32-bit 5e-7 to 8e-7,
# bfloat16 1.0 to 1.5 %; between two ways of cutting 6e-7 to 1.1e-6 (32-bit, whose sums' order follows the
# rows of a step) and 1.0 to 1.7 %
TOL = {"float32": 2e-5, "bfloat16": 2.5e-2}
TOL_SAME = {"float32": 1e-5, "bfloat16": 2.5e-2}
GAP_NATS = 0.08
CLEAR_NATS = 0.15


@pytest.fixture(scope="module")
def real_folders(tmp_path_factory):
    import bench

    out = {}
    for name, config in WIDTHS.items():
        folder = tmp_path_factory.mktemp(f"real_{name.replace('.', 'p')}")
        bench.write_folder(folder, 3, config)
        out[name] = folder
    return out


def requests_for(vocab: int) -> dict[str, list[int]]:
    g = torch.Generator().manual_seed(77)
    return {f"r{i}": torch.randint(0, vocab, (n,), generator=g).tolist() for i, n in enumerate((64, 5, 33, 48))}


_oracles: dict = {}


def oracle(name: str, folder) -> dict[str, torch.Tensor]:
    if name not in _oracles:
        config, w = plain_lfm3.read_folder(folder)
        _oracles[name] = {rid: plain_lfm3.forward_logits(config, w, ids)
                          for rid, ids in requests_for(config["vocab_size"]).items()}
    return _oracles[name]


def judge(got: torch.Tensor, want: torch.Tensor, dtype: str, what: str) -> tuple[int, int, int, int]:
    """Rows of logits against the oracle's: the relative error and the gap bound are asserted;
    returns (rows whose argmax agrees, rows, the same among the clear rows, clear rows)."""
    assert torch.isfinite(got).all(), what
    scale = want.abs().max().item()
    err = (got - want).abs().amax(dim=1)
    bad = (err > TOL[dtype] * scale).nonzero()
    assert bad.numel() == 0, (f"{what}: first wrong row {int(bad[0])} of {len(err)}: error "
                              f"{err[int(bad[0])].item():.3e}, allowed {TOL[dtype] * scale:.3e}")
    logp = torch.log_softmax(want, dim=-1)
    chosen = got.argmax(dim=-1)
    gaps = logp.max(dim=-1).values - logp.gather(1, chosen[:, None])[:, 0]
    assert gaps.max().item() <= GAP_NATS, f"{what}: a chosen token lies {gaps.max().item():.3f} nats below the best"
    top2 = want.topk(2, dim=-1).values
    clear = (top2[:, 0] - top2[:, 1]) > CLEAR_NATS
    agree = chosen == want.argmax(dim=-1)
    return int(agree.sum()), len(agree), int(agree[clear].sum()), int(clear.sum())


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", list(WIDTHS))
def test_replay_at_real_widths(name, dtype, real_folders):
    from tokenomos_b200 import ops

    folder = real_folders[name]
    reqs = requests_for(WIDTHS[name]["vocab_size"])
    want = oracle(name, folder)
    results = {}
    modes = (("whole", trace_util.whole(reqs)), ("tail", trace_util.tail_decoded(reqs, 32)),
             ("portions", trace_util.portions(reqs)), ("mixed", trace_util.mixed(reqs, live=4, seed=3)))
    for mode, steps in modes:
        per_step = trace_util.run_in_process(folder, dtype, steps, trace_util.max_live_tokens(steps, PAGE), PAGE)
        got = trace_util.collect(steps, per_step)
        counts = [judge(got[rid], ref, dtype, f"{name} {dtype} {mode} {rid}") for rid, ref in want.items()]
        agree, rows, clear_agree, clear = (sum(c[i] for c in counts) for i in range(4))
        assert agree >= (rows if dtype == "float32" else 0.94 * rows), (name, dtype, mode, agree, rows)
        assert clear_agree == clear and clear > 0, (name, dtype, mode, clear_agree, clear)
        results[mode] = got
    assert ops.gemm_tc_status() == 0 and ops.attention_prefill_tc_status() == 0
    # two ways of cutting agree far closer than either does with the oracle
    same = TOL_SAME[dtype]
    for mode in results:
        for rid, ref in want.items():
            diff = (results[mode][rid] - results["whole"][rid]).abs().max().item()
            assert diff <= same * ref.abs().max().item(), (name, dtype, mode, rid, diff)


def test_portions_behind_a_long_context_at_real_widths(real_folders):
    """The 1.2B-width cut on a 2,500-token request: whole in one step (512 attention CTAs, none
    shares its keys) against portions of 96 and 32 tokens (three tiles or one, whose keys up to
    16 CTAs share), last logits of every portion, in bfloat16; and the portions in 32-bit against
    the same in bfloat16 within the bound the two paths have against the oracle."""
    from tokenomos_b200 import ops

    folder = real_folders["1.2B"]
    g = torch.Generator().manual_seed(3)
    ids = torch.randint(0, WIDTHS["1.2B"]["vocab_size"], (2500,), generator=g).tolist()
    cuts, a = [], 0
    while a < len(ids):
        b = min(len(ids), a + (96 if len(cuts) % 2 == 0 else 32))
        cuts.append((a, b))
        a = b
    portions = [{"step": i, "entries": [{"id": "r", "tokens": ids[a:b], "want": [b - a - 1]}],
                 "end": ["r"] if b == len(ids) else []} for i, (a, b) in enumerate(cuts)]
    whole = [{"step": 0, "entries": [{"id": "r", "tokens": ids, "want": [b - 1 for _, b in cuts]}], "end": ["r"]}]

    def run(steps, dtype):
        per_step = trace_util.run_in_process(folder, dtype, steps, trace_util.max_live_tokens(steps, PAGE), PAGE)
        return trace_util.collect(steps, per_step)["r"]

    one, cut = run(whole, "bfloat16"), run(portions, "bfloat16")
    assert ops.attention_prefill_tc_status() == 0 and ops.gemm_tc_status() == 0
    scale = one.abs().max().item()
    assert (one - cut).abs().max().item() <= TOL_SAME["bfloat16"] * scale
    exact = run(portions, "float32")
    assert (exact - cut).abs().max().item() <= TOL["bfloat16"] * exact.abs().max().item()
    agree = (exact.argmax(-1) == cut.argmax(-1)).float().mean().item()
    assert agree >= 0.9, agree


def _count_routes(model) -> dict[str, int]:
    """How many products each route of every ``Linear`` of the model took so far, by matrix shape,
    plus which form the feed-forward and the conv mixer took."""
    from tokenomos_b200.parts.linear import Linear

    total: dict[str, int] = {}
    seen = set()
    for block in model.blocks:
        for part in (block.mixer, block.ffn):
            for lin in vars(part).values():
                if isinstance(lin, Linear) and id(lin) not in seen:
                    seen.add(id(lin))
                    for route, n in lin.routed.items():
                        key = f"{route} {lin.out_features}x{lin.in_features}"
                        total[key] = total.get(key, 0) + n
    for route, n in model.head.routed.items():
        total[f"{route} head"] = total.get(f"{route} head", 0) + n
    return total


def test_every_route_at_real_widths_through_generate(real_folders, monkeypatch):
    """``LLM.generate`` with captured graphs on the 1.2B-width cut at live batches of 1, 4, 5, 8,
    9, 16, 17, 40 and 64: every branch of ``Linear.route``, both forms of the feed-forward (gate/up
    with the activation in one kernel, or the product and the activation kernel) and both forms
    of the conv mixer (conv in the in-projection's epilogue, or projection and conv kernel) must
    have run, the tcgen05 kernels' error words stay clear, and every generated token is held,
    teacher-forced, to the engine's own 32-bit path (for the smallest batch also to the float64
    plain implementation)."""
    from tokenomos_b200 import LLM, SamplingParams, models, ops
    from tokenomos_b200.cache.manager import CacheManager
    from tokenomos_b200.engine.step import StepEntry, StepFunction

    folder = real_folders["1.2B"]
    vocab = WIDTHS["1.2B"]["vocab_size"]
    forms = {"swiglu fused": 0, "swiglu unfused": 0, "conv fused": 0, "conv unfused": 0}
    real_skinny, real_swiglu = ops.gemm_skinny, ops.swiglu
    real_skinny_conv, real_conv = ops.gemm_skinny_conv, ops.conv_gated

    def counted(key, fn, when=lambda *a, **k: True):
        def call(*a, **k):
            if when(*a, **k):
                forms[key] += 1
            return fn(*a, **k)
        return call

    monkeypatch.setattr(ops, "gemm_skinny", counted("swiglu fused", real_skinny, lambda *a, **k: k.get("swiglu", False)))
    monkeypatch.setattr(ops, "swiglu", counted("swiglu unfused", real_swiglu))
    monkeypatch.setattr(ops, "gemm_skinny_conv", counted("conv fused", real_skinny_conv))
    monkeypatch.setattr(ops, "conv_gated", counted("conv unfused", real_conv))

    g = torch.Generator().manual_seed(8)
    new = 6
    replies = {}
    with LLM(str(folder), work="bf16", page=PAGE, max_len=64, slots=64, pages=64 * 4 + 2,
             prefill_budget=256, graphs=True, poison=True) as llm:
        llm.engine.step_fn.capture_after = 0
        for batch in (1, 4, 5, 8, 9, 16, 17, 40, 64):
            prompts = [torch.randint(0, vocab, (3 + (7 * i + batch) % 9,), generator=g).tolist()
                       for i in range(batch)]
            outs = llm.generate(prompts, SamplingParams(max_tokens=new))
            replies[batch] = [(p, o.token_ids) for p, o in zip(prompts, outs)]
            assert all(len(o.token_ids) == new for o in outs)
        routes = _count_routes(llm.model)
        assert llm.engine.stats.decode_steps > 0 and llm.engine.stats.graph_steps > 0
    assert ops.gemm_tc_status() == 0 and ops.attention_prefill_tc_status() == 0
    # up to 8 decoded tokens a block's norms and residual adds run inside its products
    # ("skinny+norm", "skinny+add"); 9 to 16 rows take the plain weight-streaming kernel
    for key in ("skinny head", "tc head", "library head",                            # 1..8 rows, 9..64, more
                "skinny+add 2048x2048", "skinny 2048x2048", "library 2048x2048",     # out / o
                "skinny+norm 3104x2048", "skinny 3104x2048", "library 3104x2048",    # q, k, v, gate
                "skinny+add 2048x8192", "tc 2048x8192", "library 2048x8192",         # down
                "skinny+norm 16384x2048", "library 16384x2048",                      # gate / up
                "skinny+norm 6144x2048", "library 6144x2048"):                       # conv in
        assert routes.get(key, 0) > 0, (key, routes)
    assert all(n > 0 for n in forms.values()), forms

    # teacher forcing against the engine's own 32-bit path, whole sequences, one step each
    conf = models.configure(folder, work="fp32")
    model32 = models.load(folder, "cuda", conf)
    cache = CacheManager(model32.state_specs(), PAGE, 8, 2, conf.work, "cuda", max_len=64)
    step32 = StepFunction(model32, cache)
    worst, agree, total = 0.0, 0, 0
    for batch, pairs in replies.items():
        for prompt, reply in pairs[:6] + pairs[-2:]:
            cache.admit("t")
            ids = prompt + reply
            rows = list(range(len(prompt) - 1, len(ids) - 1))
            logp = torch.log_softmax(step32.run([StepEntry("t", ids, rows)]), dim=-1).cpu()
            cache.release("t")
            for i, tok in enumerate(reply):
                worst = max(worst, (logp[i].max() - logp[i, tok]).item())
                agree += int(logp[i].argmax()) == tok
                total += 1
    assert worst <= CLEAR_NATS, f"a generated token lies {worst:.3f} nats below the 32-bit path's best"
    assert agree / total >= 0.85, (agree, total)
    config, w = plain_lfm3.read_folder(folder)
    for prompt, reply in replies[1] + replies[4][:2]:
        logp = torch.log_softmax(plain_lfm3.forward_logits(config, w, prompt + reply), dim=-1)
        for i, tok in enumerate(reply):
            row = logp[len(prompt) + i - 1]
            assert (row.max() - row[tok]).item() <= CLEAR_NATS

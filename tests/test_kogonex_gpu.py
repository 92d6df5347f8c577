"""Kogonex on the GPU against the plain implementation (``tests/plain/kogonex.py``, float64).

Whole models of several small configurations, replayed whole, with a decoded tail, in portions down to
two tokens, and mixed with other requests in a pool so small that pages and state slots are used
again; every mechanism alone (a one-layer model, or its kernel with inputs made so that one key, a
sink or a window's edge decides the result); long decoding; greedy generation through the public
entry point and the scheduler.

Errors are relative: the root mean square over the vocabulary of the difference of the logits (mean
taken off) over the standard deviation of the plain model's logits.  float32 differs from float64 by
1e-6 .. 1e-5 (summation order); bfloat16 by 5e-3 .. 9e-2 (bfloat16 activations between the products; the
largest at single positions of these small random models where a sublayer's output is small before its norm).
"""

import math

import numpy as np
import pytest
import torch

from acorninfer_b200.config.model_config import (ChannelDeltaConfig, KogonexConfig, KogonexLayer, LatentAttentionConfig,
                                                 RotaryScaling, RoutedExpertsConfig)
from tests import traces
from tests.kogonex_tiny import KOGOS, make_model_dir, read_weights
from tests.paged import rows_layout, scatter_to_pages
from tests.plain import kogonex as plain
from tests.tiny import random_tokens

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = {"float32": 4e-5, "bfloat16": 0.12}
LENGTHS = [45, 38, 61, 50, 33, 29]


def rel_err(got, ref):
    d = np.asarray(got, np.float64) - np.asarray(ref, np.float64)
    d = d - d.mean()
    return math.sqrt((d ** 2).mean()) / float(np.std(ref))


@pytest.fixture(scope="module", params=list(KOGOS))
def case(request, tmp_path_factory):
    tiny = KOGOS[request.param]
    d = make_model_dir(tmp_path_factory.mktemp(request.param), tiny)
    w = read_weights(d)
    reqs = {f"r{i}": random_tokens(n, tiny["cfg"].vocab_size, 3000 + i) for i, n in enumerate(LENGTHS)}
    ref = {rid: plain.forward(tiny["cfg"].to_dict(), w, toks).numpy() for rid, toks in reqs.items()}
    return tiny, d, reqs, ref


@pytest.fixture(scope="module")
def case16(case, tmp_path_factory):
    """The same configuration with corrections that decide the experts alone: what bfloat16 runs are
    compared on (see ``make_model_dir``)."""
    tiny, _, reqs, _ = case
    d = make_model_dir(tmp_path_factory.mktemp("decisive"), tiny, decisive=True)
    w = read_weights(d)
    ref = {rid: plain.forward(tiny["cfg"].to_dict(), w, toks).numpy() for rid, toks in reqs.items()}
    return tiny, d, reqs, ref


def run_cut(tiny, model_dir, steps, dtype, max_requests=4, watch=None):
    from acorninfer_b200.engine.runner import ModelRunner
    from acorninfer_b200.replay import TraceSession

    pool = traces.max_live_tokens(steps)
    runner = ModelRunner.from_model_dir(model_dir, dtype=dtype, num_blocks=-(-pool // tiny["page_size"]),
                                        page_size=tiny["page_size"], max_requests=max_requests, max_step_tokens=4096)
    session = TraceSession(runner)

    def step(msg):
        if watch is None:
            return session.step(msg)
        out = session.step(dict(msg, end=[]))
        watch(session, msg)
        session.step({"entries": [], "end": msg["end"]})
        return out

    got = traces.collect(step, steps)
    runner.manager.assert_balanced()
    return got, runner


def check(got, ref, dtype, what):
    errs = {key: rel_err(row, ref[key[0]][key[1]]) for key, row in got.items()}
    worst = max(errs, key=errs.get)
    assert errs[worst] < TOL[dtype], f"{what}: {worst}: {errs[worst]:.3e}"


CUTS = {
    "whole": traces.whole,
    "decode_tail": lambda r: traces.decode_tail(r, tail=24),
    "portions": lambda r: traces.portions(r, sizes=(7, 2, 5, 3, 16, 2, 11, 4)),
    "mixed": lambda r: traces.mixed(r, max_live=4, seed=3, stagger=2),
}


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("cut", list(CUTS))
def test_cut_matches_plain(case, case16, cut, dtype):
    tiny, d, reqs, ref = case if dtype == "float32" else case16
    got, runner = run_cut(tiny, d, CUTS[cut](reqs), dtype)
    assert len(got) == sum(len(t) for t in reqs.values())
    check(got, ref, dtype, cut)
    if cut == "decode_tail":
        assert runner.graph_replays >= len(reqs) * 10        # single-token steps replay captured graphs


def test_cuts_agree_with_each_other_float32(case):
    """The logits at a position do not depend on how the tokens were cut into steps, on what else was
    in the batch or on which pages and slots held them, beyond rounding."""
    tiny, d, reqs, _ = case
    base, _ = run_cut(tiny, d, traces.whole(reqs), "float32")
    for cut in ("decode_tail", "portions", "mixed"):
        other, _ = run_cut(tiny, d, CUTS[cut](reqs), "float32")
        for key, row in base.items():
            assert rel_err(other[key], row) < 1e-5, f"{cut}: {key}"


def test_mixed_trace_uses_pages_and_slots_again(case):
    tiny, d, reqs, _ = case
    steps = CUTS["mixed"](reqs)
    pages: dict = {}
    slots: dict = {}

    def watch(session, msg):
        for rid, rc in session.live.items():
            slots.setdefault(rc.slot, set()).add(rid)
            for table in rc.tables:
                for page in table:
                    pages.setdefault(page, set()).add(rid)

    run_cut(tiny, d, steps, "float32", watch=watch)
    assert len(slots) <= 4 and sum(1 for users in slots.values() if len(users) >= 2) >= 1, slots
    if pages:
        assert sum(1 for users in pages.values() if len(users) >= 2) >= 2, pages


def test_first_step_of_one_token_and_requests_left_out(case):
    """A request whose first step is a single token (the bigram row of a first token, the convolution's
    zeros before the start, a window that holds one key), then portions beside another request that
    decodes and is left out of some steps."""
    tiny, d, reqs, ref = case
    a, b = reqs["r0"], reqs["r1"]
    steps = [{"entries": [{"id": "r0", "tokens": a[:1], "want": [0]}], "end": []},
             {"entries": [{"id": "r0", "tokens": a[1:3], "want": [0, 1]}, {"id": "r1", "tokens": b[:9], "want": list(range(9))}], "end": []},
             {"entries": [{"id": "r1", "tokens": b[9:10], "want": [0]}], "end": []},
             {"entries": [{"id": "r0", "tokens": a[3:20], "want": list(range(17))}, {"id": "r1", "tokens": b[10:11], "want": [0]}], "end": []},
             {"entries": [{"id": "r0", "tokens": a[20:], "want": list(range(len(a) - 20))}], "end": ["r0"]},
             {"entries": [{"id": "r1", "tokens": b[11:], "want": list(range(len(b) - 11))}], "end": ["r1"]}]
    for i, s in enumerate(steps):
        s["step"] = i
    got, _ = run_cut(tiny, d, steps, "float32")
    check(got, ref, "float32", "first token alone")


def test_long_decoding_float32(case):
    """A short prompt and 170 decoded tokens: windows pass over decoded tokens many times, pages of a
    windowed cache are given back and taken again, the recurrent state is carried all the way."""
    tiny, d, _, _ = case
    toks = random_tokens(190, tiny["cfg"].vocab_size, 77)
    ref = {"long": plain.forward(tiny["cfg"].to_dict(), read_weights(d), toks).numpy()}
    steps = traces.decode_tail({"long": toks}, tail=170)
    got, _ = run_cut(tiny, d, steps, "float32")
    check(got, ref, "float32", "long decoding")


def test_long_requests_wide_windows_over_pages(tmp_path):
    """Requests of a few hundred tokens through windows of 70 and 130 over pages of 16: the tensor-core
    attention walks several blocks of keys whose first and last are cut by the window, the windowed
    group gives pages back while a request is still fed, and the reader of the shared cache looks
    further back than the layer that writes it."""
    from tests.kogonex_tiny import KOGO_LONG
    tiny = KOGO_LONG
    reqs = {f"L{i}": random_tokens(n, tiny["cfg"].vocab_size, 600 + i) for i, n in enumerate([330, 260, 150])}
    cuts = {"whole": traces.whole, "decode_tail": lambda r: traces.decode_tail(r, tail=90),
            "portions": lambda r: traces.portions(r, sizes=(64, 3, 2, 128, 29, 16, 2, 70)),
            "mixed": lambda r: traces.mixed(r, max_live=3, seed=5, max_portion=80, stagger=1)}
    for dtype, decisive in (("float32", False), ("bfloat16", True)):
        d = make_model_dir(tmp_path / dtype, tiny, decisive=decisive)
        w = read_weights(d)
        ref = {rid: plain.forward(tiny["cfg"].to_dict(), w, toks).numpy() for rid, toks in reqs.items()}
        for cut, build in cuts.items():
            got, runner = run_cut(tiny, d, build(reqs), dtype)
            assert len(got) == sum(len(t) for t in reqs.values())
            check(got, ref, dtype, f"long, {cut}")


def follows_plain(cfg, w, prompt, ids, slack):
    logits = plain.forward(cfg.to_dict(), w, ids[:-1])
    return all(float(logits[i - 1].max() - logits[i - 1][ids[i]]) <= slack for i in range(len(prompt), len(ids)))


@pytest.mark.parametrize("dtype,slack", [("float32", 1e-4), ("bfloat16", 0.15)])
def test_greedy_generation_through_the_engine(case, case16, dtype, slack):
    """``generate``: the scheduler with a token budget (prompts cut into portions beside decoding
    requests), sampling on the device, a step ahead of the host."""
    from acorninfer_b200 import generate
    tiny, d, _, _ = case if dtype == "float32" else case16
    cfg = tiny["cfg"]
    w = read_weights(d)
    prompts = [random_tokens(n, cfg.vocab_size, 900 + n) for n in (1, 14, 23, 6, 31)]
    outs = generate(d, prompts, max_new_tokens=12, temperature=0.0, dtype=dtype, page_size=tiny["page_size"],
                    num_blocks=64, max_running=3, chunked_budget=10, watermark_blocks=0, eos_ids=())
    for p, ids in zip(prompts, outs):
        assert len(ids) == len(p) + 12 and follows_plain(cfg, w, p, ids, slack), (dtype, len(p))


def test_preemption_recomputes_state_float32(case):
    """So few pages that requests are preempted and recomputed from their first token: the recurrent
    state and the bigram's previous token start over with the slot."""
    from acorninfer_b200.generation import build_engine, generate_with_engine
    tiny, d, _, _ = case
    cfg = tiny["cfg"]
    prompts = [random_tokens(n, cfg.vocab_size, 40 + n) for n in (20, 18, 13)]
    roomy = build_engine(d, dtype="float32", page_size=tiny["page_size"], num_blocks=64, watermark_blocks=0, max_running=3)
    want = generate_with_engine(roomy, prompts, max_new_tokens=16, eos_ids=())
    pages = -(-36 // tiny["page_size"]) * 2 + 1
    tight = build_engine(d, dtype="float32", page_size=tiny["page_size"], num_blocks=pages, watermark_blocks=0, max_running=3)
    got = generate_with_engine(tight, prompts, max_new_tokens=16, eos_ids=())
    w = read_weights(d)
    for p, a, b in zip(prompts, got, want):
        assert follows_plain(cfg, w, p, a, 1e-4) and follows_plain(cfg, w, p, b, 1e-4)


# ------------------------------------------------------------------ one mechanism at a time


def _solo(mixer, mlp=None, width=48, vocab=90, bigram=False):
    return KogonexConfig(vocab_size=vocab, hidden_size=width, norm_eps=1e-5, layers=(KogonexLayer(mixer, mlp),),
                         bigram_buckets=13 if bigram else None, bigram_mul_prev=9 if bigram else 0,
                         bigram_mul_cur=4 if bigram else 0)


_TINY_DELTA = ChannelDeltaConfig(heads=1, kv_heads=1, dim=4, vdim=4, conv=1, decay_rank=2, gate_rank=2)
SOLOS = {
    "delta rule, grouped heads, 4 taps": _solo(ChannelDeltaConfig(heads=6, kv_heads=2, dim=10, vdim=28, conv=4, decay_rank=3, gate_rank=5)),
    "delta rule, heads of 72 key channels": _solo(ChannelDeltaConfig(heads=1, kv_heads=1, dim=72, vdim=8, conv=2, decay_rank=4, gate_rank=4)),
    "delta rule, heads of 136 key channels": _solo(ChannelDeltaConfig(heads=2, kv_heads=1, dim=136, vdim=20, conv=3, decay_rank=4, gate_rank=4)),
    "latent attention, window 5, scaled positions": _solo(LatentAttentionConfig(
        heads=3, dim=8, rot_dim=6, vdim=10, kv_rank=12, scale=0.4, rot_dims=6, rot_base=100.0,
        scaling=RotaryScaling(3.0, 8, 2.0, 0.5), window=5)),
    "latent attention, no window, no rotated part": _solo(LatentAttentionConfig(
        heads=2, dim=16, rot_dim=0, vdim=8, kv_rank=24, scale=0.3, rot_dims=0, rot_base=1e4, window=None)),
    "experts in groups with identity experts": _solo(_TINY_DELTA, RoutedExpertsConfig(ff=20, experts=9, identity=3, top=4, groups=6, keep=3)),
    "one expert of one": _solo(_TINY_DELTA, RoutedExpertsConfig(ff=12, experts=1, identity=0, top=1)),
    "identity experts only": _solo(_TINY_DELTA, RoutedExpertsConfig(ff=12, experts=0, identity=4, top=2, groups=2, keep=2)),
    "bigram rows": _solo(_TINY_DELTA, None, bigram=True),
}


@pytest.mark.parametrize("name", list(SOLOS))
def test_mechanism_alone(name, tmp_path):
    tiny = dict(cfg=SOLOS[name], page_size=4, seed=5)
    d = make_model_dir(tmp_path, tiny, sigma=0.3)
    w = read_weights(d)
    reqs = {f"s{i}": random_tokens(n, tiny["cfg"].vocab_size, 50 + i) for i, n in enumerate([26, 17, 9])}
    ref = {rid: plain.forward(tiny["cfg"].to_dict(), w, toks).numpy() for rid, toks in reqs.items()}
    for cut in ("whole", "portions", "mixed"):
        got, _ = run_cut(tiny, d, CUTS[cut](reqs) if cut != "portions" else traces.portions(reqs, sizes=(3, 2, 6, 2)), "float32")
        check(got, ref, "float32", f"{name}, {cut}")


def ops():
    from acorninfer_b200.kernels import ops as o
    return o


@pytest.mark.parametrize("N,top,groups,keep", [(16, 3, 2, 1), (12, 2, 4, 2), (7, 7, 1, 1), (64, 6, 8, 3), (33, 1, 3, 3), (5, 2, 5, 2)])
def test_router_choice_matches_plain(N, top, groups, keep):
    g = torch.Generator().manual_seed(N * 100 + top)
    z = torch.randn(200, N, generator=g) * 2
    corr = torch.randn(N, generator=g) * 0.05
    idx, wts = ops().moe_route(z.to(DEV), corr.to(DEV), top, groups, keep)
    idx, wts = idx.cpu(), wts.cpu()
    r = {"top": top, "groups": {"count": groups, "keep": keep}}
    for t in range(z.shape[0]):
        want = plain.route(r, z[t].double(), corr.double())
        assert [e for e, _ in want] == idx[t].tolist(), t
        assert max(abs(float(a) - float(b)) for (_, a), b in zip(want, wts[t])) < 1e-6


@pytest.mark.parametrize("N,K,scaled,limit", [(128, 64, False, 0.0), (600, 136, True, 0.0), (520, 1032, False, 7.0), (34, 72, True, 3.0)])
@pytest.mark.parametrize("tcgen05", [True, False])
def test_grouped_products_of_many_rows(N, K, scaled, limit, tcgen05, monkeypatch):
    """The paired tcgen05 kernel (tiles of 256 rows) and the mma.sync one: experts with no row, one row, a tile
    and a row more, hundreds; widths that fill no tile; factors by slot and the capped form in the epilogue.  Inputs are
    bfloat16 numbers, sums float32, one rounding to bfloat16: 2^-8 of the result and float32 sums' 2e-5 of the operands'
    norms."""
    o = ops()
    monkeypatch.setattr(o, "GROUPED_TCGEN05_MIN_ROWS", 1 if tcgen05 else 10 ** 9)
    counts = [0, 1, 256, 257, 0, 130, 515, 3, 128]
    E, slots = len(counts), sum(counts) + 9                     # nine rows of no expert at the end
    g = torch.Generator().manual_seed(N)
    rows = torch.randint(0, 700, (slots,), generator=g, dtype=torch.int32).to(DEV)
    x = torch.randn(700, K, generator=g).bfloat16().to(DEV)
    w = (torch.randn(E, N, K, generator=g) / K ** 0.5).bfloat16().to(DEV)
    scale = (torch.rand(slots, generator=g) + 0.5).to(DEV) if scaled else None
    offsets = torch.tensor([sum(counts[:e]) for e in range(E + 1)] + [slots], dtype=torch.int32, device=DEV)
    for act in (False, True):
        out = o.grouped_gemm(x, rows, w, offsets, slots, swiglu_pairs=act, slot_scale=scale,
                             **(dict(activation="capped_swish", limit=limit) if act and limit else {}))
        for e in range(E):
            a, b = sum(counts[:e]), sum(counts[:e + 1])
            want = x[rows[a:b].long()].double() @ w[e].double().T
            if scaled:
                want = want * scale[a:b, None].double()
            if act:
                gate, up = want[:, 0::2], want[:, 1::2]
                if limit:
                    gate, up = gate.clamp(max=limit), up.clamp(-limit, limit) + 1.0
                want = gate * torch.sigmoid((1.702 if limit else 1.0) * gate) * up
            got = out[a:b].double()
            assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 2e-4).all(), (e, act)
    assert o.lib().acorn_gemm_tc_pair_error() == 0


def test_grouped_products_of_many_experts(monkeypatch):
    """More experts than one launch of the tcgen05 kernel knows (512): uneven shares, some empty, at and around that one."""
    o = ops()
    E, N, K = 1100, 40, 24
    g = torch.Generator().manual_seed(0)
    counts = torch.randint(0, 200, (E,), generator=g)
    counts[[0, 511, 600, E - 1]], counts[[510, 512, 513, 1023, 1024]] = 0, torch.tensor([257, 300, 1, 5, 64])
    slots = 64 * E
    counts[700] += max(0, slots - int(counts.sum()))
    slots = int(counts.sum())
    offsets = torch.cat([torch.zeros(1, dtype=torch.int64), counts.cumsum(0)]).int().to(DEV)
    x, w = torch.randn(slots, K, generator=g).bfloat16().to(DEV), (torch.randn(E, N, K, generator=g) * K ** -0.5).bfloat16().to(DEV)
    monkeypatch.setattr(o.lib(), "acorn_grouped_gemm", lambda *a: 10001)                # the other kernel, for fewer rows an expert
    out = o.grouped_gemm(x, None, w, offsets, slots)
    off = offsets.tolist()
    for e in range(E):
        want = x[off[e]:off[e + 1]].double() @ w[e].double().T
        assert ((out[off[e]:off[e + 1]].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-4).all(), e      # as above
    assert o.lib().acorn_gemm_tc_pair_error() == 0


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-4), (torch.bfloat16, 0.15)])
@pytest.mark.parametrize("E,T,top,min_rows", [(7, 90, 2, None), (2, 300, 2, None), (12, 5, 2, None), (3, 400, 2, 10 ** 9)])
def test_grouped_products_take_each_experts_own_rows(dtype, tol, E, T, top, min_rows, monkeypatch):
    """Rows scattered over experts, some experts with no rows and some with more than a tile: every
    row against its own expert's matrix.  In bfloat16 the second shape has enough rows an expert for the
    tcgen05 kernel (tiles of 256 rows, an expert's last tile partly another's rows); the others, and the
    last with that kernel switched off, take the three tile heights of the mma.sync kernel (64, 16, 128)."""
    o = ops()
    if min_rows is not None:
        monkeypatch.setattr(o, "GROUPED_TCGEN05_MIN_ROWS", min_rows)
    g = torch.Generator().manual_seed(2)
    N, K = 50, 40
    idx = torch.randint(0, E + 2, (T, top), generator=g, dtype=torch.int32)       # two more outputs: identity experts
    idx[idx == 1] = 0                                                              # expert 1 gets nothing
    x = torch.randn(T, K, generator=g).to(dtype)
    w = torch.randn(E, N, K, generator=g).to(dtype)
    offsets, slot_of, slot_token = o.moe_plan(idx.to(DEV), E + 2)
    out = o.grouped_gemm(x.to(DEV), slot_token, w.to(DEV), offsets, T * top).float().cpu()
    off = offsets.cpu().tolist()
    assert off[-1] == T * top and off[2] == off[1]
    so = slot_of.cpu()
    for t in range(T):
        for k in range(top):
            e, s = int(idx[t, k]), int(so[t, k])
            assert off[e] <= s < off[e + 1]
            if e < E:
                assert (out[s] - x[t].float() @ w[e].float().T).abs().max() < tol
    # gate and up rows in turns: silu(gate) * up from the product's own epilogue (bfloat16) or the kernel after it
    act = o.grouped_gemm(x.to(DEV), slot_token, w.to(DEV), offsets, T * top, swiglu_pairs=True).float().cpu()
    assert act.shape == (T * top, N // 2)
    for t in range(0, T, 7):
        e, s = int(idx[t, 0]), int(so[t, 0])
        if e < E:
            gu = x[t].float() @ w[e].float().T
            want = torch.nn.functional.silu(gu[0::2]) * gu[1::2]
            assert (act[s] - want).abs().max() < tol * 4, (t, e)


def _latent_case(befores, qlens, P, d, dv, nq, window, spikes, dtype, sink_value=None, seed=0, kernel="plain"):
    """Cache rows and queries for ``attention_plain`` in the latent layout (one kv head, values = the
    first dv entries of the key rows).  ``spikes``: (row, key position): that key and all queries of the
    row get a large component along one direction, so its score stands out wherever it is seen."""
    g = torch.Generator().manual_seed(seed)
    NP = sum(-(-(b + q) // P) for b, q in zip(befores, qlens)) + 5
    lay = rows_layout(befores, qlens, P, NP, seed=seed)
    pages = torch.zeros(NP, 1, P, d, dtype=dtype, device=DEV)
    full_q, full_k = [], []
    for r, (b, q) in enumerate(zip(befores, qlens)):
        S = b + q
        k = torch.randn(S, 1, d, generator=g) * 0.3
        qq = torch.randn(S, nq, d, generator=g) * 0.3
        for (rr, j) in spikes:
            if rr == r:
                k[j, 0, d - 1] = 6.0
                qq[:, :, d - 1] = 4.0
        k = k.to(dtype).double()
        qq = qq.to(dtype).double()
        scatter_to_pages(pages, lay["tables"][r], k.to(dtype), P)
        full_q.append(qq)
        full_k.append(k)
    q_new = torch.cat([fq[b:] for fq, b in zip(full_q, befores)]).to(dtype).to(DEV).contiguous()
    sink = None if sink_value is None else torch.full((nq,), float(sink_value)) + torch.arange(nq) * 0.5
    scale = 0.5
    if kernel == "tc":
        o = ops()
        assert o.latent_attention_tc_supported(dtype, nq, d, dv, P)
        n = o.LATENT_TILE_ROWS // nq
        i32 = dict(dtype=torch.int32, device=DEV)
        tiles = torch.tensor([(r, q0) for r, length in enumerate(qlens) for q0 in range(0, length, n)], **i32)
        args = (q_new, pages, lay["block_table"], lay["page_base"], torch.tensor(np.cumsum([0] + qlens), **i32),
                torch.tensor(befores, **i32), tiles, None if sink is None else sink.to(DEV), scale, window, dv)
        out = o.latent_attention_tc(*args).float().cpu()
        for splits in (1, 3, 7):              # a tile's key blocks shared out over several blocks and merged
            again = o.latent_attention_tc(*args, splits=splits).float().cpu()
            assert (again - out).abs().max() < 2e-2, splits
    else:
        out = ops().attention_plain(q_new.view(-1, nq * d), nq * d, pages, pages, lay["block_table"], lay["page_base"],
                                    lay["token_row"], lay["positions"], lay["num_tokens"], nq, 1, d, scale, window,
                                    value_dim=dv, sink32=None if sink is None else sink.to(DEV)).float().cpu()
    want = []
    for fq, fk, b in zip(full_q, full_k, befores):
        heads = []
        for h in range(nq):
            s = fq[:, h] @ fk[:, 0].T * scale
            p = plain.windowed_sink_softmax(s, torch.tensor(-1e30, dtype=torch.float64) if sink is None else sink[h].double(), window)
            heads.append(p @ fk[:, 0, :dv])
        want.append(torch.stack(heads, 1)[b:])
    return out.view(-1, nq, dv), torch.cat(want)


@pytest.mark.parametrize("dtype,tol,kernel,d,dv,nq", [(torch.float32, 2e-5, "plain", 24, 16, 3), (torch.bfloat16, 2e-2, "plain", 24, 16, 3),
                                                      (torch.bfloat16, 2e-2, "tc", 32, 16, 3), (torch.bfloat16, 2e-2, "tc", 112, 96, 8),
                                                      (torch.bfloat16, 2e-2, "tc", 160, 144, 16)])
def test_latent_layout_attention_window_edges_far_keys_and_sink(dtype, tol, kernel, d, dv, nq):
    """A key that outweighs all others is seen up to the query window - 1 tokens after it and no
    longer, in a prompt's rows and in single decoded tokens, at page borders; a far key among hundreds
    is found without a window; a sink takes its share of every row."""
    P, W = 16, 64
    # row 0: a whole prompt; row 1: a portion after 130 cached tokens; rows 2-5: single tokens whose
    # window's first key (2, 4) or the key just before it (3, 5) is the spiked one, at a page's border or not
    befores = [0, 130, 15 + W - 1, 15 + W, 16 + W - 1, 16 + W]
    qlens = [300, 90, 1, 1, 1, 1]
    spikes = [(0, 15), (0, 16), (0, 200), (1, 100), (1, 131), (2, 15), (3, 15), (4, 16), (5, 16)]
    got, want = _latent_case(befores, qlens, P, d, dv, nq, W, spikes, dtype, sink_value=0.5, kernel=kernel)
    assert (got - want).abs().max() < tol
    # the spiked key decides the rows that see it: the decoded token of row 2 returns (nearly) its
    # value, the one of row 3, one position later, does not
    lay_tokens = np.cumsum([0] + qlens)
    assert (got[lay_tokens[2]] - got[lay_tokens[3]]).abs().max() > 0.05
    # no window: key 3 of 700 decides a decoded token's result
    got, want = _latent_case([0, 699], [40, 1], P, d, dv, nq, None, [(1, 3)], dtype, kernel=kernel)
    assert (got - want).abs().max() < tol
    # a sink that outweighs the keys leaves almost nothing
    got, want = _latent_case([5], [20], P, d, dv, nq, 8, [], dtype, sink_value=12.0, kernel=kernel)
    assert (got - want).abs().max() < tol and got.abs().max() < 0.05


@pytest.mark.parametrize("H,d,dv,P,window,sink", [(16, 448, 384, 16, 200, True), (8, 320, 192, 8, None, False), (5, 192, 128, 128, 70, True),
                                                  (64, 64, 64, 32, None, True), (1, 128, 64, 16, 64, False)])
def test_latent_attention_of_long_rows(H, d, dv, P, window, sink):
    """The tcgen05 kernel against float64: rows that end anywhere in a tile and in a block of 64 keys, single tokens,
    portions after cached keys, pages a window has given back, and pages that hold no numbers behind the last key."""
    o = ops()
    befores, qlens = [0, 130, 63, 300, 127], [333, 64, 1, 65, 193]
    NP = sum(-(-(b + q) // P) for b, q in zip(befores, qlens)) + 3
    lay = rows_layout(befores, qlens, P, NP, seed=H)
    g = torch.Generator().manual_seed(d)
    pages = torch.full((NP, 1, P, d), float("nan"), dtype=torch.bfloat16, device=DEV)
    sinks = torch.randn(H, generator=g) if sink else None
    scale, q_new, want = d ** -0.5, [], []
    table, base = lay["block_table"].clone(), lay["page_base"].clone()
    for r, (b, n) in enumerate(zip(befores, qlens)):
        k = (torch.randn(b + n, d, generator=g) * 1.5).bfloat16()
        q = (torch.randn(n, H, d, generator=g) * 1.5).bfloat16()
        gone = max(0, b - window + 1) // P if window else 0              # pages no query sees any more
        scatter_to_pages(pages, lay["tables"][r], k[:, None], P)
        for page in lay["tables"][r][:gone]:
            pages[page] = float("nan")
        table[r] = torch.roll(lay["block_table"][r], -gone)
        base[r] = gone
        q_new.append(q)
        i, j = torch.arange(b, b + n)[:, None], torch.arange(b + n)[None]
        seen = (j <= i) & (i - j < window) if window else j <= i
        s = torch.einsum("qhd,kd->hqk", q.double(), k.double()) * scale
        s = s.masked_fill(~seen, float("-inf"))
        if sink:
            s = torch.cat([s, sinks.double()[:, None, None].expand(H, n, 1)], 2)
        w = torch.softmax(s, 2)[:, :, :b + n]
        want.append(torch.einsum("hqk,kd->qhd", w, k[:, :dv].double()))
    q_new, want = torch.cat(q_new).to(DEV), torch.cat(want)
    i32 = dict(dtype=torch.int32, device=DEV)
    assert o.latent_prefill_tc_supported(torch.bfloat16, H, d, dv, P, scale)
    got = o.latent_prefill_tc(q_new, pages, table, base, torch.tensor(np.cumsum([0] + qlens), **i32), torch.tensor(befores, **i32),
                              o.latent_prefill_tiles(qlens, H), sinks.to(DEV) if sink else None, scale, window, dv).double().cpu()
    o.raise_on_kernel_error()
    # the weights and the result are rounded to 8 bits of mantissa (half a unit: 2^-9 each), a weighted mean of values up to
    # `top`; float32 scores of a few units add less than 2^-13
    top = 1.5 * 6
    assert (got - want).abs().max() < top * (2 ** -9 + 2 ** -9 + 2 ** -13)


@pytest.mark.parametrize("H,d,dv", [(32, 192, 128), (64, 448, 384), (128, 64, 64)])
def test_latent_attention_scores_that_outgrow_late(H, d, dv):
    """Rows of one tile and of one to seven blocks of 64 keys, the scores of one warp's rows (32 of the tile's 128) raised far
    beyond all before by a key of the second-to-last or of the last block: its rows rescale while the others run ahead."""
    o = ops()
    P, TQ = 16, 128 // H
    cases = [(nb, nb - 1 - back, warp) for nb in range(1, 8) for back in (0, 1) if back < nb for warp in range(4)]
    befores = [64 * nb - TQ - 3 * (i % 3) for i, (nb, _, _) in enumerate(cases)]
    NP = sum(-(-(b + TQ) // P) for b in befores) + 3
    lay = rows_layout(befores, [TQ] * len(cases), P, NP, seed=H)
    g = torch.Generator().manual_seed(d)
    pages = torch.full((NP, 1, P, d), float("nan"), dtype=torch.bfloat16, device=DEV)
    scale, q_new, want = d ** -0.5, [], []
    for r, (b, (nb, block, warp)) in enumerate(zip(befores, cases)):
        k = torch.randn(b + TQ, d, generator=g).bfloat16()
        q = torch.randn(TQ * H, d, generator=g).bfloat16()
        k[:, 0], q[:, 0] = 0, 0
        k[64 * block + 5, 0], q[32 * warp:32 * warp + 32, 0] = 8, 4 * math.sqrt(d)   # 32 in the score's units, 46 to base 2
        q = q.view(TQ, H, d)
        scatter_to_pages(pages, lay["tables"][r], k[:, None], P)
        q_new.append(q)
        seen = torch.arange(b + TQ)[None] <= torch.arange(b, b + TQ)[:, None]
        s = (torch.einsum("qhd,kd->hqk", q.double(), k.double()) * scale).masked_fill(~seen, float("-inf"))
        want.append(torch.einsum("hqk,kd->qhd", torch.softmax(s, 2), k[:, :dv].double()))
    i32 = dict(dtype=torch.int32, device=DEV)
    lens = [TQ] * len(cases)
    for _ in range(20):                 # a hand-over that comes too early need not show every time
        got = o.latent_prefill_tc(torch.cat(q_new).to(DEV), pages, lay["block_table"], lay["page_base"],
                                  torch.tensor(np.cumsum([0] + lens), **i32), torch.tensor(befores, **i32),
                                  o.latent_prefill_tiles(lens, H), None, scale, None, dv).double().cpu()
        o.raise_on_kernel_error()
        # weights and results rounded to 8 bits of mantissa as above; values up to 8; float32 scores up to 40, 2^-18 of error
        assert (got - torch.cat(want)).abs().max() < 8 * (2 ** -9 + 2 ** -9 + 2 ** -13)


@pytest.mark.parametrize("P,window", [(16, 4), (8, 1), (32, 9), (64, 20), (128, 70)])
def test_latent_attention_reads_no_rows_but_its_own(P, window):
    """Windows smaller than a page and than a block of 64 keys: what lies in the pages behind the request's last token, in
    those given back, and in the request's own rows in front of a window, is NaN and stays out."""
    o = ops()
    H, d, dv = 16, 192, 128
    befores, qlens = [100, 3, 70, 97, 250, 0, 120], [1, 2, 3, 1, 5, 40, 30]
    NP = sum(-(-(b + q) // P) for b, q in zip(befores, qlens)) + 3
    lay = rows_layout(befores, qlens, P, NP, seed=P)
    g = torch.Generator().manual_seed(P)
    pages = torch.full((NP, 1, P, d), float("nan"), dtype=torch.bfloat16, device=DEV)
    table, base = lay["block_table"].clone(), lay["page_base"].clone()
    scale, q_new, want = d ** -0.5, [], []
    for r, (b, n) in enumerate(zip(befores, qlens)):
        k, q = torch.randn(b + n, d, generator=g).bfloat16(), torch.randn(n, H, d, generator=g).bfloat16()
        k[:max(0, b - window + 1)] = float("nan")                        # rows that no query of the step reads
        scatter_to_pages(pages, lay["tables"][r], k[:, None], P)
        gone = max(0, b - window + 1) // P
        table[r], base[r] = torch.roll(lay["block_table"][r], -gone), gone
        q_new.append(q)
        for i in range(n):
            kd = k[max(0, b + i - window + 1):b + i + 1].double()
            want.append(torch.softmax(q[i].double() @ kd.T * scale, 1) @ kd[:, :dv])
    i32 = dict(dtype=torch.int32, device=DEV)
    got = o.latent_prefill_tc(torch.cat(q_new).to(DEV), pages, table, base, torch.tensor(np.cumsum([0] + qlens), **i32),
                              torch.tensor(befores, **i32), o.latent_prefill_tiles(qlens, H), None, scale, window, dv).double().cpu()
    o.raise_on_kernel_error()
    assert (got - torch.stack(want)).abs().max() < 6 * (2 ** -9 + 2 ** -9 + 2 ** -13)       # as for long rows; values up to 6


@pytest.mark.parametrize("H,d,dv,P,window", [(16, 192, 128, 16, None), (16, 448, 384, 16, 70), (1, 128, 64, 8, 100), (5, 192, 128, 64, 3), (128, 64, 64, 16, None)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_latent_attention_keeps_what_is_no_number_to_the_queries_that_read_it(H, d, dv, P, window, value):
    """An infinite value or one that is no number, at tokens anywhere in a tile and a block of 64 keys: queries that read the
    token are what float64 makes of it, the others untouched."""
    o = ops()
    befores, qlens, bad = [0, 130, 61, 10, 200], [150, 64, 9, 1, 70], [[37, 101], [131], [62, 66], [10], [150, 203]]
    NP = sum(-(-(b + q) // P) for b, q in zip(befores, qlens)) + 3
    lay = rows_layout(befores, qlens, P, NP, seed=P)
    g = torch.Generator().manual_seed(P)
    pages = torch.full((NP, 1, P, d), float("nan"), dtype=torch.bfloat16, device=DEV)
    scale, q_new, want = d ** -0.5, [], []
    for r, (b, n) in enumerate(zip(befores, qlens)):
        k, q = torch.randn(b + n, d, generator=g).bfloat16(), torch.randn(n, H, d, generator=g).bfloat16()
        k[bad[r], 7 % dv] = value
        scatter_to_pages(pages, lay["tables"][r], k[:, None], P)
        q_new.append(q)
        for i in range(n):
            kd = k[max(0, b + i - window + 1) if window else 0:b + i + 1].double()
            want.append(torch.softmax(q[i].double() @ kd.T * scale, 1) @ kd[:, :dv])
    i32, want = dict(dtype=torch.int32, device=DEV), torch.stack(want)
    got = o.latent_prefill_tc(torch.cat(q_new).to(DEV), pages, lay["block_table"], lay["page_base"],
                              torch.tensor(np.cumsum([0] + qlens), **i32), torch.tensor(befores, **i32),
                              o.latent_prefill_tiles(qlens, H), None, scale, window, dv).double().cpu()
    o.raise_on_kernel_error()
    assert torch.equal(torch.isfinite(got), torch.isfinite(want)) and bool(torch.isfinite(want).any()) and not bool(torch.isfinite(want).all())
    fine = torch.isfinite(want)
    assert (got - want)[fine].abs().max() < 6 * (2 ** -9 + 2 ** -9 + 2 ** -13)              # as for long rows; values up to 6


@pytest.mark.parametrize("H,d,dv,T,before", [(16, 448, 384, 300, 0), (4, 320, 256, 300, 0), (16, 192, 128, 64, 1500)])
@pytest.mark.parametrize("width", [1.0, 3.0])
def test_latent_attention_on_tcgen05_is_no_further_from_64_bits(H, d, dv, T, before, width):
    """Both kernels round queries, keys, weights and results to bfloat16; the distance from float64 of the tcgen05 one is no
    larger than the other's, for flat rows and for such as a few keys decide.  (Means over 2 x 10^6 roundings and more: 2 %
    of room covers their spread between seeds, measured 0.3 %.)"""
    o, P = ops(), 16
    g = torch.Generator(device=DEV).manual_seed(d)
    n = before + T
    pages = torch.zeros(-(-n // P) * P, d, device=DEV, dtype=torch.bfloat16)
    pages[:n] = torch.randn(n, d, generator=g, device=DEV) + 0.3 * torch.randn(d, generator=g, device=DEV)
    k, q = pages[:n].double(), (width * torch.randn(T, H, d, generator=g, device=DEV)).bfloat16()
    i32 = dict(dtype=torch.int32, device=DEV)
    rows = (pages.view(-1, 1, P, d), torch.arange(-(-n // P), **i32).view(1, -1), torch.zeros(1, **i32), torch.tensor([0, T], **i32),
            torch.tensor([before], **i32))
    tiles = torch.tensor([(0, t) for t in range(0, T, 64 // H)], **i32)
    general = o.latent_attention_tc(q, *rows, tiles, None, d ** -0.5, None, dv).double()
    got = o.latent_prefill_tc(q, *rows, o.latent_prefill_tiles([T], H), None, d ** -0.5, None, dv).double()
    s = torch.einsum("qhd,kd->hqk", q.double(), k) * d ** -0.5
    s = s.masked_fill(torch.arange(n, device=DEV)[None] > torch.arange(before, n, device=DEV)[:, None], float("-inf"))
    want = torch.einsum("hqk,kd->qhd", torch.softmax(s, -1), k[:, :dv])
    assert float((got - want).norm()) <= 1.02 * float((general - want).norm())


def test_bigram_rows_carry_the_previous_token_between_steps():
    o = ops()
    buckets, mp, mc, H = 11, 7, 3, 8
    table = torch.arange((buckets + 1) * H, dtype=torch.float32).view(buckets + 1, H).to(DEV)
    state = torch.zeros(3, dtype=torch.int32, device=DEV)
    seqs = {0: [5, 9, 2, 2, 7, 1], 2: [3, 3, 8, 0]}                 # by state slot
    want = {s: plain.bigram_rows(t, buckets, mp, mc) for s, t in seqs.items()}
    cuts = [{0: (0, 2), 2: (0, 1)}, {0: (2, 3)}, {2: (1, 4), 0: (3, 6)}]
    i32 = dict(dtype=torch.int32, device=DEV)
    for cut in cuts:
        ids, row, start, pos, slot = [], [], [0], [], []
        for r, (s, (a, b)) in enumerate(cut.items()):
            ids += seqs[s][a:b]
            row += [r] * (b - a)
            start.append(len(ids))
            pos.append(a)
            slot.append(s)
        x = torch.zeros(len(ids), H, device=DEV)
        o.bigram_add(x, torch.tensor(ids, **i32), torch.tensor(row, **i32), torch.tensor(start, **i32),
                     torch.tensor(pos, **i32), torch.tensor(slot, **i32), state, table, buckets, mp, mc)
        got = (x[:, 0] / H).round().int().tolist()
        t = 0
        for s, (a, b) in cut.items():
            assert got[t:t + b - a] == want[s][a:b], (cut, s)
            t += b - a


@pytest.mark.parametrize("H,KH,dim,vdim", [(4, 2, 8, 12), (3, 3, 32, 20), (2, 1, 64, 64), (6, 3, 96, 80), (2, 2, 128, 128), (1, 1, 128, 200)])
def test_delta_rule_with_channel_decays_over_chunks(H, KH, dim, vdim):
    """The recurrence over chunks of tokens against the loop over tokens in 64 bits and no further from it than three times the
    kernel that walks them: rows that end on and around an edge of a chunk (64) and of a block in it (16), unequal rows in one step, keys that
    repeat (a system far from the identity), channels from no decay to one that leaves nothing, states that were there before."""
    o = ops()
    g = torch.Generator().manual_seed(dim + vdim)
    rand = lambda *shape, scale=1.0: scale * torch.randn(*shape, generator=g)
    unit = lambda t: t / torch.sqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6)
    for lens in ([64], [65, 1, 63], [1, 200, 2, 128, 129, 5, 64, 17], [330]):
        T, slots = sum(lens), torch.randperm(10, generator=g)[:len(lens)].tolist()
        k = unit((rand(T, KH, dim, scale=0.4) + rand(KH, dim)).double())
        q = unit(rand(T, KH, dim).double()) * dim ** -0.5
        v, beta = rand(T, H, vdim).double(), torch.rand(T, H, generator=g).double()
        log2_g = -torch.exp(rand(T, H, dim, scale=2.0) - 2.0)
        log2_g[:, :, 0] = 0.0
        log2_g[T // 2, :, 1:5] = -130.0
        state = rand(10, H * dim * vdim + 4)
        f = lambda t: t.float().contiguous().to(DEV)
        starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
        i32 = lambda t: torch.tensor(t, dtype=torch.int32, device=DEV)
        assert o.channel_chunk_ok(max(lens), T, len(lens), H, dim, vdim) == (max(lens) >= 64)
        got, ends = {}, {}
        for how in ("chunks", "walk"):
            sd = state.to(DEV)
            run, decays = (o.channel_chunk, log2_g) if how == "chunks" else (o.delta_rule, torch.exp2(log2_g.double()))
            got[how] = run(f(q), f(k), f(v), f(beta), f(decays), sd, i32(starts), i32(slots), len(lens), state_off=4).double().cpu()
            ends[how] = sd.double().cpu()
        group = torch.arange(H) // (H // KH)
        qf, kf, vf, bf = (t.float().double() for t in (q, k, v, beta))
        for r, (n, slot) in enumerate(zip(lens, slots)):
            S, want = state[slot, 4:].double().view(H, dim, vdim), []
            for t in range(starts[r], starts[r] + n):
                S = torch.exp2(log2_g[t].double())[:, :, None] * S
                u = bf[t][:, None] * (vf[t] - torch.einsum("hdv,hd->hv", S, kf[t][group]))
                S = S + kf[t][group][:, :, None] * u[:, None]
                want.append(torch.einsum("hdv,hd->hv", S, qf[t][group]))
            want = torch.stack(want)
            rows = slice(starts[r], starts[r] + n)
            err = {how: float((got[how][rows] - want).norm() / want.norm()) for how in got}
            end = {how: float((ends[how][slot, 4:].view(H, dim, vdim) - S).norm() / S.norm()) for how in got}
            assert err["chunks"] < max(3 * err["walk"], 1e-6) and end["chunks"] < max(3 * end["walk"], 1e-6), (lens, r, err, end)
        untouched = [s for s in range(10) if s not in slots]
        assert torch.equal(ends["chunks"][untouched], state[untouched].double()) and torch.equal(ends["chunks"][:, :4], state[:, :4].double())


@pytest.mark.parametrize("dim,vdim,dtype", [(32, 20, torch.float32), (64, 64, torch.bfloat16), (128, 128, torch.float32), (9 * 4, 12, torch.bfloat16)])
def test_delta_rule_over_chunks_with_decays_that_leave_nothing(dim, vdim, dtype):
    """Logarithms of minus infinity and of numbers whose sums leave float32, as they are and as the prep kernel makes them of
    large weights: zeros as decays in the walk over tokens, and the same outputs and states over chunks."""
    o = ops()
    g = torch.Generator().manual_seed(dim)
    H, KH, taps = 4, 2, 3
    lens = [130, 64, 200]
    T, C = sum(lens), 2 * KH * dim + H * vdim
    starts = torch.tensor(np.cumsum([0] + lens), dtype=torch.int32, device=DEV)
    token_row = torch.repeat_interleave(torch.arange(3), torch.tensor(lens)).int().to(DEV)
    slots = torch.tensor([2, 0, 3], dtype=torch.int32, device=DEV)
    state = torch.randn(4, H * dim * vdim, generator=g)
    main = torch.randn(T, C + H, generator=g).to(dtype).to(DEV)
    conv, conv_state = torch.randn(C, taps, generator=g).to(DEV), torch.zeros(4, (taps - 1) * C, device=DEV)
    for a_log, bias in (([90.0, 0.5, 200.0, -3.0], 0.0), ([0.0, 80.0, 1.0, 85.0], 200.0)):
        up = (torch.randn(T, H * (dim + vdim), generator=g) + 1).to(DEV)
        a32, b32 = torch.tensor(a_log, device=DEV), torch.full((H * dim,), bias, device=DEV)
        prep = lambda logs: o.delta_prep(main, up, conv, conv_state, 0, a32, b32, token_row, starts, slots, H, KH, dim, vdim, taps, log2_decays=logs)
        q, k, v, beta, decays, _ = prep(False)
        logs = prep(True)[4]
        assert bool((logs < -1e30).any())
        logs[40:44, 1, :5], decays[40:44, 1, :5] = float("-inf"), 0.0
        logs[45:61, 3, 1:3], decays[45:61, 3, 1:3] = -1e38, 0.0
        ends = {how: state.to(DEV) for how in ("chunks", "walk")}
        got = o.channel_chunk(q, k, v, beta, logs, ends["chunks"], starts, slots, 3)
        want = o.delta_rule(q, k, v, beta, decays, ends["walk"], starts, slots, 3)
        assert bool(torch.isfinite(want).all())
        # both are float32 sums of the same recurrence: as far apart as either is from 64 bits (1e-6, see the test above) but for
        # the decays, rounded once as numbers and once as logarithms
        assert float((got - want).norm() / want.norm()) < 1e-5
        assert float((ends["chunks"] - ends["walk"]).norm() / ends["walk"].norm()) < 1e-5

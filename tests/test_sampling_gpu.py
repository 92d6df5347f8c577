"""The sampling kernel against the plain processing (temperature, top-k, top-p) with the
same uniform numbers, and its greedy, tie and bad-input behaviour."""

import pytest
import torch

from tests.plain import model as plain

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def run(logits, temperature, top_k, top_p, seeds, counters, logprobs=False):
    from acorninfer_b200.kernels import ops
    R = logits.shape[0]
    f = lambda v, dt: torch.tensor(v if isinstance(v, list) else [v] * R, dtype=dt, device=DEV)
    toks, lps = ops.sample(logits.to(DEV), f(temperature, torch.float32), f(top_k, torch.int32),
                           f(top_p, torch.float32), f(seeds, torch.int64), f(counters, torch.int64), logprobs)
    return toks.tolist(), (lps.tolist() if logprobs else None)


def test_greedy_takes_the_first_of_equal_maxima():
    x = torch.randn(5, 1003)
    x[0, 77] = x[0, 900] = 9.0
    x[3, 0] = 9.0
    toks, _ = run(x, 0.0, 0, 1.0, 0, 0)
    assert toks == [77] + x[1:].argmax(-1).tolist()


def test_bad_logits_are_flagged_not_sampled():
    x = torch.randn(3, 50)
    x[1, 4] = float("nan")
    x[2, 9] = float("inf")
    toks, _ = run(x, 1.0, 0, 1.0, 0, 0)
    assert toks[0] >= 0 and toks[1] == -1 and toks[2] == -1


@pytest.mark.parametrize("temperature,top_k,top_p", [(0.7, 0, 1.0), (1.0, 5, 1.0), (1.3, 0, 0.8), (0.9, 40, 0.6),
                                                     (0.5, 1, 1.0), (1.0, 0, 0.05)])
def test_sampling_matches_plain_with_the_same_uniforms(temperature, top_k, top_p):
    from acorninfer_b200.kernels import ops
    torch.manual_seed(5)
    R, V = 24, 1531
    x = 3 * torch.randn(R, V)
    seeds = list(range(100, 100 + R))
    counters = list(range(R))
    toks, lps = run(x, temperature, top_k, top_p, seeds, counters, logprobs=True)
    checked = 0
    for r in range(R):
        processed = plain.process_logits(x[r], temperature, top_k, top_p)
        u = ops.uniform(seeds[r], counters[r])
        assert 0.0 <= u < 1.0
        want, want_lp, margin = plain.sample_with_uniform(processed, u)
        assert torch.isfinite(processed[toks[r]]), "the kernel chose a token that top-k/top-p removed"
        if margin > 1e-4:                       # away from a CDF step the choice is unambiguous
            assert toks[r] == want
            assert abs(lps[r] - want_lp) < 1e-3
            checked += 1
    assert checked >= R // 2


def test_draws_follow_the_distribution_and_do_not_depend_on_the_batch():
    V = 7
    x = torch.tensor([[0.0, 1.0, 2.0, -1.0, 0.5, 1.5, -3.0]]).repeat(4000, 1)
    toks, _ = run(x, 1.0, 0, 1.0, 11, list(range(4000)))
    freq = torch.bincount(torch.tensor(toks), minlength=V).double() / 4000
    assert (freq - x[0].double().softmax(-1)).abs().max() < 0.03
    alone, _ = run(x[:1], 1.0, 0, 1.0, 11, [123])
    assert alone[0] == toks[123]


@pytest.mark.parametrize("clusters", [False, True])
@pytest.mark.parametrize("vocab", [5, 33, 4097, 19999, 20000, 32771, 151936, 360448, 360449])
def test_large_vocabularies_in_every_cut(vocab, clusters, monkeypatch):
    """Both kernels (one CTA a row, a cluster of eight CTAs a row) at vocabularies that leave some CTAs of a cluster without a
    logit, at the one from which clusters are taken, at the largest that a cluster holds and one more; rows of odd length, which
    start on 16 bytes only every fourth time; a row of equal logits, one masked down to a few tokens, one with many ties."""
    from acorninfer_b200.kernels import ops
    assert ops.sample_in_clusters(7, vocab, False) == (vocab >= 20000)
    monkeypatch.setattr(ops, "sample_in_clusters", lambda *sizes: clusters)
    R = 7
    g = torch.Generator().manual_seed(vocab)
    x = 2.5 * torch.randn(R, vocab, generator=g)
    x[4] = 0.25
    x[5, 9:] = -3.0e38
    x[6] = (x[6] * 2).round() / 2           # many equal logits
    temperature, top_k, top_p = [0.7, 1.0, 0.6, 0.0, 1.0, 1.0, 0.8], [0, 20, 50, 0, 0, 0, 1000], [0.95, 0.8, 1.0, 1.0, 0.5, 0.9, 0.9]
    seeds, counters = list(range(50, 50 + R)), [3 * i for i in range(R)]
    f = lambda v, dt: torch.tensor(v, dtype=dt, device=DEV)
    toks, lps = ops.sample(x.to(DEV), f(temperature, torch.float32), f(top_k, torch.int32), f(top_p, torch.float32),
                           f(seeds, torch.int64), f(counters, torch.int64), True)
    toks, lps = toks.tolist(), lps.tolist()
    checked = 0
    for r in range(R):
        if temperature[r] == 0:
            assert toks[r] == int(x[r].argmax())
            continue
        processed = plain.process_logits(x[r], temperature[r], top_k[r], top_p[r])
        # among equal logits at the bound of top-p the kernel keeps all, the plain one those that its sort puts last
        scaled = x[r].double() / temperature[r]
        processed = scaled.masked_fill(scaled < processed[torch.isfinite(processed)].min(), float("-inf"))
        u = ops.uniform(seeds[r], counters[r])
        want, want_lp, margin = plain.sample_with_uniform(processed, u)
        # a kept set may differ by the token at the bound of top-p, whose mass moves the CDF by as much
        if margin > 1e-6 and r != 4:
            assert toks[r] == want
            assert abs(lps[r] - want_lp) < 1e-4
            checked += 1
    assert 0 <= toks[4] < vocab and checked >= 3
    none = f([0.0] * R, torch.float32), f([0] * R, torch.int32), f([1.0] * R, torch.float32)
    seeds_, counters_ = f(seeds, torch.int64), f(counters, torch.int64)
    assert ops.sample(x.to(DEV), *none, seeds_, counters_, greedy=True)[0].tolist() == x.argmax(1).tolist()


@pytest.mark.parametrize("k", [1, 127, 128, 129, 4000])
def test_top_k_at_the_cut_by_the_warps_maxima(k):
    """The cluster kernel drops keys below the least of its 128 warps' maxima for k up to 128: rows with one large logit to a
    warp, with maxima of 0 and -0 alone, with all logits equal, and any."""
    from acorninfer_b200.kernels import ops
    V = 40000
    slice_ = (V // 8 + 3) & ~3
    x = torch.randn(4, V, generator=torch.Generator().manual_seed(k)) - 3.0
    # vectors of four by 512 threads: warp w of a CTA starts at element 128 w of its slice
    first = torch.tensor([cta * slice_ + 128 * w for cta in range(8) for w in range(16)])
    x[0, first] = torch.linspace(5.0, 6.0, 128)
    x[1] = -x[1].abs() - 1.0
    x[1, first[::2]], x[1, first[1::2]] = 0.0, -0.0
    x[2] = 1.5
    n = 400
    f = lambda v, dt: torch.full((4 * n,), v, dtype=dt, device=DEV)
    assert ops.sample_in_clusters(4 * n, V, False)
    toks = ops.sample(x.repeat_interleave(n, 0).to(DEV), f(1.0, torch.float32), f(k, torch.int32), f(1.0, torch.float32),
                      f(3, torch.int64), torch.arange(4 * n, device=DEV))[0].view(4, n).cpu()
    for r in range(4):
        kept = x[r] >= x[r].topk(k).values[-1]
        if r == 1 and k < 128:          # 0 ranks above -0 as a key where both are at the bound
            kept &= ~(torch.signbit(x[r]) & (x[r] == 0)) | (k > 64)
        assert bool(kept[toks[r].long()].all()), (r, k)
        p = torch.where(kept, x[r].double(), torch.tensor(float("-inf")).double()).softmax(0)
        # every token of a small kept set turns up as often as it should (four standard deviations)
        freq = torch.bincount(toks[r].long(), minlength=V).double() / n
        assert ((freq - p).abs() <= 4 * (p / n).sqrt() + 4 / n).all(), (r, k)


@pytest.mark.parametrize("n,spread", [(256, False), (257, False), (1024, True), (1025, True)])
@pytest.mark.parametrize("top_k,top_p", [(64, 1.0), (128, 0.5), (0, 0.5), (0, 0.0)])
def test_candidates_at_the_ends_of_the_lists(n, spread, top_k, top_p):
    """``n`` equal logits above all others, in one CTA's slice (which notes 256 candidates) or all over the row (of which
    1,024 are compared): with ties kept whole, top-k and top-p leave exactly these, each as likely as any other."""
    from acorninfer_b200.kernels import ops
    V, draws = 40000, 64
    x = torch.full((1, V), -20.0)
    at = torch.arange(n) * (39 if spread else 1) + 3
    x[0, at] = 7.25
    f = lambda v, dt: torch.full((draws,), v, dtype=dt, device=DEV)
    toks, lps = ops.sample(x.expand(draws, V).contiguous().to(DEV), f(0.8, torch.float32), f(top_k, torch.int32),
                           f(top_p, torch.float32), f(9, torch.int64), torch.arange(draws, device=DEV), True)
    u = [ops.uniform(9, i) for i in range(draws)]
    # equal probabilities of 2^44 units each: the draw is exact
    assert toks.tolist() == [int(at[int(int(v * 2 ** 24) * n // 2 ** 24)]) for v in u]
    # -ln n in float32: one rounding of the logarithm's argument and one of its result
    assert (lps.cpu().double() + torch.tensor(float(n)).double().log()).abs().max() < 4 * 2.0 ** -24 * 8


@pytest.mark.parametrize("rows,vocab", [(1, 50), (128, 700), (128, 20001), (129, 700)])
def test_parameters_among_the_launch_arguments(rows, vocab):
    """Up to 128 rows carry their parameters in the launch, more in device memory: the same tokens and log-probabilities."""
    from acorninfer_b200 import SamplingParams
    from acorninfer_b200.kernels import ops
    from acorninfer_b200.sampling.sampler import Sampler
    g = torch.Generator().manual_seed(rows)
    x = (2 * torch.randn(rows, vocab, generator=g)).to(DEV)
    params = [SamplingParams(temperature=(0.7, 0.0, 1e39, 1.3)[i % 4], top_p=(1.0, 0.4, 0.9)[i % 3], top_k=(0, 7, 1000000, 150)[i % 4],
                             seed=(1 << 62) + 5 * i) for i in range(rows)]
    counters = [i << 33 for i in range(rows)]
    f = lambda v, dt: torch.tensor(v, dtype=dt, device=DEV)
    want = ops.sample(x, f([p.temperature for p in params], torch.float64).float(), f([p.top_k for p in params], torch.int32),
                      f([p.top_p for p in params], torch.float32), f([p.seed for p in params], torch.int64), f(counters, torch.int64), True)
    got = Sampler(DEV).launch(x, params, counters, True)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    if rows > ops.SAMPLE_INLINE_ROWS:
        with pytest.raises(ops.KernelError):
            ops.sample_inline(x, [0] * rows, [0] * rows, [1.0] * rows, [1.0] * rows, [0] * rows)

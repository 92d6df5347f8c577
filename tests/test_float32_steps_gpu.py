"""The float32 path over whole steps of a model with real widths: a token's bits are a matter of its own row, however its prompt is cut
and whatever else is in the step (products on the tensor cores and on the CUDA cores, padded and replayed steps)."""

import pytest
import torch

from tests.tiny import random_tokens

pytestmark = pytest.mark.gpu


def make_runner(graphs):
    from acorninfer_b200 import ModelRunner
    from acorninfer_b200.config.presets import preset
    from acorninfer_b200.registry import config_from_dict
    raw = preset("qwen3-0.6b")
    raw.update(num_hidden_layers=2, vocab_size=1024)
    return ModelRunner.from_random(config_from_dict(raw), 5, dtype="float32", num_blocks=400, page_size=16, max_requests=90,
                                   decode_graph=graphs)


class Company:
    """Requests that share a step with the one that is looked at."""

    def __init__(self, runner, decoding, prompts):
        from acorninfer_b200.engine.batch import StepEntry
        self.entry, self.prompts, self.runner, self.made = StepEntry, prompts, runner, 0
        self.live = [runner.open(("decoding", i)) for i in range(decoding)]
        for i, rc in enumerate(self.live):
            runner.step([StepEntry(rc, random_tokens(3 + i % 5, 1024, i), [])])

    def entries(self):
        out = [self.entry(rc, [7], []) for rc in self.live]
        for n in self.prompts:
            self.made += 1
            out.insert(self.made % (len(out) + 1), self.entry(self.runner.open(("prompt", self.made)), random_tokens(n, 1024, n), []))
        return out

    def step(self, mine):
        """Logits of ``mine`` amid the company."""
        others = self.entries()
        at = len(others) // 2
        logits = self.runner.step(others[:at] + [mine] + others[at:]).clone()
        for e in others:
            if not any(e.cache is rc for rc in self.live):
                self.runner.close(e.cache)
        return logits

    def close(self):
        for rc in self.live:
            self.runner.close(rc)


@pytest.mark.parametrize("graphs", [False, True])
def test_bits_depend_on_the_row_alone(graphs):
    from acorninfer_b200.engine.batch import StepEntry
    runner = make_runner(graphs)
    tokens, answer = random_tokens(100, 1024, 77), random_tokens(4, 1024, 78)
    want = None
    for decoding, prompts in ((0, ()), (63, ()), (66, ()), (0, (40,)), (3, (2, 33)), (20, (90,))):
        company = Company(runner, decoding, prompts)
        for portions in ((100,), (64, 36), (30, 70), (2, 98)):
            rc, at, got = runner.open("mine"), 0, []
            for n in portions:
                got.append(company.step(StepEntry(rc, tokens[at:at + n], list(range(n)))))
                at += n
            for t in answer:
                got.append(company.step(StepEntry(rc, [t], [0])))
            runner.close(rc)
            got = torch.cat(got)
            if want is None:
                want = got
            assert torch.equal(got, want), (decoding, prompts, portions)
        company.close()

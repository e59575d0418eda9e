"""Decoded tokens beside portions of prompts: the two attentions of such a step run at the same
time, and every row's logits are those that its request gets in a step of its own."""
import pytest
import torch

from llmario_b200 import Model, ModelRunner, StepEntry
from llmario_b200.cli import preset_config
from llmario_b200.weights import random_tensors

DEV = "cuda:0"


@pytest.mark.gpu
@pytest.mark.parametrize("page,lengths,portions", [
    (64, [70, 500, 333, 1200, 65], [(0, 300), (40, 64), (129, 130)]),      # items of whole tiles and remainders
    (64, [900] * 24, [(0, 9), (700, 700)]),                                # one long item, a short portion
    (16, [260, 128, 31], [(0, 511), (16, 17), (5, 600)]),                  # pages whose keys are gathered first
    (64, [1500], [(0, 1500)]),                                             # more work items than SMs
])
def test_decoded_tokens_beside_portions(page, lengths, portions):
    spec = preset_config("qwen3-0.6b", 2).to_spec()
    w = random_tensors(spec, 3, torch.bfloat16, DEV)
    w["model.embed_tokens.weight"].mul_(25.0)
    model = Model(spec, w, torch.bfloat16, DEV)
    g = torch.Generator().manual_seed(len(lengths) + page)
    toks = lambda n: torch.randint(0, 150000, (n,), generator=g).tolist()  # noqa: E731
    seqs = [(toks(n), toks(1)) for n in lengths] + [(toks(a), toks(n)) for a, n in portions]
    rows = sum(len(s) for _, s in seqs)
    runner = ModelRunner(model, page_size=page, max_requests=len(seqs), max_context=4096,
                         n_pages=sum((len(a) + len(b)) // page + 2 for a, b in seqs) + 1,
                         token_budget=max(rows, 2048))
    for i, (before, _) in enumerate(seqs):
        if before:
            runner.step([StepEntry(i, before, [])])
    entries = [StepEntry(i, step, [len(step) - 1]) for i, (_, step) in enumerate(seqs)]

    def rewind(i):
        if seqs[i][0]:
            runner.cache.truncate(i, len(seqs[i][0]))
        else:
            runner.close(i)

    alone = []
    for i, e in enumerate(entries):
        alone.append(runner.step([e]).clone())
        rewind(i)
    alone = torch.cat(alone).double()
    for _ in range(3):
        both = runner.step(entries).double()
        for i in range(len(entries)):
            rewind(i)
        # two layers of bfloat16 operands whose sums are in another order: the rows of two such
        # orders differ by some 0.5 %; a row that lacks a part of its keys differs by tens
        err = (both - alone).norm(dim=1) / alone.norm(dim=1)
        assert bool((err < 0.025).all()), err

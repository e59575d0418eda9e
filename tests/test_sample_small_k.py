"""A small top-k, whose candidates are bounded by the largest logits of groups of threads: at the
edges of that rule, against the chain in float64."""
import numpy as np
import pytest
import torch

DEV = "cuda:0"


@pytest.mark.gpu
@pytest.mark.parametrize("vocab", (5, 200, 4097, 8192, 40961, 151936))
def test_small_top_k(vocab):
    """k on both sides of the rule's limit and of the vocabulary; distinct logits, ties across the k-th
    place, ties of more tokens than the sorted list holds, all of the largest in one thread's stretch."""
    from llmario_b200 import kernels
    g = torch.Generator().manual_seed(vocab)
    spike = torch.randn(vocab, generator=g)
    spike[:64] += 20.0
    kinds = [2.5 * torch.randn(vocab, generator=g), torch.round(4 * torch.randn(vocab, generator=g)) / 4,
             torch.zeros(vocab), spike]
    rows = [(l, k) for l in kinds for k in (1, 2, 40, 63, 64, 65, 200)]
    n = len(rows)
    u = torch.rand(n, generator=g, dtype=torch.float64)
    full = lambda v: torch.full((n,), v, dtype=torch.float32, device=DEV)  # noqa: E731
    out = torch.full((n,), -7, dtype=torch.int32, device=DEV)
    kernels.sample(torch.stack([r[0] for r in rows]).to(DEV), full(0.8),
                   torch.tensor([r[1] for r in rows], dtype=torch.int32, device=DEV), full(1.0), full(0.0),
                   u.to(DEV), out)
    for (l, k), ui, got in zip(rows, u.tolist(), out.tolist()):
        l = l.numpy().astype(np.float64)
        ids = np.lexsort((np.arange(vocab), -l))[:k] if k < vocab else np.arange(vocab)
        cum = np.cumsum(np.exp((l[ids] - l.max()) / 0.8))
        at = np.flatnonzero(ids == got)
        assert len(at) == 1, (k, got)
        # (the uniform may be off its stretch by the rounding of 32-bit weights: 1e-5 of their sum)
        lo = cum[at[0] - 1] if at[0] else 0.0
        assert lo - 1e-5 * cum[-1] <= ui * cum[-1] <= cum[at[0]] + 1e-5 * cum[-1], (k, got)

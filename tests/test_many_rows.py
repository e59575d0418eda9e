"""The kernels of steps with many rows, at the sizes where their tiles, remainders and runs can go
wrong, against float64 statements and against the kernels for few rows."""
import pytest
import torch

gpu = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, dtype=torch.float32, scale=1.0, seed=0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (scale * torch.randn(*shape, generator=g)).to(dtype).to(DEV)


@gpu
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("M,N,K,pad", [(1, 130, 128, 0), (16, 1024, 2048, 4), (17, 33, 1028, 0), (32, 64, 20, 8),
                                       (40, 72, 36, 0), (33, 257, 256, 0), (64, 128, 260, 0), (70, 96, 4, 0),
                                       (95, 128, 1024, 0), (129, 1000, 1040, 0), (211, 1024, 3072, 0),
                                       (130, 16500, 64, 0)])
def test_gemm_float32(M, N, K, pad, accumulate):
    """Tiles of 16 and of 32 to 64 rows, K whole and in parts, ragged N, K below one step, padded
    rows; a row's bits do not depend on how many rows there are."""
    from llmario_b200 import kernels
    a, w = rnd(M, K + pad, seed=1)[:, :K], rnd(N, K + pad, seed=2)[:, :K]
    c0 = rnd(M, N, seed=3)
    out = c0.clone()
    kernels.gemm_simt(a, w, out, accumulate)
    ref = a.double() @ w.double().T + (c0.double() if accumulate else 0)
    # every partial sum is rounded once per addition: |error| <= (K + 10) 2^-24 sum |a w|, and far
    # less on average
    size = a.abs().double() @ w.abs().double().T + (c0.abs().double() if accumulate else 0)
    assert bool(((out.double() - ref).abs() <= (K + 10) * 2 ** -24 * size).all())
    rel = float((out.double() - ref).norm() / ref.norm())
    assert rel <= 2 ** -24 * (2 + K ** 0.5)      # roundings that do not conspire
    for rows in (1, 17, 40):
        if rows < M:
            few = c0[:rows].clone()
            kernels.gemm_simt(a[:rows], w, few, accumulate)
            assert torch.equal(few, out[:rows])

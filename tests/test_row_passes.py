"""Passes over 32-bit rows in pieces of four columns: widths on both sides of what they take, rows fewer
and more than the grid's stride, against plain torch in float64."""
import pytest
import torch

gpu = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (scale * torch.randn(*shape, generator=g)).to(DEV)


@gpu
@pytest.mark.parametrize("rows,width,per", [(1, 4, 4), (3, 12, 4), (2, 10, 5), (700, 4096, 128), (5, 36, 6), (2111, 260, 20)])
def test_bias_and_decay_passes(rows, width, per):
    from llmario_b200 import kernels
    z, b, rate = rnd(rows, width, scale=3.0), rnd(width, seed=1), rnd(width // per, seed=2, scale=0.5)
    softplus = torch.nn.functional.softplus
    zb = z.double() + b.double()
    # 32-bit sums and functions: a few roundings of the exponent, of which the size is at most some 30
    tol = dict(rtol=1e-5, atol=1e-7)
    got = z.clone()
    kernels.add_bias(got, b)
    assert torch.equal(got, z + b)
    for bias, want in ((b, zb), (None, z.double())):
        got = z.clone()
        kernels.bias_sigmoid_pow(got, bias, 0.0625)
        torch.testing.assert_close(got.double(), torch.sigmoid(want) ** 0.0625, **tol)
        got = z.clone()
        kernels.rate_decay(got, rate, bias, per)
        want = torch.exp(-rate.double().exp().repeat_interleave(per) * softplus(want))
        torch.testing.assert_close(got.double(), want, **tol)


@gpu
@pytest.mark.parametrize("rows,width", [(1, 4), (3, 1020), (2, 1027), (700, 4096), (5, 4100), (3, 1024)])
@pytest.mark.parametrize("accumulate", (False, True))
def test_dual_norm_mean(rows, width, accumulate):
    from llmario_b200 import kernels
    a, b, wa, wb, y = (rnd(rows, width, seed=1), rnd(rows, width, seed=2), rnd(width, seed=3), rnd(width, seed=4),
                       rnd(rows, width, seed=5))
    unit = lambda x: x.double() * torch.rsqrt((x.double() ** 2).mean(-1, keepdim=True) + 1e-6)  # noqa: E731
    want = 0.5 * (unit(a) * wa.double() + unit(b) * wb.double()) + (y.double() if accumulate else 0)
    got = y.clone()
    kernels.dual_norm_mean(a, b, wa, wb, got, 1e-6, accumulate)
    torch.testing.assert_close(got.double(), want, rtol=1e-5, atol=2e-6)

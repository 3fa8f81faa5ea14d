"""Products with few rows (tiles of the weights, K cut over a cluster) against the fp32 references, at the edges of the
kernel's ranges: rows around the padding to 16 and the limits of the dispatch, ragged N and K, every number of parts."""
import math

import pytest
import torch

from tokenweave_b200 import ops
from tokenweave_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
BF = torch.bfloat16

# 128 outputs: 1 tile; 4096: 32 tiles, 4 parts; 5000: ragged; K 264 and 72: a k-block that ends early, no cut
SHAPES = [(128, 72), (136, 264), (1000, 2056), (4096, 4096), (5000, 1024), (20000, 512), (19336, 8200)]


def rnd(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(BF)


def near(got, want):
    """One rounding to bf16 (2^-9 of the value) behind sums in another order (1e-3 of the usual size of a result)."""
    got, want = got.float(), want.float()
    rms = want.square().mean().sqrt()
    assert ((got - want).abs() <= 2 ** -7 * want.abs() + 4e-3 * rms).all(), (got - want).abs().max().item()


@pytest.fixture(autouse=True)
def _status_clean():
    ops.reset_status()
    yield
    ops.check_status()


@pytest.mark.parametrize("N,K", SHAPES)
@pytest.mark.parametrize("M", [1, 16, 17, 63, 64, 80, 81, 112, 113, 128, 129, 160, 161, 208, 209, 224, 225, 256])
def test_plain(M, N, K):
    a, w, bias, rs = rnd(M, K), rnd(N, K, scale=K ** -0.5), rnd(N), torch.rand(M, device="cuda") + 0.5
    big = torch.zeros(M + 1, N + 8 + -N % 8, device="cuda", dtype=BF)
    out = ops.gemm(a, w, out=big[:M, :N], bias=bias, row_scale=rs)
    near(out, (a.float() @ w.float().T + bias.float()) * rs[:, None])
    assert big[M:].abs().max().item() == 0 and big[:, N:].abs().max().item() == 0
    assert torch.equal(ops.gemm(a, w, bias=bias, row_scale=rs), out)         # the order of the sums is fixed


@pytest.mark.parametrize("N,K", [(64, 72), (200, 264), (4096, 1024), (14336, 512)])
@pytest.mark.parametrize("M", [1, 33, 100, 140, 200, 224])
def test_gated_and_activations(M, N, K):
    a, w = rnd(M, K), rnd(2 * N, K, scale=K ** -0.5)
    g, u = (a.float() @ w.float().T).chunk(2, -1)
    near(ops.gemm(a, w, swiglu=True), torch.nn.functional.silu(g) * u)
    near(ops.gemm(a, w, swiglu=True, act="gelu_tanh"), torch.nn.functional.gelu(g, approximate="tanh") * u)
    rs = torch.rand(M, device="cuda") + 0.5
    g, u = (g * rs[:, None]).clamp_max(1.0), (u * rs[:, None]).clamp(-1.0, 1.0)
    near(ops.gemm(a, w, swiglu=True, act=("clamped", 1.0, 1.7), in_scale=rs), g * torch.sigmoid(1.7 * g) * (u + 1))
    y = a.float() @ w.float().T
    lo, hi = N // 2 + 3, N + 5
    want = y.clone()
    want[:, lo:hi] = y[:, lo:hi].clamp_min(0).square()
    near(ops.gemm(a, w, col_act=("relu2", lo, hi)), want)


@pytest.mark.parametrize("N,K", [(128, 144), (1000, 1040), (4096, 4096), (24, 528), (20000, 528)])
@pytest.mark.parametrize("M", [1, 31, 96, 150, 160, 208])
def test_fp8(M, N, K):
    aq, a_s = ops.quant_fp8(rnd(M, K))
    wq, w_s = ops.quant_fp8(rnd(2 * N, K, scale=K ** -0.5))
    bias = rnd(2 * N)
    y = (aq.float() @ wq.float().T) * a_s[:, None] * w_s[None]
    near(ops.gemm_fp8(aq, wq, a_s, w_s, bias=bias), y + bias.float())
    g, u = y.chunk(2, -1)
    near(ops.gemm_fp8(aq, wq, a_s, w_s, swiglu=True), torch.nn.functional.silu(g) * u)
    raw = aq.float() @ wq.float().T
    near(ops.gemm_fp8(aq, wq, None, None), raw)


@pytest.mark.parametrize("V,padded,K", [(512, 512, 256), (2000, 2048, 264), (1003, 1024, 128), (32064, 32064, 512)])
@pytest.mark.parametrize("M", [1, 24, 100, 130, 200, 256, 257])
def test_logits_are_the_converted_product(M, V, padded, K):
    a, w = rnd(M, K), rnd(padded, K, scale=K ** -0.5)
    for scale in (1.0, 0.37):
        got = ops.head_logits(a, w, V, scale)
        assert got.dtype == torch.float32 and got.shape == (M, V)
        near(got / scale, a.float() @ w.float().T[:, :V])
        if scale == 1.0:
            assert torch.equal(got, got.to(BF).float())

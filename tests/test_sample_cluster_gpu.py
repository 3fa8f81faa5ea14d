"""The cluster sampler against a sort in 64 bits: same kept set, same winner of the exponential race."""
import math

import numpy as np
import pytest
import torch

from tokenweave_b200 import ops

pytestmark = pytest.mark.gpu


def noise(seed, V):
    """Least and largest value of every element's noise -log(-log u): the fast logarithm is off by up to 2^-21.41 for arguments
    between 0.5 and 2 (CUDA's stated bound), u is rounded to 24 bits, and the outer logarithm and the sum add 1e-5."""
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + np.uint64(0x9E3779B97F4A7C15) * np.arange(1, V + 1, dtype=np.uint64)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z ^= z >> np.uint64(31)
    u = ((z >> np.uint64(40)).astype(np.float64) + 0.5) / 16777216.0
    inner, off = -np.log(u), 2.0 ** -21.41 + 2.0 ** -24
    with np.errstate(divide="ignore"):
        return -np.log(inner * (1 + 1e-6) + off) - 1e-5, -np.log(np.maximum(inner * (1 - 1e-6) - off, 0.0)) + 1e-5


def check(row, t, k, p, m, seed, got):
    """``got`` is kept and wins. The boundary of top-p may move by what rounding moves the sum (1e-5 of the mass); winners
    whose values lie closer than the noise's error may swap."""
    x = row.astype(np.float32)
    if t <= 0:
        assert got == int(np.argmax(x))
        return
    x = (x * np.float32(1 / np.float32(t))).astype(np.float64)
    V = x.size
    keep = np.ones(V, bool)
    if 0 < k < V:
        keep &= x >= np.sort(x)[V - k]
    sure = keep.copy()
    if p < 1:
        e = np.where(keep, np.exp(x - x.max()), 0.0)
        order = np.argsort(x, kind="stable")
        asc = np.cumsum(e[order])
        lim = (1 - np.float32(p)) * asc[-1]
        values = x[order]
        keep &= x >= values[min(np.searchsorted(asc, lim - 1e-5 * asc[-1], side="right"), V - 1)]
        sure &= x >= values[min(np.searchsorted(asc, lim + 1e-5 * asc[-1], side="right"), V - 1)]
    if m > 0:
        edge = x.max() + math.log(m)
        keep &= x >= edge - 1e-5
        sure &= x >= edge + 1e-5
    assert keep[got], (x[got], x[keep].min())
    least, largest = noise(seed, V)
    assert x[got] + largest[got] >= (x + least)[sure].max()


@pytest.mark.parametrize("V,ld", [(1, 1), (7, 9), (1001, 1001), (16384, 16384), (16385, 16388), (50257, 50257), (131072, 131072),
                                  (152064, 152065), (400001, 400001)])
@pytest.mark.parametrize("rows", [1, 40, 90])
def test_rows(V, ld, rows):
    r = np.random.RandomState(V + rows)
    logits = torch.from_numpy((r.randn(rows, ld) * 2.5).astype(np.float32)).cuda()[:, :V]
    t = np.where(r.rand(rows) < 0.2, 0.0, r.uniform(0.5, 1.3, rows))
    k = np.where(r.rand(rows) < 0.5, np.where(r.rand(rows) < 0.8, r.randint(1, 200, rows), r.randint(1000, 3000, rows)), 0)
    p = np.where(r.rand(rows) < 0.6, r.uniform(0.05, 0.99, rows), 1.0)
    m = np.where(r.rand(rows) < 0.3, 0.03, 0.0)
    seeds = r.randint(0, 1 << 30, rows)
    got = ops.sample(logits, ops.pack_sample_params(t, k, p, m, seeds).cuda()).tolist()
    host = logits.cpu().numpy()
    for i in range(0, rows, 1 if rows < 90 else 5):
        check(host[i], t[i], int(k[i]), float(p[i]), float(m[i]), int(seeds[i]), got[i])


@pytest.mark.parametrize("V", [300, 40000, 152064])
def test_odd_rows(V):
    """Equal logits, masked ones (-inf), only one left, nothing left, one infinite, NaN beside numbers, the type's lowest value."""
    x = torch.randn(7, V)
    x[0] = 1.25
    x[1, V // 3:] = -math.inf
    x[2] = -math.inf
    x[2, V - 2] = 3.0
    x[3] = -math.inf
    x[4, V // 2] = math.inf
    x[5, ::2] = math.nan
    x[6] = torch.finfo(torch.float32).min
    x[6, V // 5] = 0.0
    n = x.shape[0]
    for k, p, m in ((0, 1.0, 0.0), (5, 1.0, 0.0), (0, 0.9, 0.0), (50, 0.5, 0.01)):
        got = ops.sample(x.cuda(), ops.pack_sample_params([0.8] * n, [k] * n, [p] * n, [m] * n, range(n)).cuda()).tolist()
        assert 0 <= got[0] < V and got[1] < V // 3 and got[2] == V - 2 and got[3] == 0 and got[4] == V // 2
        assert got[6] == V // 5 and (got[5] % 2 == 1 or k > 0)     # top-k counts NaN among the largest
        if p == 1.0 and k == 0:
            check(x[0].numpy(), 0.8, k, p, m, 0, got[0])

"""The float32 path's linear and attention kernels at the edges of their tiles, against float64."""
import math

import pytest
import torch

import kernel_refs as R
from test_kernels_gpu import paged_case, rel_err, stream

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from mlx_lm_b200 import ops
    return ops


# rows around the few-rows kernel's limits (4, 8, 16) and the tiles' (64, 128); columns around 8 and 64; inner sizes around a
# K step (16), a segment (128), two, and sums of many segments
@pytest.mark.parametrize("M", [1, 4, 5, 8, 9, 16, 17, 64, 65, 129, 1100])
@pytest.mark.parametrize("N,K", [(7, 4), (8, 20), (65, 128), (200, 132), (64, 384), (130, 1000), (1030, 260), (24, 4100)])
def test_float32_linear(ops, M, N, K):
    """A sum of K products of magnitude 1 / sqrt(K), added in segments of 128: at most (128 + K / 128) roundings of 6e-8
    deep, a few 1e-7 over the whole result in the mean; and the same bits however many rows the call has."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w, b, res = draw(M, K), draw(N, K) / math.sqrt(K), draw(N), draw(M, N)
    want = x.double() @ w.double().T
    out = torch.empty(M, N, device="cuda")
    ops.linear_generic(x, w, b, out, stream(), residual=res)
    assert rel_err(out, want + b + res) <= 1e-6
    more = torch.empty(M + 140, N, device="cuda")
    ops.linear_generic(torch.cat([x, draw(140, K)]), w, b, more, stream(), residual=torch.cat([res, draw(140, N)]))
    assert torch.equal(more[:M], out)
    wide = draw(M, K + 4)                        # a row stride of its own, then rows that no 16-byte access can read
    for x2 in (wide[:, 4:], wide[:, 1:K + 1]):
        ops.linear_generic(x2, w, None, out, stream())
        assert rel_err(out, x2.double() @ w.double().T) <= 1e-6

"""Single rows whose scores are mixed across heads (a CTA a row with all its heads), against float64: around blocks of 64 keys, split
over CTAs or not, with every mask, and beside keys that no row may see."""
import math

import pytest
import torch

from test_wide_portions_gpu import DEV, case, i32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G,dk,dv,window,chunk,keep,gate", [
    (32, 8, 64, 64, 0, 1024, 0, "head"), (16, 4, 64, 64, 0, 100, 0, None), (64, 8, 64, 16, 70, 0, 0, "head"), (4, 1, 32, 72, 0, 0, 0, "column"),
    (8, 1, 128, 128, 200, 0, 70, None), (12, 12, 16, 8, 0, 7, 0, "head"),
])
@pytest.mark.parametrize("max_len", [0, 2048])
def test_mixed_rows(H, G, dk, dv, window, chunk, keep, gate, max_len):
    """Weights are rounded to bfloat16 (2^-9 of each, their sum too), values are of magnitude 1: a few 1e-3 at most."""
    from mlx_lm_b200 import ops
    contexts = [0, 1, 63, 64, 127, 130, 500]
    n = len(contexts)
    q, keys, values, kp, vp, table, randn = case(H, G, dk, dv, 16, False, contexts, [1] * n, H + dk)
    scale, talk = 2.0 / math.sqrt(dk), torch.eye(H, device=DEV) + 0.3 * randn(H, H)
    gt = None if gate is None else randn(n, H if gate == "head" else H * dv).bfloat16()
    want = torch.empty(n, H, dv, dtype=torch.float64, device=DEV)
    for r, p in enumerate(contexts):
        s = torch.einsum("hd,jhd->hj", q[r].double(), keys[r].repeat_interleave(H // G, dim=1)) * scale
        j = torch.arange(p + 1, device=DEV)
        ok = torch.ones_like(j, dtype=torch.bool)
        if window:
            ok &= (p - j < window) | (j < keep)
        if chunk:
            ok &= j // chunk == p // chunk
        w = torch.softmax((talk.double() @ s).masked_fill(~ok, -math.inf), dim=-1)
        want[r] = torch.einsum("hj,jhd->hd", w, values[r].repeat_interleave(H // G, dim=1))
    if gt is not None:
        want *= torch.sigmoid(gt.double().view(n, H, -1))
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    tiles = i32([(r, 1, r, p) for r, p in enumerate(contexts)] + [(0, 0, 0, 0)])
    need = ops.attention_wide_scratch(n + 1, H, dv, window, chunk, max_len, keep) if max_len else 0
    outs = []
    for first in (0, 1):                        # the second time without the first row: the same bits
        scratch = torch.full((need,), float("nan"), device=DEV) if need else None
        out = torch.full((n, H * dv), 7.0, device=DEV)
        ops.attention_wide_tiles(q.view(n, H * dk), dk, tiles[first:], n + 1 - first, 1, table, kp, vp, out, dv, H, dk, dv, scale, status,
                                 ops.current_stream(), window=window, chunk=chunk, talk=talk, gate=gt, scratch=scratch, max_len=max_len,
                                 keep_first=keep)
        outs.append(out)
    assert int(status.item()) == 0 and bool((outs[1][0] == 7.0).all()) and torch.equal(outs[0][1:], outs[1][1:])
    assert float((outs[0].double().view(n, H, dv) - want).abs().max()) < 6e-3
    short = torch.empty(n, H * dv, dtype=torch.bfloat16, device=DEV)
    ops.attention_wide_tiles(q.view(n, H * dk), dk, tiles, n + 1, 1, table, kp, vp, short, dv, H, dk, dv, scale, status,
                             ops.current_stream(), window=window, chunk=chunk, talk=talk, gate=gt, keep_first=keep)
    assert float((short.double().view(n, H, dv) - want).abs().max()) < 2e-2

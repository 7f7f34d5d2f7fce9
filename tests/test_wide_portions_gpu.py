"""The tcgen05 kernel for prompt portions with wide or mixed scores, against float64: edges of its tiles of 128 rows and blocks of 64
keys, every option, and values that no query may see."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def i32(a):
    return torch.tensor(a, dtype=torch.int32, device=DEV)


def case(H, G, dk, dv, page, shared, contexts, portions, seed):
    """Requests with ``contexts`` positions before ``portions`` new ones, in pages out of order; what nobody wrote is NaN."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    total = [c + n for c, n in zip(contexts, portions)]
    per = [(t + page - 1) // page for t in total]
    order = torch.randperm(sum(per) + 3, generator=torch.Generator().manual_seed(seed)).tolist()
    table = torch.full((len(total), max(per)), -1, dtype=torch.int32)
    kp = torch.full((sum(per) + 3, G, page, dk), float("nan"), dtype=torch.bfloat16, device=DEV)
    vp = kp if shared else torch.full((sum(per) + 3, G, page, dv), float("nan"), dtype=torch.bfloat16, device=DEV)
    keys, values, at = [], [], 0
    for r, t in enumerate(total):
        k = randn(t, G, dk).bfloat16()
        v = k[:, :, :dv] if shared else randn(t, G, dv).bfloat16()
        for p in range(per[r]):
            table[r, p] = order[at]
            n = min(page, t - p * page)
            kp[order[at], :, :n] = k[p * page:p * page + n].transpose(0, 1)
            if not shared:
                vp[order[at], :, :n] = v[p * page:p * page + n].transpose(0, 1)
            at += 1
        keys.append(k.double())
        values.append(v.double())
    return randn(sum(portions), H, dk), keys, values, kp, vp, table.to(DEV), randn


def tiles_of(contexts, portions):
    tiles, at = [], 0
    for r, (c, n) in enumerate(zip(contexts, portions)):
        tiles += [(at + a, min(128, n - a), r, c + a) for a in range(0, n, 128)]
        at += n
    return i32(tiles + [(0, 0, 0, 0)])


OPTIONS = dict(window=0, chunk=0, softcap=0.0, keep_first=0, talk=False, gate=None, shared=False, page=16)


@pytest.mark.parametrize("H,G,dk,dv,options", [
    (16, 4, 64, 64, dict(talk=True, chunk=100, gate="head")),                 # 32 tokens x 4 heads
    (32, 8, 64, 64, dict(talk=True, chunk=1024, gate="head", page=64)),       # mixed queries of 512 columns
    (6, 3, 64, 40, dict(talk=True)),                                          # 64 tokens x 2 heads, 40 value columns
    (2, 1, 128, 72, dict(talk=True, window=70)),
    (16, 1, 288, 256, dict(shared=True, window=1024)),                        # 8 tokens x 16 heads, a chunk of low halves in shared memory
    (32, 1, 288, 256, dict(shared=True, window=90, page=8)),
    (3, 1, 72, 64, dict(shared=True)),                                        # one head a CTA
    (4, 4, 96, 32, dict(window=24, keep_first=3, softcap=8.0, gate="column")),
    (8, 2, 128, 128, dict(window=100, keep_first=70, softcap=20.0)),
    (8, 2, 48, 48, dict(chunk=7, gate="column", page=32)),
    (128, 1, 64, 64, dict(gate="head")),                                      # one token a CTA
])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_wide_portions(H, G, dk, dv, options, out_dtype):
    """Weights are rounded to bfloat16 (2^-9 of each, their sum too), values are of magnitude 1: a few 1e-3 at most; a bfloat16
    result is rounded once more."""
    from mlx_lm_b200 import ops
    o = {**OPTIONS, **options}
    contexts, portions = [0, 63, 64, 130, 0], [1, 129, 64, 35, 300]
    q, keys, values, kp, vp, table, randn = case(H, G, dk, dv, o["page"], o["shared"], contexts, portions, H + dk)
    T, scale = q.shape[0], 2.0 / math.sqrt(dk)
    talk = (torch.eye(H, device=DEV) + 0.3 * randn(H, H)) if o["talk"] else None
    gate = None if o["gate"] is None else randn(T, H if o["gate"] == "head" else H * dv).bfloat16()
    want, at = torch.empty(T, H, dv, dtype=torch.float64, device=DEV), 0
    for r, (c, n) in enumerate(zip(contexts, portions)):
        k = keys[r].repeat_interleave(H // G, dim=1)
        s = torch.einsum("ihd,jhd->hij", q[at:at + n].double(), k) * scale
        if talk is not None:
            s = torch.einsum("hg,gij->hij", talk.double(), s)
        if o["softcap"]:
            s = o["softcap"] * torch.tanh(s / o["softcap"])
        i, j = torch.arange(c, c + n, device=DEV)[:, None], torch.arange(c + n, device=DEV)[None, :]
        ok = j <= i
        if o["window"]:
            ok = ok & ((i - j < o["window"]) | (j < o["keep_first"]))
        if o["chunk"]:
            ok = ok & (i // o["chunk"] == j // o["chunk"])
        p = torch.softmax(s.masked_fill(~ok, -math.inf), dim=-1)
        want[at:at + n] = torch.einsum("hij,jhd->ihd", p, values[r].repeat_interleave(H // G, dim=1))
        at += n
    if gate is not None:
        want *= torch.sigmoid(gate.double().view(T, H, -1))
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    tiles = tiles_of(contexts, portions)
    kw = dict(window=o["window"], chunk=o["chunk"], softcap=o["softcap"], keep_first=o["keep_first"], talk=talk, gate=gate)
    assert ops.attention_wide_portions_supported(q.view(T, H * dk), dk, kp, vp, H, dk, dv, talk is not None)
    outs = []
    for first in range(2):                      # the second time without the first request: the same bits
        out = torch.full((T + 2, H * dv), 7.0, dtype=out_dtype, device=DEV)
        q2 = torch.zeros(T + 2, H * dk, device=DEV)
        q2[:T] = q.view(T, H * dk)
        kw2 = dict(kw, gate=None if gate is None else torch.cat([gate, gate[:2]]))
        ops.attention_wide_portions(q2, dk, tiles[first:], len(tiles) - first, 128, table, kp, vp, out, dv, H, dk, dv, scale, status,
                                    ops.current_stream(), **kw2)
        outs.append(out)
    assert int(status.item()) == 0
    assert bool((outs[0][T:] == 7.0).all()) and bool((outs[1][0] == 7.0).all()) and torch.equal(outs[0][1:], outs[1][1:])
    err = float((outs[0][:T].double().view(T, H, dv) - want).abs().max())
    assert err < (6e-3 if out_dtype == torch.float32 else 2e-2), err


def test_wide_portions_sizes():
    """What the kernel leaves to the others: rows of no whole 16 bytes, mixed heads that are no whole chunks, pages beyond a block,
    more value columns than tensor memory has, queries that 16-byte accesses cannot read."""
    from mlx_lm_b200 import ops
    pool = lambda G, w, page=16: torch.zeros(2, G, page, w, dtype=torch.bfloat16, device=DEV)
    q = torch.zeros(4, 4096, device=DEV)
    ok = lambda k, v, H, dk, dv, talk=False, q=q, qhs=None: ops.attention_wide_portions_supported(q, qhs or dk, k, v, H, dk, dv, talk)
    assert ok(pool(2, 64), pool(2, 64), 4, 64, 64, True) and not ok(pool(2, 48), pool(2, 48), 4, 48, 48, True)
    assert not ok(pool(2, 64, 128), pool(2, 64, 128), 4, 64, 64) and not ok(pool(2, 64, 4), pool(2, 64, 4), 4, 64, 64)
    lat = pool(1, 576)
    assert not ok(lat, lat, 4, 576, 512)
    assert not ok(pool(2, 64), pool(2, 64), 4, 64, 64, q=q[:, 1:4093], qhs=64) and not ok(pool(2, 64), pool(2, 64), 4, 62, 64)


def test_a_bounded_wait_that_runs_out():
    """A build with a short limit on its waits and one arrival left out (the softmax warps are never told of a tile's first scores): the
    kernel comes back by itself and says so, and the next launch of the same library, with the switch off, is right."""
    from ctypes import c_int
    from mlx_lm_b200 import ops
    from mlx_lm_b200.ops import build
    name = "attention_wide_tcgen05:MLXB_TEST_WAIT_TIMEOUT=1"
    lib = build.load(name)
    lib.mlxb_test_withhold_arrival.argtypes, lib.mlxb_test_withhold_arrival.restype = [c_int], c_int
    H, G, d, T = 4, 2, 64, 300
    q, keys, values, kp, vp, table, _ = case(H, G, d, d, 16, False, [0], [T], 9)
    tiles, status = tiles_of([0], [T]), torch.zeros(1, dtype=torch.int32, device=DEV)
    out, want = torch.zeros(T, H * d, device=DEV), torch.zeros(T, H * d, device=DEV)
    real = ops._call
    launch = lambda o: (ops.attention_wide_portions(q.view(T, H * d), d, tiles, len(tiles), 128, table, kp, vp, o, d, H, d, d, 0.2, status,
                                                    ops.current_stream()), torch.cuda.synchronize())
    launch(want)
    assert lib.mlxb_test_withhold_arrival(1) == 0
    try:
        ops._call = lambda lib_name, *a: real(name, *a)
        launch(out)
        assert int(status.item()) == ops.ST_WAIT_TIMEOUT and not out.any()
    finally:
        ops._call = real
        assert lib.mlxb_test_withhold_arrival(0) == 0
    status.zero_()
    try:
        ops._call = lambda lib_name, *a: real(name, *a)
        launch(out)
    finally:
        ops._call = real
    assert int(status.item()) == 0 and torch.equal(out, want)

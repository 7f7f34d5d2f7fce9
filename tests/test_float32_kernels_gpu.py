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


@pytest.mark.parametrize("Hq,Hkv,Dh,page,window,sink", [(4, 4, 16, 16, 0, False), (3, 3, 36, 4, 0, True), (6, 2, 64, 16, 0, False),
                                                        (2, 1, 64, 32, 70, True), (2, 2, 100, 16, 1, False), (2, 2, 128, 64, 200, False)])
def test_float32_attention_of_portions(ops, Hq, Hkv, Dh, page, window, sink):
    """Portions around the kernel's 64 queries and the step's tiles of 128, contexts around a block of 64 keys, behind pages that
    a window gave back; rows of no tile keep what they held."""
    lens, new = [0, 63, 64, 130, 5, 300], [1, 129, 64, 35, 200, 2]
    c = paged_case(torch.float32, lens=lens, new=new, Hq=Hq, Hkv=Hkv, Dh=Dh, page=page, seed=Dh)
    # pool rows of this step's own tokens hold what paged_case put there: both sides read the pools
    if window:
        for r, n in enumerate(lens):
            for p in range(max(0, n - window + 1) // page):
                c["bt"][r, p] = -1
    dev = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in c.items()}
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    sinks = torch.randn(Hq, generator=torch.Generator().manual_seed(1)).cuda() if sink else None
    first = [sum(new[:r]) for r in range(len(new))]
    tiles = [(first[r] + a, min(128, n - a), r, lens[r] + a) for r, n in enumerate(new) if r for a in range(0, n, 128)]
    tiles = torch.tensor(tiles + [(0, 0, 0, 0)], dtype=torch.int32).cuda()
    scale = Dh ** -0.5
    q, out = dev["qkv"][:, :Hq * Dh], torch.full((c["T"], Hq * Dh), 7.0, device="cuda")
    args = (dev["bt"], dev["k_pool"], dev["v_pool"])
    ops.attention_portions_f32(q, tiles, len(tiles), *args, out, Hq, scale, window, status, stream(), sinks=sinks)
    assert int(status.item()) == 0
    assert bool((out[:1] == 7.0).all())
    row_by_row = torch.empty_like(out)
    ops.attention_generic(q, dev["positions"], dev["token_req"], *args, row_by_row, Hq, scale, window, status, stream(), sinks=sinks)
    assert rel_err(out[1:], row_by_row[1:]) <= 3e-6
    if not sink and not window:
        want = R.attention(c["qkv"][:, :Hq * Dh], c["positions"], c["token_req"], c["bt"], c["k_pool"], c["v_pool"], Hq, scale, window)
        assert rel_err(out[1:], want[1:]) <= 3e-6


@pytest.mark.parametrize("window", [0, 70])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_float32_portions_keep_values_a_query_does_not_see_out(ops, bad, window):
    """One value that is not finite: queries before its position, and queries whose window has left it behind, come out as they
    do with a finite one, bit for bit; queries that see it do not."""
    H, Dh, n, at = 2, 64, 200, 91
    c = paged_case(torch.float32, lens=[0], new=[n], Hq=H, Hkv=H, Dh=Dh, page=16, seed=4)
    dev = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in c.items()}
    tiles = torch.tensor([(0, 128, 0, 0), (128, n - 128, 0, 128)], dtype=torch.int32).cuda()
    status, q = torch.zeros(1, dtype=torch.int32, device="cuda"), dev["qkv"][:, :H * Dh]
    outs = []
    for value in (1.0, bad):
        dev["v_pool"][int(c["bt"][0, at // 16]), :, at % 16] = value
        out = torch.empty(n, H * Dh, device="cuda")
        ops.attention_portions_f32(q, tiles, 2, dev["bt"], dev["k_pool"], dev["v_pool"], out, H, Dh ** -0.5, window, status, stream())
        outs.append(out)
    sees = torch.arange(n, device="cuda") >= at
    if window:
        sees &= torch.arange(n, device="cuda") < at + window
    assert torch.equal(outs[0][~sees], outs[1][~sees])
    assert not bool(torch.isfinite(outs[1][sees]).any())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,K", [(7, 4), (65, 50), (130, 64), (64, 127), (1030, 128), (70, 132), (96, 319), (40, 320), (40, 324), (64, 1001)])
def test_linear_on_cuda_cores(ops, dtype, N, K):
    """The small products' kernel and the tiles', around the sizes where one takes over from the other: sums of exact products (of
    bfloat16 numbers) in segments of 128, the same bits however many rows the call has, bfloat16 results those sums rounded once."""
    g = torch.Generator(device="cuda").manual_seed(N + K)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda").to(dtype)
    x, w, b = draw(1100, K), draw(N, K) / math.sqrt(K), draw(N).float()
    w = w.to(dtype)
    want = x.double() @ w.double().T + b
    whole = torch.empty(1100, N, device="cuda")
    ops.linear_generic(x, w, b, whole, stream())
    assert rel_err(whole, want) <= 1e-6
    for M in (1, 17, 63, 65, 130, 600):
        out = torch.empty(M, N, device="cuda")
        ops.linear_generic(x[:M], w, b, out, stream())
        assert torch.equal(out, whole[:M])
        short = torch.empty(M, N, device="cuda", dtype=dtype)
        ops.linear_generic(x[:M], w, b, short, stream())
        assert torch.equal(short, out.to(dtype))
    wide = draw(40, K + 3)                  # a row stride and a first column that no wide access can read
    out = torch.empty(40, N, device="cuda")
    ops.linear_generic(wide[:, 1:K + 1], w, None, out, stream())
    assert rel_err(out, wide[:, 1:K + 1].double() @ w.double().T) <= 1e-6


def test_float32_steps_of_one_shape_choose_their_attention(ops, tmp_path, monkeypatch):
    """The same number of rows after few and after many positions: each step's plan has the kernel that it was recorded with."""
    from helpers import CONFIG_A, make_model_dir
    from mlx_lm_b200.engine import Engine, StepEntry
    from mlx_lm_b200.weights import load_model
    make_model_dir(tmp_path, CONFIG_A, seed=2)
    model = load_model(str(tmp_path), dtype="float32")[0]
    tokens = torch.randint(0, 512, (128,), generator=torch.Generator().manual_seed(1)).tolist()

    def go():
        engine, out, calls, real = Engine(model, page_size=16, n_pages=16, max_requests=2), [], [], ops.attention_portions_f32
        monkeypatch.setattr(ops, "attention_portions_f32", lambda *a, **k: (calls.append(len(out)), real(*a, **k)))
        for rid in range(2):
            engine.add_request(rid)
            for at in range(0, 128, 8):
                out.append(engine.step([StepEntry(rid, tokens[at:at + 8], list(range(8)))]).clone())
            engine.finish(rid)
        monkeypatch.setattr(ops, "attention_portions_f32", real)
        return torch.cat(out), set(calls), engine.n_replayed

    got, chosen, replayed = go()
    assert len(chosen) == 1 and 0 < min(chosen) < 15 and replayed == 30      # one plan in tiles, one row by row
    monkeypatch.setattr(ops, "attention_portions_f32_pays", lambda *a, **k: False)
    want, chosen, _ = go()
    assert not chosen
    assert rel_err(got, want) <= 1e-5 and torch.equal(got[:8], want[:8])

"""The chunked kernels of the state-space layer and of the gated delta rule against the recurrences in 64 bits, token by
token, and against the scans: runs that end inside and at the edges of chunks of 64 rows, states carried from step to step,
single rows left out, sizes below and at the kernels' tiles, aligned and not."""
import pytest
import torch

import plain_lelatar as plain

pytestmark = pytest.mark.gpu

DEV = "cuda"


def arrays(runs):
    """(request of each row, first row of each request): request r brings ``runs[r]`` rows; two rows of padding at the end."""
    token_req = sum(([r] * n for r, n in enumerate(runs)), []) + [-1, -1]
    first = [0]
    for n in runs:
        first.append(first[-1] + n)
    first[-1] += 2
    return torch.tensor(token_req, dtype=torch.int32, device=DEV), torch.tensor(first, dtype=torch.int32, device=DEV)


def close(got, want, scan):
    """Within 2e-5 of the result's size everywhere, and as a whole no further off than twice what the scan is, which adds in
    another order (or 2e-7, a few roundings of 32 bits)."""
    size = float(want.abs().max())
    err, of_scan = float((got.double() - want).norm() / want.norm()), float((scan.double() - want).norm() / want.norm())
    assert float((got.double() - want).abs().max()) < 2e-5 * max(1.0, size)
    assert err < max(2 * of_scan, 2e-7), (err, of_scan)


RUNS = [[(64, 1, 130), (200, 65, 2)], [(2, 63, 1), (1, 300, 128)]]


@pytest.mark.parametrize("runs", RUNS)
@pytest.mark.parametrize("H,G,N,V,shift", [(4, 2, 24, 8, 0), (2, 1, 16, 40, 0), (6, 3, 70, 12, 0), (2, 1, 128, 64, 0), (2, 2, 64, 33, 1),
                                           (1, 1, 3, 5, 0)])
def test_state_space_chunks(H, G, N, V, shift, runs):
    from mlx_lm_b200 import ops
    torch.manual_seed(H * N + V)
    R, inner, GN = 3, H * V, G * N
    dt_bias, a_log, d_skip = torch.randn(H, device=DEV) * 0.5, torch.randn(H, device=DEV) * 0.5, torch.randn(H, device=DEV)
    slots = torch.tensor([2, 0, 3], dtype=torch.int32, device=DEV)
    pools = [torch.zeros(4, H, V, N, device=DEV) for _ in range(2)]
    S = torch.zeros(R, H, N, V, dtype=torch.float64, device=DEV)
    grp = torch.arange(H, device=DEV) // (H // G)
    for step in runs:
        token_req, first = arrays(step)
        T = token_req.numel()
        wide = (torch.randn(T, inner + 2 * GN + shift, device=DEV) * 0.7).to(torch.bfloat16)
        xbc, dt_raw = wide[:, shift:], torch.randn(T, H, device=DEV).to(torch.bfloat16)
        ys = [torch.zeros(T, inner, device=DEV) for _ in range(2)]
        args = lambda i: (xbc, 0, inner, inner + GN, dt_raw, dt_bias, a_log, d_skip, pools[i], slots, token_req, first, ys[i], H, G,
                          ops.current_stream())
        ops.mamba2_chunks(*args(0))
        assert all(float(ys[0][int(first[r])].abs().max()) == 0.0 for r, n in enumerate(step) if n == 1)
        ops.mamba2_scan(*args(0), max_run=1)
        ops.mamba2_scan(*args(1))
        want = torch.zeros(T, H, V, dtype=torch.float64, device=DEV)
        x = xbc.double()
        dt = plain.softplus(dt_raw.double() + dt_bias.double())
        a = torch.exp(-torch.exp(a_log.double()) * dt)
        for t in range(T - 2):
            r, xt = int(token_req[t]), x[t, :inner].view(H, V)
            B, C = x[t, inner:inner + GN].view(G, N)[grp], x[t, inner + GN:].view(G, N)[grp]
            S[r] = a[t, :, None, None] * S[r] + (dt[t, :, None] * B)[:, :, None] * xt[:, None, :]
            want[t] = torch.einsum("hnv,hn->hv", S[r], C) + d_skip.double()[:, None] * xt
        close(ys[0].view(T, H, V), want, ys[1].view(T, H, V))
    state = lambda p: p[slots.long()].transpose(2, 3)
    close(state(pools[0]), S, state(pools[1]))
    assert float(pools[0][1].abs().max()) == 0.0


@pytest.mark.parametrize("runs", RUNS)
@pytest.mark.parametrize("H,G,K,V,shift", [(4, 2, 16, 24, 0), (2, 2, 40, 8, 0), (2, 1, 64, 64, 0), (1, 1, 64, 33, 1), (3, 1, 7, 5, 0)])
@pytest.mark.parametrize("slow", [False, True])
def test_gated_delta_chunks(H, G, K, V, shift, runs, slow):
    """``slow``: keys that repeat, strong updates and hardly any decay, so that the triangular system is far from the identity."""
    from mlx_lm_b200 import ops
    torch.manual_seed(H * K + V)
    R, n_in = 3, 2 * G * K + H * V
    dt_bias, a_log = torch.randn(H, device=DEV) * 0.5 - (6.0 if slow else 0.0), torch.randn(H, device=DEV) * 0.5
    slots = torch.tensor([2, 0, 3], dtype=torch.int32, device=DEV)
    pools = [torch.zeros(4, H, V, K, device=DEV) for _ in range(2)]
    S = torch.zeros(R, H, K, V, dtype=torch.float64, device=DEV)
    grp = torch.arange(H, device=DEV) // (H // G)
    for step in runs:
        token_req, first = arrays(step)
        T = token_req.numel()
        wide = torch.randn(T, n_in + shift, device=DEV)
        if slow:
            wide[:, shift + G * K:shift + 2 * G * K] = wide[:1, shift + G * K:shift + 2 * G * K] + 0.3 * wide[:, shift + G * K:shift + 2 * G * K]
        wide = wide.to(torch.bfloat16)
        qkv = wide[:, shift:]
        b_raw = (torch.randn(T, H, device=DEV) + (3.0 if slow else 0.0)).to(torch.bfloat16)
        a_raw = torch.randn(T, H, device=DEV).to(torch.bfloat16)
        os_ = [torch.zeros(T, H * V, device=DEV) for _ in range(2)]
        args = lambda i: (qkv, 0, G * K, 2 * G * K, b_raw, a_raw, dt_bias, a_log, pools[i], slots, token_req, first, os_[i], H, G,
                          ops.current_stream())
        ops.gated_delta_chunks(*args(0))
        assert all(float(os_[0][int(first[r])].abs().max()) == 0.0 for r, n in enumerate(step) if n == 1)
        ops.gated_delta_scan(*args(0), max_run=1)
        ops.gated_delta_scan(*args(1))
        want = torch.zeros(T, H, V, dtype=torch.float64, device=DEV)
        x = qkv.double()
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
        q, k = unit(x[:, :G * K].reshape(T, G, K)) * K ** -0.5, unit(x[:, G * K:2 * G * K].reshape(T, G, K))
        v, beta = x[:, 2 * G * K:].reshape(T, H, V), torch.sigmoid(b_raw.double())
        decay = torch.exp(-torch.exp(a_log.double()) * plain.softplus(a_raw.double() + dt_bias.double()))
        for t in range(T - 2):
            r, kt, qt = int(token_req[t]), k[t, grp], q[t, grp]
            S[r] = decay[t, :, None, None] * S[r]
            u = beta[t, :, None] * (v[t] - torch.einsum("hkv,hk->hv", S[r], kt))
            S[r] = S[r] + kt[:, :, None] * u[:, None, :]
            want[t] = torch.einsum("hkv,hk->hv", S[r], qt)
        close(os_[0].view(T, H, V), want, os_[1].view(T, H, V))
    state = lambda p: p[slots.long()].transpose(2, 3)
    close(state(pools[0]), S, state(pools[1]))


BAD = [(70, 40, float("inf")), (3, 90, float("nan")), (64, 15, float("-inf"))]      # row, place among the row's inputs, value


@pytest.mark.parametrize("row,place,value", BAD)
@pytest.mark.parametrize("where", ["x", "B", "C", "dt"])
def test_state_space_rows_before_one_that_is_not_finite(row, place, value, where):
    """An infinity or a NaN in one row: the rows before it are those of a finite row, bit for bit, as token by token; where it
    goes into the state, so are the columns of the state that it does not reach, and those it reaches are not finite."""
    from mlx_lm_b200 import ops
    H, N, V, T = 2, 128, 64, 130
    torch.manual_seed(row)
    consts = [torch.randn(H, device=DEV) * 0.5 for _ in range(3)]
    token_req, first = arrays((T,))
    xbc0 = (torch.randn(T + 2, H * V + 2 * N, device=DEV) * 0.7).to(torch.bfloat16)
    dt0 = torch.randn(T + 2, H, device=DEV).to(torch.bfloat16)
    got = {}
    for kernel in ("chunks", "scan"):
        for v in (1.0, value):
            xbc, dt = xbc0.clone(), dt0.clone()
            if where == "dt":
                dt[row, 0] = abs(v)
            else:
                xbc[row, {"x": 0, "B": H * V, "C": H * V + N}[where] + place % 64] = v
            S, y = torch.zeros(1, H, V, N, device=DEV), torch.zeros(T + 2, H * V, device=DEV)
            f = ops.mamba2_chunks if kernel == "chunks" else ops.mamba2_scan
            f(xbc, 0, H * V, H * V + N, dt, *consts, S, torch.zeros(1, dtype=torch.int32, device=DEV), token_req, first, y, H, 1,
              ops.current_stream())
            got[kernel, v == 1.0] = y, S
    for kernel in ("chunks", "scan"):
        (y, S), (fy, fS) = got[kernel, False], got[kernel, True]
        assert torch.equal(y[:row], fy[:row])
        assert not bool(torch.isfinite(y[row]).all())
        # what the value does not reach (other columns, other heads), and what it does, as token by token
        reached = torch.isfinite(got["scan", False][0])
        assert torch.equal(torch.isfinite(y), reached)
        assert torch.equal(torch.isfinite(S), torch.isfinite(got["scan", False][1]))


def test_state_space_chunks_from_a_state_that_is_not_finite():
    """What comes out of an infinite entry of the state, or of one near the largest number, is what it is token by token."""
    from mlx_lm_b200 import ops
    H, N, V, T = 1, 64, 32, 40
    torch.manual_seed(9)
    consts = [torch.full((H,), -6.0, device=DEV), torch.zeros(H, device=DEV), torch.zeros(H, device=DEV)]
    token_req, first = arrays((T,))
    xbc = (torch.randn(T + 2, H * V + 2 * N, device=DEV) * 0.7).to(torch.bfloat16)
    xbc[:, H * V + N + 7] = 2.0 ** -20
    dt, ys = torch.zeros(T + 2, H, device=DEV, dtype=torch.bfloat16), []
    for f in (ops.mamba2_scan, ops.mamba2_chunks):
        S, y = torch.zeros(1, H, V, N, device=DEV), torch.zeros(T + 2, H * V, device=DEV)
        S[0, 0, 3, 5], S[0, 0, 4, 5], S[0, 0, 5, 7] = float("inf"), float("-inf"), 3.3e38
        f(xbc, 0, H * V, H * V + N, dt, *consts, S, torch.zeros(1, dtype=torch.int32, device=DEV), token_req, first, y, H, 1,
          ops.current_stream())
        ys.append((y[:T], S))
    for got, want in zip(ys[1], ys[0]):
        finite = torch.isfinite(want)
        assert bool(finite.any()) and not bool(finite.all())
        assert torch.equal(torch.where(finite, 0.0, got), torch.where(finite, 0.0, want))
        assert float((got - want)[finite].abs().max()) <= 2e-5 * float(want[finite].abs().max())


@pytest.mark.parametrize("row,place,value", BAD)
@pytest.mark.parametrize("where", ["v", "k", "q", "a", "b"])
def test_gated_delta_rows_before_one_that_is_not_finite(row, place, value, where):
    """As for the state-space layer; a decay's or an update strength's input is a NaN (an infinity gives a finite gate)."""
    from mlx_lm_b200 import ops
    H, K, V, T = 2, 64, 64, 130
    torch.manual_seed(row)
    consts = [torch.randn(H, device=DEV) * 0.5 for _ in range(2)]
    token_req, first = arrays((T,))
    qkv0 = torch.randn(T + 2, 2 * K + H * V, device=DEV).to(torch.bfloat16)
    ab0 = [torch.randn(T + 2, H, device=DEV).to(torch.bfloat16) for _ in range(2)]
    got = {}
    for kernel in ("chunks", "scan"):
        for v in (1.0, value):
            qkv, (a, b) = qkv0.clone(), (t.clone() for t in ab0)
            if where in "ab":
                (a if where == "a" else b)[row, 0] = v if v == 1.0 else float("nan")
            else:
                qkv[row, {"q": 0, "k": K, "v": 2 * K}[where] + place % 64] = v
            S, o = torch.zeros(1, H, V, K, device=DEV), torch.zeros(T + 2, H * V, device=DEV)
            f = ops.gated_delta_chunks if kernel == "chunks" else ops.gated_delta_scan
            f(qkv, 0, K, 2 * K, b, a, *consts, S, torch.zeros(1, dtype=torch.int32, device=DEV), token_req, first, o, H, 1,
              ops.current_stream())
            got[kernel, v == 1.0] = o, S
    for kernel in ("chunks", "scan"):
        (o, S), (fo, fS) = got[kernel, False], got[kernel, True]
        assert torch.equal(o[:row], fo[:row])
        assert not bool(torch.isfinite(o[row]).all())
        assert torch.equal(torch.isfinite(o), torch.isfinite(got["scan", False][0]))
        assert torch.equal(torch.isfinite(S), torch.isfinite(got["scan", False][1]))


def test_gated_delta_chunks_forget_at_an_infinite_step():
    """A decay of zero: what the state held is gone, and what follows is finite and as token by token."""
    from mlx_lm_b200 import ops
    H, K, V, T = 1, 32, 32, 70
    torch.manual_seed(5)
    consts = [torch.randn(H, device=DEV) * 0.5 for _ in range(2)]
    token_req, first = arrays((T,))
    qkv = torch.randn(T + 2, 2 * K + V, device=DEV).to(torch.bfloat16)
    a, b = (torch.randn(T + 2, H, device=DEV).to(torch.bfloat16) for _ in range(2))
    a[21, 0] = a[22, 0] = float("inf")
    outs = []
    for f in (ops.gated_delta_scan, ops.gated_delta_chunks):
        S, o = torch.ones(1, H, V, K, device=DEV), torch.zeros(T + 2, V, device=DEV)
        f(qkv, 0, K, 2 * K, b, a, *consts, S, torch.zeros(1, dtype=torch.int32, device=DEV), token_req, first, o, H, 1,
          ops.current_stream())
        outs.append((o[:T], S))
    for got, want in zip(outs[1], outs[0]):
        assert bool(torch.isfinite(want).all())
        assert float((got - want).abs().max()) <= 2e-5 * float(want.abs().max())


@pytest.mark.parametrize("kind", ["state space", "delta rule"])
def test_steps_of_single_rows_keep_the_order_of_kernels(kind):
    """A grid that finds no run of several rows ends no earlier than the kernel before it, whose result the kernel behind reads."""
    from mlx_lm_b200 import ops
    H, R = 4, 16
    a, w = torch.randn(128, 8192, device=DEV), torch.randn(2048, 8192, device=DEV)
    c, got, stream = torch.zeros(128, 2048, device=DEV), torch.zeros(128, 2048, device=DEV), ops.current_stream()
    rows = torch.arange(128, dtype=torch.int32, device=DEV)
    req, first = torch.arange(R, dtype=torch.int32, device=DEV), torch.arange(R + 1, dtype=torch.int32, device=DEV)
    x, g = torch.randn(R, 3 * H * 32, device=DEV).to(torch.bfloat16), torch.randn(R, H, device=DEV).to(torch.bfloat16)
    consts, S, y = [torch.zeros(H, device=DEV) for _ in range(3)], torch.zeros(R, H, 32, 32, device=DEV), torch.zeros(R, H * 32, device=DEV)
    for _ in range(10):
        c.zero_()
        ops.linear_generic(a, w, None, c, stream)
        if kind == "state space":
            ops.mamba2_chunks(x, 0, H * 32, 2 * H * 32, g, *consts, S, req, req, first, y, H, H, stream)
        else:
            ops.gated_delta_chunks(x, 0, H * 32, 2 * H * 32, g, g, *consts[:2], S, req, req, first, y, H, H, stream)
        ops.gather_rows(c, rows, got, stream)
        torch.cuda.synchronize()
        assert torch.equal(got, c) and float(c[-1].abs().max()) > 0
    assert float(y.abs().max()) == 0.0


@pytest.mark.parametrize("kind", ["state space", "delta rule"])
def test_every_run_goes_one_way(kind):
    """A rule that sends runs of 20 rows and less through the scan: with the requests that bring several rows listed, both kernels
    together leave what the scan alone does."""
    from mlx_lm_b200 import ops
    torch.manual_seed(2)
    H, N, V, runs = 4, 32, 48, (1, 20, 70, 2, 21, 1)
    rule = ops.ChunkRule(0, 10, 205, 0)
    assert [rule.chunks(n) for n in runs] == [False, False, True, False, True, False]
    token_req, first = arrays(runs)
    T, R = token_req.numel(), len(runs)
    slots = torch.arange(R, dtype=torch.int32, device=DEV)
    listed = torch.tensor([2, 4, 1, 3, -1, -1], dtype=torch.int32, device=DEV)
    x, g = torch.randn(T, H * V + 2 * H * N, device=DEV).to(torch.bfloat16), torch.randn(T, H, device=DEV).to(torch.bfloat16)
    consts = [torch.randn(H, device=DEV) * 0.5 for _ in range(3)]
    S0, out = torch.randn(R, H, V, N, device=DEV) * 0.1, []
    for both in (True, False):
        S, y = S0.clone(), torch.zeros(T, H * V, device=DEV)
        if kind == "state space":
            args = (x, 0, H * V, H * V + H * N, g, *consts, S, slots, token_req, first, y, H, H, ops.current_stream())
            chunks, scan = ops.mamba2_chunks, ops.mamba2_scan
        else:
            args = (x, 0, H * N, 2 * H * N, g, g, *consts[:2], S, slots, token_req, first, y, H, H, ops.current_stream())
            chunks, scan = ops.gated_delta_chunks, ops.gated_delta_scan
        if both:
            chunks(*args, requests=listed, rule=rule)
            assert [bool(y[int(first[r])].any()) for r in range(R)] == [rule.chunks(n) for n in runs]
            scan(*args, max_run=1, rule=rule)
        else:
            scan(*args)
        out.append((y, S))
    for got, want in zip(*out):
        assert float((got - want).abs().max()) <= 2e-5 * float(want.abs().max())
    for r, n in enumerate(runs):                       # what the scan did, it did as alone
        if not rule.chunks(n):
            assert torch.equal(out[0][0][int(first[r]):int(first[r]) + n], out[1][0][int(first[r]):int(first[r]) + n])
            assert torch.equal(out[0][1][r], out[1][1][r])


def test_a_plan_belongs_to_its_runs(tmp_path, monkeypatch):
    """Steps of the same shape (rows, requests, tiles) whose runs go different ways: each re-issues a plan of its own."""
    from lelatar_cases import CONFIG_Q, make_dir, tokens
    from mlx_lm_b200 import ops
    from mlx_lm_b200.engine import Engine, StepEntry
    from mlx_lm_b200.weights import load_model
    make_dir(tmp_path, CONFIG_Q, seed=3)
    model = load_model(str(tmp_path), dtype="bfloat16")[0]
    steps = [(50, 14), (40, 24), (47, 17), (60, 3), (33, 18), (50, 14)]

    def go(limit):
        rule = ops.ChunkRule(0, 10, 10 * limit, 0)
        monkeypatch.setattr(ops, "chunk_rule", lambda *layer, sms=148: rule if any(rule.chunks(n) for n in layer[-1]) else None)
        engine, out, calls = Engine(model, page_size=16, n_pages=64, max_requests=4, max_len=512), [], []
        real = ops.mamba2_chunks
        monkeypatch.setattr(ops, "mamba2_chunks", lambda *a, **k: (calls.append(1), real(*a, **k)))
        for i, lengths in enumerate(steps):
            for r in range(2):
                engine.add_request((i, r))
            out.append(engine.step([StepEntry((i, r), tokens(n, CONFIG_Q["vocab"], n), [n - 1]) for r, n in enumerate(lengths)]).clone())
            for r in range(2):
                engine.finish((i, r))
        monkeypatch.setattr(ops, "mamba2_chunks", real)
        return torch.stack(out), len(calls), engine.n_replayed

    want, n, replayed = go(1 << 20)
    assert n == 0 and replayed == len(steps) - 1
    got, n, replayed = go(45)
    assert n > 0 and replayed == len(steps) - 2
    assert float((got - want).abs().max()) <= 0.06 * float(want.abs().max())
    by_rows = [bool((got[i] == want[i]).all()) for i in range(len(steps))]
    assert by_rows[1] and by_rows[4] and not all(by_rows)


def test_short_prompts_launch_no_chunks(tmp_path, monkeypatch):
    from lelatar_cases import CONFIG_Q, make_dir, tokens
    from mlx_lm_b200 import ops
    from mlx_lm_b200.engine import Engine, StepEntry
    from mlx_lm_b200.weights import load_model
    make_dir(tmp_path, CONFIG_Q, seed=3)
    engine = Engine(load_model(str(tmp_path), dtype="bfloat16")[0], page_size=16, n_pages=64, max_requests=4, max_len=512)
    seen = []
    for name in ("mamba2_chunks", "gated_delta_chunks"):
        monkeypatch.setattr(ops, name, lambda *a, name=name, real=getattr(ops, name), **k: (seen.append(name), real(*a, **k)))
    for rid, n in (("short", 8), ("long", 200)):
        engine.add_request(rid)
        engine.step([StepEntry(rid, tokens(n, CONFIG_Q["vocab"], n), [n - 1])])
        assert bool(seen) == (rid == "long")

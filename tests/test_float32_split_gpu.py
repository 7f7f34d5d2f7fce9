"""The float32 linear kernel on tensor cores (operands in three bfloat16 parts) at the edges of its tiles and blocks, against float64."""
import math

import pytest
import torch

from helpers import CONFIG_C, make_model_dir, random_tokens
from test_kernels_gpu import rel_err, stream

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from mlx_lm_b200 import ops
    return ops


@pytest.mark.parametrize("width", ["64", "128"])
@pytest.mark.parametrize("M,N,K", [(1, 64, 256), (17, 7, 4), (127, 65, 60), (128, 128, 64), (129, 130, 68), (300, 200, 1000),
                                   (257, 1030, 260), (1100, 512, 128), (64, 3072, 132), (40, 24, 4100)])
def test_float32_linear_in_parts(ops, M, N, K, width, monkeypatch):
    """What is left out of a product is 2^-25.4 of it in the mean square (2^-22 at worst) and of either sign, a block of 64 of K takes four
    cut-off sums of 2^-23 at most, the blocks' sums K / 64 roundings of 2^-24: a few 1e-7 over the whole result at most; the same bits for
    both tile widths and however many rows of this kernel."""
    monkeypatch.setenv("MLXB_SPLIT_BN", width)
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w, b, res = draw(M, K), draw(N, K) / math.sqrt(K), draw(N), draw(M, N)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    want = x.double() @ w.double().T
    out = torch.empty(M, N, device="cuda")
    ops.linear_split(x, w, None, out, status, stream())
    assert rel_err(out, want) <= 5e-7
    if M < 130:
        more = torch.empty(M + 140, N, device="cuda")
        monkeypatch.setenv("MLXB_SPLIT_BN", "128" if width == "64" else "64")
        ops.linear_split(torch.cat([x, draw(140, K)]), w, None, more, status, stream())
        assert torch.equal(more[:M], out)
    ops.linear_split(x, w, b, out, status, stream(), epilogue=ops.EPI_GELU_NEW, residual=res)
    plain = torch.empty(M, N, device="cuda")
    ops.linear_generic(x, w, b, plain, stream(), epilogue=ops.EPI_GELU_NEW, residual=res)
    assert rel_err(out, plain) <= 1e-6
    inplace = res.clone()
    ops.linear_split(x, w, None, inplace, status, stream(), residual=inplace)
    assert rel_err(inplace, want + res) <= 5e-7
    wide = draw(M, K + 4)                            # a row stride of its own
    ops.linear_split(wide[:, 4:], w, b, out, status, stream())
    assert rel_err(out, wide[:, 4:].double() @ w.double().T + b) <= 1e-6
    assert int(status.item()) == 0


def test_float32_linear_in_parts_of_numbers_at_the_ends(ops):
    """Infinities, NaN, numbers that bfloat16 rounds to infinity, and tiny ones: as in plain float32."""
    g = torch.Generator(device="cuda").manual_seed(1)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w = draw(200, 512), draw(130, 512) / 16
    x[3, 5], x[7, 9], w[11, 20], x[50, 1] = math.inf, math.nan, -math.inf, 3.4e38
    w[12], w[13, 5], w[14, 5] = w[12].bfloat16().float(), 0.0, 0.5
    w[:, 1].clamp_(-0.5, 0.5)
    x[60] *= 1e-30
    status, out, plain = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.empty(200, 130, device="cuda"), torch.empty(200, 130, device="cuda")
    ops.linear_split(x, w, None, out, status, stream())
    ops.linear_generic(x, w, None, plain, stream())
    assert int(status.item()) == 0
    assert torch.equal(torch.isnan(out), torch.isnan(plain)) and torch.equal(torch.isinf(out), torch.isinf(plain))
    assert torch.equal(out[torch.isinf(out)], plain[torch.isinf(plain)])
    fine = torch.isfinite(plain)
    assert bool(fine[50].any()) and bool(fine[60].any())
    for r in (0, 50, 60, 199):
        assert rel_err(out[r][fine[r]], plain[r][fine[r]]) <= 1e-6


def test_float32_linear_in_parts_with_many_rows_that_are_not_finite(ops):
    """Every number of such rows among the 32 that a warp finishes: as in plain float32, and the other rows' bits as without them."""
    M, N, K = 300, 150, 260
    g = torch.Generator(device="cuda").manual_seed(6)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda") / 16
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, clean, plain = (torch.empty(M, N, device="cuda") for _ in range(3))
    ops.linear_split(x, w, None, clean, status, stream())
    bad = list(range(32)) + [40] + list(range(64, 71)) + list(range(97, 100)) + [130]
    x[:32, 3], x[40], x[64:71, 259], x[97:100, 7] = math.nan, math.nan, math.inf, -math.inf
    x[130], x[130, 1] = 0.0, 3.4e38                  # bfloat16 rounds it to infinity
    ops.linear_split(x, w, None, out, status, stream())
    ops.linear_generic(x, w, None, plain, stream())
    assert int(status.item()) == 0
    others = [r for r in range(M) if r not in bad]
    assert torch.equal(out[others], clean[others])
    assert torch.equal(torch.isnan(out), torch.isnan(plain)) and torch.equal(torch.isinf(out), torch.isinf(plain))
    assert torch.equal(out[64:100][torch.isinf(plain[64:100])], plain[64:100][torch.isinf(plain[64:100])])
    assert rel_err(out[130], plain[130]) <= 1e-6
    b, res = torch.randn(N, generator=g, device="cuda"), torch.randn(M, N, generator=g, device="cuda")
    inplace, want = res.clone(), res.clone()
    ops.linear_split(x, w, b, inplace, status, stream(), epilogue=ops.EPI_GELU_NEW, residual=inplace)
    ops.linear_generic(x, w, b, want, stream(), epilogue=ops.EPI_GELU_NEW, residual=want)
    assert torch.equal(torch.isnan(inplace), torch.isnan(want)) and torch.equal(torch.isinf(inplace), torch.isinf(want))
    assert rel_err(inplace[130], want[130]) <= 1e-6 and rel_err(inplace[others], want[others]) <= 1e-6


def test_a_bounded_wait_that_runs_out(ops):
    """A build with a short limit on its waits and one arrival left out (the sums' warps are never told of the first accumulator): the
    kernel comes back by itself and says so, and the next launch of the same library, with the switch off, is right."""
    from ctypes import c_int, c_void_p
    from mlx_lm_b200.ops import build
    name = "gemm_split:MLXB_TEST_WAIT_TIMEOUT=1"
    lib = build.load(name)
    lib.mlxb_test_withhold_arrival.argtypes, lib.mlxb_test_withhold_arrival.restype = [c_int], c_int
    M, N, K = 300, 200, 512
    g = torch.Generator(device="cuda").manual_seed(2)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    out, status = torch.zeros(M, N, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")

    def launch():
        ops._call(name, "mlxb_linear_split", [c_void_p] * 5 + [c_int] * 6 + [c_void_p, c_void_p], x.data_ptr(), w.data_ptr(), None, None,
                  out.data_ptr(), M, N, K, K, N, ops.EPI_NONE, status.data_ptr(), stream())
        torch.cuda.synchronize()

    assert lib.mlxb_test_withhold_arrival(1) == 0
    try:
        launch()
        assert int(status.item()) == ops.ST_WAIT_TIMEOUT and not out.any()
    finally:
        assert lib.mlxb_test_withhold_arrival(0) == 0
    status.zero_()
    launch()
    assert int(status.item()) == 0 and rel_err(out, x.double() @ w.double().T) <= 5e-7


def test_rows_of_a_step_whatever_others_share_it(tmp_path):
    """A float32 engine: the logits of a request that brings one token, and of one that brings several, have the same bits alone and
    beside others, few or many, before or behind them among the step's entries."""
    from mlx_lm_b200.engine import Engine, StepEntry
    from mlx_lm_b200.weights import load_model
    make_model_dir(str(tmp_path), CONFIG_C, 11, peaky=3.0)
    model, _ = load_model(str(tmp_path), dtype="float32", device="cuda:0")
    V, N = CONFIG_C["vocab_size"], 40
    engine = Engine(model, page_size=16, n_pages=4 * N + 64, max_requests=N + 1)
    for r in range(N):
        engine.add_request(r)
        engine.step([StepEntry(r, random_tokens(20 + r, V, r))])
    engine.add_request("p")
    prompt = random_tokens(270, V, 77)
    first, rest = prompt[:170], prompt[170:]

    def logits(ones, place=None, wanted=(0, 99)):
        entries = [StepEntry(r, [3 * r + 1], [0]) for r in ones]
        if place is not None:
            engine.step([StepEntry("p", first)])
            entries.insert(place, StepEntry("p", rest, list(wanted)))
        got = engine.step(entries)
        by, at = {}, 0
        for e in entries:
            by[e.rid] = got[at:at + len(e.want)].clone()
            at += len(e.want)
        for r in ones:
            engine.cache.truncate(r, 20 + r)
        engine.cache.truncate("p", 0)
        return by

    alone = {r: logits([r])[r] for r in range(N)}
    portion = logits([], 0)["p"]
    assert float((alone[0] - alone[1]).abs().max()) > 1e-3
    for ones, place in ((range(16), None), (range(17), None), (range(N), None), ([5], 0), (range(17), 17), (range(N), 3), ([2, 1], 1)):
        by = logits(list(ones), place)
        for r in ones:
            assert torch.equal(by[r], alone[r]), (r, len(ones), place)
        if place is not None:
            assert torch.equal(by["p"], portion), (len(ones), place)
    every = logits([4], 0, range(100))["p"]                     # more wanted rows: the output head runs more rows
    assert torch.equal(every[[0, 99]], portion)
    engine.check_status()

"""The gated delta rule in two passes (what needs no state for all chunks of a run side by side): everything that is asked of the
one kernel, by its own tests, and the choice between the two."""
import pytest
import torch

import test_recurrent_chunks_gpu as one

pytestmark = pytest.mark.gpu


@pytest.fixture
def two_passes(monkeypatch):
    from mlx_lm_b200 import ops
    real, calls = ops.gated_delta_chunks, []

    def wrapped(*a, requests=None, **k):
        n = a[9].numel() if requests is None else requests.numel()
        scratch = torch.full((ops.gated_delta_chunks_scratch(ops.delta_chunk_jobs(a[0].shape[0], n), a[13]),), float("nan"), device="cuda")
        calls.append(n)
        return real(*a, requests=requests, scratch=scratch, **k)
    monkeypatch.setattr(ops, "gated_delta_chunks", wrapped)
    yield calls
    assert calls


@pytest.mark.parametrize("runs", one.RUNS)
@pytest.mark.parametrize("H,G,K,V,shift", [(4, 2, 16, 24, 0), (2, 2, 40, 8, 0), (2, 1, 64, 64, 0), (1, 1, 64, 33, 1), (3, 1, 7, 5, 0)])
@pytest.mark.parametrize("slow", [False, True])
def test_against_the_recurrence(H, G, K, V, shift, runs, slow, two_passes):
    one.test_gated_delta_chunks(H, G, K, V, shift, runs, slow)


@pytest.mark.parametrize("row,place,value", one.BAD)
@pytest.mark.parametrize("where", ["v", "k", "q", "a", "b"])
def test_rows_before_one_that_is_not_finite(row, place, value, where, two_passes):
    one.test_gated_delta_rows_before_one_that_is_not_finite(row, place, value, where)


def test_an_infinite_step(two_passes):
    one.test_gated_delta_chunks_forget_at_an_infinite_step()


def test_order_of_kernels_and_of_runs(two_passes):
    one.test_steps_of_single_rows_keep_the_order_of_kernels("delta rule")
    one.test_every_run_goes_one_way("delta rule")


def test_error_against_64_bits_is_no_larger():
    """1000 rows, random and slow: no further from 64 bits than the one kernel, up to the tenth that the order of roundings moves."""
    from mlx_lm_b200 import ops
    errors = {}
    for slow in (False, True):
        H, K, V, T = 4, 64, 64, 1000
        torch.manual_seed(11)
        dt_bias, a_log = torch.randn(H, device="cuda") * 0.5 - (6.0 if slow else 0.0), torch.randn(H, device="cuda") * 0.5
        token_req, first = one.arrays((T,))
        wide = torch.randn(T + 2, 2 * K + H * V, device="cuda")
        if slow:
            wide[:, K:2 * K] = wide[:1, K:2 * K] + 0.3 * wide[:, K:2 * K]
        qkv = wide.to(torch.bfloat16)
        b = (torch.randn(T + 2, H, device="cuda") + (3.0 if slow else 0.0)).to(torch.bfloat16)
        a = torch.randn(T + 2, H, device="cuda").to(torch.bfloat16)
        x = qkv.double()
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
        q, k = unit(x[:, :K]) * K ** -0.5, unit(x[:, K:2 * K])
        v, beta = x[:, 2 * K:].view(-1, H, V), torch.sigmoid(b.double())
        decay = torch.exp(-torch.exp(a_log.double()) * one.plain.softplus(a.double() + dt_bias.double()))
        S, want = torch.zeros(H, K, V, dtype=torch.float64, device="cuda"), torch.zeros(T, H, V, dtype=torch.float64, device="cuda")
        for t in range(T):
            S = decay[t, :, None, None] * S
            u = beta[t, :, None] * (v[t] - torch.einsum("hkv,k->hv", S, k[t]))
            S = S + k[t][None, :, None] * u[:, None, :]
            want[t] = torch.einsum("hkv,k->hv", S, q[t])
        scratch = torch.empty(ops.gated_delta_chunks_scratch(ops.delta_chunk_jobs(T + 2, 1), H), device="cuda")
        for name, f, kw in (("two", ops.gated_delta_chunks, dict(scratch=scratch)), ("one", ops.gated_delta_chunks, {}),
                            ("scan", ops.gated_delta_scan, {})):
            state, o = torch.zeros(1, H, V, K, device="cuda"), torch.zeros(T + 2, H * V, device="cuda")
            f(qkv, 0, K, 2 * K, b, a, dt_bias, a_log, state, torch.zeros(1, dtype=torch.int32, device="cuda"), token_req, first, o, H, 1,
              ops.current_stream(), **kw)
            errors[slow, name] = (float((o[:T].view(T, H, V) - want).norm() / want.norm()),
                                  float((state[0].transpose(1, 2) - S).norm() / S.norm()))
    print(errors)
    for slow in (False, True):
        for two, one_kernel in zip(errors[slow, "two"], errors[slow, "one"]):
            assert two < 1.1 * one_kernel, errors

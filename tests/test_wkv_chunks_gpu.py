"""The wkv recurrence with the chunks of a run side by side, against the recurrence in float64 token by token."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def i32(a):
    return torch.tensor(a, dtype=torch.int32, device=DEV)


def reference(r, k, v, d, u, S):
    w, o = torch.exp(-torch.exp(d)), torch.empty(r.shape[0], *v.shape[1:], dtype=torch.float64, device=DEV)
    for t in range(r.shape[0]):
        kv = k[t, :, :, None] * v[t, :, None, :]
        o[t] = torch.einsum("hk,hkv->hv", r[t], S + u[:, :, None] * kv)
        S = w[t, :, :, None] * S + kv
    return o, S


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,K,V,runs", [
    (2, 64, 64, [1, 63, 64, 65, 128, 129, 300]),      # around a chunk, several chunks
    (3, 16, 16, [70, 1, 200]), (2, 32, 34, [130, 17]), (1, 128, 70, [65, 192]), (1, 256, 130, [66, 5]),
    (2, 64, 64, [1] * 40 + [100] + [1] * 7),          # requests beyond a warp's lanes
    (1, 64, 64, [1] * 33 + [577, 64, 3700, 1]),       # the states of all chunks before the second pass
    (2, 48, 48, [70, 3]), (2, 64, 63, [70, 3]),       # token by token: rows that are no power of two, odd columns
])
def test_wkv_chunks(dtype, H, K, V, runs):
    """Float32 products and sums: an output is a sum of K products, a state of as many terms as its decays let through; the
    same state and outputs as token by token up to roundings of 6e-8 each."""
    from mlx_lm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(K + V + len(runs))
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    T, pad = sum(runs), 2
    Kp, Vp = (K * H + 7) // 8 * 8, (V * H + 7) // 8 * 8
    rkv = randn(T + pad, 2 * Kp + Vp).to(dtype)
    d = randn(T + pad, H * K) * 1.5 - 1.5
    u, n = randn(H, K) * 0.5, len(runs)
    pool = randn(n + 3, H, V, K)
    slots = torch.randperm(n + 3, generator=torch.Generator().manual_seed(n))[:n].tolist()
    token_req = i32([r for r, m in enumerate(runs) for _ in range(m)] + [-1] * pad)
    first = [0]
    for m in runs:
        first.append(first[-1] + m)
    first = i32(first[:-1] + [T + pad])               # rows that pad the step belong to nobody
    before, scan_pool = pool.clone(), pool.clone()
    o, by_token = (torch.full((T + pad, H * V), 7.0, device=DEV) for _ in range(2))
    long_rows = T + pad - n                           # all but the first of every request
    scratch = torch.full((max(4, ops.wkv_chunks_scratch(long_rows, H, K, V)),), float("nan"), device=DEV)
    args = (rkv, 0, Kp, 2 * Kp, d, u)
    ops.wkv_chunks(*args, pool, i32(slots), token_req, first, o, H, scratch, ops.current_stream(), long_rows=long_rows)
    ops.wkv_scan(*args, scan_pool, i32(slots), token_req, first, by_token, H, ops.current_stream())
    at = 0
    for i, m in enumerate(runs):
        part = lambda a, w: rkv[at:at + m, a:a + H * w].double().view(m, H, w)
        want, S = reference(part(0, K), part(Kp, K), part(2 * Kp, V), d[at:at + m].double().view(m, H, K), u.double(),
                            before[slots[i]].double().transpose(1, 2))
        for got, states in ((o, pool), (by_token, scan_pool)):
            got = got[at:at + m].double().view(m, H, V)
            assert float((got - want).norm() / want.norm()) < 1e-6
            end = states[slots[i]].double().transpose(1, 2)
            assert float((end - S).norm() / S.norm()) < 1e-6
        at += m
    assert bool((o[T:] == 7.0).all())
    rest = [s for s in range(n + 3) if s not in slots]
    assert torch.equal(pool[rest], before[rest])


def test_wkv_chunks_of_a_run_beside_others():
    """A run's bits do not depend on the step's rows, with the states of all chunks made before the second pass or walked through by it."""
    from mlx_lm_b200 import ops
    H, K, runs = 2, 64, [700, 3600]
    g = torch.Generator(device=DEV).manual_seed(5)
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    rkv, d, u = randn(sum(runs), 3 * H * K), randn(sum(runs), H * K), randn(H, K)
    outs = []
    for T, first in ((700, [0, 700]), (4300, [0, 700, 4300])):
        n = len(first) - 1
        o, pool = torch.empty(T, H * K, device=DEV), torch.zeros(n, H, K, K, device=DEV)
        scratch = torch.empty(ops.wkv_chunks_scratch(T, H, K, K), device=DEV)
        ops.wkv_chunks(rkv[:T], 0, H * K, 2 * H * K, d[:T], u, pool, i32(list(range(n))),
                       i32([0] * 700 + [1] * (T - 700)), i32(first), o, H, scratch, ops.current_stream())
        outs.append((o[:700], pool[0]))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


def test_wkv_chunks_keep_what_is_not_finite_to_the_rows_behind_it():
    from mlx_lm_b200 import ops
    H, K, T, at = 2, 64, 200, 70
    g = torch.Generator(device=DEV).manual_seed(3)
    randn = lambda *s: torch.randn(*s, generator=g, device=DEV)
    rkv, d, u = randn(T, 3 * H * K), randn(T, H * K), randn(H, K)
    outs = []
    for bad in (1.0, float("nan")):
        rkv[at, H * K + 5] = bad                      # a key of the first head
        o, pool = torch.empty(T, H * K, device=DEV), torch.zeros(1, H, K, K, device=DEV)
        scratch = torch.empty(ops.wkv_chunks_scratch(T, H, K, K), device=DEV)
        ops.wkv_chunks(rkv, 0, H * K, 2 * H * K, d, u, pool, i32([0]), i32([0] * T), i32([0, T]), o, H, scratch, ops.current_stream())
        outs.append(o)
    assert torch.equal(outs[0][:at], outs[1][:at]) and torch.equal(outs[0][:, K:], outs[1][:, K:])
    assert not bool(torch.isfinite(outs[1][at:, :K]).any())

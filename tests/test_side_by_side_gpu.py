"""Single rows and portions of one step whose kernels run side by side: the same bits as one after the other."""
import pytest
import torch

from test_kernels_gpu import paged_case, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,singles,portion", [(16, 5, 40), (20, 31, 256), (12, 100, 300), (2, 3, 129)])
def test_rows_beside_portions(H, singles, portion):
    """With the queries, and the pages of all rows, written by a kernel right before (what both kernels have to wait for), and the
    results read by one right after."""
    from mlx_lm_b200 import ops
    lens, new = [70 + 7 * i for i in range(singles)] + [130], [1] * singles + [portion]
    c = paged_case(torch.bfloat16, lens=lens, new=new, Hq=H, Hkv=H, Dh=64, page=16, seed=H)
    dev = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in c.items()}
    T, D = c["T"], H * 64
    status, scale = torch.zeros(1, dtype=torch.int32, device="cuda"), 64 ** -0.5
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    tiles = i32([(singles + a, min(128, portion - a), singles, 130 + a) for a in range(0, portion, 128)])
    rows, row_tiles = i32(list(range(singles))), i32([(r, 1, r, lens[r]) for r in range(singles)])
    scratch = torch.zeros(ops.attention_decode_scratch(singles, H, 64, 1024), device="cuda")
    counters = torch.zeros(singles * H, dtype=torch.int32, device="cuda")
    src = dev["qkv"].contiguous()
    kp, vp = dev["k_pool"], dev["v_pool"]
    junk = torch.randn(2048, 2048, device="cuda")

    def go(beside, on_tensor_cores, qkv):
        out = torch.full((T, D), 7.0, dtype=torch.bfloat16, device="cuda")
        args = (dev["bt"], kp, vp, out, H, scale, 0, status, stream())
        ops.kv_write(qkv[:, D:2 * D], qkv[:, 2 * D:], dev["positions"], dev["token_req"], dev["bt"], kp, vp, status, stream())
        q = qkv[:, :D]
        portions = lambda: ops.attention_portions(q, tiles, len(tiles), *args, beside=beside)
        if beside:
            portions()
        else:
            torch.cuda.synchronize()
        if on_tensor_cores:
            ops.attention_rows(q, row_tiles, singles, *args, beside=beside)
        else:
            ops.attention_decode(q, dev["positions"], dev["token_req"], dev["bt"], kp, vp, out, H, scale, 0, scratch, counters, 1024, status,
                                 stream(), rows=rows, beside=beside)
        if not beside:
            torch.cuda.synchronize()
            portions()
            torch.cuda.synchronize()
        copy = torch.empty_like(out)
        ops.gather_rows(out, torch.arange(T, dtype=torch.int32, device="cuda"), copy, stream())
        return copy

    for on_tensor_cores in (False, True):
        for k in range(8):
            qkv = torch.roll(src, k, 0).contiguous()         # other queries, keys and values at the same places
            want = go(False, on_tensor_cores, qkv)
            kp_now = kp.clone()
            go(False, on_tensor_cores, torch.zeros_like(qkv))
            for _ in range(3):
                junk @ junk
                got = go(True, on_tensor_cores, qkv)
                assert torch.equal(got, want), (on_tensor_cores, k)
            assert torch.equal(kp, kp_now)
    assert int(status.item()) == 0

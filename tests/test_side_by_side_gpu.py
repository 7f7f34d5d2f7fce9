"""Single rows and portions of one step whose kernels run side by side: the same bits as one after the other."""
import numpy as np
import pytest
import torch

from helpers import CONFIG_C, Trace, make_model_dir, max_live_tokens, mixed_schedule, random_tokens, run_trace
from test_kernels_gpu import paged_case, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,singles,portion", [(16, 5, 40), (20, 31, 256), (12, 100, 300), (2, 3, 129)])
def test_rows_beside_portions(H, singles, portion):
    """The queries (one buffer, every time other contents) and the pages of all rows are written by kernels of the library right before,
    the results read by one right after.  Contexts of up to 950 positions: a row's own position lies in any of the batches of keys
    that the kernel of few rows reads one after the other."""
    from mlx_lm_b200 import ops
    lens, new = [70 + 211 * i % 881 for i in range(singles)] + [130], [1] * singles + [portion]
    c = paged_case(torch.bfloat16, lens=lens, new=new, Hq=H, Hkv=H, Dh=64, page=16, seed=H)
    dev = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in c.items()}
    T, D = c["T"], H * 64
    status, scale = torch.zeros(1, dtype=torch.int32, device="cuda"), 64 ** -0.5
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    tiles = i32([(singles + a, min(128, portion - a), singles, 130 + a) for a in range(0, portion, 128)])
    rows, row_tiles = i32(list(range(singles))), i32([(r, 1, r, lens[r]) for r in range(singles)])
    scratch = torch.zeros(ops.attention_decode_scratch(singles, H, 64, 1024), device="cuda")
    counters = torch.zeros(singles * H, dtype=torch.int32, device="cuda")
    src, every_row = dev["qkv"].contiguous(), torch.arange(T, dtype=torch.int32, device="cuda")
    kp, vp = dev["k_pool"], dev["v_pool"]
    qkv = torch.zeros_like(src)
    junk = torch.randn(2048, 2048, device="cuda")

    def go(beside, on_tensor_cores, source):
        out = torch.full((T, D), 7.0, dtype=torch.bfloat16, device="cuda")
        copy = torch.empty_like(out)
        args = (dev["bt"], kp, vp, out, H, scale, 0, status, stream())
        junk @ junk                                          # (what is launched next is on its way before the device gets to it)
        ops.gather_rows(source, every_row, qkv, stream())
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
        ops.gather_rows(out, every_row, copy, stream())
        return copy

    for on_tensor_cores in (False, True):
        for k in range(8):
            source = torch.roll(src, k, 0).contiguous()      # other queries, keys and values at the same places
            want = go(False, on_tensor_cores, source)
            kp_now = kp.clone()
            for _ in range(3):
                go(False, on_tensor_cores, torch.zeros_like(source))
                assert not qkv.any() and not torch.equal(kp, kp_now)
                got = go(True, on_tensor_cores, source)
                assert torch.equal(got, want), (on_tensor_cores, k)
                assert torch.equal(kp, kp_now)
    assert int(status.item()) == 0


def test_mixed_steps_replayed(tmp_path):
    """The same mixed steps three times through one engine, recorded and replayed, and once with every kernel waiting for the one before
    it (MLXB_PDL=0, in a process of its own): the same bits."""
    from mlx_lm_b200.engine import Engine, StepEntry
    from mlx_lm_b200.weights import load_model
    make_model_dir(str(tmp_path / "model"), CONFIG_C, 7, peaky=3.0)
    V = CONFIG_C["vocab_size"]
    model, _ = load_model(str(tmp_path / "model"), dtype="bfloat16", device="cuda:0")
    engine = Engine(model, page_size=16, n_pages=256, max_requests=8)
    lengths = (300, 17, 290)
    for r, n in enumerate(lengths):
        engine.add_request(r)
        engine.step([StepEntry(r, random_tokens(n, V, r))])
    engine.add_request(3)
    seen, replayed = [], engine.n_replayed
    for _ in range(3):
        seen.append([])
        for k in range(3):
            entries = [StepEntry(r, [k + r], [0]) for r in range(3)]
            seen[-1].append(engine.step(entries + [StepEntry(3, random_tokens(100, V, 50 + k), [0, 99])]).clone())
        for r, n in enumerate(lengths + (0,)):
            engine.cache.truncate(r, n)
    engine.check_status()
    assert engine.n_replayed - replayed >= 6
    for again in seen[1:]:
        assert all(torch.equal(a, b) for a, b in zip(seen[0], again))
    trace = Trace()
    reqs = {f"r{i}": random_tokens(n, V, 20 + i) for i, n in enumerate((130, 300, 290))}
    mixed_schedule(trace, list(reqs.items()), seed=3, sizes=(1, 130, 1, 1, 16, 1, 1, 100, 1, 2, 65, 1, 1))
    outs = [run_trace(str(tmp_path / "model"), trace, "bfloat16", str(tmp_path / name), max_tokens=max_live_tokens(trace), env=env)
            for name, env in (("beside", None), ("after", {"MLXB_PDL": "0"}))]
    assert len(outs[0]) == sum(len(t) for t in reqs.values()) and outs[0].keys() == outs[1].keys()
    assert all(np.array_equal(outs[0][k], outs[1][k]) for k in outs[0])

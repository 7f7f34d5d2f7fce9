"""Which runs of the gated delta rule go through it in two passes (``ops.chunks_side_by_side``), and which single rows' attention runs
beside that of portions (``ops.rows_beside_pay``)."""
import torch

from mlx_lm_b200 import ops

DELTA = ("delta", 16, 64, 64)


def test_long_runs_of_few_states_go_in_two_passes():
    assert ops.chunks_side_by_side(*DELTA, (1024, 1024)) and ops.chunks_side_by_side(*DELTA, (200,))
    assert not ops.chunks_side_by_side(*DELTA, (128,)) and not ops.chunks_side_by_side(*DELTA, (64,) * 4)
    assert not ops.chunks_side_by_side(*DELTA, ())


def test_what_has_no_two_passes_takes_none():
    assert not ops.chunks_side_by_side("delta", 16, 65, 64, (1024,))       # no chunked kernel for such states
    assert not ops.chunks_side_by_side("mamba2", 32, 128, 64, (1024,))
    assert not ops.chunks_side_by_side(*DELTA, (40000,))                   # their scratch memory has a limit


def test_the_limit_counts_what_is_allocated():
    """Short runs fill few of the chunks that their rows and requests may have; the memory is for all of those."""
    jobs = ops.delta_chunk_jobs(512 * 64, 512)
    assert jobs * 16 > ops.DELTA_CHUNK_HEADS and not ops.chunks_side_by_side(*DELTA, (64,) * 512)
    assert ops.chunks_side_by_side(*DELTA, (1024, 1024), jobs=512) and not ops.chunks_side_by_side(*DELTA, (1024, 1024), jobs=513)
    runs = [1, 64, 65, 130, 191, 2]
    assert sum(-(-n // 64) for n in runs) <= ops.delta_chunk_jobs(sum(runs), len(runs))


def test_scratch_memory_grows_up_to_its_limit():
    from mlx_lm_b200.engine import Workspace
    ws = Workspace("cpu")
    f = lambda n: ws.flat("x", n, torch.float32, most=10000).numel()
    assert [f(3000), f(3000), f(3001), f(6001), f(9000), f(10000)] == [3000, 3000, 6000, 10000, 10000, 10000]
    assert ws.flat("y", 3000, torch.float32).numel() == 3000 and ws.flat("y", 3001, torch.float32).numel() == 6000


def test_many_rows_do_not_run_beside_few_tiles():
    assert ops.rows_beside_pay(1, 1, 16) and ops.rows_beside_pay(64, 1, 25) and ops.rows_beside_pay(128, 8, 25)
    assert not ops.rows_beside_pay(128, 1, 16) and not ops.rows_beside_pay(128, 2, 20)

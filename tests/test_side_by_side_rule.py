"""Which runs of the gated delta rule go through it in two passes (``ops.chunks_side_by_side``)."""
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

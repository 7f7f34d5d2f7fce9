"""Choices between kernels that depend on a step's portions: which runs of rows go through a recurrence token by token and which in
chunks (``ops.chunk_rule``), and whether float32 portions run in tiles (``ops.attention_portions_f32_pays``)."""
import pytest

from mlx_lm_b200 import ops

MAMBA, DELTA = ("mamba2", 32, 128, 64), ("delta", 16, 64, 64)


@pytest.mark.parametrize("layer", [MAMBA, DELTA, ("mamba2", 16, 16, 32), ("delta", 64, 64, 128)])
@pytest.mark.parametrize("requests", [1, 4, 32])
def test_short_runs_go_token_by_token(layer, requests):
    assert ops.chunk_rule(*layer, (8,) * requests) is None
    assert ops.chunk_rule(*layer, (2,) * requests) is None


def test_long_runs_go_in_chunks():
    assert ops.chunk_rule(*MAMBA, (64,)) is ops.CHUNKS
    assert ops.chunk_rule(*MAMBA, (1024, 1024)) is ops.CHUNKS
    assert ops.chunk_rule(*DELTA, (1024, 1024)) is ops.CHUNKS
    # 256 states of the delta rule fill the SMs token by token, and wait for them in chunks
    assert ops.chunk_rule(*DELTA, (100,) * 16) is None


def test_a_step_with_both():
    rule = ops.chunk_rule(*MAMBA, (300, 5, 20, 2))
    assert rule is not None and rule is not ops.CHUNKS
    assert rule.chunks(300) and not rule.chunks(5) and not rule.chunks(1)
    assert all(isinstance(v, int) and 0 <= v < 1 << 31 for v in rule)


def test_what_the_chunked_kernels_do_not_take():
    assert ops.chunk_rule("mamba2", 32, 129, 64, (1024,)) is None
    assert ops.chunk_rule("delta", 16, 65, 64, (1024,)) is None
    assert ops.chunk_rule(*MAMBA, ()) is None


@pytest.mark.parametrize("heads,dim", [(4, 16), (16, 64), (16, 128)])
def test_float32_attention_of_few_keys_goes_row_by_row(heads, dim):
    pays = lambda portions, window=0: ops.attention_portions_f32_pays(heads, dim, window, portions)
    assert not pays([(0, 2)]) and not pays([(0, 8)] * 4) and not pays([(8, 2)])
    assert pays([(0, 64)]) and pays([(0, 300), (0, 5)]) and pays([(1000, 2)]) and pays([(0, 1024)] * 2)
    assert not pays([(1000, 2)], window=4)              # rows that see four keys

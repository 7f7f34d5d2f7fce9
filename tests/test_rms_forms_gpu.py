"""RMS norms and stream updates in every form of their kernels (whole rows, parts, gated parts, sums without a norm) at the edges of what
a warp or a block holds, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("Dg", [4, 64, 132, 512, 516, 1024, 2052, 8192, 8196, 1001])
@pytest.mark.parametrize("groups,gate_mode,weighted,gathered", [
    (1, 0, True, False), (1, 0, False, False), (2, 0, True, False), (3, 0, False, False), (1, 1, True, False), (2, 2, True, False),
    (2, 1, False, False), (1, 0, True, True), (1, 0, False, True)])
def test_rmsnorm_forms(Dg, groups, gate_mode, weighted, gathered):
    """A float32 norm rounds its sum, its root and each product: a few 6e-8."""
    from mlx_lm_b200 import ops
    D, R = Dg * groups, 9
    g = torch.Generator(device=DEV).manual_seed(Dg + groups)
    x, gate = torch.randn(R, D, generator=g, device=DEV), torch.randn(R, D, generator=g, device=DEV)
    for period in ({D, Dg} if weighted else {D}):
        w = torch.randn(period, generator=g, device=DEV) if weighted else None
        rows = [3, 0, 8, -1, R, 3] if gathered else list(range(R))
        out = torch.full((len(rows), D), 7.0, device=DEV)
        ops.rmsnorm(x, w, out, 1e-5, ops.current_stream(), offset=1.0, groups=groups, period=period, gate=gate if gate_mode else None,
                    gate_mode=gate_mode, rows=torch.tensor(rows, dtype=torch.int32, device=DEV) if gathered else None)
        v, silu = x.double().view(R, groups, Dg), torch.nn.functional.silu(gate.double()).view(R, groups, Dg)
        if gate_mode == ops.GATE_BEFORE:
            v = v * silu
        v = v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5)
        v = v * (1.0 + w.double().repeat(D // period).view(groups, Dg)) if weighted else v
        if gate_mode == ops.GATE_AFTER:
            v = v * silu
        want = v.reshape(R, D)
        for i, r in enumerate(rows):
            if 0 <= r < R:
                assert rel(out[i], want[r]) < 1e-6, (i, period)
            else:
                assert not out[i].any()


@pytest.mark.parametrize("D", [4, 64, 128, 132, 1024, 4100, 8192, 8196, 1001])
@pytest.mark.parametrize("one,two,second", [(False, False, False), (True, False, False), (False, False, True), (False, True, True), (True, True, True)])
def test_residual_update_forms(D, one, two, second):
    from mlx_lm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(D)
    x, y1, y2 = (torch.randn(7, D, generator=g, device=DEV) for _ in range(3))
    w1, w2 = (torch.randn(D, generator=g, device=DEV) for _ in range(2))
    norm = lambda y, w: y.double() / torch.sqrt((y.double() ** 2).mean(-1, keepdim=True) + 1e-5) * w.double()
    want = x.double() + 0.5 * ((norm(y1, w1) if one else y1.double()) + ((norm(y2, w2) if two else y2.double()) if second else 0.0))
    cast = torch.empty(7, D, dtype=torch.bfloat16, device=DEV)
    ops.residual_update(x, y1, ops.current_stream(), w1=w1 if one else None, y2=y2 if second else None, w2=w2 if two else None, scale=0.5,
                        eps=1e-5, cast_out=cast)
    assert rel(x, want) < 1e-6 and torch.equal(cast, x.bfloat16())

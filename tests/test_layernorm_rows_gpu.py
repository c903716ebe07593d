"""Layernorm on both sides of the row count from which gamma and beta are requested after the reductions (one block of eight
rows per SM), against float64: f32 rows of unit scale, two-pass statistics, stay within 2e-5 for values up to 16."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [64, 508, 512, 516, 1024])
@pytest.mark.parametrize("R", [1, 9, 1184, 1185, 1300])
def test_rows(ctx, R, C):
    rng = np.random.default_rng(R + C)
    x = (rng.standard_normal((R, C)) * 2 + 0.5).astype(np.float32)
    g, b = [(1 + 0.2 * rng.standard_normal(C)).astype(np.float32) for _ in range(2)], [rng.standard_normal(C).astype(np.float32) for _ in range(2)]
    tx, tg, tb = ctx.upload(x, R, C), [ctx.upload(v, 1, C) for v in g], [ctx.upload(v, 1, C) for v in b]
    ln = lambda a, i: (a - a.mean(1, keepdims=True)) / np.sqrt(a.var(1, keepdims=True) + 1e-5) * g[i] + b[i]  # noqa: E731
    want = ln(x.astype(np.float64), 0)
    assert np.abs(ctx.download(ctx.layernorm(tx, tg[0], tb[0])).reshape(R, C) - want).max() < 2e-5
    y, z = ctx.layernormChain(tx, tg[0], tb[0], tg[1], tb[1])
    assert np.abs(ctx.download(y).reshape(R, C) - want).max() < 2e-5
    # the second result may exist as the f16 operand alone: half a unit in the last place of values below 16
    assert np.abs(ctx.download(z).reshape(R, C) - ln(want, 1)).max() < 8e-3

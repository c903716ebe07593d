"""Relative-position attention at the edges of its key tiles and of the split of a window's queries over CTAs, against
float64.  Operands and probabilities are f16 (2^-11 each) under f32 sums: a score of order 1 from products with 128 terms of
0.09 and 1.0 moves by less than 2e-3, which moves the average of values below 3 by less than 1e-2."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (1, 1, T): three CTAs per head; 64 pairs: two; 152 pairs: one.  T around multiples of 48, the step of the tile count.
@pytest.mark.parametrize("W,H,T", [(1, 1, 16), (1, 1, 31), (1, 2, 48), (1, 2, 49), (1, 1, 96), (1, 1, 97), (1, 2, 144), (1, 1, 145),
                                   (1, 1, 191), (8, 8, 33), (8, 8, 134), (19, 8, 47), (19, 8, 150)])
def test_tiles_and_query_split(ctx, W, H, T):
    rng = np.random.default_rng(W * 1000 + T)
    HD, S = 128, H * 128
    qkv = rng.standard_normal((W * T, 3 * S)).astype(np.float32)
    qkv[:, :S] /= np.sqrt(HD)
    pos = rng.standard_normal((2 * T - 1, S)).astype(np.float32)
    u, v = (rng.standard_normal((2, S)) * 0.02).astype(np.float32)
    got = ctx.download(ctx.attnFusedQKV(ctx.upload(qkv, W * T, 3 * S), ctx.upload(pos, 2 * T - 1, S), ctx.upload(u, 1, S),
                                        ctx.upload(v, 1, S), H, HD, W)).reshape(W, T, H, HD)
    q, k, val = (qkv[:, i * S:(i + 1) * S].astype(np.float64).reshape(W, T, H, HD) for i in range(3))
    p4, u4, v4 = pos.astype(np.float64).reshape(-1, H, HD), u.reshape(H, HD), v.reshape(H, HD)
    s = np.einsum("wihd,wjhd->whij", q + u4, k)
    rel = np.einsum("wihd,phd->whip", q + v4, p4)
    i, j = np.indices((T, T))
    s += rel[:, :, i, T - 1 - i + j]
    e = np.exp(s - s.max(-1, keepdims=True))
    want = np.einsum("whij,wjhd->wihd", e / e.sum(-1, keepdims=True), val)
    assert np.abs(got - want).max() < 1e-2

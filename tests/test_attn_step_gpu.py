"""One-pass attention of one query per stream against the separate ops and against float64.

Bound: a score is a sum of HD <= 128 products, off by at most HD * 2^-24 * sum|q k| ~ 1e-5 at unit-scale scores, which
moves a softmax weight by that relative amount; the weighted sum of |v| <= 6 values then stays within 1e-4 of float64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(q, k, v, H, HD, W):
    Tk = k.shape[0] // W
    q4 = q.astype(np.float64).reshape(W, H, HD)
    k4, v4 = (t.astype(np.float64).reshape(W, Tk, H, HD) for t in (k, v))
    s = np.einsum("whd,wjhd->whj", q4, k4)
    p = np.exp(s - s.max(-1, keepdims=True))
    return np.einsum("whj,wjhd->whd", p / p.sum(-1, keepdims=True), v4).reshape(W, H * HD)


# windows, keys, heads, head width: one key, edges of the row octets and of the 64-key rounds, a ragged last strip, the
# narrowest and widest heads, split and unsplit key ranges
@pytest.mark.parametrize("W,Tk,H,HD", [(1, 1, 20, 64), (1, 7, 3, 64), (1, 65, 20, 64), (1, 1500, 20, 64), (3, 129, 5, 32),
                                       (2, 64, 7, 4), (64, 200, 20, 64), (70, 33, 1, 128), (5, 191, 9, 16)])
def test_step_matches_f64_and_ops(ctx, W, Tk, H, HD):
    rng = np.random.default_rng(W * 1000 + Tk)
    D = H * HD
    q = (rng.standard_normal((W, D)) / np.sqrt(HD)).astype(np.float32)
    k, v = (rng.standard_normal((W * Tk, D)).astype(np.float32) for _ in range(2))
    tq, tk, tv = ctx.upload(q, W, D), ctx.upload(k, W * Tk, D), ctx.upload(v, W * Tk, D)
    for _ in range(2):  # the second launch finds the tickets as the first left them
        got = ctx.download(ctx.attnStep(tq, tk, tv, H, HD, W)).reshape(W, D)
        assert np.abs(got - _reference(q, k, v, H, HD, W)).max() < 1e-4
    ops = ctx.download(ctx.bmmPV(ctx.softmax(ctx.bmmQK(tq, tk, None, H, HD, W)), tv, H, HD, W)).reshape(W, D)
    assert np.abs(got - ops).max() < 1e-4


@pytest.mark.parametrize("S,n,NH,HD", [(1, 0, 20, 64), (1, 130, 20, 64), (3, 8, 5, 32), (64, 15, 20, 64), (70, 63, 2, 64)])
def test_append_step(ctx, S, n, NH, HD):
    rng = np.random.default_rng(S * 100 + n)
    D = NH * HD
    qkv = (rng.standard_normal((S, 3 * D)) / HD ** 0.25).astype(np.float32)
    ck, cv = (rng.standard_normal((n + 3, S * D)).astype(np.float32) for _ in range(2))
    tk, tv = ctx.upload(ck, n + 3, S * D), ctx.upload(cv, n + 3, S * D)
    got = ctx.download(ctx.attnStepAppend(ctx.upload(qkv, S, 3 * D), tk, tv, n, NH, HD)).reshape(S, D)
    for c, t, part in ((ck, tk, 1), (cv, tv, 2)):
        c[n] = qkv[:, part * D:(part + 1) * D].reshape(-1)
        assert np.array_equal(ctx.download(t).reshape(n + 3, S * D), c)
    want = _reference(qkv[:, :D].reshape(1, -1), ck[:n + 1], cv[:n + 1], S * NH, HD, 1).reshape(S, D)
    assert np.abs(got - want).max() < 1e-4


@pytest.mark.parametrize("Tk", [5, 700])
def test_infinities_and_nans_as_in_the_separate_ops(ctx, Tk):
    H, HD, D = 8, 32, 256
    rng = np.random.default_rng(Tk)
    q = np.abs(rng.standard_normal((1, D))).astype(np.float32) + 0.1
    k, v = (rng.standard_normal((Tk, D)).astype(np.float32) for _ in range(2))
    k[0, 0:32] = -np.inf           # head 0: one masked key
    k[:, 32:64] = -np.inf          # head 1: every key masked
    k[Tk - 1, 64:96] = np.inf      # head 2
    k[2, 96] = np.nan              # head 3
    k[0, 128:160] = np.float32(-3.4e38)  # head 4: the type's lowest value (the score overflows to -inf)
    v[1, 160] = np.inf             # head 5
    k[:4, 192:224] = -np.inf       # head 6: a run of masked keys
    tq, tk, tv = ctx.upload(q, 1, D), ctx.upload(k, Tk, D), ctx.upload(v, Tk, D)
    got = ctx.download(ctx.attnStep(tq, tk, tv, H, HD))
    ops = ctx.download(ctx.bmmPV(ctx.softmax(ctx.bmmQK(tq, tk, None, H, HD)), tv, H, HD))
    np.testing.assert_allclose(got, ops, atol=1e-4, rtol=0, equal_nan=True)


def test_shapes_outside_the_kernel_are_declined(ctx):
    t = ctx.alloc(2, 96)
    assert ctx.attnStep(t, t, t, 2, 48, 1) is None  # two queries per window
    assert ctx.attnStep(t, t, t, 2, 48, 2) is None  # head width not a power of two

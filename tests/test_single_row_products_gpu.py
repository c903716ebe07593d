"""One row against f16 and int8 weights: the forms of the kernel (two batches of 8 or 16 rows, 64 or 128 columns, three or four
blocks an SM) at their edges against float64, and the rate at which wide matrices are read."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# K and N: one quad of columns; slices shorter than a batch, ending inside one, of exactly two; more than the 2048 rows held at a
# time; strips of 64 and 128 columns with a remainder; grids of up to three blocks an SM, between three and four, and more
@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("K,N", [(4096, 4), (64, 260), (127, 132), (128, 2304), (129, 2308), (1280, 2300), (1000, 1284), (2049, 516), (20000, 64),
                                 (520, 30724), (1280, 14340), (250, 57344), (513, 38400), (1280, 20484)])
def test_edges(ctx, K, N, int8):
    rng = np.random.default_rng(K + N)
    x = rng.standard_normal(K).astype(np.float32)
    if int8:
        q = rng.integers(-127, 128, (K, N), dtype=np.int8)
        sc = (rng.uniform(0.2, 1.0, N) / (73.3 * np.sqrt(K))).astype(np.float32)
        got = ctx.matmulInt8(ctx.upload(x, 1, K), ctx.uploadBytes(q.view(np.uint8).reshape(-1)), ctx.upload(sc, 1, N), N, K)
        want = x.astype(np.float64) @ q * sc
    else:
        w = (rng.standard_normal((K, N), dtype=np.float32) / np.float32(np.sqrt(K))).astype(np.float16)
        got = ctx.matmul(ctx.upload(x, 1, K), ctx.uploadF16(w.astype(np.float32), K, N))
        want = x.astype(np.float64) @ w
    # f32 sums of K terms of order K^-1/2 in at least eight parts: below sqrt(K) * 2^-24 of a result of order 1, five sigma
    assert np.abs(ctx.download(got) - want).max() < 5 * np.sqrt(K) * 2.0 ** -24 + 5e-7


@pytest.mark.parametrize("int8", [False, True])
def test_infinities_stay_where_they_are(ctx, int8):
    """Rows past the end of a slice meet a zero activation and are not read: a row of infinities behind the matrix, or an infinite
    activation, touches nothing else."""
    K, N = 200, 260
    x = np.ones(K, np.float32)
    x[K - 1] = np.inf
    w = np.zeros((K, N), np.float32)
    w[K - 1, 0], w[K - 1, 1:] = 1.0, 2.0
    if int8:
        got = ctx.matmulInt8(ctx.upload(x, 1, K), ctx.uploadBytes(w.astype(np.int8).view(np.uint8).reshape(-1)), ctx.upload(np.ones(N), 1, N), N, K)
    else:
        got = ctx.matmul(ctx.upload(x, 1, K), ctx.uploadF16(w, K, N))
    assert np.isposinf(ctx.download(got)).all()


@pytest.mark.parametrize("int8,K,N,bound_us", [(False, 1280, 51868, 36), (False, 5120, 10240, 34), (True, 1280, 51868, 21.5), (True, 2560, 20484, 21.5)])
def test_wide_matrices_are_streamed(ctx, int8, K, N, bound_us):
    """Bounds between what these take (23, 20, 16 and 16 us on one B200) and what 16 loads of a lane with a bound per row took
    (48, 47, 27 and 26 us)."""
    raw = np.random.default_rng(1).integers(-127, 128, (K, N), dtype=np.int8)
    x, sc = ctx.upload(np.ones(K, np.float32), 1, K), ctx.upload(np.ones(N, np.float32), 1, N)
    ws = [ctx.uploadBytes(raw.view(np.uint8).reshape(-1)) if int8 else ctx.uploadF16(raw.astype(np.float32), K, N) for _ in range(3)]

    def body():
        for _ in range(4):
            for w in ws:
                ctx.freeTensor(ctx.matmulInt8(x, w, sc, N, K) if int8 else ctx.matmul(x, w))

    body()
    batch, _ = ctx.recordBatch(body)
    best = 1e9
    for _ in range(8):
        ctx.sync()
        t0 = time.perf_counter()
        for _ in range(5):
            batch.launch()
        ctx.sync()
        best = min(best, (time.perf_counter() - t0) / 60)
    batch.free()
    for w in ws:
        (ctx.freeBytes if int8 else ctx.freeTensor)(w)
    assert best < bound_us * 1e-6, best

"""int4 products of 1 to 16 rows against float64 on the exact weights (q - zp) * scale.

The mma.sync form (5 rows on): rows as f16 value + residue (2^-22 of each value), exact weights, f32 sums of a block's 32 terms
times its scale: with |a| ~ 1 and weights of norm ~1 per column the result, of order 1, is off by less than 3e-5.  The dp4a
form (1 to 4 rows): two int8 digits, 2^-15 of the row maximum ~4 on every value: below 2e-3."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one block; a K slice not a multiple of four blocks; slices of 16, 20, 32, 36, 64 blocks; a last slice that is short; one
# column group, several per warp, two passes; rows that do not fill the tile; K that ends inside a block
@pytest.mark.parametrize("M,K,N", [(16, 32, 8), (5, 96, 16), (16, 2016, 64), (16, 2048, 8192), (7, 2080, 264), (16, 4096, 520), (9, 4128, 128),
                                   (16, 8192, 2048), (16, 8160, 72), (11, 2560, 5128), (16, 1000, 40), (6, 2050, 48),
                                   (1, 8192, 2048), (1, 2560, 1288), (1, 512, 2360), (3, 4096, 1100), (4, 2048, 2376)])
def test_few_rows(ctx, M, K, N):
    rng = np.random.default_rng(K + N)
    nblk = (K + 31) // 32
    a = rng.standard_normal((M, K)).astype(np.float32)
    q = rng.integers(0, 16, (N, nblk * 32))
    z = rng.integers(0, 16, (N, (nblk + 1) // 2 * 2))
    sc = (rng.uniform(0.25, 1.0, (N, nblk)) / (4.6 * np.sqrt(K))).astype(np.float32)
    w = (q.reshape(N, nblk, 32) - z[:, :nblk, None]) * sc.astype(np.float64)[:, :, None]
    want = a.astype(np.float64) @ w.reshape(N, -1)[:, :K].T
    packed = (q[:, 0::2] | (q[:, 1::2] << 4)).astype(np.uint8)
    zp = (z[:, 0::2] | (z[:, 1::2] << 4)).astype(np.uint8)
    ctx.startProfile(16)
    got = ctx.download(ctx.matmulNBits(ctx.upload(a, M, K), ctx.uploadBytes(packed.reshape(-1)), ctx.upload(sc, 1, sc.size),
                                       ctx.uploadBytes(zp.reshape(-1)), N)).reshape(M, N)
    labels = [e["label"] for e in ctx.endProfile()]
    small = N * K < 1 << 18  # little work: the any-shape kernel, exact too
    assert small or ("nbits_mma" if M > 4 else "gemv_nbits") in labels, labels
    assert np.abs(got - want).max() < (3e-5 if M > 4 else 2e-3) * max(1.0, np.abs(want).max() / 4)


def _int4(ctx, K, N, rng):
    nblk = K // 32
    return (ctx.uploadBytes(rng.integers(0, 256, N * nblk * 16, dtype=np.uint8)), ctx.upload(np.full(N * nblk, 0.01, np.float32), 1, N * nblk),
            ctx.uploadBytes(np.full(N * ((nblk + 1) // 2), 0x88, np.uint8)))


# (three weight sets: small ones stay in L2, which favours the copy)
# what the default rule takes against the product on the f16 copy: at most a fifth slower (1.8 to 2.2 times as slow when every
# width streamed the 4-bit weights), and far faster where the columns are few
@pytest.mark.parametrize("M,K,N,at_most", [(16, 1536, 16384, 1.2), (5, 2048, 20480, 1.2), (16, 8192, 4096, 1.2), (16, 4096, 16384, 1.2),
                                           (16, 2048, 8192, 1.3), (16, 1024, 2048, 0.8), (16, 4096, 2048, 0.8), (12, 8192, 2304, 0.95),
                                           (12, 5120, 2560, 1.2), (12, 1536, 8192, 1.2), (12, 512, 24576, 1.2)])
def test_the_rule_takes_the_faster_form(ctx, M, K, N, at_most):
    import time

    rng = np.random.default_rng(K)
    x, ws = ctx.upload(rng.standard_normal((M, K)).astype(np.float32), M, K), [_int4(ctx, K, N, rng) for _ in range(3)]

    def body():
        for _ in range(4):
            for w in ws:
                ctx.freeTensor(ctx.matmulNBits(x, *w, N))

    times = {}
    try:
        for rows in (16, 0):
            ctx.setOption("nbits_mma_rows", rows)
            body()
            batch, _ = ctx.recordBatch(body)
            best = 1e9
            for _ in range(6):
                ctx.sync()
                t0 = time.perf_counter()
                for _ in range(5):
                    batch.launch()
                ctx.sync()
                best = min(best, time.perf_counter() - t0)
            times[rows] = best
            batch.free()
    finally:
        ctx.setOption("nbits_mma_rows", 16)
    assert times[16] < at_most * times[0], times


def test_a_wide_product_first_used_in_a_recording(ctx):
    """The f16 copy is not started inside a recording: the streaming kernel takes the product there, eager calls the copy."""
    rng = np.random.default_rng(3)
    M, K, N = 16, 1024, 16384
    a, w = rng.standard_normal((M, K)).astype(np.float32), _int4(ctx, K, N, rng)
    x = ctx.upload(a, M, K)
    batch, y = ctx.recordBatch(lambda: ctx.matmulNBits(x, *w, N))
    batch.launch()
    recorded = ctx.download(y)
    batch.free()
    eager = ctx.download(ctx.matmulNBits(x, *w, N))
    assert np.linalg.norm(recorded - eager) < 1e-3 * np.linalg.norm(eager)  # weights exact, and rounded to f16


# one to four rows on both sides of K = 2048, fewer and more columns than the SMs have warps for
@pytest.mark.parametrize("M", [1, 2, 4])
@pytest.mark.parametrize("K,N", [(32, 8192), (2048, 515), (2048, 4730), (2080, 515), (2080, 2370), (2080, 4740)])
def test_one_to_four_rows(ctx, M, K, N):
    test_few_rows(ctx, M, K, N)

"""Products whose tiles fit one wave of the SMs: the choice of tile height and K split, ring stages of two K chunks (int8), and the
vector form of the int8 digit pass, at the edges of what each takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# two K chunks per ring stage of the int8 form against one: an unsplit sum and a split one, several tiles per CTA, the fewest
# chunks, a remainder of rows and columns
@pytest.mark.parametrize("kind,M,K,N", [("i8", 512, 4096, 1024), ("i8", 100, 4096, 1024), ("i8", 17, 512, 520), ("i8", 300, 1280, 520), ("i8", 16, 5120, 1280),
                                        ("i8", 33, 2048, 1000), ("i8", 48, 1024, 20000)])
def test_wide_stages_bit_for_bit(ctx, kind, M, K, N):
    rng = np.random.default_rng(M + N)
    a = ctx.upload(rng.standard_normal((M, K)).astype(np.float32), M, K)
    add = ctx.upload(rng.standard_normal((M, N)).astype(np.float32), M, N)
    w = (ctx.uploadBytes(rng.integers(-127, 128, (K, N), dtype=np.int8).view(np.uint8).reshape(-1)),
         ctx.upload(np.full(N, 0.01, np.float32), 1, N), N, K)
    outs, labels = [], []
    try:
        for wide in (1, 0):
            ctx.setOption("tc_wide_stages", wide)
            ctx.startProfile(16)
            ctx.linearStep(a, *w)
            labels.append({e["label"] for e in ctx.endProfile()})
            outs.append([ctx.download(ctx.linearStep(a, *w, act="silu")), ctx.download(ctx.linearStep(a, *w, add=add))])
    finally:
        ctx.setOption("tc_wide_stages", 1)
    assert "tc_gemm_i8_wide" in labels[0] and "tc_gemm_i8" in labels[1], labels  # each is the form it says it is
    assert np.array_equal(outs[0][0], outs[1][0]) and np.array_equal(outs[0][1], outs[1][1])


# f32 weights (residue planes, sums of 2^-20 terms), int8 weights with three digits (2^-22 of the row maximum): heights and
# splits chosen on both sides of 64 and 128 rows, K chunks that do not divide by the split, one row and a remainder
@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("M,K,N", [(300, 4096, 1024), (300, 2080, 1024), (100, 4096, 1000), (40, 2112, 2048), (129, 1056, 260), (17, 4100, 512),
                                   (600, 2048, 1024)])
def test_tile_and_split_choices(ctx, M, K, N, int8):
    rng = np.random.default_rng(M + K)
    a = rng.standard_normal((M, K)).astype(np.float32)
    add = rng.standard_normal((M, N)).astype(np.float32)
    ctx.setOption("int8_limbs", 3)
    try:
        if int8:
            q = rng.integers(-127, 128, (K, N), dtype=np.int8)
            sc = (rng.uniform(0.2, 1.0, N) / (73.3 * np.sqrt(K))).astype(np.float32)
            got = ctx.linearStep(ctx.upload(a, M, K), ctx.uploadBytes(q.view(np.uint8).reshape(-1)), ctx.upload(sc, 1, N), N, K,
                                 add=ctx.upload(add, M, N))
            want = a.astype(np.float64) @ (q * sc.astype(np.float64)) + add
        else:
            w = (rng.standard_normal((K, N)) / np.sqrt(K)).astype(np.float32)
            got = ctx.matmul(ctx.upload(a, M, K), ctx.upload(w, K, N), add=ctx.upload(add, M, N))
            want = a.astype(np.float64) @ w.astype(np.float64) + add
        got = ctx.download(got).reshape(M, N)
    finally:
        ctx.setOption("int8_limbs", 2)
    # results of order 1; the tensor core's accumulator drops at most 2^-22 of the sum per step of K / 8 to K / 32 steps
    assert np.abs(got - want).max() < 2e-4


@pytest.mark.parametrize("K", [68, 1024, 1028, 2048, 4092, 8192, 8196, 1027])
def test_digit_pass_of_whole_quads(ctx, K):
    """Quads in registers (K % 4 == 0, up to 8192) and the general form beside it.  Three digits carry a row to 2^-22 of its
    maximum: over the largest |a| ~ 4.5, |w| <= 127 and sqrt(K) growth the sum is off by less than 1e-6 of K."""
    rng = np.random.default_rng(K)
    M, N = 9, 128
    a = rng.standard_normal((M, K)).astype(np.float32)
    a[3] = 0
    q = rng.integers(-127, 128, (K, N), dtype=np.int8)
    ctx.setOption("int8_limbs", 3)
    ctx.setOption("gemv_rows", 0)
    try:
        got = ctx.download(ctx.matmulInt8(ctx.upload(a, M, K), ctx.uploadBytes(q.view(np.uint8).reshape(-1)),
                                          ctx.upload(np.full(N, 0.01, np.float32), 1, N), N, K)).reshape(M, N)
    finally:
        ctx.setOption("int8_limbs", 2)
        ctx.setOption("gemv_rows", 4)
    assert np.abs(got - 0.01 * (a.astype(np.float64) @ q)).max() < 1e-6 * K
    assert not got[3].any()


# parts: how many sums K is kept in at least.  The operands are f16 values, so what is left is the accumulator: a step adds 16
# products and drops less than 2^-25 of the sum on average, and a part takes K / 16 / parts steps.
@pytest.mark.parametrize("M,K,N,parts", [(65, 1024, 1024, 4), (200, 1024, 1024, 4), (375, 1024, 1024, 2), (128, 2048, 2048, 4),
                                         (250, 2048, 2048, 2), (65, 4096, 1024, 8), (100, 1024, 4096, 2), (70, 512, 2048, 2),
                                         (190, 1000, 1000, 2), (360, 5120, 1280, 2)])
def test_a_sum_stays_in_parts(ctx, M, K, N, parts):
    rng = np.random.default_rng(M + K)
    a, w = (rng.standard_normal(s).astype(np.float16).astype(np.float32) for s in ((M, K), (K, N)))
    add = rng.standard_normal((M, N)).astype(np.float32)
    want = a.astype(np.float64) @ w.astype(np.float64)
    ta, tw = ctx.upload(a, M, K), ctx.uploadF16(w, K, N)
    for got, ref in ((ctx.matmul(ta, tw), want), (ctx.matmul(ta, tw, add=ctx.upload(add, M, N)), want + add)):
        err = ctx.download(got).reshape(M, N) - ref
        assert np.linalg.norm(err) / np.linalg.norm(ref) < K / 16 / parts * 2.0 ** -25


@pytest.mark.parametrize("M,K,N", [(100, 1024, 4096), (200, 4096, 1024), (60, 1024, 1024)])
def test_silu_of_one_wave_int8_products(ctx, M, K, N):
    """Three digits carry a row to 2^-22 of its maximum and the activation is x / (1 + exp(-x)) in f32, so results of order 1
    stay within 1e-5, which the epilogue that computes it by an approximate tanh leaves."""
    rng = np.random.default_rng(M)
    a = rng.standard_normal((M, K)).astype(np.float32)
    q = rng.integers(-127, 128, (K, N), dtype=np.int8)
    sc = np.full(N, 1 / (73.3 * np.sqrt(K)), np.float32)
    ctx.setOption("int8_limbs", 3)
    try:
        got = ctx.download(ctx.matmulInt8(ctx.upload(a, M, K), ctx.uploadBytes(q.view(np.uint8).reshape(-1)), ctx.upload(sc, 1, N), N, K,
                                          act="silu")).reshape(M, N)
    finally:
        ctx.setOption("int8_limbs", 2)
    z = a.astype(np.float64) @ (q * sc.astype(np.float64))
    assert np.abs(got - z / (1 + np.exp(-z))).max() < 1e-5


# tile height and K split of the plain rule (the shortest tile of at least 64 rows that keeps one wave, then the widest split):
# what is chosen instead is no slower (it was 8 to 11 % slower where a tall tile left a split fewer than three ring stages)
@pytest.mark.parametrize("M,K,N,rows,split", [(100, 1024, 4096, 64, 2), (804, 5120, 1280, 64, 1), (200, 2048, 2048, 64, 2), (300, 4096, 1024, 64, 2)])
def test_choices_against_the_plain_rule(ctx, M, K, N, rows, split):
    import time

    rng = np.random.default_rng(K)
    x = ctx.upload(rng.standard_normal((M, K)).astype(np.float32), M, K)
    ws = [ctx.upload(rng.standard_normal((K, N)).astype(np.float32), K, N) for _ in range(3)]

    def body():
        for _ in range(4):
            for w in ws:
                ctx.freeTensor(ctx.matmul(x, w))

    def best_of():
        body()
        batch, _ = ctx.recordBatch(body)
        best = 1e9
        for _ in range(8):
            ctx.sync()
            t0 = time.perf_counter()
            for _ in range(3):
                batch.launch()
            ctx.sync()
            best = min(best, time.perf_counter() - t0)
        batch.free()
        return best

    chosen = best_of()
    ctx.setOption("tc_tile_rows", rows)
    ctx.setOption("tc_split_k", split)
    try:
        plain = best_of()
    finally:
        ctx.setOption("tc_tile_rows", 0)
        ctx.setOption("tc_split_k", 0)
    assert chosen < 1.05 * plain, (chosen, plain)

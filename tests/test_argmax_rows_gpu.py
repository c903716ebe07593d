"""Row argmax on both sides of the rule that picks its block size, first maximum of a row, and how long rows of few columns take."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,C", [(1, 1), (3, 31), (7, 257), (600, 1000), (1, 8191), (592, 8192), (593, 8192), (2, 16383), (600, 16384), (5, 51866)])
def test_first_maximum(ctx, R, C):
    rng = np.random.default_rng(R + C)
    x = rng.integers(-50, 50, (R, C + 2)).astype(np.float32)  # many ties
    x[:, C:] = 1000.0  # columns past the ones asked for
    x[R // 2, :C] = -np.inf
    x[0, C // 2:C] = np.nan if C > 1 else 1.0
    got = ctx.download(ctx.argmaxRowsIndex(ctx.upload(x, R, C + 2), C)).reshape(R, 2)
    want = np.argmax(np.where(np.isnan(x[:, :C]), -np.inf, x[:, :C]), axis=1)
    assert np.array_equal(got[:, 0], want.astype(np.float32))
    assert np.array_equal(got[:, 1], np.where(np.isnan(x), -np.inf, x)[np.arange(R), want])


def test_many_short_rows_share_the_sms(ctx):
    """8192 rows of 1000 columns: 33 MB, 14.6 us in blocks of 256 threads (53.6 in blocks of 1024); twice that is the bound."""
    R, C = 8192, 1000
    x = ctx.alloc(R, C)

    def body():
        for _ in range(20):
            ctx.freeTensor(ctx.argmaxRowsIndex(x))

    body()
    batch, _ = ctx.recordBatch(body)
    best = 1e9
    for _ in range(8):
        ctx.sync()
        t0 = time.perf_counter()
        for _ in range(5):
            batch.launch()
        ctx.sync()
        best = min(best, (time.perf_counter() - t0) / 100)
    batch.free()
    assert best < 30e-6, best

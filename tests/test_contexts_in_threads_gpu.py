"""Contexts of one device in several host threads: every launch finds the shared-memory limit that it needs."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_few_row_int4_products_side_by_side(pkg):
    """Each thread repeats one product, each of them with another amount of shared memory for the same kernels."""
    errors = []

    def work(K, rows):
        c = pkg.CudaContext(0)
        try:
            rng = np.random.default_rng(K)
            N, nblk = 512, K // 32
            w = (c.uploadBytes(rng.integers(0, 256, N * nblk * 16, dtype=np.uint8)), c.upload(np.full(N * nblk, 0.01, np.float32), 1, N * nblk),
                 c.uploadBytes(np.full(N * ((nblk + 1) // 2), 0x88, np.uint8)))
            xs = [c.upload(rng.standard_normal((M, K)).astype(np.float32), M, K) for M in rows]
            want = [c.download(c.matmulNBits(x, *w, N)) for x in xs]
            for _ in range(5000):
                for x in xs:
                    c.freeTensor(c.matmulNBits(x, *w, N))
            for x, y in zip(xs, want):
                assert np.array_equal(c.download(c.matmulNBits(x, *w, N)), y)
        except Exception as e:  # noqa: BLE001 - reported by the test's own thread
            errors.append(repr(e))
        finally:
            c.destroy()

    threads = [threading.Thread(target=work, args=a) for a in ((1024, (16, 4)), (2016, (16, 4)), (8192, (16, 4)), (6144, (16, 4)))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors

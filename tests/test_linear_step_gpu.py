"""One linear layer of a decoding step, add + act(layernorm(x) @ W + bias), against float64.

Bound: f32 sums of K products of unit-scale rows with columns of norm ~1 (2^-24 * sqrt(K) rounding steps of the partial
sums, the layernorm's statistics and its scaling) stay within 2e-5 of a result of order 1 for K <= 8192."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _erf_gelu(x):  # the approximation of the activation table (src/gpu/kernels/actf.js:5-22)
    z = x * 0.70710678118654752
    t = 1 / (1 + 0.3275911 * np.abs(z))
    y = 1 - (((((1.061405429 * t - 1.453152027) * t) + 1.421413741) * t - 0.284496736) * t + 0.254829592) * t * np.exp(-z * z)
    return 0.5 * x * (1 + np.where(z >= 0, y, -y))


# a single quad of columns, strips with a remainder, one and several K slices, K slices with a remainder, the longest row
# the layernorm takes, a row longer than that (separate ops), many columns on one slice, two rows (separate ops)
@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("M,K,N", [(1, 4096, 4), (1, 1280, 132), (1, 1280, 1280), (1, 132, 5120), (1, 2052, 260), (1, 516, 640),
                                   (1, 4096, 1280), (1, 5120, 1280), (1, 128, 51868), (1, 1280, 3840), (2, 1280, 256), (1, 66, 512)])
@pytest.mark.parametrize("norm", [False, True])
def test_linear_step(ctx, M, K, N, int8, norm):
    rng = np.random.default_rng(K * 7 + N)
    x = (rng.standard_normal((M, K)) + 0.3).astype(np.float32)
    g, b = (1 + 0.1 * rng.standard_normal(K)).astype(np.float32), (0.1 * rng.standard_normal(K)).astype(np.float32)
    bias, add = rng.standard_normal(N).astype(np.float32), rng.standard_normal((M, N)).astype(np.float32)
    if int8:
        q = rng.integers(-127, 128, (K, N), dtype=np.int8)
        sc = (rng.uniform(0.2, 1.0, N) / (73.3 * np.sqrt(K))).astype(np.float32)
        w64, args = q.astype(np.float64) * sc, (ctx.uploadBytes(q.view(np.uint8).reshape(-1)), ctx.upload(sc, 1, N), N, K)
    else:
        w16 = (rng.standard_normal((K, N)) / np.sqrt(K)).astype(np.float16)
        w64, args = w16.astype(np.float64), (ctx.uploadF16(w16.astype(np.float32), K, N),)
    a = x.astype(np.float64)
    if norm:
        a = (a - a.mean(1, keepdims=True)) / np.sqrt(a.var(1, keepdims=True) + 1e-5) * g + b
    want = _erf_gelu(a @ w64 + bias) + add
    ctx.setOption("int8_limbs", 3)  # f32-grade digits where two rows take the tensor cores
    try:
        got = ctx.download(ctx.linearStep(ctx.upload(x, M, K), *args, norm=(ctx.upload(g, 1, K), ctx.upload(b, 1, K)) if norm else None,
                                          bias=ctx.upload(bias, 1, N), act="gelu_erf", add=ctx.upload(add, M, N)))
    finally:
        ctx.setOption("int8_limbs", 2)
    assert np.abs(got.reshape(M, N) - want).max() < 2e-5


def test_linear_step_checks_its_operands(ctx, pkg):
    x, w = ctx.alloc(1, 128), ctx.uploadF16(np.zeros(128 * 256, np.float32), 128, 256)
    with pytest.raises(pkg.CudaError):
        ctx.linearStep(ctx.alloc(1, 64), w)
    with pytest.raises(pkg.CudaError):
        ctx.linearStep(x, w, add=ctx.alloc(1, 128))
    with pytest.raises(pkg.CudaError):
        ctx.linearStep(x, w, bias=ctx.alloc(1, 128))


def test_stale_handles_are_refused_unread(ctx, pkg):
    """A handle is looked up before what it points at is read: an address that was never a tensor's (nothing is mapped there)
    is an error, not a crash."""
    gone = pkg.Tensor(0x40, 1, 256)
    for M in (1, 2):
        x, w, n = ctx.alloc(M, 128), ctx.uploadF16(np.zeros(128 * 256, np.float32), 128, 256), ctx.alloc(1, 128)
        for kw in (dict(add=gone), dict(bias=gone), dict(norm=(gone, n)), dict(norm=(n, gone))):
            with pytest.raises(pkg.CudaError):
                ctx.linearStep(x, w, **kw)
        with pytest.raises(pkg.CudaError):
            ctx.linearStep(x, gone)
        with pytest.raises(pkg.CudaError):
            ctx.linearStep(gone, w)

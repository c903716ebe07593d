"""TDT decoding at the edges of the prediction network's window chunks (8 windows, 32): ids and frames as the CPU decoder's."""
import numpy as np
import pytest

from oracle.tdt_oracle import TdtOracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [1, 7, 8, 9, 33])
def test_window_chunks(ctx, pkg, W):
    from fluidaudio_web_b200.engines import tdt_decoder as td

    T = 21
    w = td.synth_tdt_weights(5)
    proj = np.random.default_rng(W).standard_normal((W, T, 640)).astype(np.float32)
    want = TdtOracle(w, int8=True, threads=8).decode_proj_batch(proj, W, T)
    dec = td.TdtDecoder(ctx, w)
    try:
        for _ in range(2):  # the second decode finds the handle's read-back buffers as the first left them
            got = dec.decode_proj(ctx.upload(proj.reshape(W * T, 640), W * T, 640), W, T)
            for (gi, gf), (wi, wf) in zip(got, want):
                assert gi.tolist() == wi.tolist() and gf.tolist() == wf.tolist()
    finally:
        dec.free()
    assert sum(len(i) for i, _ in want) > 0

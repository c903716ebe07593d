"""The native layer loops issue the members of the host loops: same results, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one short window (few-row products), a group whose q|k|v stays f32, one that keeps it packed, frames past the attention kernel
@pytest.mark.parametrize("W,samples", [(1, 59200), (3, 64000), (2, 171200), (1, 320000)])
def test_conformer_blocks(ctx, pkg, W, samples):
    from fluidaudio_web_b200.engines import fastconformer as fc, synth

    enc = fc.load_encoder(ctx, synth.encoder_weights(dict(synth.PARAKEET_06B, layers=2), seed=4))
    mel = ctx.logMelWindows(ctx.upload(synth.synth_audio(W, samples=samples, seed=5), W, samples), 128)
    layers = enc["layers"]
    enc["layers"] = [{k: v for k, v in w.items() if k != "native"} for w in layers]
    host, t0 = fc.encode_batch(ctx, enc, mel)
    host = ctx.download(host)
    seen = []
    enc["layers"] = layers
    got, t1 = fc.encode_batch(ctx, enc, mel, layer_hook=lambda L, x: seen.append((L, x.rows)))
    assert t0 == t1 and [s[0] for s in seen] == [0, 1]
    assert np.array_equal(ctx.download(got), host)
    # an encoder put together from another one's layers runs those layers, and half the blocks in each loop are the same blocks
    last = dict(enc, layers=layers[1:], cfg=dict(enc["cfg"], layers=1), _posProj={})
    plain = dict(last, layers=[{k: v for k, v in layers[1].items() if k != "native"}], _posProj={})
    assert np.array_equal(*(ctx.download(fc.encode_batch(ctx, e, mel)[0]) for e in (last, plain)))
    enc["layers"] = [{k: v for k, v in layers[0].items() if k != "native"}, layers[1]]
    assert np.array_equal(ctx.download(fc.encode_batch(ctx, enc, mel)[0]), host)


@pytest.mark.parametrize("quant", [None, "int8"])
@pytest.mark.parametrize("S", [1, 3])
@pytest.mark.parametrize("NH", [4, 16])  # head widths 64 and 16
def test_decoder_tokens(ctx, pkg, quant, S, NH):
    from fluidaudio_web_b200.engines import synth, whisper_decoder as wd

    cfg = dict(D=256, NH=NH, FFN=1024, layers=2, VOCAB=2003, maxPos=40, Tenc=96)
    dec = wd.load_decoder(ctx, synth.decoder_weights(cfg, seed=11), NH, quant=quant)
    states = ctx.upload(np.concatenate(synth.encoder_states(cfg, S, seed=13)), S * cfg["Tenc"], cfg["D"])
    layers, runs = dec["layers"], []
    for with_native in (True, False):
        if not with_native:
            dec["layers"] = [{k: v for k, v in w.items() if k != "native"} for w in layers]
        kv = wd.cross_kv_streams(ctx, dec, states)
        st = wd.decode_init_streams(ctx, dec, S, 8)
        runs.append([wd.decode_next_streams(ctx, dec, kv, st, [t] * S, want_logits=True)[1] for t in (1, 7, 3)])
    for a, b in zip(*runs):
        assert np.array_equal(a, b)


def test_decode_next_gives_its_row_back(ctx, pkg):
    from fluidaudio_web_b200.engines import synth, whisper_decoder as wd

    cfg = dict(D=256, NH=4, FFN=1024, layers=2, VOCAB=2003, maxPos=40, Tenc=96)
    dec = wd.load_decoder(ctx, synth.decoder_weights(cfg, seed=11), 4)
    kv = wd.cross_kv(ctx, dec, ctx.upload(synth.encoder_states(cfg, 1, seed=13)[0], cfg["Tenc"], cfg["D"]))
    st = wd.decode_init(ctx, dec, 16)
    for t in range(3):
        wd.decode_next(ctx, dec, kv, st, t)
    before = ctx.memStats()
    for t in range(5):
        wd.decode_next(ctx, dec, kv, st, t)
    assert ctx.memStats() ["created"] == before["created"]


@pytest.mark.parametrize("S", [1, 3])
def test_decoder_tokens_with_heads_that_the_one_pass_attention_declines(ctx, pkg, S):
    """Head width 48: the native loop's separate members, same bits as the host loop, and no handle left behind."""
    from fluidaudio_web_b200.engines import synth, whisper_decoder as wd

    cfg = dict(D=192, NH=4, FFN=768, layers=2, VOCAB=2003, maxPos=40, Tenc=96)
    dec = wd.load_decoder(ctx, synth.decoder_weights(cfg, seed=17), 4)
    states = ctx.upload(np.concatenate(synth.encoder_states(cfg, S, seed=13)), S * cfg["Tenc"], cfg["D"])
    kv, layers, runs = wd.cross_kv_streams(ctx, dec, states), dec["layers"], []
    for native in (True, False):
        if not native:
            dec["layers"] = [{k: v for k, v in w.items() if k != "native"} for w in layers]
        st = wd.decode_init_streams(ctx, dec, S, 8)
        before = ctx.handleCount()
        runs.append([wd.decode_next_streams(ctx, dec, kv, st, [t] * S, want_logits=True)[1] for t in (1, 7, 3)])
        assert not native or ctx.handleCount() == before
    for a, b in zip(*runs):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("W,samples", [(1, 59200), (3, 64000)])
def test_conformer_blocks_when_the_one_kernel_attention_is_off(ctx, pkg, W, samples):
    from fluidaudio_web_b200.engines import fastconformer as fc, synth

    enc = fc.load_encoder(ctx, synth.encoder_weights(dict(synth.PARAKEET_06B, layers=2), seed=4))
    mel = ctx.logMelWindows(ctx.upload(synth.synth_audio(W, samples=samples, seed=5), W, samples), 128)
    layers = enc["layers"]
    ctx.setOption("attn_one_kernel", 0)
    try:
        native = ctx.download(fc.encode_batch(ctx, enc, mel)[0])
        before, arena = ctx.handleCount(), ctx.pushArena()
        fc.encode_batch(ctx, enc, mel)
        ctx.popArena(arena)
        assert ctx.handleCount() == before
        enc["layers"] = [{k: v for k, v in w.items() if k != "native"} for w in layers]
        assert np.array_equal(ctx.download(fc.encode_batch(ctx, enc, mel)[0]), native)
    finally:
        ctx.setOption("attn_one_kernel", 1)


def _no_native(layers):
    return [{k: v for k, v in w.items() if k != "native"} for w in layers]


@pytest.mark.parametrize("W,samples", [(1, 59200), (2, 171200)])  # fewer than 256 rows, more
def test_a_replaced_matrix_of_an_encoder_layer_is_the_one_that_runs(ctx, pkg, W, samples):
    from fluidaudio_web_b200.engines import fastconformer as fc, synth

    cfg = dict(synth.PARAKEET_06B, layers=2)
    enc, other = (fc.load_encoder(ctx, synth.encoder_weights(cfg, seed=s)) for s in (4, 9))
    mel = ctx.logMelWindows(ctx.upload(synth.synth_audio(W, samples=samples, seed=5), W, samples), 128)
    run = lambda e: ctx.download(fc.encode_batch(ctx, e, mel)[0])  # noqa: E731
    seen = [run(enc)]
    row = lambda v: ctx.upload(np.full(1024, v, np.float32), 1, 1024)  # noqa: E731
    new = dict({k: other["layers"][0][k] for k in ("ff1w1", "q", "pw2T")}, lnatt=(row(2.0), row(0.1)), vb=row(0.5))
    for key in new:
        old = enc["layers"][0][key]
        enc["layers"][0][key] = new[key]
        got = run(enc)
        parts = dict(enc, layers=[{k: v for k, v in w.items() if k not in ("qkv", "qkvb", "qkv_of")} for w in _no_native(enc["layers"])])
        near = run(parts)  # the host loop over the entries themselves
        assert np.linalg.norm(got - near) < 2e-3 * np.linalg.norm(near)
        assert np.linalg.norm(got - seen[0]) > 2e-2 * np.linalg.norm(near)
        enc["layers"][0][key] = old
        assert np.array_equal(run(enc), seen[0])
    derived = dict(enc, layers=[dict(enc["layers"][0], ff1w1=other["layers"][0]["ff1w1"]), enc["layers"][1]])
    assert not np.array_equal(run(derived), seen[0]) and np.array_equal(run(enc), seen[0])
    ctx.freeTensor(enc["layers"][0]["lnconv"][0])
    with pytest.raises(pkg.CudaError):
        run(enc)


@pytest.mark.parametrize("quant", [None, "int8"])
@pytest.mark.parametrize("S", [1, 2])
def test_a_replaced_matrix_of_a_decoder_layer_is_the_one_that_runs(ctx, pkg, quant, S):
    from fluidaudio_web_b200.engines import synth, whisper_decoder as wd

    cfg = dict(D=256, NH=4, FFN=1024, layers=2, VOCAB=2003, maxPos=40, Tenc=96)
    dec, other = (wd.load_decoder(ctx, synth.decoder_weights(cfg, seed=s), 4, quant=quant) for s in (11, 12))
    kv = wd.cross_kv_streams(ctx, dec, ctx.upload(np.concatenate(synth.encoder_states(cfg, S, seed=13)), S * cfg["Tenc"], cfg["D"]))

    def run(layers):
        st = wd.decode_init_streams(ctx, dec, S, 8)
        return np.stack([wd.decode_next_streams(ctx, dict(dec, layers=layers), kv, st, [t] * S, want_logits=True)[1] for t in (1, 7, 3)])

    first = run(dec["layers"])
    row = lambda v: ctx.upload(np.full(256, v, np.float32), 1, 256)  # noqa: E731
    new = dict({k: other["layers"][1][k] for k in ("f1w", "svw", "cow")}, ln2=(row(3.0), row(0.5)), svb=row(0.5), cob=row(0.5))
    for key in new:
        old = dec["layers"][1][key]
        dec["layers"][1][key] = new[key]
        got = run(dec["layers"])
        near = run([{k: v for k, v in w.items() if not k.startswith("sqkv")} for w in _no_native(dec["layers"])])
        assert np.linalg.norm(got - near) < 1e-3 * np.linalg.norm(near)
        assert np.linalg.norm(got - first) > 5e-3 * np.linalg.norm(near)
        dec["layers"][1][key] = old
        assert np.array_equal(run(dec["layers"]), first)
    ctx.freeTensor(dec["layers"][0]["ln1"][0])
    ctx.freeTensor(dec["layers"][0]["ln1"][1])
    with pytest.raises(pkg.CudaError):
        run(dec["layers"])

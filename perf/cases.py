"""The work whose speed counts, as a user's program has this package do it.

Four kinds of case, each through the public entry points:

  blocks    a chain of feed-forward blocks (layernorm, up projection, activation, down projection, residual; the int8
            member takes no residual, the int4 member neither that nor an activation) with int4, int8, f16 or f32
            weights, recorded once and replayed per pass, the way a decode loop or a fixed-shape forward keeps its
            recording.
  encoder   16 kHz samples on the device -> log-mel -> the 24-layer 0.6B FastConformer encoder -> frames.
  decoder   the KV-cached decoder of the large-v3-turbo shape: cross K/V of the clips, then token after token.  The
            token that is fed is the given one, as with a forced prompt or when scoring a transcript, so that two
            correct implementations see the same sequence; the pick is made all the same.
  tdt       encoder frames -> joint projection -> greedy TDT decoding in lock-step -> token ids and emission frames.

Weights of the three models are random with a fixed seed, loaded once per process as a server loads them; everything a
pass reads besides them is made from the seed that prepare() is given.
"""
import importlib
import math

import numpy as np
import torch

fa = importlib.import_module("fluidaudio-web_b200")
fastconformer = importlib.import_module("fluidaudio-web_b200.engines.fastconformer")
whisper_decoder = importlib.import_module("fluidaudio-web_b200.engines.whisper_decoder")
tdt_decoder = importlib.import_module("fluidaudio-web_b200.engines.tdt_decoder")
synth = importlib.import_module("fluidaudio-web_b200.engines.synth")

ENC = synth.PARAKEET_06B
DEC = synth.WHISPER_TURBO_DEC
WEIGHT_BYTES = {"int4": 0.5 + 4.0 / 32 + 0.5 / 32, "int8": 1.0, "f16": 2.0, "f32": 4.0}


def listed():
    return [
        # one token through int4 projections (the decode sizes K = 2048, N = 8192 and back): latency and the weight stream
        {"name": "int4_row1", "kind": "blocks", "weights": "int4", "rows": 1, "width": 2048, "hidden": 8192, "blocks": 4},
        # sixteen streams through the same matrices
        {"name": "int4_rows16", "kind": "blocks", "weights": "int4", "rows": 16, "width": 2048, "hidden": 8192, "blocks": 4},
        # prefill-size int8 products, 512 x 1024 x 4096 and back
        {"name": "int8_rows512", "kind": "blocks", "weights": "int8", "rows": 512, "width": 1024, "hidden": 4096, "blocks": 6},
        # encoder feed-forward halves over a ragged number of frames (about five windows)
        {"name": "f16_rows937", "kind": "blocks", "weights": "f16", "rows": 937, "width": 1024, "hidden": 4096, "blocks": 6},
        # f32 weights, which the interface computes in f32: one window and a half of frames
        {"name": "f32_rows300", "kind": "blocks", "weights": "f32", "rows": 300, "width": 1024, "hidden": 4096, "blocks": 3},
        # a short utterance on its own: a user who waits for the answer
        {"name": "encoder_clip", "kind": "encoder", "windows": 1, "samples": 59200},
        # a group of windows of a recording that does not fill 15 s
        {"name": "encoder_group6", "kind": "encoder", "windows": 6, "samples": 171200},
        # the batch that fills a GPU: 32 windows of 15 s
        {"name": "encoder_batch32", "kind": "encoder", "windows": 32, "samples": 240000},
        # one clip, token by token, int8 weights
        {"name": "decoder_stream1_int8", "kind": "decoder", "weights": "int8", "streams": 1, "tokens": 16},
        # 64 clips in lock-step, f16 weights
        {"name": "decoder_streams64_f16", "kind": "decoder", "weights": "f16", "streams": 64, "tokens": 16},
        # the decode of one short utterance
        {"name": "tdt_clip", "kind": "tdt", "windows": 1, "frames": 47},
        # the decode of a batch of 32 full windows
        {"name": "tdt_batch32", "kind": "tdt", "windows": 32, "frames": 188},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["blocks", "blocks", "encoder", "decoder", "tdt"])
    if kind == "blocks":
        weights = rng.choice(["int4", "int8", "f16", "f32"])
        lo, hi = {"int4": (1, 64), "int8": (1, 2048), "f16": (1, 6016), "f32": (16, 1024)}[weights]
        step = 32 if weights == "int4" else 8
        width = rng.randrange(512 // step, 2560 // step + 1) * step
        hidden = min(8192, _log_int(rng, width, 4 * width) // step * step)
        return {"kind": kind, "weights": weights, "rows": _log_int(rng, lo, hi), "width": width, "hidden": hidden,
                "blocks": rng.randint(2, 5)}
    if kind == "encoder":
        return {"kind": kind, "windows": _log_int(rng, 1, 32), "samples": rng.randint(32000, 240000)}
    if kind == "decoder":
        return {"kind": kind, "weights": rng.choice(["f16", "int8"]), "streams": _log_int(rng, 1, 48), "tokens": rng.randint(6, 16)}
    return {"kind": kind, "windows": _log_int(rng, 1, 32), "frames": rng.randint(25, 188)}


# ---- engines: contexts and weights, loaded once ----------------------------------------------------------------------

_ENGINES = {}


def _engine(key, make):
    if key not in _ENGINES:
        _ENGINES[key] = make()
    return _ENGINES[key]


def _normal(gen, shape, std=1.0):
    return torch.randn(shape, generator=gen, device="cuda") * std


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _encoder():
    gen = _generator(3)
    D, F, S, fs = ENC["D"], ENC["DFF"], ENC["Csub"], ENC["melBins"] // 8
    host = lambda t: t.cpu().numpy()  # noqa: E731
    mat = lambda *shape, fan: host(_normal(gen, shape, fan ** -0.5))  # noqa: E731
    w = {"c0w": mat(S, 1, 3, 3, fan=9), "c1w": mat(S, 1, 3, 3, fan=9), "c2w": mat(S, S, 1, 1, fan=S),
         "c3w": mat(S, 1, 3, 3, fan=9), "c4w": mat(S, S, 1, 1, fan=S), "linw": mat(S * fs, D, fan=S * fs),
         "linb": host(_normal(gen, D, 0.02))}
    w.update({"c%db" % i: host(_normal(gen, S, 0.02)) for i in range(5)})
    for L in range(ENC["layers"]):
        g = "L%d_" % L
        for n in ("lnff1", "lnatt", "lnconv", "lnff2", "lnout"):
            w[g + n + "_w"], w[g + n + "_b"] = np.ones(D, np.float32), np.zeros(D, np.float32)
        for n in ("ff1", "ff2"):
            w[g + n + "w1"], w[g + n + "w2"] = mat(D, F, fan=D), mat(F, D, fan=F)
        for n in ("q", "k", "v", "pos", "out"):
            w[g + n] = mat(D, D, fan=D)
        for n in ("pbu", "pbv"):
            w[g + n] = host(_normal(gen, (ENC["H"], ENC["HD"]), 0.02))
        w[g + "pw1"], w[g + "pw2"] = mat(2 * D, D, 1, fan=D), mat(D, D, 1, fan=D)
        w[g + "dw"], w[g + "dwb"] = mat(D, 1, ENC["dwK"], fan=ENC["dwK"]), host(_normal(gen, D, 0.02))
    ctx = fa.CudaContext(0)
    return ctx, fastconformer.load_encoder(ctx, w)


def _decoder(weights):
    ctx = fa.CudaContext(0)
    w = _engine("decoder weights", lambda: synth.decoder_weights(DEC))
    dec = whisper_decoder.load_decoder(ctx, w, DEC["NH"], "int8" if weights == "int8" else None)
    return ctx, whisper_decoder.resident_tables(ctx, dec)


def _tdt():
    ctx = fa.CudaContext(0)
    return ctx, tdt_decoder.TdtDecoder(ctx, tdt_decoder.synth_tdt_weights())


class _Buffer:
    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f4", "version": 3}


def _view(ctx, t):
    """A tensor of the context as a torch tensor on the same memory."""
    return torch.as_tensor(_Buffer(ctx.devicePtr(t), (t.rows, t.cols)), device="cuda")


def _fill(ctx, values):
    """A tensor of the context that holds `values`, a torch tensor on the GPU."""
    t = ctx.alloc(*values.shape)
    _view(ctx, t).copy_(values)
    torch.cuda.synchronize()
    return t


class _State:
    """What one case keeps; its tensors go back to the context's pool with it."""

    def __init__(self, ctx, case):
        self.ctx, self.case, self.tensors, self.bytes, self.graph, self.out = ctx, case, [], [], None, []

    def keep(self, t):
        self.tensors.append(t)
        return t

    def keep_bytes(self, b):
        self.bytes.append(b)
        return b

    def release_outputs(self):
        for t in self.out:
            self.ctx.freeTensor(t)
        self.out = []

    def __del__(self):
        try:
            self.ctx.sync()
            self.release_outputs()
            if self.graph is not None:
                self.graph.free()
            for t in self.tensors:
                self.ctx.freeTensor(t)
            for b in self.bytes:
                self.ctx.freeBytes(b)
        except Exception:  # the process is ending
            pass


# ---- blocks ------------------------------------------------------------------------------------------------------------

def _weight(s, gen, kind, K, N):
    """A [K, N] matrix in the storage asked for, gain about 1."""
    ctx = s.ctx
    if kind == "int4":
        nblk = K // 32
        q = torch.randint(0, 256, (N * nblk * 16,), generator=gen, device="cuda", dtype=torch.uint8)
        top = 2.0 / (4.6 * math.sqrt(K))
        sc = (torch.rand(N * nblk, generator=gen, device="cuda") * (0.75 * top) + 0.25 * top).half().float()
        zp = np.full(N * ((nblk + 1) // 2), 0x88, np.uint8)
        return (s.keep_bytes(ctx.uploadBytes(q.cpu().numpy())), s.keep(ctx.upload(sc.cpu().numpy(), 1, N * nblk)),
                s.keep_bytes(ctx.uploadBytes(zp)), N, K)
    if kind == "int8":
        q = torch.randint(-127, 128, (K * N,), generator=gen, device="cuda", dtype=torch.int8)
        top = 2.0 / (73.3 * math.sqrt(K))
        sc = torch.rand(N, generator=gen, device="cuda") * (0.9 * top) + 0.1 * top
        return s.keep_bytes(ctx.uploadBytes(q.cpu().numpy())), s.keep(ctx.upload(sc.cpu().numpy(), 1, N)), N, K
    w = _normal(gen, (K, N), K ** -0.5).cpu().numpy()
    return (s.keep(ctx.uploadF16(w, K, N) if kind == "f16" else ctx.upload(w, K, N)),)


def _block(s, x, up, down, bias_up, bias_down):
    ctx, kind = s.ctx, s.case["weights"]
    n = ctx.layernorm(x, *s.norm)
    if kind == "int4":
        h = ctx.matmulNBits(n, up[0], up[1], up[2], up[3])
        return ctx.matmulNBits(h, down[0], down[1], down[2], down[3])
    if kind == "int8":
        h = ctx.matmulInt8(n, up[0], up[1], up[2], up[3], bias=bias_up, act="silu")
        return ctx.matmulInt8(h, down[0], down[1], down[2], down[3], bias=bias_down)
    h = ctx.matmul(n, up[0], bias=bias_up, act="silu")
    return ctx.matmul(h, down[0], bias=bias_down, add=x)


def _prepare_blocks(case, seed):
    ctx = _engine("blocks", lambda: fa.CudaContext(0))
    s, gen = _State(ctx, case), _generator(seed)
    D, F = case["width"], case["hidden"]
    s.x = s.keep(_fill(ctx, _normal(gen, (case["rows"], D))))
    s.norm = (s.keep(_fill(ctx, _normal(gen, (1, D), 0.05) + 1)), s.keep(_fill(ctx, _normal(gen, (1, D), 0.02))))
    s.layers = [(_weight(s, gen, case["weights"], D, F), _weight(s, gen, case["weights"], F, D),
                 s.keep(_fill(ctx, _normal(gen, (1, F), 0.02))), s.keep(_fill(ctx, _normal(gen, (1, D), 0.02))))
                for _ in range(case["blocks"])]

    def forward():
        arena = ctx.pushArena()
        y = s.x
        for layer in s.layers:
            y = _block(s, y, *layer)
        ctx.pin(y)
        ctx.popArena(arena)
        return y

    ctx.freeTensor(forward())  # handles do their one-time work on first use
    s.graph, y = ctx.recordBatch(forward)
    s.keep(y)
    ctx.sync()
    s.result = _view(ctx, y)
    return s


def _run_blocks(s):
    s.graph.launch()
    return s.result


# ---- encoder -----------------------------------------------------------------------------------------------------------

def _audio(gen, windows, samples):
    """Pink noise of unit RMS times an amplitude, plus one to four tones, as in engines/synth.py."""
    f = torch.fft.rfftfreq(samples, 1 / 16000.0, device="cuda").clamp_min(16000.0 / samples)
    x = torch.fft.irfft(torch.fft.rfft(_normal(gen, (windows, samples))) * f.rsqrt(), samples)
    uniform = lambda *shape: torch.rand(shape, generator=gen, device="cuda")  # noqa: E731
    x = x / x.square().mean(1, keepdim=True).sqrt() * (0.05 + 0.45 * uniform(windows, 1))
    t = torch.arange(samples, device="cuda") / 16000.0
    for k in range(4):
        there = (uniform(windows, 1) < (1.0 if k == 0 else 0.5)).float()
        amp, freq, phase = 0.05 + 0.45 * uniform(windows, 1), 100 + 3900 * uniform(windows, 1), 2 * math.pi * uniform(windows, 1)
        x = x + there * amp * torch.sin(2 * math.pi * freq * t + phase)
    return x.contiguous()


def _prepare_encoder(case, seed):
    ctx, enc = _engine("encoder", _encoder)
    s = _State(ctx, case)
    s.enc = enc
    s.audio = s.keep(_fill(ctx, _audio(_generator(seed), case["windows"], case["samples"])))
    return s


def _run_encoder(s):
    ctx = s.ctx
    s.release_outputs()
    arena = ctx.pushArena()
    x, _ = fastconformer.encode_batch(ctx, s.enc, ctx.logMelWindows(s.audio, ENC["melBins"]))
    ctx.pin(x)
    ctx.popArena(arena)
    s.out = [x]
    return _view(ctx, x)


# ---- decoder -----------------------------------------------------------------------------------------------------------

def _prepare_decoder(case, seed):
    ctx, dec = _engine("decoder " + case["weights"], lambda: _decoder(case["weights"]))
    s, gen = _State(ctx, case), _generator(seed)
    S, n = case["streams"], case["tokens"]
    s.dec = dec
    s.states = s.keep(_fill(ctx, _normal(gen, (S * DEC["Tenc"], DEC["D"]))))
    ids = torch.randint(0, DEC["VOCAB"], (n, S), generator=gen, device="cuda")
    if S == 1:
        s.ids = [int(i) for i in ids[:, 0].cpu()]
        s.cache = whisper_decoder.decode_init(ctx, dec, n)
    else:
        s.ids = [s.keep(_fill(ctx, ids[i].float().reshape(S, 1))) for i in range(n)]
        s.cache = whisper_decoder.decode_init_streams(ctx, dec, S, n)
    for t in s.cache["selfK"] + s.cache["selfV"]:
        s.keep(t)
    return s


def _run_decoder_one(s):
    ctx, dec = s.ctx, s.dec
    kv = whisper_decoder.cross_kv(ctx, dec, s.states)
    s.cache["n"] = 0
    logits = [whisper_decoder.decode_next(ctx, dec, kv, s.cache, i) for i in s.ids]
    for c in kv:
        ctx.freeTensor(c["k"])
        ctx.freeTensor(c["v"])
    return {"logits": logits, "pick": int(np.argmax(logits[-1]))}


def _run_decoder_streams(s):
    ctx, dec, vocab = s.ctx, s.dec, DEC["VOCAB"]
    s.release_outputs()
    kv = whisper_decoder.cross_kv_streams(ctx, dec, s.states)
    out = []
    for n, ids in enumerate(s.ids):
        arena = ctx.pushArena()
        x = ctx.embedRows(dec["embedDev"], dec["posDev"], ids, n)
        logits = whisper_decoder.step_streams(ctx, dec, kv, s.cache, x, n)
        pick = ctx.argmaxRowsIndex(logits, vocab)
        s.out += [ctx.pin(logits), ctx.pin(pick)]
        ctx.popArena(arena)
        out.append((_view(ctx, logits)[:, :vocab], _view(ctx, pick)))
    for c in kv:
        ctx.freeTensor(c["k"])
        ctx.freeTensor(c["v"])
    return {"logits": [lg for lg, _ in out], "best": [p[:, 1] for _, p in out]}


# ---- tdt ---------------------------------------------------------------------------------------------------------------

def _prepare_tdt(case, seed):
    ctx, dec = _engine("tdt", _tdt)
    s = _State(ctx, case)
    s.dec = dec
    s.frames = s.keep(_fill(ctx, _normal(_generator(seed), (case["windows"] * case["frames"], tdt_decoder.ENC_D))))
    return s


def _run_tdt(s):
    W, T = s.case["windows"], s.case["frames"]
    arena = s.ctx.pushArena()
    found = s.dec.decode_proj(s.dec.project(s.frames), W, T)
    s.ctx.popArena(arena)
    most = 10 * T  # ten symbols per frame at most
    ids, at = np.full((W, most), -1, np.int32), np.full((W, most), -1, np.int32)
    for w, (i, f) in enumerate(found):  # one row per window
        ids[w, :i.size], at[w, :i.size] = i, f
    return {"ids": ids, "frames": at, "counts": np.array([i.size for i, _ in found], np.int32)}


# ---- the interface -----------------------------------------------------------------------------------------------------

def prepare(case, seed):
    return {"blocks": _prepare_blocks, "encoder": _prepare_encoder, "decoder": _prepare_decoder, "tdt": _prepare_tdt}[case["kind"]](case, seed)


def run(state):
    kind = state.case["kind"]
    if kind == "decoder":
        return _run_decoder_one(state) if state.case["streams"] == 1 else _run_decoder_streams(state)
    return {"blocks": _run_blocks, "encoder": _run_encoder, "tdt": _run_tdt}[kind](state)


def work(case):
    if case["kind"] == "blocks":
        n, M, D, F = case["blocks"], case["rows"], case["width"], case["hidden"]
        return {"bytes": n * (2 * D * F * WEIGHT_BYTES[case["weights"]] + 4 * (D + F)) + 8 * M * D, "flops": 4.0 * n * M * D * F}
    if case["kind"] == "encoder":
        W, N = case["windows"], case["samples"]
        D, F, S, mel = ENC["D"], ENC["DFF"], ENC["Csub"], ENC["melBins"]
        T = N // 160
        t1, t2, t3 = (T + 1) // 2, (T + 3) // 4, (T + 7) // 8
        stem = S * (9 * t1 * mel / 2 + (9 + S) * t2 * mel / 4 + (9 + S) * t3 * mel / 8) + t3 * (S * mel / 8) * D
        block = t3 * (4 * D * F + 4 * D * D + 3 * D * D + ENC["dwK"] * D) + 3 * t3 * t3 * D + (2 * t3 - 1) * D * D / W
        weights = ENC["layers"] * (4 * D * F + 8 * D * D) + S * mel / 8 * D
        return {"bytes": 2.0 * weights + 4.0 * W * (N + t3 * D), "flops": 2.0 * W * (stem + ENC["layers"] * block)}
    if case["kind"] == "decoder":
        S, n, L, D, F, V, Te = case["streams"], case["tokens"], DEC["layers"], DEC["D"], DEC["FFN"], DEC["VOCAB"], DEC["Tenc"]
        w = WEIGHT_BYTES[case["weights"]]
        step = L * (6 * D * D + 2 * D * F) + D * V
        cross = 2 * L * D * D
        return {"bytes": w * (cross + n * step) + 4.0 * S * Te * D * (1 + 2 * L * (1 + n)) + 4.0 * S * n * V,
                "flops": 2.0 * S * (Te * cross + n * (step + 2 * L * Te * D))}
    W, T, H, V, E = case["windows"], case["frames"], tdt_decoder.HID, tdt_decoder.LOGITS, tdt_decoder.ENC_D
    # one look at the joint for each frame; the weights of the prediction network and the joint read once
    return {"bytes": H * V + 4.0 * 13 * H * H + 2.0 * E * H + 4.0 * W * T * E, "flops": 2.0 * W * T * H * (V + E)}


def tolerance(case):
    # Four times the largest distance seen: blocks from the same chain in f64, the encoder and the decoder from themselves
    # with value + residue operands throughout (encoder: also from the unfused op sequence), over sizes of these ranges.
    if case["kind"] == "blocks":
        return {"rel": {"int4": 2.4e-3, "int8": 1.8e-3, "f16": 1.3e-3, "f32": 1.5e-4}[case["weights"]]}
    if case["kind"] == "encoder":
        return {"rel": 1.3e-3}
    if case["kind"] == "decoder":
        return {"rel": {"f16": 1.5e-4, "int8": 8e-4}[case["weights"]]}
    return {"differ": 5e-4}  # whole values: a pick between two logits that tie in f32 may fall either way

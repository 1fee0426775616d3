"""Performance cases: the transcription path stage by stage and as whole calls, through the public Python API.

Stages: log-mel frontend (`ParakeetFeatureExtractor.extract_device`), encoder (`encode_device`, whole stacks, single
blocks and the FP8 option), TDT decode (`tdt_decode_device`), voice-activity network (`SileroVad.process`).  Whole calls:
`TranscriptionPipeline.run` and `LongFormTranscriptionPipeline.run_with_config` from host audio.

Audio is the seeded sinusoid + noise distribution of `scriptrs_b200.synth`.  Encoder weights are seeded N(0, 0.02) with
identity norms.  The predictor / joint weights are built so that decisions have the margins of a trained model (see
`_decoder_weights`): tokens then do not hang on rounding, and the confidences carry the numerics.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import scriptrs_b200 as sb
from scriptrs_b200 import synth

D, HEADS, FF, H, VOCAB = 1024, 8, 4096, 640, 1025
BLANK = VOCAB - 1
MAX_CLIP = 240_000  # samples: 15 s, the model's longest chunk
VAD_WINDOW = 512


# ------------------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # a voice command or dictation turn: one clip, nothing to batch with
        dict(name="frontend_clip_15s", kind="frontend", clips=1, samples=240_000, ragged=False, int16=False),
        # a WAV ingest batch: 16-bit PCM, clips of every length, most of them at odd places of the buffer
        dict(name="frontend_i16_ragged", kind="frontend", clips=97, samples=239_357, ragged=True, int16=True),
        # the bulk feature extraction benchmark: 1024 clips of 30 s
        dict(name="frontend_1024x30s", kind="frontend", clips=1024, samples=480_000, ragged=False, int16=False),
        # the whole encoder on one chunk: what an interactive caller waits for
        dict(name="encoder_clip_15s", kind="encoder", layers=24, clips=1, frames=1501, ragged=False, fp8=False),
        # a serving batch: 32 clips of 10 s through 24 blocks
        dict(name="encoder_32x10s", kind="encoder", layers=24, clips=32, frames=1001, ragged=False, fp8=False),
        # one Conformer block behind the sub-sampling at bulk size: the chunks of two hours of audio
        dict(name="encoder_block_2h", kind="encoder", layers=1, clips=560, frames=1497, ragged=False, fp8=False),
        # the FP8 option (its default product), clips of mixed length
        dict(name="encoder_fp8_ragged", kind="encoder", layers=4, clips=141, frames=1501, ragged=True, fp8=True),
        # decode of one clip: latency of a step-by-step loop
        dict(name="decode_clip", kind="decode", clips=1, frames=188, ragged=False),
        # decode of an hour of chunks
        dict(name="decode_1h", kind="decode", clips=280, frames=187, ragged=True),
        # voice activity of a ten-minute recording from host memory: one long recurrence
        dict(name="vad_10min", kind="vad", samples=9_600_123),
        # the simplest user program: one utterance in, transcript out
        dict(name="pipeline_clip_11s", kind="pipeline", samples=176_543),
        # an hour-long recording through the long-form pipeline
        dict(name="longform_1h", kind="longform", samples=57_600_000, vad=False),
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frontend", "frontend", "encoder", "block", "fp8", "decode", "decode", "vad", "pipeline", "longform"])
    ragged = rng.random() < 0.6
    if kind == "frontend":
        return dict(kind="frontend", clips=_between(rng, 1, 1024), samples=_between(rng, 1_600, 480_000), ragged=ragged,
                    int16=rng.random() < 0.4)
    if kind == "encoder":
        return dict(kind="encoder", layers=24, clips=_between(rng, 1, 32), frames=rng.randint(60, 1001), ragged=ragged, fp8=False)
    if kind == "block":
        return dict(kind="encoder", layers=1, clips=_between(rng, 1, 560), frames=rng.randint(60, 1497), ragged=ragged, fp8=False)
    if kind == "fp8":
        return dict(kind="encoder", layers=4, clips=_between(rng, 2, 141), frames=rng.randint(200, 1501), ragged=ragged, fp8=True)
    if kind == "decode":
        return dict(kind="decode", clips=_between(rng, 1, 280), frames=rng.randint(12, 188), ragged=ragged)
    if kind == "vad":
        return dict(kind="vad", samples=_between(rng, 16_000, 9_600_000))
    if kind == "pipeline":
        return dict(kind="pipeline", samples=_between(rng, 16_000, MAX_CLIP))
    return dict(kind="longform", samples=_between(rng, 480_000, 28_800_000), vad=rng.random() < 0.3)


def _lengths(case, what):
    """Sizes of the clips; ragged batches spread over a third of the longest upwards."""
    n, most = case["clips"], case[what]
    if not case["ragged"]:
        return [most] * n
    return [most] + [max(1, int(most * (0.34 + 0.66 * ((i * 0.6180339887) % 1.0)))) for i in range(1, n)]


def _offsets(lengths):
    return np.concatenate([np.zeros(1, np.int64), np.cumsum(np.asarray(lengths, np.int64))])


def _sub(t):
    return (t - 1) // 2 + 1


def _enc_frames(t):
    return _sub(_sub(_sub(t)))


# ---------------------------------------------------------------------------------------------------------- weights
def _randn(shape, std, seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return torch.randn(*shape, generator=g, device=device) * std


_encoder_cache = {}
_decoder_cache = {}


def _encoder_weights(layers):
    """Seeded N(0, 0.02) matrices and biases, identity norms; a shallow stack is the first blocks of the deep one."""
    if layers not in _encoder_cache:
        w = {}
        for i, (name, shape) in enumerate(synth.encoder_weight_shapes(layers).items()):
            if ".norm" in name or "norm_" in name:
                one = name.endswith(("weight", "running_var"))
                w[name] = torch.ones(*shape, device="cuda") if one else torch.zeros(*shape, device="cuda")
            else:
                w[name] = _randn(shape, 0.02, 1000 + i)
        _encoder_cache[layers] = w
    return _encoder_cache[layers]


# Joint dimensions: token patterns from the predictor, durations and blank from the encoder row, durations from the predictor
_TOK, _EDUR, _BLK, _PDUR = slice(0, 580), slice(580, 600), slice(600, 620), slice(620, 640)
_LIVE = 96  # tokens that the built model uses; the others keep a small random output row


def _lstm(w, x, h, c):
    """Two LSTM layers, gate order i, f, g, o; x [B, 640], h and c lists of [B, 640] in the dtype of w."""
    ho, co = [], []
    for layer in range(2):
        g = x @ w["predictor.lstm.weight_ih"][layer].T + h[layer] @ w["predictor.lstm.weight_hh"][layer].T
        g = g + w["predictor.lstm.bias_ih"][layer] + w["predictor.lstm.bias_hh"][layer]
        i, f, n, o = g.split(H, 1)
        cn = torch.sigmoid(f) * c[layer] + torch.sigmoid(i) * torch.tanh(n)
        x = torch.sigmoid(o) * torch.tanh(cn)
        ho.append(x)
        co.append(cn)
    return ho, co


def _decoder_weights():
    """Predictor / joint weights with a trained model's margins.  After token t the predictor asks for a token next(t) and
    a duration; an encoder row whose entries 600..619 are large asks for the blank, and its entries 580..599 for the
    blank's duration.  Everything else is small seeded noise, which moves the confidences and not the decisions."""
    if _decoder_cache:
        return _decoder_cache
    w = {n: _randn(s, 0.05, 50 + i) for i, (n, s) in enumerate(synth.DECODER_SHAPES.items())}
    w["predictor.embedding"] = _randn((VOCAB, H), 1.0, 71)
    w["predictor.lstm.weight_hh"] = _randn((2, 4 * H, H), 0.015, 72)
    w["predictor.lstm.bias_ih"][:, H:2 * H] -= 2.0  # a short memory
    g = torch.Generator().manual_seed(73)
    chain = torch.cat([torch.randperm(_LIVE, generator=g), torch.tensor([BLANK])])  # the blank stands for the start
    following = chain[:_LIVE].roll(-1)
    pattern = (torch.rand(_LIVE + 1, 580, generator=g) < 0.3).double().cuda()
    pattern[_LIVE] = pattern[_LIVE - 1]  # from the start as from the chain's last token
    dur = torch.multinomial(torch.tensor([0.03, 0.35, 0.30, 0.20, 0.12]), _LIVE + 1, replacement=True, generator=g)
    want = torch.zeros(_LIVE + 1, H, dtype=torch.float64, device="cuda")
    want[:, _TOK] = 2.0 * pattern - 1.0
    want[:, _PDUR] = -2.0
    for d in range(5):
        want[(dur == d).cuda(), 620 + 4 * d:624 + 4 * d] = 2.0
    w64 = {k: v.double() for k, v in w.items()}
    zero = [torch.zeros(_LIVE + 1, H, dtype=torch.float64, device="cuda")] * 2
    h, _ = _lstm(w64, w64["predictor.embedding"][chain.cuda()], zero, zero)
    w["joint.pred.weight"] = (torch.linalg.pinv(h[1]) @ want).T.float()
    w["joint.pred.bias"] = torch.zeros(H, device="cuda")
    enc = _randn((H, D), 0.008, 74)
    bias = torch.zeros(H, device="cuda")
    enc[_PDUR] = 0.0
    for j in range(580, 620):
        enc[j] = 0.0
        enc[j, j] = 1.0
        bias[j] = -6.0
    w["joint.enc.weight"], w["joint.enc.bias"] = enc, bias
    out = _randn((VOCAB + 5, H), 0.02, 75)
    out[:, 580:] = 0.0
    out[following.cuda(), _TOK] += ((pattern[:_LIVE] - 0.3) * (8.0 / 122.0)).float()
    out[BLANK, _BLK] = 0.1
    out[VOCAB:, _TOK] *= 0.2
    for d in range(5):
        out[VOCAB + d, 580 + 4 * d:584 + 4 * d] = 1.0
        out[VOCAB + d, 620 + 4 * d:624 + 4 * d] = 1.0
    w["joint.out.weight"] = out
    w["joint.out.bias"] = _randn((VOCAB + 5,), 0.02, 76)
    _decoder_cache.update(w)
    return _decoder_cache


def _host(w):
    return {k: v.cpu().numpy() for k, v in w.items()}


_handles = {}  # contexts with their models, kept for the life of a user's program


def _context(layers=0, fp8=False, vad=None):
    """One context per model: encoder blocks (with predictor and joint), the FP8 option, or a voice-activity network."""
    key = (layers, fp8, vad)
    if key not in _handles:
        ctx = sb.Context(0)
        if layers:
            w = dict(_encoder_weights(layers), **_decoder_weights())
            sb.load_model(ctx, _host(w), layers, has_encoder=True, has_decoder=True, fp8_weights=fp8)
            if layers != 24:
                _encoder_cache.pop(layers)
        elif vad is None:
            sb.load_model(ctx, _host(_decoder_weights()), 0, has_encoder=False, has_decoder=True)
        if fp8:
            ctx.set_option("fp8", 1)
        net = None
        if vad is not None:
            net = sb.SileroVad(ctx, weights=synth.seeded_vad_weights(5) if vad == "seeded" else synth.energy_vad_weights())
        _handles[key] = (ctx, net)
    return _handles[key]


# ----------------------------------------------------------------------------------------------------------- inputs
def _pcm(lengths, seed, int16=False):
    """One packed buffer of clips, each with sinusoids of its own."""
    most = max(lengths)
    packed = torch.empty(int(sum(lengths)), dtype=torch.int16 if int16 else torch.float32, device="cuda")
    at, step = 0, max(1, (1 << 27) // most)
    for i in range(0, len(lengths), step):
        block = synth.clip_batch_torch(min(step, len(lengths) - i), most, (seed * 7919 + i) % (1 << 31), "cuda", silent_every=0)
        if int16:
            block = (block * 32767.0).round_().to(torch.int16)
        for k, n in enumerate(lengths[i:i + step]):
            packed[at:at + n] = block[k, :n]
            at += n
    return packed


def _recording(n, seed, sparse=False):
    """A host recording.  sparse: sound and near-silence, for the voice-activity mode."""
    x = synth.long_audio_torch(n, seed % (1 << 31), "cuda")
    if sparse:
        x += _randn((n,), 1e-4, seed % (1 << 31) + 1)
    return x.cpu().numpy()


def _features(frames, seed):
    """Normalised log-mel rows of one clip per length, packed; made with torch so that they are inputs like any other."""
    out = torch.empty(int(sum(frames)), 128, device="cuda")
    at = 0
    for i in range(0, len(frames), 32):
        part = frames[i:i + 32]
        pcm = synth.clip_batch_torch(len(part), 160 * (max(part) - 1) + 80, (seed * 104729 + i) % (1 << 31), "cuda", silent_every=0)
        for k, t in enumerate(part):
            out[at:at + t] = _logmel(pcm[k, :160 * (t - 1) + 80], torch.float32)
            at += t
    return out


def _encoder_rows(lengths, seed):
    """Rows as a trained encoder hands them to the joint: unit variance; about two of three frames ask for the blank."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed % (1 << 31))
    n = int(sum(lengths))
    x = torch.randn(n, D, generator=g, device="cuda")
    blank = torch.rand(n, generator=g, device="cuda") < 0.65
    dur = torch.multinomial(torch.tensor([0.25, 0.45, 0.18, 0.08, 0.04], device="cuda"), n, replacement=True, generator=g)
    ask = torch.zeros(n, 40, device="cuda")
    ask[blank, 20:] = 12.0
    for d in range(5):
        ask[blank & (dur == d), 4 * d:4 * d + 4] = 12.0
    x[:, 580:620] += ask
    return x


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frontend":
        lengths = _lengths(case, "samples")
        frames = [n // 160 + 1 for n in lengths]
        return dict(kind=kind, extractor=sb.ParakeetFeatureExtractor(_context(vad="seeded")[0]), pcm=_pcm(lengths, seed, case["int16"]),
                    offsets=_offsets(lengths), feats=torch.empty(sum(frames), 128, device="cuda"), int16=case["int16"])
    if kind == "encoder":
        frames = _lengths(case, "frames")
        rows = sum(_enc_frames(t) for t in frames)
        return dict(kind=kind, ctx=_context(case["layers"], case["fp8"])[0], feats=_features(frames, seed), offsets=_offsets(frames),
                    out=torch.empty(rows, D, device="cuda"))
    if kind == "decode":
        lengths = _lengths(case, "frames")
        return dict(kind=kind, ctx=_context()[0], rows=_encoder_rows(lengths, seed), offsets=_offsets(lengths),
                    width=2 * case["frames"] + 10)
    if kind == "vad":
        return dict(kind=kind, net=_context(vad="seeded")[1], audio=_recording(case["samples"], seed))
    ctx, _ = _context(24)
    vocab = sb.Vocabulary.from_tokens(["▁w%d" % i if i % 3 == 0 else "s%d" % i for i in range(BLANK)] + ["<blk>"])
    pipe = sb.TranscriptionPipeline(ctx, vocab)
    width = case["samples"] // 1000 + 16
    if kind == "pipeline":
        return dict(kind=kind, pipe=pipe, width=width, audio=_pcm([case["samples"]], seed).cpu().numpy())
    config = sb.LongFormConfig(mode=sb.LongFormMode.Vad if case["vad"] else sb.LongFormMode.Fast)
    if case["vad"]:
        sb.SileroVad(ctx, weights=synth.energy_vad_weights())
    return dict(kind=kind, pipe=sb.LongFormTranscriptionPipeline(pipe), config=config, width=width,
                audio=_recording(case["samples"], seed, sparse=case["vad"]))


def _dense(rows, width):
    """Streams of different lengths as one zero-filled array."""
    out = np.zeros((len(rows), width), rows[0].dtype)
    for i, r in enumerate(rows):
        out[i, :len(r)] = r[:width]
    return out


def _tokens(r, width):
    """Tokens and confidences of a transcript, zero-filled: their number depends on the recording in the voice-activity mode."""
    return [_dense([v], width)[0] for v in (r.token_ids, r.starts, r.ends, r.confidences)]


def run(state):
    kind = state["kind"]
    if kind == "frontend":
        state["extractor"].extract_device(state["pcm"].data_ptr(), state["offsets"], state["feats"].data_ptr(), int16=state["int16"])
        return state["feats"]
    if kind == "encoder":
        sb.encode_device(state["ctx"], state["feats"].data_ptr(), state["offsets"], state["out"].data_ptr())
        return state["out"]
    if kind == "decode":
        clips = sb.tdt_decode_device(state["ctx"], state["rows"].data_ptr(), state["offsets"])
        return [_dense([c[k] for c in clips], state["width"]) for k in ("tokens", "frames", "durations", "conf")]
    if kind == "vad":
        return state["net"].process(state["audio"])
    if kind == "pipeline":
        return _tokens(state["pipe"].run(state["audio"]), state["width"])
    return _tokens(state["pipe"].run_with_config(state["audio"], state["config"]), state["width"])


# ------------------------------------------------------------------------------------------------- work and tolerance
def _encoder_work(frames, layers):
    flops = 0.0
    for t in frames:
        t1 = _sub(t)
        t2 = _sub(t1)
        t3 = _sub(t2)
        flops += 2 * (t1 * 64 * 256 * 9 + t2 * 32 * 256 * (9 + 256) + t3 * 16 * 256 * (9 + 256) + t3 * 4096 * D)
        # feed-forward twice, QKV, output, pointwise convolutions, depthwise; attention: q k, q p over 2 t - 1, p v
        flops += layers * 2 * (t3 * D * (4 * FF + 3 * D + D + 2 * D + D + 9) + D * t3 * (t3 + 2 * t3 - 1 + t3))
    weights = 2 * (2 * 65536 + 4096 * D) + layers * 2 * (4 * D * FF + 8 * D * D)  # bf16; relative-position table projected once
    return dict(bytes=weights + sum(4 * 128 * t + 4 * D * _enc_frames(t) for t in frames), flops=flops)


def _decode_work(lengths):
    frames = float(sum(lengths))
    steps = frames / 1.3  # about 1.3 frames a step
    weights = 4 * (2 * 4 * H * 2 * H + H * H + (VOCAB + 5) * H + H * D)
    flops = 2 * (steps * (2 * 4 * H * 2 * H + H * H + (VOCAB + 5) * H) + frames * H * D)
    return dict(bytes=weights + 4 * D * frames + 20 * steps * 0.35, flops=flops)


def work(case):
    kind = case["kind"]
    if kind == "frontend":
        lengths = _lengths(case, "samples")
        frames = sum(n // 160 + 1 for n in lengths)
        # window, real 512-point transform, power, 257 + 255 filterbank taps, logarithm, statistics
        return dict(bytes=(2 if case["int16"] else 4) * sum(lengths) + 512 * frames, flops=frames * (400 + 2.5 * 512 * 9 + 257 * 3 + 2 * 512 + 128 * 6))
    if kind == "encoder":
        return _encoder_work(_lengths(case, "frames"), case["layers"])
    if kind == "decode":
        return _decode_work(_lengths(case, "frames"))
    if kind == "vad":
        windows = -(-case["samples"] // VAD_WINDOW)
        return dict(bytes=4 * case["samples"] + 4 * windows + 1.3e6, flops=windows * (1.2e6 + 2 * 128 * 512))
    if kind == "pipeline":
        chunks = [case["samples"]]
    else:
        stride, length = 206_080, 239_360
        chunks = [min(length, case["samples"] - at) for at in range(0, max(1, case["samples"] - 32_000), stride)]
        if case["vad"]:
            chunks = [int(0.7 * n) for n in chunks]
    frames = [n // 160 + 1 for n in chunks]
    enc, dec = _encoder_work(frames, 24), _decode_work([_enc_frames(t) for t in frames])
    return dict(bytes=4 * case["samples"] + enc["bytes"] + dec["bytes"], flops=enc["flops"] + dec["flops"])


def tolerance(case):
    kind = case["kind"]
    if kind == "frontend":
        return dict(rel=2e-5, max=1e-3)  # f32 transform and statistics; the logarithm of near-empty cells
    if kind == "encoder":
        return dict(rel=0.03 if case["layers"] > 1 else 0.016, max=0.3)  # bf16 operands through a stack of blocks
    if kind == "decode":
        return dict(rel=2e-4, max=2e-3, differ=0.001)  # split products: 2^-16 of an operand
    if kind == "vad":
        return dict(rel=2e-5, max=5e-4)  # f32 recurrence
    return dict(rel=0.01, max=0.1, differ=0.002)  # confidences behind the bf16 encoder


# ------------------------------------------------------------------------------------------------------------ 64 bits
_tables = {}


def _mel_tables():
    """Hann window of 400 (symmetric) and the 128 x 257 Slaney filterbank."""
    if not _tables:
        _tables["window"] = torch.from_numpy(0.5 - 0.5 * np.cos(2.0 * np.pi * np.arange(400) / 399.0)).cuda()
        top = 15.0 + math.log(8.0) / 0.06875177742094912
        mel = np.linspace(0.0, top, 130)
        edge = np.where(mel < 15.0, mel * 200.0 / 3.0, 1000.0 * np.exp((mel - 15.0) * 0.06875177742094912))
        hz = np.arange(257) * 31.25
        up = (hz[None] - edge[:-2, None]) / (edge[1:-1] - edge[:-2])[:, None]
        down = (edge[2:, None] - hz[None]) / (edge[2:] - edge[1:-1])[:, None]
        bank = np.maximum(0.0, np.minimum(up, down)) * (2.0 / (edge[2:] - edge[:-2]))[:, None]
        _tables["bank"] = torch.from_numpy(bank).cuda()
    return _tables["window"], _tables["bank"]


def _logmel(x, dtype=torch.float64):
    """One clip -> normalised log-mel [T, 128]."""
    window, bank = _mel_tables()
    x = x.to(dtype)
    y = x.clone()
    y[1:] -= 0.97 * x[:-1] if dtype != torch.float64 else float(np.float32(0.97)) * x[:-1]
    y = torch.nn.functional.pad(y, (256, 256))
    frames = y.unfold(0, 512, 160)[:, :400] * window.to(dtype)
    power = torch.fft.rfft(frames, n=512).abs().square()
    v = torch.log(power @ bank.to(dtype).T + 2.0 ** -24)
    return (v - v.mean(0)) / (v.std(0, unbiased=True) + 1e-5)


def _conv3(x, w, b):
    """Depthwise 3 x 3, stride 2, padding 1 over [T, F, C]."""
    t, f, _ = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    to, fo = _sub(t), _sub(f)
    y = sum(p[i:i + 2 * to - 1:2, j:j + 2 * fo - 1:2] * w[:, 0, i, j] for i in range(3) for j in range(3))
    return y + b


def _encode(w, feats):
    """One clip [T, 128] -> [T', 1024] in 64 bits; w: the named weights (converted layer by layer)."""
    f = {k: v.double() for k, v in w.items() if k.startswith("subsampling")}
    p = torch.nn.functional.pad(feats.double()[None, None], (1, 1, 1, 1))[0, 0]
    patches = p.unfold(0, 3, 2).unfold(1, 3, 2).reshape(_sub(feats.shape[0]), 64, 9)
    x = torch.relu(patches @ f["subsampling.layers.0.weight"].reshape(256, 9).T + f["subsampling.layers.0.bias"])
    for dw, pw in ((2, 3), (5, 6)):
        x = _conv3(x, f["subsampling.layers.%d.weight" % dw], f["subsampling.layers.%d.bias" % dw])
        x = torch.relu(x @ f["subsampling.layers.%d.weight" % pw].reshape(256, 256).T + f["subsampling.layers.%d.bias" % pw])
    x = x.transpose(1, 2).reshape(x.shape[0], -1) @ f["subsampling.linear.weight"].T + f["subsampling.linear.bias"]
    return x


def _blocks(w, layers, xs):
    """The Conformer blocks over a list of clips [T', 1024]."""
    bounds = _offsets([x.shape[0] for x in xs])
    x = torch.cat(xs)
    most = max(len(v) for v in xs)
    ang = torch.arange(most - 1, -most, -1, device="cuda").double()[:, None] / 10000.0 ** (torch.arange(0, D, 2, device="cuda").double() / D)
    pos = torch.stack([ang.sin(), ang.cos()], -1).reshape(2 * most - 1, D)
    for i in range(layers):
        p = "layers.%d." % i
        f = {k[len(p):]: v.double() for k, v in w.items() if k.startswith(p)}
        lin = lambda v, n: v @ f[n + ".weight"].reshape(f[n + ".weight"].shape[0], -1).T + f[n + ".bias"]  # noqa: E731
        norm = lambda v, n: torch.nn.functional.layer_norm(v, (D,), f[n + ".weight"], f[n + ".bias"], 1e-5)  # noqa: E731
        ff = lambda v, n: lin(torch.nn.functional.silu(lin(v, n + ".linear1")), n + ".linear2")  # noqa: E731
        x = x + 0.5 * ff(norm(x, "norm_feed_forward1"), "feed_forward1")
        y = norm(x, "norm_self_att")
        q, k, v = (lin(y, "self_attn.%s_proj" % n).reshape(-1, HEADS, D // HEADS).transpose(0, 1) for n in "qkv")
        r = (pos @ f["self_attn.relative_k_proj.weight"].T).reshape(-1, HEADS, D // HEADS).transpose(0, 1)
        o = torch.empty_like(x)
        for a, b in zip(bounds[:-1], bounds[1:]):
            t = int(b - a)
            ac = (q[:, a:b] + f["self_attn.bias_u"][:, None]) @ k[:, a:b].transpose(1, 2)
            bd = (q[:, a:b] + f["self_attn.bias_v"][:, None]) @ r[:, most - t:most + t - 1].transpose(1, 2)
            at = t - 1 - (torch.arange(t, device="cuda")[:, None] - torch.arange(t, device="cuda")[None])
            s = torch.softmax((ac + bd.gather(2, at.expand(HEADS, t, t))) / math.sqrt(D // HEADS), -1)
            o[a:b] = (s @ v[:, a:b]).transpose(0, 1).reshape(t, D)
        x = x + lin(o, "self_attn.o_proj")
        y = lin(norm(x, "norm_conv"), "conv.pointwise_conv1")
        y = y[:, :D] * torch.sigmoid(y[:, D:])
        z = torch.empty_like(y)
        for a, b in zip(bounds[:-1], bounds[1:]):
            e = torch.nn.functional.pad(y[a:b], (0, 0, 4, 4))
            z[a:b] = sum(e[j:j + int(b - a)] * f["conv.depthwise_conv.weight"][:, 0, j] for j in range(9))
        z = z + f["conv.depthwise_conv.bias"]
        z = (z - f["conv.norm.running_mean"]) / torch.sqrt(f["conv.norm.running_var"] + 1e-5) * f["conv.norm.weight"] + f["conv.norm.bias"]
        x = x + lin(torch.nn.functional.silu(z), "conv.pointwise_conv2")
        x = x + 0.5 * ff(norm(x, "norm_feed_forward2"), "feed_forward2")
        x = norm(x, "norm_out")
    return x


def _decode(rows, offsets):
    """Greedy TDT decode in 64 bits: the confidences of each clip."""
    w = {k: v.double() for k, v in _decoder_weights().items()}
    n = len(offsets) - 1
    start = torch.as_tensor(offsets[:-1]).cuda()
    length = torch.as_tensor(np.diff(offsets)).cuda()
    enc = rows.double() @ w["joint.enc.weight"].T + w["joint.enc.bias"]
    h, c = ([torch.zeros(n, H, dtype=torch.float64, device="cuda")] * 2 for _ in range(2))
    token = torch.full((n,), BLANK, device="cuda")
    at, symbols = torch.zeros(n, dtype=torch.int64, device="cuda"), torch.zeros(n, dtype=torch.int64, device="cuda")
    conf, kept = [], []
    for step in range(11 * int(length.max()) + 2):
        alive = at < length
        if step % 8 == 0 and not bool(alive.any()):
            break
        hn, cn = _lstm(w, w["predictor.embedding"][token], h, c)
        pred = hn[1] @ w["joint.pred.weight"].T + w["joint.pred.bias"]
        z = torch.relu(enc[start + torch.minimum(at, length - 1)] + pred)
        logits = z @ w["joint.out.weight"].T + w["joint.out.bias"]
        p, t = torch.softmax(logits[:, :VOCAB], 1).max(1)
        d = logits[:, VOCAB:].argmax(1)
        emit = alive & (t != BLANK)
        conf.append(p)
        kept.append(emit)
        h = [torch.where(emit[:, None], a, b) for a, b in zip(hn, h)]
        c = [torch.where(emit[:, None], a, b) for a, b in zip(cn, c)]
        token = torch.where(emit, t, token)
        symbols = symbols + emit
        on = (d > 0) | (t == BLANK) | (symbols >= 10)
        at = torch.where(alive, at + torch.where(d > 0, d, on.long()), at)
        symbols = torch.where(on, torch.zeros_like(symbols), symbols)
    conf, kept = torch.stack(conf, 1), torch.stack(kept, 1)
    return [p[k].cpu().numpy() for p, k in zip(conf, kept)]


def _vad(audio):
    """Window probabilities in 64 bits: contexts, spectra and convolutions at once, the recurrence window by window."""
    w = {k: torch.from_numpy(v).double() for k, v in synth.seeded_vad_weights(5).items()}
    n = -(-audio.size // VAD_WINDOW)
    x = np.concatenate([audio, np.full(n * VAD_WINDOW - audio.size, audio[-1], np.float32)]).astype(np.float64)
    x = torch.from_numpy(np.concatenate([np.zeros(64), x])).unfold(0, 576, VAD_WINDOW).cuda()
    e = []
    for part in x.split(16384):
        y = torch.cat([part, part[:, -65:-1].flip(1)], 1).unfold(1, 256, 128)
        s = y @ w["stft.forward_basis_buffer"].reshape(258, 256).T.cuda()
        y = torch.sqrt(s[..., :129] ** 2 + s[..., 129:] ** 2)
        for i, stride in enumerate((1, 2, 2, 1)):
            k = w["encoder.%d.reparam_conv.weight" % i].cuda()
            y = torch.nn.functional.pad(y, (0, 0, 1, 1)).unfold(1, 3, stride)
            y = torch.relu(y.reshape(y.shape[0], y.shape[1], -1) @ k.reshape(k.shape[0], -1).T + w["encoder.%d.reparam_conv.bias" % i].cuda())
        e.append(y[:, 0] @ w["decoder.rnn.weight_ih"].T.cuda() + (w["decoder.rnn.bias_ih"] + w["decoder.rnn.bias_hh"]).cuda())
    gates = torch.cat(e).cpu().numpy()
    hh = np.ascontiguousarray(w["decoder.rnn.weight_hh"].numpy())
    h, c = np.zeros(128), np.zeros(128)
    out = np.empty((n, 128))
    for k in range(n):
        g = gates[k] + hh @ h
        s = 1.0 / (1.0 + np.exp(-g))
        c = s[128:256] * c + s[:128] * np.tanh(g[256:384])
        h = s[384:] * np.tanh(c)
        out[k] = h
    v = np.maximum(out, 0.0) @ w["decoder.decoder.2.weight"].reshape(128).numpy() + w["decoder.decoder.2.bias"].item()
    return 1.0 / (1.0 + np.exp(-v))


def exact(case, seed):
    kind = case["kind"]
    if kind == "longform":
        return None  # hundreds of chunks and the merge of their tokens
    state = prepare(case, seed)
    if kind == "frontend":
        o = state["offsets"]
        x = state["pcm"]
        clip = lambda a, b: (x[a:b].double() / 32767.0).float() if case["int16"] else x[a:b]  # noqa: E731
        return torch.cat([_logmel(clip(a, b)) for a, b in zip(o[:-1], o[1:])])
    if kind == "encoder":
        o, w = state["offsets"], _encoder_weights(case["layers"])
        xs = [_encode(w, state["feats"][a:b]) for a, b in zip(o[:-1], o[1:])]
        return torch.cat([_blocks(w, case["layers"], xs[i:i + 64]) for i in range(0, len(xs), 64)])
    if kind == "decode":
        return [None, None, None, _dense(_decode(state["rows"], state["offsets"]), state["width"])]
    if kind == "vad":
        return _vad(state["audio"])
    w = _encoder_weights(24)
    rows = _blocks(w, 24, [_encode(w, _logmel(torch.from_numpy(state["audio"]).cuda()))])
    return [None, None, None, _dense(_decode(rows, _offsets([rows.shape[0]])), state["width"])[0]]

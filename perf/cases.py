"""The work whose speed this framework is kept to, as a user's program asks for it through the public entry points.

Every case is a dict of plain values; ``listed()`` names the standing ones, ``draw(rng)`` gives another of the same
ranges.  Five kinds of work:

``offline``     ``ConformerCTC.forward_offline`` / ``forward_offline_packed``: a batch of utterances, features to
                log-probs.  The whole range from one short voice command to a full batch of long recordings, both model
                widths, 16-bit types and the 8-bit Linear kinds.
``stream``      ``forward_chunk_paged`` or its graph-replayed form: streams that begin, send chunk after chunk and hold
                their keys / values in pages, 16-bit or fp8.  A pass is one session of every stream.
``fast``        ``FastConformerEncoder.forward_ctc``: the 24-layer, 1024-wide encoder on ragged batches.
``fast_stream`` ``FastConformerEncoder.forward_chunk``: sessions of the same encoder chunk by chunk.
``fbank``       ``features.batched_fbank``: waveforms to normalised log-mel features.
``operators``   one Conformer layer call by call through the drop-in operators, which is how a host engine uses the
                package after ``install``.

Weights are random and fixed: a program loads its model once and then serves many batches, so a model is built once per
process and shared by the states.  What the seed makes are the inputs, and the order in which a batch's lengths come.
Greedy tokens are left out of the outputs: with random weights many frames are near ties, and two correct bf16
implementations differ there.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

import oasr_b200 as ob
from oasr_b200.encoder import ConformerConfig, ConformerCTC
from oasr_b200.fastconformer import FastConformerEncoder
from oasr_b200.features import FbankConfig, batched_fbank
from oasr_b200.weights import fastconformer_param_spec, param_spec, subsampled_bins

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
_CHUNK = 16                    # encoder frames of a streaming step
_HISTORY = 256                 # cached frames of a Conformer stream
_WINDOW = 4 * (_CHUNK - 1) + 7  # feature frames a Conformer chunk reads (67)

# hidden, heads, ffn, layers, kernel, sliding window, lookahead, mel bins, subsampling channels, vocabulary
_FAST = (1024, 8, 4096, 24, 9, 57, 3, 128, 256, 1024)


def listed():
    return [
        # a voice command: one utterance of 3 s, where launches and latency are all there is
        {"name": "offline_single", "kind": "offline", "d_model": 512, "utts": 1, "shortest": 317, "longest": 317,
         "padded": False, "dtype": "bf16", "quant": "none"},
        # a handful of utterances through the smaller model, padded in and out as the reference's default path has it
        {"name": "offline_few", "kind": "offline", "d_model": 256, "utts": 4, "shortest": 400, "longest": 1000,
         "padded": True, "dtype": "fp16", "quant": "none"},
        # a transcription job's pack of short utterances with W8A8 Linears
        {"name": "offline_pack_int8", "kind": "offline", "d_model": 512, "utts": 45, "shortest": 100, "longest": 1300,
         "padded": False, "dtype": "bf16", "quant": "int8"},
        # a transcription job's full batch, 2 to 20 s each
        {"name": "offline_batch", "kind": "offline", "d_model": 512, "utts": 64, "shortest": 200, "longest": 2000,
         "padded": False, "dtype": "bf16", "quant": "none"},
        # one live stream, each chunk waited for by a person
        {"name": "stream_single", "kind": "stream", "streams": 1, "chunks": 12, "graph": False, "kv": "bf16", "dtype": "bf16"},
        # an ordinary server load with a number of streams that changes from step to step
        {"name": "stream_some", "kind": "stream", "streams": 37, "chunks": 20, "graph": False, "kv": "bf16", "dtype": "bf16"},
        # a full server: a fixed batch replayed as a graph, fp8 pages, sessions long enough to evict pages
        {"name": "stream_full_fp8", "kind": "stream", "streams": 256, "chunks": 20, "graph": True, "kv": "fp8", "dtype": "bf16"},
        # FastConformer: a few recordings with fp8 Linears
        {"name": "fast_few_fp8", "kind": "fast", "utts": 9, "shortest": 500, "longest": 3000, "quant": "fp8"},
        # FastConformer: a full batch, 5 to 30 s each
        {"name": "fast_batch", "kind": "fast", "utts": 128, "shortest": 500, "longest": 3000, "quant": "none"},
        # FastConformer live streams
        {"name": "fast_stream", "kind": "fast_stream", "streams": 24, "chunks": 5},
        # the features of a batch of recordings, 16 kHz
        {"name": "fbank_batch", "kind": "fbank", "utts": 64, "shortest": 32000, "longest": 320000},
        # a layer by operators on a padded batch, the drop-in use
        {"name": "operators_layer", "kind": "operators", "utts": 8, "frames": 249, "dtype": "fp16"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("offline", "offline", "stream", "stream", "fast", "fast_stream", "fbank", "operators"))
    if kind == "offline":
        utts, longest = _log_int(rng, 1, 64), _log_int(rng, 100, 2000)
        return {"kind": kind, "d_model": rng.choice((256, 512, 512)), "utts": utts,
                "shortest": longest if utts == 1 else _log_int(rng, 67, longest), "longest": longest,
                "padded": rng.random() < 0.5, "dtype": rng.choice(("bf16", "bf16", "fp16")),
                "quant": rng.choice(("none", "none", "none", "fp8", "int8"))}
    if kind == "stream":
        return {"kind": kind, "streams": _log_int(rng, 1, 256), "chunks": rng.randint(4, 20), "graph": rng.random() < 0.4,
                "kv": rng.choice(("bf16", "fp8")), "dtype": "bf16"}
    if kind == "fast":
        utts, longest = _log_int(rng, 1, 110), _log_int(rng, 300, 3000)
        return {"kind": kind, "utts": utts, "shortest": longest if utts == 1 else _log_int(rng, 200, longest), "longest": longest,
                "quant": rng.choice(("none", "none", "fp8", "int8"))}
    if kind == "fast_stream":
        return {"kind": kind, "streams": _log_int(rng, 1, 64), "chunks": rng.randint(2, 6)}
    if kind == "fbank":
        utts, longest = _log_int(rng, 1, 64), _log_int(rng, 8000, 320000)
        return {"kind": kind, "utts": utts, "shortest": longest if utts == 1 else _log_int(rng, 4000, longest), "longest": longest}
    return {"kind": kind, "utts": _log_int(rng, 1, 32), "frames": _log_int(rng, 16, 500), "dtype": rng.choice(("bf16", "fp16"))}


def _lengths(case):
    """The batch's lengths, ascending: the shortest and the longest of the case and ragged ones spread between them."""
    n, lo, hi = case["utts"], case["shortest"], case["longest"]
    if n == 1:
        return [hi]
    r = random.Random(1000003 * n + 1009 * lo + hi)
    return sorted([lo, hi] + [r.randint(lo, hi) for _ in range(n - 2)])


def _shuffled_lengths(case, seed):
    lengths = _lengths(case)
    random.Random(seed).shuffle(lengths)
    return lengths


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


# ------------------------------------------------------------------ models, built once per process
def _random_tensor(shape, std, mean, g):
    return (torch.randn(shape, generator=g, device="cuda") * std + mean).cpu()


def _conformer_config(d_model, causal):
    return ConformerConfig(input_size=80, d_model=d_model, heads=d_model // 64, ffn=2048, layers=12, kernel=15, vocab=5008, causal=causal)


@functools.lru_cache(maxsize=None)
def _conformer(d_model, causal, dtype, quant):
    cfg = _conformer_config(d_model, causal)
    g = _generator(1234)
    params = {}
    for name, shape, what in param_spec(cfg):
        if what == "matrix":
            params[name] = _random_tensor(shape, 0.02, 0.0, g)
        elif what in ("gain", "var"):
            params[name] = _random_tensor(shape, 0.05, 1.0, g)
        else:
            params[name] = _random_tensor(shape, 0.05, 0.0, g)
    return ConformerCTC(cfg, params, device="cuda", dtype=_DTYPES[dtype], quant=None if quant == "none" else quant)


@functools.lru_cache(maxsize=None)
def _kv_scales(dtype):
    """Scales of the fp8 pages, calibrated on a few chunks as at a server's start."""
    windows = torch.randn(4, 16, _WINDOW, 80, generator=_generator(99), device="cuda")
    return _conformer(512, True, dtype, "none").calibrate_kv_scales(list(windows), _CHUNK, margin=1.5)


@functools.lru_cache(maxsize=None)
def _fast(quant, dtype="bf16"):
    hidden, heads, ffn, layers, kernel, window, lookahead, mels, channels, vocab = _FAST
    g = _generator(1234)
    params = {}
    for name, shape, what in fastconformer_param_spec(hidden, heads, ffn, layers, kernel, False):
        params[name] = _random_tensor(shape, 0.02 if what == "w" else 0.1, 1.0 if what == "g" else 0.0, g)
    s = "subsampling."
    front = [(s + "conv_in.weight", (channels, 3, 3, 1)), (s + "conv_in.bias", (channels,))]
    for i in range(2):
        p = f"{s}layers.{i}."
        front += [(p + "depthwise_conv.weight", (channels, 3, 3, 1)), (p + "depthwise_conv.bias", (channels,)),
                  (p + "pointwise_conv.weight", (channels, 1, 1, channels)), (p + "pointwise_conv.bias", (channels,))]
    front += [(s + "linear.weight", (hidden, channels * subsampled_bins(mels))), (s + "linear.bias", (hidden,))]
    for name, shape in front:
        fan_in = math.prod(shape[1:]) if len(shape) > 1 else 0
        params[name] = _random_tensor(shape, math.sqrt(2.0 / fan_in) if fan_in else 0.1, 0.0, g)
    params["ctc.ctc_lo.weight"] = _random_tensor((vocab, hidden), 0.02, 0.0, g)
    params["ctc.ctc_lo.bias"] = torch.zeros(vocab)
    enc = FastConformerEncoder(hidden, heads, ffn, layers, kernel, window, lookahead, mels, channels, params, dtype=_DTYPES[dtype])
    if quant != "none":
        enc.stack.set_quant(quant)
    return enc


@functools.lru_cache(maxsize=None)
def _layer_weights(dtype):
    """One Conformer layer's operator parameters (d 512, 8 heads, FFN 2048, kernel 15)."""
    d, f, k, dt = 512, 2048, 15, _DTYPES[dtype]
    g = _generator(4321)
    mat = lambda *s: (torch.randn(*s, generator=g, device="cuda") * 0.04).to(dt)
    vec = lambda n, mean: (torch.randn(n, generator=g, device="cuda") * 0.05 + mean).to(dt)
    norm = lambda: (vec(d, 1.0), vec(d, 0.0))
    return {"norms": [norm() for _ in range(5)], "ff1": (mat(f, d), vec(f, 0.0), mat(d, f), vec(d, 0.0)),
            "qkv": (mat(3 * d, d), vec(3 * d, 0.0)), "out": (mat(d, d), vec(d, 0.0)), "pw1": (mat(2 * d, d), vec(2 * d, 0.0)),
            "dw": (mat(k, d), vec(d, 0.0)), "bn": (vec(d, 1.0), vec(d, 0.0), vec(d, 0.0), vec(d, 1.0).abs()),
            "pw2": (mat(d, d), vec(d, 0.0)), "ff2": (mat(f, d), vec(f, 0.0), mat(d, f), vec(d, 0.0))}


# ------------------------------------------------------------------ states
def prepare(case, seed):
    kind = case["kind"]
    g = _generator(seed)
    if kind == "offline":
        lengths = _shuffled_lengths(case, seed)
        return {"case": case, "model": _conformer(case["d_model"], False, case["dtype"], case["quant"]), "lengths": lengths,
                "features": torch.randn(len(lengths), max(lengths), 80, generator=g, device="cuda")}
    if kind == "stream":
        B, n = case["streams"], case["chunks"]
        model = _conformer(512, True, case["dtype"], "none")
        cache = model.new_streaming_cache(B, _HISTORY, chunk_frames=_CHUNK, seed=5,
                                          kv_scales=_kv_scales(case["dtype"]) if case["kv"] == "fp8" else None)
        feats = torch.randn(B, 64 * n + 3, 80, generator=g, device="cuda")
        state = {"case": case, "model": model, "cache": cache, "slots": list(range(B)),
                 "windows": [feats[:, 64 * c:64 * c + _WINDOW].contiguous() for c in range(n)]}
        if case["graph"]:
            model.forward_chunk_paged(state["windows"][0], state["slots"], cache)
            state["step"] = model.graphed_chunk_forward(cache, B, _WINDOW)
            # the graph's outputs are overwritten by its next replay: a decoder's own copy of every chunk
            state["log_probs"] = torch.empty(n, B, _CHUNK, model.cfg.vocab_padded, device="cuda")
        return state
    if kind == "fast":
        lengths = _shuffled_lengths(case, seed)
        return {"case": case, "encoder": _fast(case["quant"]), "lengths": lengths,
                "features": torch.randn(len(lengths), max(lengths), _FAST[7], generator=g, device="cuda")}
    if kind == "fast_stream":
        B, n = case["streams"], case["chunks"]
        enc = _fast("none")
        feats = torch.randn(n, B, 8 * _CHUNK, _FAST[7], generator=g, device="cuda")
        return {"case": case, "encoder": enc, "cache": enc.new_streaming_cache(B, chunk_frames=_CHUNK), "slots": list(range(B)),
                "chunks": list(feats)}
    if kind == "fbank":
        lengths = _shuffled_lengths(case, seed)
        B, T = len(lengths), max(lengths)
        # a few drifting tones over noise, at the scale of 16-bit samples
        t = torch.arange(T, device="cuda", dtype=torch.float32)[None] / 16000.0
        waves = 300.0 * torch.randn(B, T, generator=g, device="cuda")
        for _ in range(3):
            f0, level = (torch.rand(B, 1, generator=g, device="cuda") for _ in range(2))
            waves += 3000.0 * level * torch.sin(2 * math.pi * ((100.0 + 3000.0 * f0) * t + 40.0 * f0 * t * t))
        cmvn = (torch.randn(80, generator=g, device="cuda") * 0.5 + 12.0, torch.rand(80, generator=g, device="cuda") * 0.2 + 0.2)
        return {"case": case, "waves": waves, "lengths": torch.tensor(lengths), "cmvn": cmvn, "config": FbankConfig()}
    B, T, dt = case["utts"], case["frames"], _DTYPES[case["dtype"]]
    r = random.Random(seed)
    lens = [T] + [r.randint(max(1, T // 2), T) for _ in range(B - 1)]
    mask = torch.arange(T, device="cuda")[None, :] < torch.tensor(lens, device="cuda")[:, None]
    return {"case": case, "weights": _layer_weights(case["dtype"]), "x": torch.randn(B, T, 512, generator=g, device="cuda").to(dt),
            "bias": torch.randn(B, 8, T, T, generator=g, device="cuda").to(dt),
            "lens": torch.tensor(lens, dtype=torch.int32, device="cuda"), "mask": mask.unsqueeze(-1)}


# ------------------------------------------------------------------ one pass
def run(state):
    return _RUN[state["case"]["kind"]](state)


def _run_offline(s):
    if s["case"]["padded"]:
        return s["model"].forward_offline(s["features"], s["lengths"])
    log_probs, out_lengths, _ = s["model"].forward_offline_packed(s["features"], s["lengths"], padded_output=False)
    return log_probs, out_lengths


def _run_stream(s):
    model, cache, slots = s["model"], s["cache"], s["slots"]
    for slot in slots:
        cache.reset_stream(slot)
    if "step" not in s:
        return [model.forward_chunk_paged(window, slots, cache) for window in s["windows"]]
    for i, window in enumerate(s["windows"]):
        log_probs, _ = s["step"](window, slots)
        s["log_probs"][i].copy_(log_probs)
    return s["log_probs"]


def _run_fast(s):
    log_probs, out_lengths = s["encoder"].forward_ctc(s["features"], s["lengths"], padded_output=False)
    return log_probs, np.array(out_lengths)


def _run_fast_stream(s):
    for slot in s["slots"]:
        s["cache"].reset_stream(slot)
    return [s["encoder"].forward_chunk(chunk, s["slots"], s["cache"]) for chunk in s["chunks"]]


def _run_fbank(s):
    return batched_fbank(s["waves"], s["lengths"], s["config"], s["cmvn"])


def _run_operators(s):
    w, x, case = s["weights"], s["x"], s["case"]
    B, T, H, D = case["utts"], case["frames"], 8, 64
    n = w["norms"]
    w1, b1, w2, b2 = w["ff1"]
    y = ob.gemm(ob.gemm_activation(ob.layer_norm(x, *n[0]), w1, b1, 2), w2, b2)
    h, x = ob.add_layer_norm_residual(y, x, *n[1], alpha=0.5)
    qkv = ob.gemm(h, *w["qkv"]).view(B, T, 3, H, D).permute(2, 0, 3, 1, 4)
    att = ob.fmha(qkv[0], qkv[1], qkv[2], softmax_scale=D ** -0.5, attn_bias=s["bias"], cache_seqlens=s["lens"])
    y = ob.gemm(att.transpose(1, 2).reshape(B, T, H * D), *w["out"])
    h, x = ob.add_layer_norm_residual(y, x, *n[2])
    y = ob.glu(ob.gemm(h, *w["pw1"]))
    y = ob.batch_norm_swish(ob.depthwise_conv1d(y, *w["dw"], padding=7, mask=s["mask"]), *w["bn"])
    h, x = ob.add_layer_norm_residual(ob.gemm(y, *w["pw2"]), x, *n[3])
    w1, b1, w2, b2 = w["ff2"]
    y = ob.gemm(ob.gemm_activation(h, w1, b1, 2), w2, b2)
    return ob.add_layer_norm_residual(y, x, *n[4], alpha=0.5)


_RUN = {"offline": _run_offline, "stream": _run_stream, "fast": _run_fast, "fast_stream": _run_fast_stream, "fbank": _run_fbank,
        "operators": _run_operators}


# ------------------------------------------------------------------ what a pass cannot do without
def _conformer_work(d, ffn, layers, kernel, vocab, f2, tokens, attention_keys, weight_byte, frames_in, out_rows, kv_bytes):
    """One forward over ``tokens`` frames; ``attention_keys`` = keys summed over all query frames."""
    linear = 4 * ffn * d + 3 * d * d + d * d + 2 * d * d + d * d          # multiply-adds of a layer's Linears per token
    front = 9 * d * d * f2 + f2 * d * d + 2 * 9 * 39 * d
    flops = 2.0 * tokens * (layers * (linear + kernel * d) + front + vocab * d) + 6.0 * layers * d * attention_keys
    weights = layers * (linear * weight_byte + 2 * d * d) + 2.0 * (9 * d * d + f2 * d * d + vocab * d)
    return {"bytes": weights + 4.0 * 80 * frames_in + 4.0 * vocab * out_rows + kv_bytes, "flops": flops}


def work(case):
    kind = case["kind"]
    if kind == "offline":
        lengths = _lengths(case)
        outs = [max((n - 3) // 4, 0) for n in lengths]
        cfg = _conformer_config(case["d_model"], False)
        padded = len(outs) * max(outs) if case["padded"] else sum(outs)
        return _conformer_work(cfg.d_model, cfg.ffn, cfg.layers, cfg.kernel, cfg.vocab_padded, 19, sum(outs), sum(n * n for n in outs),
                               2 if case["quant"] == "none" else 1, sum(lengths), padded, 0.0)
    if kind == "stream":
        B, n = case["streams"], case["chunks"]
        keys = [min(c * _CHUNK, _HISTORY) + _CHUNK for c in range(n)]
        total = {"bytes": 0.0, "flops": 0.0}
        for k in keys:       # every chunk is a call of its own: weights and cached keys / values are read again
            kv = 12.0 * 2 * B * k * 512 * (1 if case["kv"] == "fp8" else 2)
            w = _conformer_work(512, 2048, 12, 15, 5008, 19, B * _CHUNK, B * _CHUNK * k, 2, B * _WINDOW, B * _CHUNK, kv)
            total = {m: total[m] + w[m] for m in total}
        return total
    if kind in ("fast", "fast_stream"):
        hidden, _, ffn, layers, kernel, window, lookahead, mels, channels, vocab = _FAST
        linear = 4 * ffn * hidden + 4 * hidden * hidden + 3 * hidden * hidden
        bins = [mels // 2 + 1, mels // 4 + 1, subsampled_bins(mels)]
        per_frame = 4 * bins[0] * 9 * channels + (2 * bins[1] + bins[2]) * (9 * channels + channels * channels) + \
            bins[2] * channels * hidden
        weights = 2.0 * (bins[2] * channels * hidden + 2 * channels * channels)
        span = window + lookahead        # the most keys a frame sees
        if kind == "fast":
            outs = []
            for n in _lengths(case):
                for _ in range(3):
                    n = n // 2 + 1
                outs.append(n)
            tokens, keys = sum(outs), sum(n * min(n, span) for n in outs)
            weight_byte = 2 if case["quant"] == "none" else 1
            b = layers * (linear * weight_byte + 2.0 * hidden * hidden) + weights + 2.0 * vocab * hidden + \
                4.0 * mels * sum(_lengths(case)) + 4.0 * vocab * tokens
            fl = 2.0 * tokens * (layers * (linear + kernel * hidden) + per_frame + vocab * hidden) + 6.0 * layers * hidden * keys
            return {"bytes": b, "flops": fl}
        B, n = case["streams"], case["chunks"]
        tokens = B * _CHUNK
        b = fl = 0.0
        for c in range(n):
            k = min(c * _CHUNK, 64) + _CHUNK
            b += layers * linear * 2.0 + weights + 4.0 * mels * 8 * tokens + 4.0 * hidden * tokens + layers * 4.0 * B * k * hidden
            fl += 2.0 * tokens * (layers * (linear + kernel * hidden) + per_frame) + 6.0 * layers * hidden * tokens * min(k, span)
        return {"bytes": b, "flops": fl}
    if kind == "fbank":
        lengths, cfg = _lengths(case), FbankConfig()
        frames = [max(0, (n - cfg.frame_length_samples) // cfg.frame_shift_samples + 1) for n in lengths]
        fft = 2.5 * 512 * 9 + 4 * 400 + 3 * 257 + 2 * 514           # real FFT, window, power, mel filters
        return {"bytes": 4.0 * sum(lengths) + 4.0 * 80 * len(lengths) * max(frames), "flops": fft * sum(frames)}
    B, T, d, f = case["utts"], case["frames"], 512, 2048
    M = B * T
    linear = 4 * f * d + 3 * d * d + d * d + 2 * d * d + d * d
    return {"bytes": 2.0 * linear + 3 * 2.0 * M * d + 2.0 * B * 8 * T * T, "flops": 2.0 * M * (linear + 15 * d) + 4.0 * B * T * T * d}


def tolerance(case):
    """What the 16-bit (8-bit) roundings inside the path leave between two correct implementations.  The log-probs sit at
    -ln(vocabulary), about -8.6 and -7, with a spread of a few tenths, so their relative error is small; the hidden states
    of the streaming FastConformer are layer-normalised."""
    kind, quant = case["kind"], case.get("quant", "none")
    if kind in ("offline", "stream"):
        return {"none": {"rel": 6e-4, "max": 4e-3}, "int8": {"rel": 1.2e-3, "max": 8e-3}, "fp8": {"rel": 3e-3, "max": 2e-2}}[quant]
    if kind == "fast":       # 24 layers, every Linear's input rounded again
        return {"rel": 2e-3, "max": 1.2e-2} if quant == "none" else {"rel": 1.2e-2, "max": 7e-2}
    if kind == "fast_stream":
        return {"rel": 2e-2, "max": 0.15}
    if kind == "fbank":      # 32-bit sums, then a logarithm: a weak band under a strong tone loses digits
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 7e-3, "max": 5e-2} if case["dtype"] == "bf16" else {"rel": 1e-3, "max": 8e-3}

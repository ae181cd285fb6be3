"""Timed work of this framework, through the calls that its trainer, scorer and translator make.

Every case is one of five kinds:

* ``train_text``   one ``TrainEngine.train_step`` of a text Transformer (forward, backward, clipping, AdamW), host batch in;
* ``train_audio``  the same for the two speech models: a Whisper model on 30 s windows of 80 log-mel bins, and a wav2vec 2.0
  encoder on raw 16 kHz audio with an mBART-50 decoder;
* ``score``        gold scoring (``model.decode``): forward pass, log-probability of every target token;
* ``translate``    beam search of a text Transformer from a host batch to hypotheses on the host;
* ``transcribe``   beam search of a Whisper model from log-mel windows on the host to hypotheses on the host.

Model sizes are those of ``bench.py`` (the tiny and the big Transformer), ``bench_speech.py`` (Whisper-large-v2's width,
wav2vec2-large + mBART-50) and the option table's defaults (512 wide, 8 heads, 2048 in the feed-forward blocks); lengths are
theirs too (20 to 100 tokens, 30 s windows, utterances of 5 to 20 s).  All weights come from the seed.
"""
import functools
import math

import numpy as np
import torch

from nmtgminor_b200 import ops
from nmtgminor_b200.data.dataset import Batch, collate
from nmtgminor_b200.data.synthetic import synthetic_dict
from nmtgminor_b200.inference.beam_search import BeamConfig, beam_search
from nmtgminor_b200.models.factory import build_model
from nmtgminor_b200.options import default_options
from nmtgminor_b200.parallel.flat import FlatParameterStore
from nmtgminor_b200.train.engine import TrainEngine

BOS, EOS, FIRST = 2, 3, 4
SMOOTHING, LR, DECAY, CLIP = 0.1, 1e-4, 0.01, 5.0
PAD_PARAM, PAD_TOTAL = 64, 256        # the flat buffers align every parameter, and their end


def _text(kind, name, layers, dim, heads, ffn, vocab, sentences, lo, hi, **more):
    return dict({"name": name, "kind": kind, "layers": layers, "dim": dim, "heads": heads, "ffn": ffn, "vocab": vocab,
                 "sentences": sentences, "lo": lo, "hi": hi}, **more)


def listed():
    return [
        # a tiny model and 32 short pairs: what a step costs beyond its arithmetic (development runs, small corpora)
        _text("train_text", "train tiny", 2, 256, 4, 1024, 8000, 32, 10, 50, act="relu", dropout=0.1),
        # the default model size with a small batch, without dropout (the last epochs of a fine-tuning run)
        _text("train_text", "train base", 6, 512, 8, 2048, 32000, 64, 20, 100, act="relu", dropout=0.0),
        # the flagship: Transformer-big, about 8200 target tokens
        _text("train_text", "train big", 6, 1024, 16, 4096, 32000, 136, 20, 100, act="relu", dropout=0.1),
        # document-level pairs: sequences of several hundred tokens, GELU
        _text("train_text", "train documents", 6, 512, 8, 2048, 32000, 17, 200, 500, act="gelu", dropout=0.1),
        # speech recognition with Whisper-large-v2's layers (12 + 12 of its 32 + 32): 1500 encoder frames an utterance
        {"name": "train whisper", "kind": "train_audio", "model": "whisper", "layers": 12, "dim": 1280, "heads": 20, "ffn": 5120,
         "vocab": 51865, "utterances": 8, "lo": 18, "hi": 446, "dropout": 0.1},
        # speech translation: wav2vec2-large on 5 to 20 s of raw audio, 12-layer mBART-50 decoder
        {"name": "train wav2vec2", "kind": "train_audio", "model": "wav2vec2", "layers": 12, "dim": 1024, "heads": 16, "ffn": 4096,
         "vocab": 250054, "utterances": 6, "lo": 10, "hi": 120, "dropout": 0.1},
        # rescoring / perplexity of a corpus: forward passes over large batches
        _text("score", "score big", 6, 1024, 16, 4096, 32000, 128, 20, 100, act="relu"),
        # one request of an online translator: latency
        _text("translate", "translate one sentence", 6, 1024, 16, 4096, 32000, 1, 20, 100, act="relu", beam=4, normalize=True),
        # offline translation of a test set in batches of 64
        _text("translate", "translate batch", 6, 1024, 16, 4096, 32000, 64, 20, 100, act="relu", beam=4, normalize=False),
        # transcription of 30 s windows, a batch of long recordings
        {"name": "transcribe", "kind": "transcribe", "model": "whisper", "layers": 12, "dim": 1280, "heads": 20, "ffn": 5120,
         "vocab": 51865, "utterances": 8, "beam": 4, "steps": 100, "normalize": False},
    ]


def _between(rng, lo, hi):
    """Whole number from ``lo`` to ``hi``, even over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["train_text", "train_text", "train_text", "train_audio", "train_audio", "score", "translate", "translate",
                       "transcribe"])
    dim, heads = rng.choice([(256, 4), (512, 8), (768, 12), (1024, 16)])
    layers, vocab = rng.randint(2, 6), _between(rng, 4000, 32000) // 2 * 2      # the output bias takes an even vocabulary
    if kind == "train_audio" and rng.random() < 0.5:
        return {"kind": kind, "model": "wav2vec2", "layers": rng.randint(3, 12), "dim": 1024, "heads": 16, "ffn": 4096,
                "vocab": _between(rng, 8000, 250054), "utterances": rng.randint(1, 6), "lo": 10, "hi": rng.randint(20, 120),
                "dropout": rng.choice([0.0, 0.1])}
    if kind in ("train_audio", "transcribe"):
        dim, heads = rng.choice([(512, 8), (768, 12), (1024, 16), (1280, 20)])
        case = {"kind": kind, "model": "whisper", "layers": _between(rng, 2, 12), "dim": dim, "heads": heads, "ffn": 4 * dim,
                "vocab": 51865, "utterances": rng.randint(1, 8)}
        if kind == "train_audio":
            return dict(case, lo=18, hi=rng.randint(40, 446), dropout=rng.choice([0.0, 0.1]))
        return dict(case, beam=rng.randint(1, 5), steps=rng.randint(20, 100), normalize=rng.random() < 0.5)
    case = {"kind": kind, "layers": layers, "dim": dim, "heads": heads, "ffn": 4 * dim, "vocab": vocab}
    if kind == "translate":
        hi = rng.randint(20, 100)
        return dict(case, sentences=_between(rng, 1, 64), lo=rng.randint(5, 20), hi=hi, act=rng.choice(["relu", "gelu"]),
                    beam=rng.randint(1, 6), normalize=rng.random() < 0.5)
    hi = _between(rng, 20, 500)
    lo = max(1, int(hi * rng.uniform(0.2, 0.9)))
    most = max(2, 2 * 8200 // (lo + hi))
    return dict(case, sentences=_between(rng, max(1, most // 30), most), lo=lo, hi=hi, act=rng.choice(["relu", "gelu", "silu"]),
                **({"dropout": rng.choice([0.0, 0.1])} if kind == "train_text" else {}))


# ---------------------------------------------------------------------------------------------------------------------
# inputs and weights, from the seed alone
# ---------------------------------------------------------------------------------------------------------------------
def _lengths(case, n, lo, hi, salt):
    """Sequence lengths of a case: the same for every seed, so that every batch of a case is the same amount of work."""
    r = np.random.RandomState(1000 * salt + n)
    return r.randint(lo, hi + 1, size=n)


def _pairs(case, seed):
    r = np.random.RandomState(seed % (1 << 31))
    n = case["sentences"]
    ids = lambda m: torch.from_numpy(r.randint(FIRST, case["vocab"], size=m).astype(np.int64))
    src = [ids(m) for m in _lengths(case, n, case["lo"], case["hi"], 1)]
    wrap = lambda t: torch.cat([torch.tensor([BOS]), t, torch.tensor([EOS])])
    return src, [wrap(ids(m)) for m in _lengths(case, n, case["lo"], case["hi"], 2)]


def _utterances(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["model"] == "whisper":
        return [f.cpu() for f in torch.randn(case["utterances"], 3000, 80, device="cuda", generator=g)]
    return [(torch.randn(int(m), 1, device="cuda", generator=g) * 0.1).cpu() for m in _lengths(case, case["utterances"], 80000, 320000, 3)]


def _transcripts(case, seed):
    r = np.random.RandomState((seed + 7) % (1 << 31))
    return [torch.from_numpy(np.concatenate([[BOS], r.randint(FIRST, case["vocab"], size=m), [EOS]]).astype(np.int64))
            for m in _lengths(case, case["utterances"], case["lo"], case["hi"], 4)]


def _text_shapes(case):
    """Parameters of the text Transformer in the order of the module tree: [(name, shape)]."""
    d, f, v = case["dim"], case["ffn"], case["vocab"]
    norm = lambda p: [(p + ".weight", (d,)), (p + ".bias", (d,))]
    ffn = lambda p: norm(p + "ffn_norm") + [(p + "ffn.fc1.weight", (f, d)), (p + "ffn.fc1.bias", (f,)), (p + "ffn.fc2.weight", (d, f)),
                                            (p + "ffn.fc2.bias", (d,))]
    out = [("encoder.embed.weight", (v, d))]
    for i in range(case["layers"]):
        p = "encoder.layers.%d." % i
        out += norm(p + "attn_norm") + [(p + "attn.qkv.weight", (3 * d, d)), (p + "attn.out.weight", (d, d))] + ffn(p)
    out += norm("encoder.final_norm")
    for i in range(case["layers"]):
        p = "decoder.layers.%d." % i
        out += norm(p + "self_norm") + [(p + "self_attn.qkv.weight", (3 * d, d)), (p + "self_attn.out.weight", (d, d))]
        out += norm(p + "cross_norm") + [(p + "cross_attn.q.weight", (d, d)), (p + "cross_attn.kv.weight", (2 * d, d)),
                                         (p + "cross_attn.out.weight", (d, d))] + ffn(p)
    out += norm("decoder.final_norm")
    if case["kind"] == "translate":
        out.append(("generator.weight", (v, d)))      # else tied to the embedding
    return out + [("generator.bias", (v,))]


def _values(named_shapes, seed, emb_std, res_std):
    """Weights as a trained model has them, roughly: matrices keep the scale of their input, the projections that feed the
    residual stream (``out``, ``fc2``) are smaller, LayerNorm gains near one.  Rounded to bf16, so that the working copies are exact."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = {}
    for name, shape in named_shapes:
        w = torch.randn(shape, device="cuda", generator=g)
        if len(shape) == 1 and "norm" in name:
            w = w * 0.05 + (1.0 if name.endswith("weight") else 0.0)
        elif len(shape) == 1:
            w = w * (0.02 * res_std if name.endswith("out.bias") or name.endswith("fc2.bias") else 0.02)
        elif name.endswith("embed.weight") or name.endswith("embed.pos") or name == "generator.weight":
            w = w * emb_std
        elif name.endswith("out.weight") or name.endswith("fc2.weight"):
            w = w * (res_std / math.sqrt(shape[1]))
        else:
            w = w * (1.0 / math.sqrt(math.prod(shape[1:])))
        out[name] = w.bfloat16().float()
    return out


def _text_weights(case, seed):
    d = case["dim"]
    w = _values(_text_shapes(case), seed, d ** -0.5, 0.5)
    if case["kind"] == "translate":
        # A trained model is sure of most of its words.  Word t makes the generator prefer one other word, its successor, with a
        # probability of roughly 0.9 (the decoder's states keep some of the embedding of the word that they were fed).
        words = case["vocab"] - FIRST
        order = torch.randperm(words, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed + 1)) + FIRST
        gen = w["generator.weight"]
        gen[order] = w["encoder.embed.weight"][order.roll(1)]
        gen[order[0]] += w["encoder.embed.weight"][BOS]
        w["generator.weight"] = (gen * (24.0 / math.sqrt(d))).bfloat16().float()
        w["generator.bias"].zero_()
    return w


@functools.lru_cache(maxsize=8)
def _vocabulary(n):
    return synthetic_dict(n)


def _options(case, more):
    p = str(case.get("dropout", 0.0))
    opt = default_options(["-layers", str(case["layers"]), "-model_size", str(case["dim"]), "-n_heads", str(case["heads"]), "-inner_size",
                           str(case["ffn"]), "-dropout", p, "-attn_dropout", p, "-emb_dropout", p, "-label_smoothing", str(SMOOTHING), "-optim",
                           "adam", "-weight_decay", str(DECAY), "-learning_rate", str(LR), "-update_method", "regular", "-max_grad_norm",
                           str(CLIP), "-fp16", "-bf16"] + more)
    return opt


def _model(case, seed):
    """The model with the weights of the seed, its parameters on the GPU, and its options."""
    d = _vocabulary(case["vocab"])
    text = "sentences" in case
    if text:
        more = ["-model", "transformer", "-ffn_activation", case["act"], "-join_embedding"]
        more += [] if case["kind"] == "translate" else ["-tie_weights"]
    elif case["model"] == "whisper":
        more = ["-model", "whisper"]
    else:
        more = ["-model", "wav2vec2_bert", "-dec_pretrained_model", "mbart50"]
    opt = _options(case, more)
    with torch.device("cuda"):
        model = build_model(opt, {"src": d, "tgt": d})
    named = dict(model.named_parameters())
    if text:
        weights = _text_weights(case, seed)
    else:
        # Whisper's output layer is its embedding: small rows, and residual branches of their size, make it prefer one word, too
        small = 26.0 / case["dim"] if case["model"] == "whisper" else 0.6 / math.sqrt(case["dim"])
        res = 0.46 * small / math.sqrt(case["layers"]) if case["model"] == "whisper" else 0.5
        weights = _values([(n, tuple(p.shape)) for n, p in named.items()], seed, small, res)
    assert set(named) == set(weights), sorted(set(named) ^ set(weights))
    with torch.no_grad():
        for n, p in named.items():
            p.copy_(weights[n])
    return model, opt


def prepare(case, seed):
    torch.manual_seed(seed)
    ops.manual_seed(seed)
    ops.ext().get_seed_tensor(torch.cuda.current_device()).zero_()      # dropout masks from the seed, whatever ran before
    device = torch.device("cuda", torch.cuda.current_device())
    model, opt = _model(case, seed)
    kind = case["kind"]
    if kind in ("train_text", "score"):
        src, tgt = _pairs(case, seed)
        batch = collate(src, tgt, padded=kind == "score", packed=True, **({"static_shapes": True} if kind == "train_text" else {"round_to": 1}))
    elif kind == "train_audio":
        batch = collate(_utterances(case, seed), _transcripts(case, seed), src_type="audio", padded=True, packed=True, round_to=16)
    elif kind == "translate":
        batch = collate(_pairs(case, seed)[0], None, padded=True, packed=True, round_to=1)
    else:
        batch = collate(_utterances(case, seed), None, src_type="audio", padded=True, packed=True, round_to=1)
    state = {"kind": kind, "host": batch.pin_memory().tensors, "device": device}
    if kind in ("train_text", "train_audio"):
        state["engine"] = TrainEngine(model, opt, device=device, cuda_graph=True)
        return state
    FlatParameterStore(model, device)
    for b in model.buffers():
        b.data = b.data.to(device)
    state["model"] = model.eval()
    if kind == "translate":
        model.renew_buffer(2 * case["hi"] + 16)
        state["search"] = BeamConfig(beam_size=case["beam"], max_len=2 * case["hi"] + 10, dynamic_max_len=True, normalize=case["normalize"],
                                     alpha=1.0 if case["normalize"] else 0.0)
    elif kind == "transcribe":
        state["search"] = BeamConfig(beam_size=case["beam"], max_len=case["steps"], min_len=case["steps"], normalize=case["normalize"],
                                     alpha=1.0 if case["normalize"] else 0.0)
    return state


def run(state):
    batch = Batch(dict(state["host"]))          # as a loader hands it over: tensors in pinned host memory
    if "engine" in state:
        engine = state["engine"]
        loss, correct = engine.train_step(batch)
        return {"loss": loss, "correct": correct, "weights": engine.store.master, "mean": engine.optim.exp_avg, "square": engine.optim.exp_avg_sq}
    batch = batch.cuda(state["device"])
    if state["kind"] == "score":
        _, sentences, tokens = state["model"].decode(batch)
        return {"sentences": sentences, "tokens": tokens}
    found = beam_search(state["model"], batch, state["search"])
    best = [h[0] for h in found]
    words = np.zeros((len(best), max(len(h.tokens) for h in best)), dtype=np.int64)
    for i, h in enumerate(best):
        words[i, :len(h.tokens)] = h.tokens
    return {"words": words, "scores": np.array([h.score for h in best])}


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def _stack(tokens, pairs, d, ffn, memory=None, cross_pairs=0, kv_rows=None):
    """Multiply-adds of one layer's forward pass: projections, attention over ``pairs`` query-key pairs, feed-forward."""
    n = tokens * (4 * d * d + 2 * d * ffn) + 2 * pairs * d
    if memory is not None:
        n += 2 * tokens * d * d + 2 * (memory if kv_rows is None else kv_rows) * d * d + 2 * cross_pairs * d
    return n


def work(case):
    d, f, v, layers = case["dim"], case["ffn"], case["vocab"], case["layers"]
    kind = case["kind"]
    if "sentences" in case:
        n = case["sentences"]
        a = _lengths(case, n, case["lo"], case["hi"], 1).astype(float)
        b = _lengths(case, n, case["lo"], case["hi"], 2).astype(float) + 1
        front, enc_layers, enc_d, enc_f, enc_params = 0.0, layers, d, f, layers * (4 * d * d + 2 * d * f) + v * d
    elif case["model"] == "whisper":
        n = case["utterances"]
        a, b = np.full(n, 1500.0), (np.zeros(n) if kind == "transcribe" else _lengths(case, n, case["lo"], case["hi"], 4) + 1.0)
        front, enc_layers, enc_d, enc_f = n * (3000 * 3 * 80 * d + 1500 * 3 * d * d), layers, d, f
        enc_params = layers * (4 * d * d + 2 * d * f) + 3 * d * (80 + d)
    else:
        n = case["utterances"]
        samples = _lengths(case, n, 80000, 320000, 3).astype(float)
        a, b = np.floor(samples / 320), _lengths(case, n, case["lo"], case["hi"], 4) + 1.0
        enc_layers, enc_d, enc_f = 24, 1024, 4096
        front = float(samples.sum()) * (512 * 10 / 5 + 512 * 512 * 3 * (1 / 10 + 1 / 20 + 1 / 40 + 1 / 80) + 512 * 512 * 2 * (1 / 160 + 1 / 320))
        position = float(a.sum()) * 1024 * 64 * 128
        front, enc_params = front + 3 * position, enc_layers * (4 * enc_d * enc_d + 2 * enc_d * enc_f) + 64 * 128 * 1024 + 512 * 1024
    dec_params = layers * (8 * d * d + 2 * d * f) + v * d
    enc = front + enc_layers * _stack(a.sum(), (a * a).sum(), enc_d, enc_f)
    params = enc_params + dec_params - (v * d if "sentences" in case and kind != "translate" else 0)
    if kind in ("translate", "transcribe"):
        k = case["beam"]
        steps = np.floor(1.5 * a + 10) if kind == "translate" else np.full(n, float(case["steps"]))
        flops = enc + 2 * layers * a.sum() * d * d
        flops += k * (steps.sum() * (layers * (6 * d * d + 2 * d * f) + v * d) + layers * 2 * d * ((steps * steps / 2).sum() + (steps * a).sum()))
        # each step reads the decoder's weights, the keys and values so far and those of the source, and writes one more position
        t = steps.max()
        reads = t * 2 * dec_params + layers * 4 * d * (k * (steps * steps / 2).sum() + (steps * a).sum())
        return {"bytes": float(2 * enc_params + reads), "flops": float(2 * flops)}
    dec = layers * _stack(b.sum(), (b * b).sum() / 2, d, f, memory=a.sum(), cross_pairs=(a * b).sum()) + b.sum() * v * d
    if kind == "score":
        return {"bytes": float(2 * params + 8 * (a.sum() + 2 * b.sum())), "flops": float(2 * (enc + dec))}
    # bf16 weights in, fp32 weights and two moments in and out, bf16 weights out
    return {"bytes": float(params * (2 + 24 + 2) + 8 * (a.sum() + 2 * b.sum())), "flops": float(6 * (enc + dec))}


def tolerance(case):
    # bf16 operands, 32-bit sums.  Measured: text models against 64 bits 0.0002 to 0.0024; the speech models' gradients 0.011 apart
    # (single values 0.77 of the root mean square) between two orders of the 32-bit sums in a few of the forward products, for their 36
    # layers pass the last bit of bf16 on; a search with 2^-9 of noise on every weight: scores 0.0016 apart, the same words.
    if case["kind"] == "train_audio":
        return {"rel": 0.03, "max": 0.99}
    if case["kind"] == "train_text":
        return {"rel": 0.015, "max": 0.9}
    return {"rel": 0.01, "differ": 0.005}


# ---------------------------------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------------------------------
def _positions(n, d):
    half = d // 2
    freq = torch.exp(torch.arange(half, dtype=torch.float32) * -(math.log(10000.0) / (half - 1)))
    angle = torch.arange(n, dtype=torch.float32)[:, None] * freq[None, :]
    return torch.cat([angle.sin(), angle.cos()], 1).cuda().double()


def _norm(w, p, x):
    return torch.nn.functional.layer_norm(x, x.shape[-1:], w[p + ".weight"], w[p + ".bias"], 1e-5)


def _attend(q, k, v, heads, keep):
    b, n, d = q.shape
    split = lambda t: t.view(b, t.shape[1], heads, d // heads).transpose(1, 2)
    s = split(q) @ split(k).transpose(-1, -2) / math.sqrt(d // heads)
    return (s.masked_fill(~keep, -math.inf).softmax(-1) @ split(v)).transpose(1, 2).reshape(b, n, d)


def _feed(case, w, p, x):
    act = {"relu": torch.relu, "gelu": torch.nn.functional.gelu, "silu": torch.nn.functional.silu}[case["act"]]
    h = act(_norm(w, p + "ffn_norm", x) @ w[p + "ffn.fc1.weight"].T + w[p + "ffn.fc1.bias"])
    return x + h @ w[p + "ffn.fc2.weight"].T + w[p + "ffn.fc2.bias"]


def _pad(seqs):
    n = max(len(s) for s in seqs)
    return torch.stack([torch.cat([s, s.new_zeros(n - len(s))]) for s in seqs]).cuda()


def _exact_logits(case, w, src, tgt_in):
    """Decoder logits of the real target positions, sentence by sentence: [tokens, vocabulary]."""
    d, heads = case["dim"], case["heads"]
    s, t = _pad(src), _pad(tgt_in)
    pos = _positions(max(s.shape[1], t.shape[1]), d)
    emb = w["encoder.embed.weight"]
    look = lambda ids: emb[ids] * math.sqrt(d) + pos[: ids.shape[1]]
    real = (s != 0)[:, None, None, :]
    x = look(s)
    for i in range(case["layers"]):
        p = "encoder.layers.%d." % i
        q, k, v = (_norm(w, p + "attn_norm", x) @ w[p + "attn.qkv.weight"].T).chunk(3, -1)
        x = x + _attend(q, k, v, heads, real) @ w[p + "attn.out.weight"].T
        x = _feed(case, w, p, x)
    memory = _norm(w, "encoder.final_norm", x)
    past = torch.ones(t.shape[1], t.shape[1], dtype=torch.bool, device="cuda").tril()[None, None]
    x = look(t)
    for i in range(case["layers"]):
        p = "decoder.layers.%d." % i
        q, k, v = (_norm(w, p + "self_norm", x) @ w[p + "self_attn.qkv.weight"].T).chunk(3, -1)
        x = x + _attend(q, k, v, heads, past) @ w[p + "self_attn.out.weight"].T
        q = _norm(w, p + "cross_norm", x) @ w[p + "cross_attn.q.weight"].T
        k, v = (memory @ w[p + "cross_attn.kv.weight"].T).chunk(2, -1)
        x = x + _attend(q, k, v, heads, real) @ w[p + "cross_attn.out.weight"].T
        x = _feed(case, w, p, x)
    x = _norm(w, "decoder.final_norm", x)
    x = torch.cat([x[i, : len(t)] for i, t in enumerate(tgt_in)])
    return x @ w["encoder.embed.weight"].T + w["generator.bias"]


def _flat(tensors):
    """The layout of the flat buffers: every parameter on a boundary of its own, zeros between them."""
    parts = []
    for t in tensors:
        t = t.reshape(-1)
        parts += [t, t.new_zeros(-len(t) % PAD_PARAM)]
    n = sum(len(p) for p in parts)
    return torch.cat(parts + [parts[0].new_zeros(-n % PAD_TOTAL)])


def exact(case, seed):
    if case["kind"] not in ("train_text", "score") or case.get("dropout", 0.0) > 0:
        return None           # a search, masks that the kernels draw, or a model of hundreds of layers' work in 64 bits
    src, tgt = _pairs(case, seed)
    w = {n: t.double() for n, t in _text_weights(case, seed).items()}
    labels = torch.cat([t[1:] for t in tgt]).cuda()
    if case["kind"] == "score":
        with torch.no_grad():
            logp = _exact_logits(case, w, src, [t[:-1] for t in tgt]).log_softmax(-1)
        gold = logp.gather(1, labels[:, None])[:, 0]
        tokens = gold.new_zeros(max(len(t) for t in tgt) - 1, len(tgt))
        for i, part in enumerate(gold.split([len(t) - 1 for t in tgt])):
            tokens[: len(part), i] = part
        return {"sentences": tokens.sum(0), "tokens": tokens}
    for t in w.values():
        t.requires_grad_(True)
    logits = _exact_logits(case, w, src, [t[:-1] for t in tgt])
    logp = logits.log_softmax(-1)
    loss = -((1 - SMOOTHING) * logp.gather(1, labels[:, None]).sum() + SMOOTHING * logp.mean(-1).sum())
    loss.backward()
    correct = (logits.argmax(-1) == labels).sum().double().reshape(1)
    flat = _flat([t.detach() for t in w.values()])
    grad = _flat([t.grad for t in w.values()])
    # the padding word's own row takes no gradient from the embedding; it takes one from the output layer, as every word does
    norm = grad.norm()
    if norm > CLIP:
        grad = grad * (CLIP / (norm + 1e-6))
    mean, square = 0.1 * grad, 0.003 * grad * grad
    step = (mean / 0.1) / ((square / 0.003).sqrt() + 1e-9) + DECAY * flat
    return {"loss": loss.detach().reshape(1), "correct": correct, "weights": flat - LR * step, "mean": mean, "square": square}

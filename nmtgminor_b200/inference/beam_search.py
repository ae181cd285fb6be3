"""Batched beam search with a fixed ``[sentences, beam]`` layout that never leaves the device.

Every step: the model scores the last symbol of all ``B * beam`` hypotheses (incremental key/value
caches), the ``2 * beam`` best continuations per sentence are taken from the flattened ``beam * V`` scores,
continuations ending in EOS are moved into a per-sentence table of finished hypotheses (kept sorted, best
``beam`` only), the first ``beam`` non-EOS continuations become the new active set and the decoder caches
are re-indexed accordingly.  A sentence stops when it has ``beam`` finished hypotheses and its best active
score can no longer enter the table; the loop ends when all sentences stopped or ``max_len`` is reached.
The batch is not shrunk when sentences finish (static shapes keep the step graph-capturable); finished
sentences simply stop contributing.  On a GPU a search without constraints runs as one captured CUDA graph per step
(``_DeviceSearch``); the others read from the device only every fourth step (the "all sentences done" flag), with finished
sentences masked in between.  On the CPU one ``any()`` per step skips the merge of finished hypotheses when no EOS was produced.

Constraints supported: minimum length, maximum length (absolute or ``a * src_len + b``), length-normalised
scores (``score / len^alpha``), n-gram blocking, forced target prefixes, banned first tokens, vocabulary
masks, sampling instead of top-k.

Functional counterpart of the reference's ``FastTranslator._translate_batch``
(onmt/inference/fast_translator.py:428-1010) and ``BeamSearch.step`` (onmt/inference/search.py:62-106).
"""
from __future__ import annotations

import threading
from dataclasses import dataclass, field
from typing import List, Optional

import torch


@dataclass
class BeamConfig:
    beam_size: int = 4
    n_best: int = 1
    max_len: int = 256
    min_len: int = 1
    dynamic_max_len: bool = False
    len_a: float = 1.5          # max_len = len_a * src_len + len_b when dynamic
    len_b: float = 10.0
    alpha: float = 0.0          # length-penalty exponent (0 = raw sum of log-probabilities)
    normalize: bool = False
    no_repeat_ngram_size: int = 0
    bos: int = 2
    eos: int = 3
    pad: int = 0
    sampling: bool = False
    sampling_temperature: float = 1.0
    diversity_rate: float = 0.0  # > 0: sibling-rank penalty (the k-th best continuation of a hypothesis loses k * rate)
    vocab_mask: Optional[torch.Tensor] = None   # bool [V], True = allowed
    fused_step: bool = True     # CUDA: fused log-softmax + top-k kernel when no constraint needs full log-probabilities
    cuda_graph: bool = True     # CUDA + fused_step: replay whole search steps as a captured graph


@dataclass
class Hypothesis:
    tokens: List[int]
    score: float
    positional_scores: List[float] = field(default_factory=list)


def _block_ngrams(tokens, step, lprobs, n, pad):
    """Set to -inf every symbol that would complete an n-gram already present in its hypothesis."""
    if n <= 0 or step + 1 < n:
        return lprobs
    hist = tokens[:, :step + 1]
    R = hist.shape[0]
    if n == 1:
        lprobs.scatter_(1, hist, float("-inf"))
        return lprobs
    prefix = hist[:, -(n - 1):]                                   # last n-1 symbols
    windows = hist.unfold(1, n, 1)                                # [R, W, n]
    match = (windows[:, :, :n - 1] == prefix[:, None, :]).all(-1)  # [R, W]
    banned = windows[:, :, n - 1]
    rows = torch.arange(R, device=tokens.device)[:, None].expand_as(banned)
    lprobs[rows[match], banned[match]] = float("-inf")
    return lprobs


def _masked_topk(lprobs, cfg, step, max_rows, prefix_tokens, banned_first, tokens, scores, B, K):
    """Reference step: apply the length / prefix / n-gram constraints to ``lprobs`` [R, V] and pick 2K candidates."""
    device = lprobs.device
    R = B * K
    V = lprobs.shape[1]
    lprobs[:, cfg.pad] = float("-inf")
    if cfg.vocab_mask is not None:
        lprobs.masked_fill_(~cfg.vocab_mask[None, :].to(device), float("-inf"))
    if step < cfg.min_len:
        lprobs[:, cfg.eos] = float("-inf")
    force_eos = (step >= max_rows)                             # at the length limit only EOS may follow
    if force_eos.any():
        keep = lprobs[:, cfg.eos].clone()
        lprobs[force_eos] = float("-inf")
        lprobs[force_eos, cfg.eos] = keep[force_eos]
    if prefix_tokens is not None and step < prefix_tokens.shape[1]:
        want = prefix_tokens[:, step].repeat_interleave(K)
        forced = want != cfg.pad
        if forced.any():
            keep = lprobs.gather(1, want[:, None]).squeeze(1)
            lprobs[forced] = float("-inf")
            lprobs[forced, want[forced]] = keep[forced]
    if banned_first is not None and step == 0:
        lprobs[:, banned_first] = float("-inf")
    lprobs = _block_ngrams(tokens, step, lprobs, cfg.no_repeat_ngram_size, cfg.pad)
    if cfg.diversity_rate > 0 and step > 0:
        # diverse beam search: only the best 2K continuations of a hypothesis can be selected, so ranking those suffices
        top_v, top_i = lprobs.topk(min(2 * K, V), dim=1)
        penalty = torch.arange(top_v.shape[1], device=device, dtype=lprobs.dtype) * cfg.diversity_rate
        lprobs = lprobs.scatter(1, top_i, top_v - penalty[None, :])

    cand = scores[:, :, None] + lprobs.view(B, K, V)            # [B, K, V]
    flat = cand.view(B, K * V)
    if cfg.sampling and step > 0:
        probs = torch.softmax(lprobs.view(B, K, V) / cfg.sampling_temperature, -1)
        samp = torch.multinomial(probs.view(R, V), 2).view(B, K * 2)
        beam_of = torch.arange(K, device=device).repeat_interleave(2)[None, :].expand(B, -1)
        top_idx = beam_of * V + samp
        top_scores = flat.gather(1, top_idx)
    else:
        top_scores, top_idx = flat.topk(min(2 * K, K * V), dim=1)
    return top_scores, top_idx, V


def _replayable(model, state) -> bool:
    """Whether every step of ``model`` is its decoder's static step over fused key/value caches, so that a captured step sees
    everything it needs at fixed addresses."""
    from ..models.layers import SelfAttention
    from ..models.transformer import Seq2SeqBase
    dec = getattr(model, "decoder", None)
    if dec is None or not hasattr(dec, "step_static") or getattr(type(model), "step", None) is not Seq2SeqBase.step:
        return False
    if getattr(dec, "language_embedding", None) is not None or getattr(dec, "adapters", None) is not None:
        return False
    attn = [m for m in dec.modules() if isinstance(m, SelfAttention)]
    return (len(attn) == len(state.buffers) and all(type(m).step is SelfAttention.step and not m.rotary and m.dim // m.heads == 64 for m in attn)
            and state.context.is_cuda and state.context.dtype == torch.bfloat16)


class _StepPools:
    """Table sets, and the graphs captured over them, of one model in one state.  A graph has the address of every tensor baked in that
    its step reads besides its own tables.  The state is those addresses, so that a graph is replayed only on a model whose tensors
    lie where they lay; one that has moved (a longer position table, a new weight store, a layer replaced) gets a new object.

    Searches may run in several threads: a set belongs to one search at a time, and the lock guards the sets and the captures."""

    MAX_KEPT = 4
    lock = threading.RLock()
    streams = {}             # device index -> the stream that captures run on

    @classmethod
    def capture_stream(cls, device):
        """A stream of the process that no other thread can be working on: its launches would end up in the graph."""
        from .. import ops
        with cls.lock:
            if device.index not in cls.streams:
                cls.streams[device.index] = torch.cuda.ExternalStream(ops.ext().make_stream(device.index), device=device)
            return cls.streams[device.index]

    def __init__(self, state):
        self.state = state
        self.sets = {}

    def take(self, key):
        with self.lock:
            return self.sets.pop(key, None)

    def put(self, key, kept):
        with self.lock:
            self.sets.pop(key, None)             # of two searches of one geometry the later one's set stays
            while len(self.sets) >= self.MAX_KEPT:
                self.sets.pop(next(iter(self.sets)))
            self.sets[key] = kept

    @classmethod
    def of(cls, model, device, modules=None):
        """The pool of ``model`` as it is now, and the tensors that its steps read: a search holds on to them, since another thread may
        replace the position table meanwhile.  ``modules``: those of the decoder, if they are at hand."""
        emb = getattr(model.decoder, "embed", None)
        modules = list(model.decoder.modules()) if modules is None else modules
        reads = [emb._pos_table(device) if hasattr(emb, "_pos_table") else None]
        generator = getattr(model, "generator", None)
        for m in (*modules, *(generator.modules() if generator is not None else ())):
            if m._parameters or m._buffers:
                for t in (*m._parameters.values(), *m._buffers.values()):
                    reads += (t, getattr(t, "work", None))
        state = [m.training for m in modules]
        state += [None if t is None else (t.data_ptr(), t.shape, t.dtype) for t in reads]
        with cls.lock:
            pools = model.__dict__.get("_decode_pools")
            if pools is None or pools.state != state:
                pools = model.__dict__["_decode_pools"] = cls(state)
        return pools, reads

    def __reduce__(self):           # a copied or saved model starts without
        return type(None), ()


class _DeviceSearch:
    """A search whose steps never leave the device: embedding, decoder layers over preallocated caches, output projection, best
    continuations and all bookkeeping (finished hypotheses, next active set, ancestors of every cached position) read and
    write tables at fixed addresses, so one captured CUDA graph is replayed per step.  Hypotheses are not moved when they
    are re-ranked: every step leaves a (word, parent, score) record, the words of the finished ones are traced back at the end,
    and attention finds a hypothesis's past through a table of cache rows.

    Tables, caches and the graph are kept on the model for later batches of the same geometry; a search takes its set out of the pool
    and puts it back when its results are on the host, so concurrent searches have sets of their own."""

    @staticmethod
    def capacity(T: int) -> int:
        """Cached positions for ``T`` steps, rounded so that batches share a geometry."""
        return (T + 2 + 63) // 64 * 64

    def __init__(self, model, state, cfg, K: int, B: int, T: int, max_len_per):
        dev = state.context.device
        R = B * K
        self.model, self.state, self.cfg, self.K, self.B, self.T = model, state, cfg, K, B, T
        cap = self.capacity(T)
        emb = getattr(model.decoder, "embed", None)
        if emb is not None and hasattr(emb, "renew"):
            emb.renew(cap)
        from ..models.layers import SelfAttention
        modules = list(model.decoder.modules())
        widths = [m.dim for m in modules if isinstance(m, SelfAttention)]
        cross = [b for b in state.buffers if "c_k" in b]
        src_cap = (max(b["c_k"].shape[1] for b in cross) + 63) // 64 * 64 if cross else 0
        self.key = (B, K, cap, src_cap, len(state.buffers), str(dev), cfg.pad, cfg.eos)
        self.pools, self.reads = _StepPools.of(model, dev, modules)
        pool = self.pools.take(self.key)
        if pool is None:
            with torch.inference_mode(False), torch.no_grad():      # kept tables serve callers in either mode
                mk = lambda shape, dt: torch.zeros(shape, dtype=dt, device=dev)
                i32, f32, i64 = torch.int32, torch.float32, torch.int64
                pool = {"graph": None, "warm": 0, "tables": [
                    mk(3, i32), mk(cap + 1, f32), mk(B, i32), mk(R, f32), mk(R, torch.uint8), mk(B, torch.uint8), mk(R, i64), mk(R, i64),
                    mk((R, cap), i32), mk(B, i32), mk((B, K), f32), mk((B, K), i32), mk((B, K), i32), mk((B, K), f32),
                    mk((cap, R), i32), mk((cap, R), i32), mk((cap, R), f32)], "layers": []}
                for buf, H in zip(state.buffers, widths):
                    keep = {name: torch.empty(R, cap, H, dtype=torch.bfloat16, device=dev) for name in ("k", "v")}
                    if "c_k" in buf:
                        shape = (B, src_cap, buf["c_k"].shape[2])
                        keep.update(c_k=mk(shape, torch.bfloat16), c_v=mk(shape, torch.bfloat16), c_len=mk(B, i32))
                    pool["layers"].append(keep)
                pool["done_host"] = [torch.zeros(B, dtype=torch.uint8, pin_memory=True) for _ in range(2)]
        self.pool = pool
        (ctl, inv_norm, max_rows, scores, force, done, tok, pos_rows, anc, fin_count, fin_score) = pool["tables"][:11]
        self.tok, self.pos_rows, self.done = tok, pos_rows, done
        # `normalize` alone decides the stop rule; scores are divided only if there is a length penalty as well
        ctl.copy_(torch.tensor([T, cfg.min_len, int(bool(cfg.normalize))], dtype=torch.int32))
        # reciprocal of the length penalty in the precision of a division by a host scalar
        penalty = bool(cfg.normalize and cfg.alpha > 0)
        inv_norm[1:T + 2].copy_(1.0 / torch.tensor([float(n) ** cfg.alpha if penalty else 1.0 for n in range(1, T + 2)], dtype=torch.float32))
        max_rows.copy_(max_len_per)
        scores.fill_(float("-inf"))
        scores.view(B, K)[:, 0] = 0.0                       # only the first hypothesis is alive at step 0
        force.copy_(torch.where(max_len_per <= 0, 1, 2 if cfg.min_len > 0 else 0).repeat_interleave(K))
        tok.fill_(cfg.bos)
        fin_score.fill_(float("-inf"))
        for t in (done, pos_rows, fin_count):
            t.zero_()
        for buf, keep in zip(state.buffers, pool["layers"]):
            if "c_k" in buf:
                ts = buf["c_k"].shape[1]
                keep["c_k"][:, :ts].copy_(buf["c_k"])
                keep["c_v"][:, :ts].copy_(buf["c_v"])
                keep["c_len"].copy_(buf["c_len"])
            buf.update(keep)
            buf.update(anc=anc, pos_rows=pos_rows, beam=K, cap=cap)

    def _body(self):
        from .. import ops
        ops.ext().set_step_overlap(True)        # this thread's launches
        try:
            with ops.step_sums:
                hidden = self.model.decoder.step_static(self.tok, self.pos_rows, self.state)
                logits = self.model.generator(hidden)
            if logits.dtype not in (torch.float32, torch.bfloat16):
                logits = logits.float()
            ops.ext().beam_step(logits, self.pool["tables"], self.K, self.cfg.pad, self.cfg.eos)
        finally:
            ops.ext().set_step_overlap(False)

    def _step(self):
        pool = self.pool
        if pool["warm"] < 2:                    # lazy initialisation happens outside the capture
            pool["warm"] += 1
            return self._body()
        while pool["graph"] is None:
            with _StepPools.lock:               # one capture at a time
                self.pools, self.reads = _StepPools.of(self.model, self.tok.device)
                g = torch.cuda.CUDAGraph()
                torch.cuda.synchronize()
                with torch.cuda.graph(g, stream=_StepPools.capture_stream(self.tok.device), capture_error_mode="thread_local"):
                    self._body()                # captured, not run
                # another thread may have renewed the position table meanwhile: then this graph reads another one than is held
                if _StepPools.of(self.model, self.tok.device)[0] is self.pools:
                    pool["graph"] = g
        pool["graph"].replay()

    def run(self):
        """All steps, then per sentence the ``n_best`` finished hypotheses, best first."""
        with torch.cuda.device(self.tok.device):        # events and captures belong to the model's device, whichever is current
            return self._run()

    def _run(self):
        from .. import ops
        cfg, K = self.cfg, self.K
        seen = None
        for step in range(self.T + 1):
            self._step()
            if step % 4 == 3 and step < self.T:
                # "all sentences done", read four steps late so that the device never waits for the host
                if seen is not None:
                    seen[0].synchronize()
                    if bool(seen[1].all()):
                        break
                host = self.pool["done_host"][(step // 4) & 1]
                host.copy_(self.done, non_blocking=True)
                event = torch.cuda.Event()
                event.record()
                seen = (event, host)
        tables = self.pool["tables"]
        n = max(1, min(cfg.n_best, K))
        words, word_scores = ops.ext().beam_trace(tables, K, cfg.pad, cfg.eos, n)
        scores, last = tables[10][:, :n].cpu(), tables[11][:, :n].cpu()
        longest = int(last.masked_fill(scores == float("-inf"), 0).max()) + 1
        words, word_scores = words[:, :, :longest].cpu(), word_scores[:, :, :longest].cpu()
        self.pools.put(self.key, self.pool)
        results = []
        for b in range(self.B):
            hyps = []
            for k in range(min(cfg.n_best, K)):
                if torch.isfinite(scores[b, k]):
                    m = int(last[b, k]) + 1
                    hyps.append(Hypothesis(words[b, k, :m].tolist(), float(scores[b, k]), word_scores[b, k, :m].tolist()))
            results.append(hyps or [Hypothesis([cfg.eos], float("-inf"))])
        return results


@torch.no_grad()
def beam_search(model, batch, cfg: BeamConfig, prefix_tokens: Optional[torch.Tensor] = None,
                banned_first: Optional[torch.Tensor] = None) -> List[List[Hypothesis]]:
    """Decode every sentence of ``batch``; returns ``n_best`` hypotheses per sentence (best first)."""
    K = cfg.beam_size
    state = model.create_decoder_state(batch, K)
    # batch size / source lengths come from the encoder output, so audio batches (no packed source) work too
    device = state.context.device
    B = state.context.shape[0] // K
    src_len = (~state.src_pad_mask).sum(1)[::K].to(torch.float32)
    if cfg.dynamic_max_len:
        max_len_per = (cfg.len_a * src_len + cfg.len_b).clamp(max=cfg.max_len).long()
    else:
        max_len_per = torch.full((B,), cfg.max_len, device=device, dtype=torch.long)
    T = int(max_len_per.max().item())
    # fused step: log-softmax, masks and the per-sentence top-2K in two kernels, no [R, V] log-probabilities
    fused = (device.type == "cuda" and cfg.fused_step and getattr(model, "supports_logits_step", False)
             and not cfg.sampling and cfg.no_repeat_ngram_size <= 0 and cfg.vocab_mask is None and 2 * K <= 64
             and cfg.diversity_rate <= 0)
    if (fused and cfg.cuda_graph and prefix_tokens is None and banned_first is None and _replayable(model, state)
            and B * K * _DeviceSearch.capacity(T) < 2 ** 31):       # cache rows are addressed with 32 bits
        return _DeviceSearch(model, state, cfg, K, B, T, max_len_per).run()
    R = B * K
    tokens = torch.full((R, T + 2), cfg.pad, dtype=torch.long, device=device)
    tokens[:, 0] = cfg.bos
    pos_scores = torch.zeros((R, T + 2), dtype=torch.float32, device=device)
    scores = torch.zeros((B, K), dtype=torch.float32, device=device)
    scores[:, 1:] = float("-inf")                                  # only beam 0 is alive at step 0
    fin_scores = torch.full((B, K), float("-inf"), device=device)
    fin_tokens = torch.full((B, K, T + 2), cfg.pad, dtype=torch.long, device=device)
    fin_pos = torch.zeros((B, K, T + 2), dtype=torch.float32, device=device)
    fin_len = torch.zeros((B, K), dtype=torch.long, device=device)
    fin_count = torch.zeros(B, dtype=torch.long, device=device)
    done = torch.zeros(B, dtype=torch.bool, device=device)
    base = (torch.arange(B, device=device) * K)[:, None]
    max_rows = max_len_per.repeat_interleave(K)

    if hasattr(state, "set_cache_capacity") and device.type == "cuda":
        state.set_cache_capacity(T + 2)
    for step in range(T + 1):
        use_fused = (fused and not (prefix_tokens is not None and step < prefix_tokens.shape[1])
                     and not (banned_first is not None and step == 0))
        if use_fused:
            from .. import ops
            logits = model.step(tokens[:, :step + 1], state, logits_only=True)["logits"]
            V = logits.shape[1]
            if logits.dtype not in (torch.float32, torch.bfloat16):
                logits = logits.float()
            top_scores, top_idx, _ = ops.ext().beam_topk(logits, scores.reshape(-1).contiguous(),
                                                         (step >= max_rows).to(torch.uint8), K, cfg.pad, cfg.eos,
                                                         step < cfg.min_len)
            lprobs = None
        else:
            top_scores = None
            out = model.step(tokens[:, :step + 1], state)
            lprobs = out["log_prob"].float()                       # [R, V]
        if lprobs is not None:
            top_scores, top_idx, V = _masked_topk(lprobs, cfg, step, max_rows, prefix_tokens, banned_first, tokens, scores, B, K)
        cand_beam = top_idx // V
        cand_tok = top_idx % V
        C = top_scores.shape[1]
        is_eos = (cand_tok == cfg.eos) & torch.isfinite(top_scores)
        # an EOS candidate only counts when it is within the top `beam` of the step (fairseq convention)
        is_eos &= torch.arange(C, device=device)[None, :] < K
        is_eos &= ~done[:, None]

        # ---- finalize: merge EOS candidates into the sorted table of finished hypotheses ---------
        # on a GPU the merge runs whenever EOS is possible instead of asking the device (`any()` would stall the host)
        if step >= cfg.min_len and (device.type == "cuda" or bool(is_eos.any())):
            length = step + 1                                      # symbols after BOS, including EOS
            norm = (float(length) ** cfg.alpha) if (cfg.normalize and cfg.alpha > 0) else 1.0
            new_scores = torch.where(is_eos, top_scores / norm, torch.full_like(top_scores, float("-inf")))
            src_rows = (base + cand_beam).view(-1)
            new_tok = tokens[src_rows].view(B, C, T + 2).clone()
            new_tok[:, :, step + 1] = cfg.eos
            new_pos = pos_scores[src_rows].view(B, C, T + 2).clone()
            new_pos[:, :, step + 1] = top_scores - scores.gather(1, cand_beam)
            all_scores = torch.cat([fin_scores, new_scores], 1)
            order = all_scores.argsort(dim=1, descending=True, stable=True)[:, :K]
            gather3 = order[:, :, None].expand(-1, -1, T + 2)
            fin_tokens = torch.cat([fin_tokens, new_tok], 1).gather(1, gather3)
            fin_pos = torch.cat([fin_pos, new_pos], 1).gather(1, gather3)
            fin_len = torch.cat([fin_len, torch.full((B, C), length, device=device, dtype=torch.long)], 1).gather(1, order)
            fin_scores = all_scores.gather(1, order)
            fin_count = (fin_count + is_eos.sum(1)).clamp(max=K)

        # ---- next active set: first K non-EOS candidates -----------------------------------------
        alive_key = torch.where(cand_tok == cfg.eos, torch.full_like(top_scores, float("-inf")), top_scores)
        act_scores, act_pos = alive_key.topk(K, dim=1)
        act_beam = cand_beam.gather(1, act_pos)
        act_tok = cand_tok.gather(1, act_pos)
        reorder = (base + act_beam).view(-1)
        tokens = tokens.index_select(0, reorder)
        pos_scores = pos_scores.index_select(0, reorder)
        tokens[:, step + 1] = act_tok.view(-1)
        pos_scores[:, step + 1] = (act_scores - scores.gather(1, act_beam)).view(-1)
        scores = act_scores
        state.reorder(reorder)

        # ---- stopping ------------------------------------------------------------------------------
        best_possible = scores[:, 0] / ((float(T + 1) ** cfg.alpha) if (cfg.normalize and cfg.alpha > 0) else 1.0)
        worst_fin = fin_scores[:, K - 1]
        stop_early = (best_possible <= worst_fin) if cfg.normalize else torch.ones_like(done)
        done = done | ((fin_count >= K) & stop_early) | ~torch.isfinite(scores[:, 0])
        scores = torch.where(done[:, None], torch.full_like(scores, float("-inf")), scores)
        if (device.type != "cuda" or step % 4 == 3 or step == T) and bool(done.all()):
            break

    fin_scores_c, fin_tokens_c, fin_len_c, fin_pos_c = fin_scores.cpu(), fin_tokens.cpu(), fin_len.cpu(), fin_pos.cpu()
    results: List[List[Hypothesis]] = []
    for b in range(B):
        hyps = []
        for k in range(min(cfg.n_best, K)):
            if not torch.isfinite(fin_scores_c[b, k]):
                continue
            n = int(fin_len_c[b, k])
            hyps.append(Hypothesis(fin_tokens_c[b, k, 1:n + 1].tolist(), float(fin_scores_c[b, k]),
                                   fin_pos_c[b, k, 1:n + 1].tolist()))
        if not hyps:
            hyps.append(Hypothesis([cfg.eos], float("-inf")))
        results.append(hyps)
    return results


@torch.no_grad()
def greedy_search(model, batch, max_len: int = 256, bos: int = 2, eos: int = 3, pad: int = 0) -> List[List[int]]:
    state = model.create_decoder_state(batch, 1)
    B = state.context.shape[0]
    device = state.context.device
    tokens = torch.full((B, max_len + 2), pad, dtype=torch.long, device=device)
    tokens[:, 0] = bos
    finished = torch.zeros(B, dtype=torch.bool, device=device)
    for step in range(max_len + 1):
        lp = model.step(tokens[:, :step + 1], state)["log_prob"]
        lp[:, pad] = float("-inf")
        nxt = lp.argmax(-1)
        nxt = torch.where(finished, torch.full_like(nxt, pad), nxt)
        tokens[:, step + 1] = nxt
        finished |= nxt == eos
        if bool(finished.all()):
            break
    out = []
    for row in tokens[:, 1:].tolist():
        seq = []
        for t in row:
            if t == pad:
                break
            seq.append(t)
            if t == eos:
                break
        out.append(seq)
    return out

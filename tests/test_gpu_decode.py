"""Beam-step, cache and single-query attention kernels against PyTorch."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from nmtgminor_b200 import ops


def _dev():
    return torch.device("cuda", 0)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("V", [50, 4096, 32000])
def test_beam_topk_matches_torch(dtype, V):
    torch.manual_seed(0)
    dev = _dev()
    B, K = 5, 4
    R = B * K
    logits = torch.randn(R, V, device=dev).to(dtype)
    scores = torch.randn(R, device=dev)
    scores[3] = float("-inf")
    force = torch.zeros(R, dtype=torch.uint8, device=dev)
    force[6] = 1
    pad, eos = 0, 3
    for ban in (False, True):
        os_, oi, lse = ops.ext().beam_topk(logits, scores, force, K, pad, eos, ban)
        lp = torch.log_softmax(logits.float(), -1)
        assert torch.allclose(lse, torch.logsumexp(logits.float(), -1), atol=1e-4)
        lp[:, pad] = float("-inf")
        if ban:
            lp[:, eos] = float("-inf")
        keep = torch.log_softmax(logits.float(), -1)[6, eos]
        lp[6] = float("-inf")
        lp[6, eos] = keep
        tot = (lp + scores[:, None]).view(B, K * V)
        rs, ri = tot.topk(2 * K, dim=1)
        assert torch.allclose(os_, rs, atol=1e-4, rtol=1e-5)
        finite = torch.isfinite(rs)
        # ties are rare with random inputs; compare indices where the scores are distinct
        same = (oi == ri) | ~finite
        if dtype == torch.float32:
            assert same.float().mean().item() > 0.97
        got = tot.gather(1, oi.clamp(0, K * V - 1))
        assert torch.allclose(got[finite], rs[finite], atol=1e-4)


def test_gather_rows_and_cache_append():
    dev = _dev()
    R, cap, hid = 6, 10, 128
    src = torch.randn(R, cap, hid, device=dev).bfloat16()
    dst = torch.zeros_like(src)
    index = torch.tensor([5, 0, 0, 3, 2, 2], device=dev)
    ops.ext().gather_rows(src, dst, index, 4 * hid)
    assert torch.equal(dst[:, :4], src[index][:, :4]) and dst[:, 4:].abs().sum() == 0
    ops.ext().gather_rows(src, dst, index, -1)
    assert torch.equal(dst, src[index])
    kc, vc = torch.zeros(R, cap, hid, device=dev).bfloat16(), torch.zeros(R, cap, hid, device=dev).bfloat16()
    kv = torch.randn(R, 3 * hid, device=dev).bfloat16()
    ops.ext().cache_append(kv[:, hid:2 * hid], kv[:, 2 * hid:], kc, vc, 7)
    assert torch.equal(kc[:, 7], kv[:, hid:2 * hid]) and torch.equal(vc[:, 7], kv[:, 2 * hid:]) and kc[:, :7].abs().sum() == 0


@pytest.mark.parametrize("kv_div", [1, 4])
@pytest.mark.parametrize("cap,length", [(16, 1), (160, 37), (1500, 1500)])
def test_decode_attention(kv_div, cap, length):
    torch.manual_seed(1)
    dev = _dev()
    R, heads = 8, 4
    hid = heads * 64
    q = torch.randn(R, 3 * hid, device=dev).bfloat16()[:, :hid]             # strided rows
    kc = torch.randn(R // kv_div, cap, hid, device=dev).bfloat16()
    vc = torch.randn(R // kv_div, cap, hid, device=dev).bfloat16()
    lengths = torch.randint(1, length + 1, (R // kv_div,), device=dev, dtype=torch.int32)
    lengths[0] = length
    scale = 1 / 8.0
    for lens in (None, lengths):
        out = ops.ext().decode_attn(q, kc, vc, lens, length, heads, scale)
        qf = q.float().view(R, heads, 64)
        kf = kc.float().view(-1, cap, heads, 64).repeat_interleave(kv_div, 0)
        vf = vc.float().view(-1, cap, heads, 64).repeat_interleave(kv_div, 0)
        s = torch.einsum("rhd,rjhd->rhj", qf, kf) * scale
        ln = (lens if lens is not None else torch.full_like(lengths, length)).repeat_interleave(kv_div)
        mask = torch.arange(cap, device=dev)[None, None, :] >= ln[:, None, None]
        p = torch.softmax(s.masked_fill(mask, float("-inf")), -1)
        ref = torch.einsum("rhj,rjhd->rhd", p, vf).reshape(R, hid)
        assert torch.allclose(out.float(), ref, atol=2e-2, rtol=2e-2)


def test_fused_beam_search_matches_unfused_and_cpu():
    """Preallocated caches + single-query attention + fused top-k give the hypotheses of the plain PyTorch path."""
    import copy

    from nmtgminor_b200.data.dataset import collate
    from nmtgminor_b200.data.synthetic import synthetic_dict
    from nmtgminor_b200.inference.beam_search import BeamConfig, beam_search
    from nmtgminor_b200.models.transformer import Transformer
    from nmtgminor_b200.options import default_options
    from nmtgminor_b200.parallel.flat import FlatParameterStore

    torch.manual_seed(0)
    d = synthetic_dict(500)
    opt = default_options(["-model_size", "256", "-layers", "2", "-n_heads", "4", "-inner_size", "512", "-tie_weights",
                           "-join_embedding", "-ffn_activation", "relu"])
    model = Transformer(opt, {"src": d, "tgt": d}).eval()
    # sharpen the output distribution so that bf16 rounding cannot flip the ranking
    with torch.no_grad():
        model.generator.weight.mul_(6.0)
    gpu = copy.deepcopy(model)
    FlatParameterStore(gpu, "cuda")
    for b in gpu.buffers():
        b.data = b.data.cuda()
    g = torch.Generator().manual_seed(1)
    src = [torch.randint(4, 500, (int(n),), generator=g) for n in (7, 12, 5, 9, 3)]
    batch = collate(src, None, padded=True, packed=True, round_to=1)
    gbatch = copy.deepcopy(batch).cuda("cuda")
    res = {}
    for name, fused, graph in (("fused", True, False), ("graph", True, True), ("plain", False, False)):
        cfg = BeamConfig(beam_size=4, n_best=2, max_len=20, min_len=2, fused_step=fused, cuda_graph=graph)
        res[name] = beam_search(gpu, gbatch, cfg)
    assert ops.check_status() == 0
    for other in ("plain", "graph"):
        for a, b in zip(res["fused"], res[other]):
            assert [h.tokens for h in a] == [h.tokens for h in b], other
            for ha, hb in zip(a, b):
                assert abs(ha.score - hb.score) < 5e-2
                assert len(ha.positional_scores) == len(ha.tokens)
    cpu = beam_search(model, batch, BeamConfig(beam_size=4, n_best=2, max_len=20, min_len=2))
    agree = sum(a[0].tokens == c[0].tokens for a, c in zip(res["fused"], cpu))
    assert agree >= 4, "best hypotheses differ between the bf16 GPU path and the fp32 CPU path"


@pytest.mark.parametrize("B,K,heads,cap,pos", [(1, 1, 1, 64, 0), (3, 2, 2, 64, 1), (2, 4, 3, 64, 33), (5, 3, 2, 192, 130), (2, 6, 1, 320, 319), (1, 12, 2, 64, 40)])
def test_step_self_attention(B, K, heads, cap, pos):
    """Append + attention through a table of ancestor rows: first position, block edges, several CTAs per sentence."""
    g = torch.Generator(device="cuda").manual_seed(pos + K)
    R, hid = B * K, heads * 64
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    qkv, kc, vc = rnd(R, 3 * hid + 8)[:, :3 * hid], rnd(R, cap, hid), rnd(R, cap, hid)
    anc = (torch.randint(0, K, (B, K, cap), device="cuda", generator=g) + torch.arange(B, device="cuda")[:, None, None] * K).int().view(R, cap).contiguous()
    before = kc.clone(), vc.clone()
    out = ops.ext().decode_self(qkv, kc, vc, anc, torch.full((R,), pos, dtype=torch.long, device="cuda"), K, heads, 0.125)
    q, k, v = (t.double().view(R, heads, 64) for t in qkv.split(hid, 1))
    take = lambda c: torch.stack([c[anc[:, j].long(), j] for j in range(pos)], 1).double().view(R, pos, heads, 64) if pos else k.new_zeros(R, 0, heads, 64)
    keys, vals = torch.cat([take(before[0]), k[:, None]], 1), torch.cat([take(before[1]), v[:, None]], 1)
    p = torch.softmax(torch.einsum("rhd,rjhd->rhj", q, keys) * 0.125, -1)
    want = torch.einsum("rhj,rjhd->rhd", p, vals).reshape(R, hid)
    assert (out.double() - want).abs().max() < 2 ** -8 * want.abs().max()          # one rounding to bf16 of a 32-bit result
    before[0][:, pos], before[1][:, pos] = qkv[:, hid:2 * hid], qkv[:, 2 * hid:]
    assert torch.equal(kc, before[0]) and torch.equal(vc, before[1])


@pytest.mark.parametrize("B,K,heads,cap", [(1, 1, 1, 31), (2, 4, 2, 100), (1, 5, 2, 513), (3, 2, 4, 1500), (2, 9, 1, 1536), (1, 4, 16, 4096)])
def test_step_cross_attention(B, K, heads, cap):
    """One sentence's hypotheses over its shared keys, the long ones cut over a cluster; lengths 0, 1 and full among them."""
    g = torch.Generator(device="cuda").manual_seed(cap)
    hid = heads * 64
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    q, k, v = rnd(B * K, hid), rnd(B, cap, hid), rnd(B, cap, hid)
    for lens in ([cap] * B, [1] * B, [0] * B, [(cap * (i + 2)) // (B + 3) for i in range(B)]):
        out = ops.ext().decode_cross(q, k, v, torch.tensor(lens, dtype=torch.int32, device="cuda"), heads, 0.125)
        for b, n in enumerate(lens):
            qb, kb, vb = q[b * K:(b + 1) * K].double().view(K, heads, 64), k[b, :n].double().view(n, heads, 64), v[b, :n].double().view(n, heads, 64)
            want = torch.einsum("khj,jhd->khd", torch.softmax(torch.einsum("khd,jhd->khj", qb, kb) * 0.125, -1), vb).reshape(K, hid)
            assert (out[b * K:(b + 1) * K].double() - want).abs().max() <= 2 ** -8 * want.abs().max() + 1e-6


@pytest.mark.parametrize("K,pos", [(1, 15), (1, 16), (3, 17), (5, 255), (7, 256), (8, 31), (8, 513), (9, 257), (17, 16)])
def test_step_attention_tiles(K, pos):
    """Edges of the key blocks (16), of the staged ancestors (256) and of the eight queries of a CTA, with a past that the hypotheses
    share at first; a hypothesis whose past is not a number leaves the others of its sentence alone."""
    g = torch.Generator(device="cuda").manual_seed(pos * K)
    B, heads = 2, 2
    R, hid, cap = B * K, heads * 64, (pos + 64) // 64 * 64
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    qkv, kc, vc = rnd(R, 3 * hid), rnd(R, cap, hid), rnd(R, cap, hid)
    own = torch.arange(R, device="cuda").view(B, K, 1)
    anc = torch.where(torch.arange(cap, device="cuda") < pos // 2, own[:, :1], own).int().view(R, cap).contiguous()
    if K > 1:
        vc[1, pos // 2:], kc[1, pos // 2:] = float("nan"), float("nan")
    out = ops.ext().decode_self(qkv, kc.clone(), vc.clone(), anc, torch.full((R,), pos, dtype=torch.long, device="cuda"), K, heads, 0.125)
    q, k, v = (t.double().view(R, heads, 64) for t in qkv.split(hid, 1))
    take = lambda c: torch.stack([c[anc[:, j].long(), j] for j in range(pos)], 1).double().view(R, pos, heads, 64)
    keys, vals = torch.cat([take(kc), k[:, None]], 1), torch.cat([take(vc), v[:, None]], 1)
    want = torch.einsum("rhj,rjhd->rhd", torch.softmax(torch.einsum("rhd,rjhd->rhj", q, keys) * 0.125, -1), vals).reshape(R, hid)
    if K > 1:
        assert out[1].isnan().all()
        out[1], want[1] = 0, 0
    assert (out.double() - want).abs().max() < 2 ** -8 * want.abs().max()          # one rounding to bf16 of a 32-bit result
    # the same queries over keys that all of them share, from rows that do not start on 16 bytes
    shift = torch.zeros(R, hid + 8, dtype=torch.bfloat16, device="cuda")[:, 3:hid + 3]
    shift.copy_(qkv[:, :hid])
    kb, vb = rnd(B, pos, hid), rnd(B, pos, hid)
    out = ops.ext().decode_cross(shift, kb, vb, torch.tensor([pos, pos - 3], dtype=torch.int32, device="cuda"), heads, 0.125)
    for b, n in enumerate((pos, pos - 3)):
        qb, kk, vv = q[b * K:(b + 1) * K], kb[b, :n].double().view(n, heads, 64), vb[b, :n].double().view(n, heads, 64)
        want = torch.einsum("khj,jhd->khd", torch.softmax(torch.einsum("khd,jhd->khj", qb, kk) * 0.125, -1), vv).reshape(K, hid)
        assert (out[b * K:(b + 1) * K].double() - want).abs().max() < 2 ** -8 * want.abs().max()


def _compare_searches(dtype, B, K, V, T, min_len, normalize, alpha, end_bias=None, open_words=None):
    from types import SimpleNamespace

    from nmtgminor_b200.inference import beam_search as bs
    g = torch.Generator(device="cuda").manual_seed(V + T)
    ld = (V + 7) // 8 * 8
    by_word = torch.randn(V, ld, device="cuda", generator=g)
    by_word[:, 3] += 1.5                                   # EOS is likely enough to end hypotheses early
    by_step = torch.randn(T + 2, ld, device="cuda", generator=g)
    if end_bias is not None:                               # EOS is a weak continuation at first and a strong one from step 4 on
        h = torch.Generator().manual_seed(V + T)
        by_word, by_step = torch.randn(V, ld, generator=h), torch.randn(T + 2, ld, generator=h)
        by_word[:, 3] += 1.5 + end_bias
        by_word[torch.arange(V), torch.randint(4, V, (V,), generator=h)] += 6
        by_step[:4, 3], by_step[4:, 3] = 0.0, by_step[4:, 3] + 12
        by_word, by_step = by_word.cuda(), by_step.cuda()
    if open_words is not None:                             # all other words are impossible
        closed = torch.ones(ld, dtype=torch.bool, device="cuda")
        closed[open_words] = False
        by_word[:, closed] = float("-inf")
    logits_of = lambda tok, step: (by_word[tok] + by_step[step]).to(dtype)[:, :V]
    lens = torch.randint(2, 9, (B,), device="cuda", generator=g)

    class State:
        buffers = []

        def __init__(self):
            self.context = torch.zeros(B * K, 8, 4, device="cuda")
            self.src_pad_mask = (torch.arange(8, device="cuda")[None] >= lens[:, None]).repeat_interleave(K, 0)

        def reorder(self, index):
            pass

    model = SimpleNamespace(supports_logits_step=True, decoder=torch.nn.Module(), create_decoder_state=lambda batch, k: State())
    model.step = lambda tokens, state, logits_only=False: {"logits": logits_of(tokens[:, -1], tokens.shape[1] - 1)}
    cfg = bs.BeamConfig(beam_size=K, n_best=K, max_len=T, min_len=min_len, dynamic_max_len=True, len_a=1.0, len_b=T - 8, normalize=normalize,
                        alpha=alpha)
    want = bs.beam_search(model, None, cfg)
    limit = (lens.float() + T - 8).clamp(max=T).long()

    class Search(bs._DeviceSearch):
        def _body(self):
            step = int(self.pos_rows[0])
            ops.ext().beam_step(logits_of(self.tok, min(step, T + 1)), self.pool["tables"], K, cfg.pad, cfg.eos)

        _step = _body

    for _ in range(2):                                      # the second search takes the first one's tables
        got = Search(model, State(), cfg, K, B, int(limit.max()), limit).run()
        for a, b in zip(want, got):
            assert [h.tokens for h in a] == [h.tokens for h in b]
            for x, y in zip(a, b):
                assert abs(x.score - y.score) <= 2e-5 * max(1.0, abs(x.score)) or x.score == y.score
                assert torch.allclose(torch.tensor(x.positional_scores), torch.tensor(y.positional_scores), atol=2e-4)
    cfg.normalize = not normalize
    return want, bs.beam_search(model, None, cfg)          # the same under the other stop rule


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,K,V,T,min_len,normalize", [(1, 1, 40, 6, 0, False), (3, 4, 50, 12, 1, False), (5, 4, 4097, 9, 3, True),
                                                       (2, 6, 8200, 7, 0, True), (2, 32, 5000, 5, 1, False), (4, 3, 1000, 10, 10, True)])
def test_device_search_matches_host_bookkeeping(dtype, B, K, V, T, min_len, normalize):
    """The step kernels against the tensor statements of the same search, on logits that depend on the last word and the step."""
    _compare_searches(dtype, B, K, V, T, min_len, normalize, 0.6 if normalize else 0.0)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K,V,count", [(1, 4096, 4), (4, 9000, 12), (4, 13000, 60), (16, 9000, 40)])
def test_device_search_among_few_possible_words(dtype, K, V, count):
    """Pieces of the vocabulary without a possible word, and warps with fewer of them than are wanted."""
    words = torch.cat([torch.tensor([3]), torch.linspace(4, V - 1, count).long()])
    _compare_searches(dtype, 3, K, V, 8, 1, False, 0.0, open_words=words.cuda())


def test_steps_of_very_many_rows():
    """More rows than a grid has blocks along its second dimension: attention over the past and over the source, and a whole search."""
    R, hid = 66000, 64
    g = torch.Generator(device="cuda").manual_seed(1)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    k, v, q = rnd(R, 16, hid), rnd(R, 16, hid), rnd(R, hid)
    out = ops.ext().decode_cross(q, k, v, torch.full((R,), 16, dtype=torch.int32, device="cuda"), 1, 0.125)
    want = torch.einsum("rj,rjd->rd", torch.softmax(torch.einsum("rd,rjd->rj", q.float(), k.float()) * 0.125, -1), v.float())
    assert (out.float() - want).abs().max() <= 2 ** -7 * want.abs().max()          # one rounding to bf16, 32-bit sums on both sides
    qkv = rnd(R, 3 * hid)
    anc = torch.arange(R, dtype=torch.int32, device="cuda")[:, None].expand(R, 16).contiguous()
    keys, vals = torch.cat([k[:, :15], qkv[:, None, hid:2 * hid]], 1).float(), torch.cat([v[:, :15], qkv[:, None, 2 * hid:]], 1).float()
    out = ops.ext().decode_self(qkv, k, v, anc, torch.full((R,), 15, dtype=torch.long, device="cuda"), 1, 1, 0.125)
    want = torch.einsum("rj,rjd->rd", torch.softmax(torch.einsum("rd,rjd->rj", qkv[:, :hid].float(), keys) * 0.125, -1), vals)
    assert (out.float() - want).abs().max() <= 2 ** -7 * want.abs().max()
    _compare_searches(torch.bfloat16, R // 2, 2, 40, 3, 0, False, 0.0)


@pytest.mark.parametrize("B,K,V,alpha,end_bias", [(8, 2, 50, 0.0, 2.0), (6, 3, 50, 0.0, 2.0), (6, 3, 50, -0.5, 2.0), (8, 4, 300, 0.0, 3.0)])
def test_device_search_stop_rule_without_penalty(B, K, V, alpha, end_bias):
    """`normalize` without a length penalty: the search goes on after `beam` hypotheses have ended while a better one can still come."""
    found, first_ended = _compare_searches(torch.float32, B, K, V, 24, 0, True, alpha, end_bias)
    assert any([h.tokens for h in a] != [h.tokens for h in b] for a, b in zip(found, first_ended)), "the inputs must tell the two rules apart"


def _successor_model(seed, device="cuda"):
    """A small Transformer on the GPU in which every word prefers one other word."""
    from nmtgminor_b200.data.synthetic import synthetic_dict
    from nmtgminor_b200.models.transformer import Transformer
    from nmtgminor_b200.options import default_options
    from nmtgminor_b200.parallel.flat import FlatParameterStore
    torch.manual_seed(seed)
    d = synthetic_dict(300)
    opt = default_options(["-model_size", "256", "-layers", "3", "-n_heads", "4", "-inner_size", "512", "-ffn_activation", "relu"])
    model = Transformer(opt, {"src": d, "tgt": d}).eval()
    with torch.no_grad():
        # every word prefers its successor by a wide margin, so that rounding does not change the best hypothesis
        order = torch.randperm(296) + 4
        model.generator.weight[order] = 1.5 * model.decoder.embed.weight[order.roll(1)]
        model.generator.weight[order[0]] += 1.5 * model.decoder.embed.weight[2]
    model.store = FlatParameterStore(model, device)
    for b in model.buffers():
        b.data = b.data.to(device)
    return model


@pytest.mark.parametrize("beam", [1, 2, 5])
def test_replayed_search_matches_the_stepwise_one(beam):
    """Captured steps against the same search launched kernel by kernel, over enough steps and batches that the replays matter; with
    one hypothesis per sentence the encoder's keys have as many rows as there are hypotheses."""
    from nmtgminor_b200.data.dataset import collate
    from nmtgminor_b200.inference.beam_search import BeamConfig, beam_search
    model = _successor_model(beam)
    g = torch.Generator().manual_seed(3)
    for _ in range(3):
        src = [torch.randint(4, 300, (int(n),), generator=g) for n in torch.randint(3, 40, (7,), generator=g)]
        batch = collate(src, None, padded=True, packed=True, round_to=1).cuda("cuda")
        res = [beam_search(model, batch, BeamConfig(beam_size=beam, max_len=40, min_len=30, cuda_graph=c)) for c in (False, True)]
        for a, b in zip(*res):
            assert a[0].tokens == b[0].tokens
            # the logits are bf16 of up to 32: one rounding that falls the other way moves a score by 2^-3; two of them
            assert abs(a[0].score - b[0].score) <= 0.25
    assert ops.check_status() == 0


def test_replayed_search_follows_the_model():
    """A second search of the same geometry after the model moved: a longer position table, and a new weight store with other weights.  The
    old tensors stay allocated and are overwritten, as if something else had been put there."""
    from nmtgminor_b200.data.dataset import collate
    from nmtgminor_b200.inference.beam_search import BeamConfig, beam_search
    from nmtgminor_b200.parallel.flat import FlatParameterStore
    model = _successor_model(5)
    g = torch.Generator().manual_seed(4)
    src = [torch.randint(4, 300, (int(n),), generator=g) for n in (9, 20, 5)]
    batch = collate(src, None, padded=True, packed=True, round_to=1).cuda("cuda")
    search = lambda graph: [h[0] for h in beam_search(model, batch, BeamConfig(beam_size=2, max_len=30, min_len=20, cuda_graph=graph))]

    def same():
        for a, b in zip(search(True), search(False)):
            assert a.tokens == b.tokens and abs(a.score - b.score) <= 0.25          # the tolerance of the test above
    same()
    first = [h.tokens for h in search(True)]
    old = model.decoder.embed._pos_work
    model.renew_buffer(5000)
    old.normal_(0.0, 3.0)
    same()
    old = model.store
    with torch.no_grad():
        order = torch.randperm(296, generator=g) + 4
        for p in (model.generator.weight, model.decoder.embed.weight):
            p[4:] = p[order.to(p.device)]                  # words change their names
    model.store = FlatParameterStore(model, "cuda")
    old.work.zero_()
    same()
    assert [h.tokens for h in search(True)] != first
    assert ops.check_status() == 0


def test_searches_in_several_threads():
    """Four threads with geometries of their own and one that two of them share: captures, a position table that grows under the others, and
    a pool that overflows.  Every result is the one of a search alone."""
    from concurrent.futures import ThreadPoolExecutor

    from nmtgminor_b200.data.dataset import collate
    from nmtgminor_b200.inference.beam_search import BeamConfig, beam_search
    g = torch.Generator().manual_seed(8)
    jobs = []
    for i, (n, beam, longest) in enumerate(((3, 2, 30), (5, 4, 70), (1, 3, 1100), (4, 1, 130), (2, 2, 30), (3, 2, 30))):
        src = [torch.randint(4, 300, (int(m),), generator=g) for m in torch.randint(3, 40, (n,), generator=g)]
        cfg = BeamConfig(beam_size=beam, max_len=longest, min_len=25)
        jobs.append((collate(src, None, padded=True, packed=True, round_to=1).cuda("cuda"), cfg))
    flat = lambda found: [(h.tokens, h.score) for hyps in found for h in hyps]
    alone = _successor_model(9)
    want = [flat(beam_search(alone, *job)) for job in jobs]
    shared = _successor_model(9)
    with ThreadPoolExecutor(4) as threads:
        for _ in range(3):
            got = [f.result(timeout=120) for f in [threads.submit(lambda j: flat(beam_search(shared, *j)), job) for job in jobs]]
            assert got == want
    assert len(shared.__dict__["_decode_pools"].sets) <= 4
    assert ops.check_status() == 0


def test_search_in_and_out_of_inference_mode():
    """Tables that were made under torch.inference_mode serve a search outside of it."""
    from nmtgminor_b200.data.dataset import collate
    from nmtgminor_b200.inference.beam_search import BeamConfig, beam_search
    model = _successor_model(11)
    batch = collate([torch.arange(4, 20)], None, padded=True, packed=True, round_to=1).cuda("cuda")
    search = lambda: [(h.tokens, h.score) for h in beam_search(model, batch, BeamConfig(beam_size=2, max_len=20, min_len=10))[0]]
    with torch.inference_mode():
        want = search()
    assert search() == want
    with torch.inference_mode():
        assert search() == want


@pytest.mark.parametrize("n_best", [-1, 0, 1, 9])
def test_number_of_hypotheses_asked_for(n_best):
    """None, one and more than the beam: the same lists from the replayed and the kernel-by-kernel search."""
    from nmtgminor_b200.data.dataset import collate
    from nmtgminor_b200.inference.beam_search import BeamConfig, beam_search
    model = _successor_model(12)
    batch = collate([torch.arange(4, 20), torch.arange(30, 36)], None, padded=True, packed=True, round_to=1).cuda("cuda")
    a, b = (beam_search(model, batch, BeamConfig(beam_size=2, n_best=n_best, max_len=20, min_len=10, cuda_graph=c)) for c in (True, False))
    assert [len(x) for x in a] == [len(x) for x in b] == [max(1, min(n_best, 2))] * 2
    assert [x[0].tokens for x in a] == [x[0].tokens for x in b]


def test_scores_do_not_depend_on_the_batch():
    """A sentence is scored to the same bits alone (few rows, few tiles) and beside eleven others, and so are its encoder states."""
    from nmtgminor_b200.data.dataset import collate
    model = _successor_model(13)
    g = torch.Generator().manual_seed(2)
    ids = lambda n: torch.randint(4, 300, (int(n),), generator=g)
    src = [ids(n) for n in torch.randint(20, 100, (12,), generator=g)]
    tgt = [torch.cat([torch.tensor([2]), ids(n), torch.tensor([3])]) for n in torch.randint(20, 100, (12,), generator=g)]
    pack = lambda s, t: collate(s, t, padded=True, packed=True, round_to=1).cuda("cuda")
    _, _, tokens = model.decode(pack(src, tgt))
    with torch.no_grad():
        context, seqs = model.encode(pack(src, tgt))
        for i in range(12):
            _, _, alone = model.decode(pack(src[i:i + 1], tgt[i:i + 1]))
            n = len(tgt[i]) - 1
            assert torch.equal(alone[:n, 0], tokens[:n, i])
            states, _ = model.encode(pack(src[i:i + 1], None))
            at = int(seqs.cu[i])
            assert torch.equal(states[:len(src[i])], context[at:at + len(src[i])])


def test_search_on_another_device_than_the_current_one():
    """The flags that end a search early are waited for on the model's device."""
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    from nmtgminor_b200.data.dataset import collate
    from nmtgminor_b200.inference.beam_search import BeamConfig, beam_search
    cfg = BeamConfig(beam_size=3, max_len=200, min_len=30)
    batches = [collate([torch.arange(4, 4 + n), torch.arange(30, 36)], None, padded=True, packed=True, round_to=1) for n in (9, 20, 30)]
    found = []
    for device in ("cuda:0", "cuda:1"):
        model = _successor_model(14, device)
        found.append([[h[0].tokens for h in beam_search(model, b.cuda(device), cfg)] for b in batches])
    assert found[0] == found[1]


def test_searches_keep_no_weights():
    """Between searches nothing holds the weights that the captured steps read: a replaced store is freed."""
    import gc

    from nmtgminor_b200.data.dataset import collate
    from nmtgminor_b200.inference.beam_search import BeamConfig, beam_search
    from nmtgminor_b200.parallel.flat import FlatParameterStore
    model = _successor_model(15)
    batch = collate([torch.arange(4, 20)], None, padded=True, packed=True, round_to=1).cuda("cuda")
    search = lambda: beam_search(model, batch, BeamConfig(beam_size=2, max_len=20, min_len=10))[0][0].tokens
    want = search()
    assert search() == want
    gc.collect()
    before = torch.cuda.memory_allocated()
    model.store = FlatParameterStore(model, "cuda")
    gc.collect()
    assert torch.cuda.memory_allocated() - before < model.store.work.numel()
    assert search() == want


def test_unaligned_caches_are_refused():
    """The caches are read with 16-byte loads: one that starts inside such a unit is an error on the host."""
    e, R, hid = ops.ext(), 4, 128
    flat = torch.zeros(R * 8 * hid + 8, device="cuda").bfloat16()
    good, bad = flat[:R * 8 * hid].view(R, 8, hid), flat[1:R * 8 * hid + 1].view(R, 8, hid)
    q, qkv, lens = torch.zeros(R, hid, device="cuda").bfloat16(), torch.zeros(R, 3 * hid, device="cuda").bfloat16(), torch.ones(R, dtype=torch.int32, device="cuda")
    anc, pos = torch.zeros(R, 8, dtype=torch.int32, device="cuda"), torch.zeros(R, dtype=torch.long, device="cuda")
    for k, v in ((bad, good), (good, bad)):
        for call in (lambda: e.decode_cross(q, k, v, lens, 2, 0.125), lambda: e.decode_attn(q, k, v, lens, 8, 2, 0.125),
                     lambda: e.decode_self(qkv, k, v, anc, pos, 2, 2, 0.125), lambda: e.cache_append(q, q, k, v, 0)):
            with pytest.raises(RuntimeError, match="16-byte"):
                call()


def test_position_table_first_needed_in_a_capture():
    """A captured call that meets a renewed table converts it for itself: calls outside of the graph must not get its memory, which only
    a replay fills."""
    from nmtgminor_b200.models.layers import PackedSeqs
    emb = _successor_model(16).decoder.embed
    at = torch.arange(50, device="cuda")
    seqs = PackedSeqs(torch.full((50,), 7, device="cuda"), at, torch.tensor([0, 50], dtype=torch.int32, device="cuda"), 50)
    with torch.no_grad():
        want = emb(seqs)
        emb.renew(3000)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = emb(seqs)
        assert torch.equal(emb(seqs), want)
        graph.replay()
        assert torch.equal(out, want) and torch.equal(emb(seqs), want)


def test_captures_have_a_stream_of_their_own():
    """torch hands out 32 streams of a priority in turn: none of them may be the one that searches capture on, since another thread's launches
    on it would be captured instead of run."""
    from nmtgminor_b200.inference.beam_search import _StepPools
    device = torch.device("cuda", torch.cuda.current_device())
    others = {torch.cuda.Stream(priority=p).cuda_stream for p in (0, -1) for _ in range(80)} | {torch.cuda.current_stream().cuda_stream}
    assert _StepPools.capture_stream(device).cuda_stream not in others
    assert _StepPools.capture_stream(device) is _StepPools.capture_stream(device)


@pytest.mark.parametrize("M,N,K,norm,act", [(1, 8, 8, True, "none"), (8, 24, 40, True, "relu"), (7, 3072, 256, True, "none"), (6, 4096, 1024, True, "gelu"), (16, 4096, 1024, False, "gelu"),
                                            (8, 5120, 1280, True, "silu"), (17, 5120, 1280, False, "silu"), (32, 1280, 1272, False, "silu"), (4, 2056, 512, True, "relu"), (4, 9472, 768, True, "none"), (12, 9472, 768, False, "none"),
                                            (5, 512, 512, False, "none"), (8, 1280, 1280, False, "relu"), (3, 1024, 4096, False, "none"), (8, 2368, 5120, False, "none"),
                                            (1, 256, 1544, False, "gelu"), (7, 768, 3072, False, "none"), (32, 520, 520, False, "none"), (13, 1280, 1280, False, "none")])
def test_step_linear(M, N, K, norm, act):
    """LayerNorm, product, bias, activation and residual of a decoding step in one kernel: ragged tiles of rows, features and K."""
    g = torch.Generator(device="cuda").manual_seed(M * N + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, w, bias, res, gamma, beta = rnd(M, K), rnd(N, K) * K ** -0.5, rnd(N), rnd(M, N), rnd(K), rnd(K)
    for b, r in ((bias, res), (None, None)):
        out = ops.ext().step_linear(x, gamma if norm else None, beta if norm else None, 1e-5, w, b, r, ops.ACT_IDS[act])
        h = ops.ext().layernorm_fwd(x, gamma, beta, 1e-5)[0] if norm else x          # the same bf16 values
        y = h.double() @ w.double().t() + (b.double() if b is not None else 0)
        y = {"none": lambda t: t, "relu": torch.relu, "gelu": torch.nn.functional.gelu, "silu": torch.nn.functional.silu}[act](y)
        y = y + (r.double() if r is not None else 0)
        # one rounding to bf16 of a 32-bit sum of K products (2^-24 each step, of the sum of magnitudes)
        size = h.double().abs() @ w.double().abs().t()
        assert ((out.double() - y).abs() <= 2 ** -8 * y.abs() + K ** 0.5 * 2 ** -22 * size + 1e-5).all()
    assert ops.ext().step_linear(x.float(), None, None, 0.0, w, None, None, 0) is None
    assert ops.ext().step_linear(rnd(33, K), None, None, 0.0, w, None, None, 0) is None


def test_step_linear_normalises_as_the_layernorm_kernel_does():
    g = torch.Generator(device="cuda").manual_seed(5)
    for K in (8, 256, 520, 1024, 1280):
        x, gamma, beta = (torch.randn(*s, device="cuda", generator=g).bfloat16() for s in ((7, K), (K,), (K,)))
        eye = torch.eye(K, device="cuda").bfloat16()
        assert torch.equal(ops.ext().step_linear(x * 3 + 1, gamma, beta, 1e-5, eye, None, None, 0), ops.ext().layernorm_fwd(x * 3 + 1, gamma, beta, 1e-5)[0])


def _opposite_pairs(rows, T, hid, g):
    """Keys in pairs of equal rows, anywhere in the past, whose values have opposite signs: attention over them is exactly 0."""
    at = torch.randperm(T, device="cuda", generator=g)
    k, v = (torch.randn(rows, T // 2, hid, device="cuda", generator=g).bfloat16() for _ in range(2))
    keys, values = (torch.empty(rows, T, hid, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    keys[:, at], values[:, at] = torch.cat([k, k], 1), torch.cat([v, -v], 1)
    return keys, values


@pytest.mark.parametrize("kind,B,K,heads,T,adds", [("cross", 64, 4, 16, 200, 9), ("cross", 16, 4, 20, 1500, 18), ("self", 64, 4, 16, 82, 5),
                                                   ("self", 4, 1, 8, 1002, 16)])
def test_step_attention_sums_in_32_bits(kind, B, K, heads, T, adds):
    """What is left of an exact 0 is the rounding of the sums.  `adds` 32-bit additions (blocks of 16 keys of a warp, then warps and shares)
    round to nearest, 0.58 x 2^-24 of the sum so far each (root mean square); the sums so far are a random walk to the root of the terms'
    squares.  A quarter more for what a block loses inside."""
    g = torch.Generator(device="cuda").manual_seed(T)
    e, hid, total, size = ops.ext(), heads * 64, 0.0, 0.0
    for _ in range(3):
        rows = B if kind == "cross" else B * K
        keys, values = _opposite_pairs(rows, T, hid, g)
        qkv = torch.randn(B * K, 3 * hid, device="cuda", generator=g).bfloat16()
        if kind == "cross":
            out = e.decode_cross(qkv[:, :hid].contiguous(), keys, values, torch.full((B,), T, dtype=torch.int32, device="cuda"), heads, 0.125)
            keys, values = keys.repeat_interleave(K, 0), values.repeat_interleave(K, 0)
        else:
            qkv[:, hid:2 * hid], qkv[:, 2 * hid:] = keys[:, -1], values[:, -1]
            anc = torch.arange(B * K, dtype=torch.int32, device="cuda")[:, None].expand(B * K, T + 6).contiguous()
            kc, vc = (torch.cat([t, t.new_zeros(rows, 6, hid)], 1) for t in (keys, values))
            out = e.decode_self(qkv, kc, vc, anc, torch.full((B * K,), T - 1, device="cuda"), K, heads, 0.125)
        split = lambda t: t.float().view(B * K, T, heads, 64)
        w = (torch.einsum("rhd,rjhd->rhj", qkv[:, :hid].float().view(B * K, heads, 64), split(keys)) * 0.125).softmax(-1)
        size += torch.einsum("rhj,rjhd->rhd", w.square(), split(values).square()).mean().item()
        total += out.double().square().mean().item()
    assert total ** 0.5 <= 1.25 * 0.58 * 2 ** -24 * (size * adds / 2) ** 0.5


@pytest.mark.parametrize("K", [1, 3, 9])
def test_infinite_values_of_a_step(K):
    """An infinite value under a positive weight makes its own output infinite and no other one."""
    g = torch.Generator(device="cuda").manual_seed(K)
    B, heads, T, e = 2, 2, 40, ops.ext()
    R, hid, inf = B * K, heads * 64, float("inf")
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    q, k, v = rnd(R, hid), rnd(B, T, hid), rnd(B, T, hid)
    clean = e.decode_cross(q, k, v, torch.full((B,), T, dtype=torch.int32, device="cuda"), heads, 0.125).view(R, hid)
    v[0, 5, 70], v[1, 39, 3] = inf, -inf
    out = e.decode_cross(q, k, v, torch.full((B,), T, dtype=torch.int32, device="cuda"), heads, 0.125).view(R, hid)
    want = clean.clone()
    want[:K, 70], want[K:, 3] = inf, -inf
    assert torch.equal(out, want)
    qkv, kc, vc = rnd(R, 3 * hid), rnd(R, 64, hid), rnd(R, 64, hid)
    anc = torch.arange(R, dtype=torch.int32, device="cuda")[:, None].expand(R, 64).contiguous()
    anc[:, :32] = anc[:, :32] // K * K                       # a beginning that a sentence's hypotheses share
    pos = torch.full((R,), T - 1, device="cuda")
    step = lambda: e.decode_self(qkv, kc.clone(), vc.clone(), anc, pos, K, heads, 0.125).view(R, hid)
    want = step()
    vc[0, 20, 7], vc[R - 1, 35, 100], qkv[K - 1, 2 * hid + 9] = inf, inf, -inf
    want[:K, 7], want[R - 1, 100], want[K - 1, 9] = inf, inf, -inf
    assert torch.equal(step(), want)


@pytest.mark.parametrize("B,heads,cap,pos", [(30, 16, 64, 50), (30, 16, 192, 131), (28, 16, 128, 127), (56, 16, 320, 300), (3, 2, 64, 40)])
def test_step_self_attention_of_one_hypothesis(B, heads, cap, pos):
    """Greedy searches on either side of every line between two, four and eight warps to a CTA."""
    test_step_self_attention(B, 1, heads, cap, pos)

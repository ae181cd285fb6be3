"""Launches that overlap the kernel before them: every dependence between neighbours holds, in a stream and in a captured graph."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from nmtgminor_b200 import ops


def _chain(rows, width, sync):
    """Products, norms, dropout and attention, each over what the one before wrote, in two buffers that are overwritten while the kernel
    before still reads the other.  `sync` waits behind every launch."""
    g = torch.Generator(device="cuda").manual_seed(rows + width)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, w = rnd(rows, width), [rnd(width, width) * width ** -0.5 for _ in range(3)]
    gain, shift = 1 + 0.1 * rnd(width), 0.1 * rnd(width)
    a, b, grad = torch.empty_like(x), torch.empty_like(x), torch.zeros(width, width, device="cuda")
    wait = torch.cuda.synchronize if sync else (lambda: None)
    e = ops.ext()
    outs = []

    def run():
        outs.clear()
        src = x
        for i in range(6):
            ops.gemm(src, w[i % 3], a)
            wait()
            y, mean, rstd = e.layernorm_fwd(a, gain, shift, 1e-5)
            wait()
            ops.gemm(y, w[(i + 1) % 3], b)
            wait()
            ops.gemm(b, w[(i + 2) % 3], a, residual=y)              # overwrites what the norm before read
            wait()
            dg, db = torch.zeros(width, device="cuda"), torch.zeros(width, device="cuda")
            wait()
            dx = e.layernorm_bwd(a, b, mean, rstd, gain, y, dg, db)
            wait()
            z = e.dropout_add(dx, a, 0.1, 7, i)
            wait()
            ops.gemm(z, dx, grad, a_mn_major=True, b_mn_major=True)
            wait()
            b.copy_(z)                                             # a launch of another library between them
            wait()
            src = b
            outs.append((z.clone(), grad.clone(), db.clone()))
    return run, outs


@pytest.mark.parametrize("rows,width", [(40, 64), (300, 256), (1000, 512), (2100, 1024)])
def test_overlapped_chain_equals_the_waited_one(rows, width):
    run, outs = _chain(rows, width, True)
    run()
    torch.cuda.synchronize()
    want = [tuple(t.clone() for t in o) for o in outs]
    run, outs = _chain(rows, width, False)
    for reserve in (0, 16):                    # with SMs set aside nothing overlaps
        ops.ext().set_sm_reserve(reserve)
        try:
            for _ in range(3):
                run()
                torch.cuda.synchronize()
                for got, ref in zip(outs, want):
                    assert torch.equal(got[0], ref[0]) and (reserve or torch.equal(got[1], ref[1]))
        finally:
            ops.ext().set_sm_reserve(0)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    for _ in range(5):
        graph.replay()
    torch.cuda.synchronize()
    for got, ref in zip(outs, want):
        assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])
        assert torch.allclose(got[2], ref[2], rtol=1e-4, atol=1e-3)          # column sums meet in any order
    assert ops.check_status() == 0


@pytest.mark.parametrize("length,batch", [(20, 3), (100, 40), (200, 5)])
def test_overlapped_attention_equals_the_waited_one(length, batch):
    heads, width = 4, 256
    g = torch.Generator(device="cuda").manual_seed(length)
    x = torch.randn(batch * length, width, device="cuda", generator=g).bfloat16()
    w = [(torch.randn(3 * width, width, device="cuda", generator=g) * width ** -0.5).bfloat16() for _ in range(2)]
    cu = torch.arange(0, batch * length + 1, length, dtype=torch.int32, device="cuda")
    res = []
    for sync in (True, False, False):
        wait = torch.cuda.synchronize if sync else (lambda: None)
        src = x
        for i in range(4):
            qkv = torch.empty(batch * length, 3 * width, dtype=torch.bfloat16, device="cuda")
            ops.gemm(src, w[i % 2], qkv)
            wait()
            leaf = qkv.requires_grad_()
            out = ops.self_attention(leaf, cu, heads, length, True, 0.0, True)
            wait()
            grad, = torch.autograd.grad(out, leaf, out.detach())
            wait()
            src = (grad[:, :width].contiguous() + out.detach()).contiguous()
            wait()
        res.append(src)
    torch.cuda.synchronize()
    if length <= 128:
        assert torch.equal(res[0], res[1]) and torch.equal(res[0], res[2])
    else:                       # gradients of the queries meet in any order
        assert (res[0].float() - res[1].float()).abs().max() <= 2 ** -5 * res[0].float().abs().max()


class _Waiting:
    """The extension, with a wait for the device behind every call."""

    def __init__(self, inner):
        self.inner = inner

    def __getattr__(self, name):
        f = getattr(self.inner, name)

        def call(*args, **kwargs):
            out = f(*args, **kwargs)
            torch.cuda.synchronize()
            return out
        return call


def _tables(B, K, cap, steps):
    mk = lambda shape, dt: torch.zeros(shape, dtype=dt, device="cuda")
    R, i32, f32, i64 = B * K, torch.int32, torch.float32, torch.int64
    t = [mk(3, i32), mk(cap + 1, f32), mk(B, i32), mk(R, f32), mk(R, torch.uint8), mk(B, torch.uint8), mk(R, i64), mk(R, i64), mk((R, cap), i32),
         mk(B, i32), mk((B, K), f32), mk((B, K), i32), mk((B, K), i32), mk((B, K), f32), mk((cap, R), i32), mk((cap, R), i32), mk((cap, R), f32)]
    t[0].copy_(torch.tensor([steps, 3, 1]))
    t[1].fill_(1.0)
    t[2].fill_(steps)
    t[3].fill_(float("-inf"))
    t[3].view(B, K)[:, 0] = 0.0
    t[4].fill_(2)                     # no sentence ends at once
    t[6].fill_(2)
    t[10].fill_(float("-inf"))
    return t


def _search_steps(B, K, width, source, vocab, steps):
    """The launches of a decoding layer's steps, straight from the kernels: look-up (launched plainly), norms, products, attention over the past
    and the source, best continuations, which rewrite the ancestors and positions that the next step reads before its first wait."""
    g = torch.Generator(device="cuda").manual_seed(B * 100 + K + width)
    rnd = lambda *s, by=1.0: (torch.randn(*s, device="cuda", generator=g) * by).bfloat16()
    R, heads, cap = B * K, width // 64, 64
    words, gain, shift = rnd(vocab, width), 1 + rnd(width, by=0.1), rnd(width, by=0.1)
    mat = lambda n, k: rnd(n, k, by=k ** -0.5)
    qkv_w, out_w, q_w, out2_w, fc1, fc2, last = (mat(3 * width, width), mat(width, width), mat(width, width), mat(width, width), mat(4 * width, width),
                                                 mat(width, 4 * width), mat(vocab, width) * 4)
    ck, cv = rnd(B, source, width), rnd(B, source, width)
    lens = torch.randint(1, source + 1, (B,), device="cuda", generator=g).int()
    lens[0] = source
    first = _tables(B, K, cap, steps)
    tables = [t.clone() for t in first]
    kc, vc = (torch.zeros(R, cap, width, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    outs = []

    def product(e, x, w, act=0, residual=None, norm=False):
        y = e.step_linear(x, gain if norm else None, shift if norm else None, 1e-5, w, None, residual, act)
        if y is None:
            y = ops.empty_rows(R, w.shape[0], "cuda")
            e.gemm(e.layernorm_fwd(x, gain, shift, 1e-5)[0] if norm else x, False, w, False, y, None, residual, None, None, act, 0.0, 0, 0, 1.0, False, True, 0, 0,
                   None, None, None)
        return y

    def run(e):
        outs.clear()
        for t, f in zip((*tables, kc, vc), (*first, torch.zeros_like(kc), torch.zeros_like(vc))):
            t.copy_(f)
        for _ in range(steps):
            x = words.index_select(0, tables[6])
            e.set_step_overlap(True)
            try:
                ctx = e.decode_self(product(e, x, qkv_w, norm=True), kc, vc, tables[8], tables[7], K, heads, 0.125).view(R, width)
                x = product(e, ctx, out_w, residual=x)
                ctx = e.decode_cross(product(e, x, q_w, norm=True), ck, cv, lens, heads, 0.125).view(R, width)
                x = product(e, ctx, out2_w, residual=x)
                x = product(e, product(e, x, fc1, act=1, norm=True), fc2, residual=x)
                logits = product(e, e.layernorm_fwd(x, gain, shift, 1e-5)[0], last)
                e.beam_step(logits, tables, K, 0, 3)
            finally:
                e.set_step_overlap(False)
            outs.append((logits, [t.clone() for t in tables]))
    return run, outs


@pytest.mark.parametrize("B,K,width,source,vocab", [(1, 1, 64, 1, 40), (1, 4, 128, 17, 515), (2, 4, 1024, 100, 9001), (1, 8, 320, 300, 5000), (3, 9, 256, 40, 700),
                                                   (1, 16, 1280, 1500, 4099), (20, 2, 192, 33, 600), (9, 5, 128, 700, 300)])
def test_overlapped_search_steps_equal_the_waited_ones(B, K, width, source, vocab):
    """What a step's kernels fetch before they wait (weights, gains, ancestors, positions, keys and values of the past and the source) is
    there: a captured chain of steps gives the bits of one that waits behind every launch."""
    steps = 8
    run, outs = _search_steps(B, K, width, source, vocab, steps)
    with torch.no_grad():
        run(_Waiting(ops.ext()))
        want = [(a.clone(), [t.clone() for t in b]) for a, b in outs]
        assert len({tuple(b[6].tolist()) for _, b in want}) > 1 or vocab < 50          # the words change from step to step
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run(ops.ext())
        for _ in range(4):
            graph.replay()
            torch.cuda.synchronize()
            for (got, tables), (logits, ref) in zip(outs, want):
                assert torch.equal(got, logits)
                for a, b in zip(tables, ref):
                    assert torch.equal(a, b)
    assert ops.check_status() == 0


@pytest.mark.parametrize("sentences,beam,width", [(1, 4, 256), (1, 1, 512), (5, 5, 512), (20, 4, 1024)])
def test_overlapped_search_equals_the_waited_one(sentences, beam, width, monkeypatch):
    """A replayed search and one that waits behind every launch: the same words and scores to the last bit."""
    from nmtgminor_b200.data.dataset import collate
    from nmtgminor_b200.data.synthetic import synthetic_dict
    from nmtgminor_b200.inference import beam_search as search
    from nmtgminor_b200.models.transformer import Transformer
    from nmtgminor_b200.options import default_options
    from nmtgminor_b200.parallel.flat import FlatParameterStore
    torch.manual_seed(width)
    d = synthetic_dict(700)
    model = Transformer(default_options(["-model_size", str(width), "-layers", "2", "-n_heads", str(width // 64), "-inner_size", str(4 * width), "-ffn_activation",
                                         "gelu"]), {"src": d, "tgt": d}).eval()
    FlatParameterStore(model, "cuda")
    for b in model.buffers():
        b.data = b.data.cuda()
    g = torch.Generator().manual_seed(beam)
    src = [torch.randint(4, 700, (int(n),), generator=g) for n in torch.randint(3, 90, (sentences,), generator=g)]
    batch = collate(src, None, padded=True, packed=True, round_to=1).cuda("cuda")
    find = lambda: [[(h.tokens, h.score, h.positional_scores) for h in hyps] for hyps in
                    search.beam_search(model, batch, search.BeamConfig(beam_size=beam, n_best=beam, max_len=40, min_len=5))]
    found = [find(), find()]
    inner = ops.ext()
    monkeypatch.setattr(search._DeviceSearch, "_step", search._DeviceSearch._body)
    monkeypatch.setattr(ops, "ext", lambda: _Waiting(inner))
    want = find()
    assert found == [want, want]
    assert ops.check_status() == 0

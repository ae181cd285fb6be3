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

"""tcgen05 GEMM against fp32 matmul: operand layouts, ragged shapes, epilogues, split-K."""
import pytest
import torch

from nmtgminor_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(params=[0, 1], ids=["pair", "single"], autouse=True)
def gemm_variant(request):
    """0 = automatic (CTA-pair kernel for M > 128), 1 = single-CTA kernel only."""
    ops.ext().set_gemm_variant(request.param)
    yield request.param
    ops.ext().set_gemm_variant(0)


def _rel_err(got, want):
    got, want = got.float(), want.float()
    return ((got - want).abs().max() / (want.abs().max() + 1e-6)).item()


def _status_ok():
    s = ops.check_status()
    assert s == 0, "kernel status word = %d (a bounded wait timed out)" % s


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 512), (1000, 1032, 264), (8192, 1024, 1024), (77, 3072, 1024),
                                   (300, 128, 4096), (4096, 32000, 1024)])
def test_gemm_k_major(M, N, K):
    torch.manual_seed(0)
    a = torch.randn(M, K, device=DEV).bfloat16()
    b = torch.randn(N, K, device=DEV).bfloat16()
    out = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    ops.gemm(a, b, out)
    torch.cuda.synchronize()
    _status_ok()
    want = a.float() @ b.float().t()
    assert _rel_err(out, want) < 1e-2


@pytest.mark.parametrize("a_mn,b_mn", [(False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(128, 128, 128), (512, 1024, 640), (1000, 264, 1000), (1024, 4096, 8192)])
def test_gemm_mn_major(a_mn, b_mn, M, N, K):
    torch.manual_seed(1)
    A = torch.randn(M, K, device=DEV).bfloat16()
    B = torch.randn(N, K, device=DEV).bfloat16()
    a = A.t().contiguous() if a_mn else A
    b = B.t().contiguous() if b_mn else B
    out = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    ops.gemm(a, b, out, a_mn_major=a_mn, b_mn_major=b_mn)
    torch.cuda.synchronize()
    _status_ok()
    assert _rel_err(out, A.float() @ B.float().t()) < 1e-2


@pytest.mark.parametrize("force_bn", [128, 256])
def test_gemm_tile_widths(force_bn):
    torch.manual_seed(2)
    a = torch.randn(640, 512, device=DEV).bfloat16()
    b = torch.randn(768, 512, device=DEV).bfloat16()
    out = torch.empty(640, 768, device=DEV, dtype=torch.bfloat16)
    ops.gemm(a, b, out, force_bn=force_bn)
    _status_ok()
    assert _rel_err(out, a.float() @ b.float().t()) < 1e-2


@pytest.mark.parametrize("act", [0, 1, 2, 3])
def test_gemm_bias_act_residual_preact(act):
    torch.manual_seed(3)
    M, N, K = 513, 1024, 256
    a = torch.randn(M, K, device=DEV).bfloat16()
    b = (torch.randn(N, K, device=DEV) / 16).bfloat16()
    bias = torch.randn(N, device=DEV).bfloat16()
    res = torch.randn(M, N, device=DEV).bfloat16()
    out = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    pre = torch.empty_like(out)
    ops.gemm(a, b, out, bias=bias, residual=res, preact=pre, act=act)
    _status_ok()
    z = a.float() @ b.float().t() + bias.float()
    f = [lambda t: t, torch.relu, torch.nn.functional.gelu, torch.nn.functional.silu][act]
    assert _rel_err(pre, z) < 1e-2
    assert _rel_err(out, f(z) + res.float()) < 1.5e-2


def test_gemm_dropout_epilogue_matches_dropout_kernel():
    torch.manual_seed(4)
    M, N, K = 256, 512, 128
    a = torch.randn(M, K, device=DEV).bfloat16()
    b = torch.randn(N, K, device=DEV).bfloat16()
    plain = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    dropped = torch.empty_like(plain)
    ops.gemm(a, b, plain)
    ops.gemm(a, b, dropped, dropout_p=0.25, seed=99, stream_id=3)
    same_mask = ops.ext().dropout_add(plain, None, 0.25, 99, 3)
    _status_ok()
    assert _rel_err(dropped, same_mask) < 1e-2
    frac = (dropped == 0).float().mean().item()
    assert abs(frac - 0.25) < 0.02


@pytest.mark.parametrize("act,name", [(5, "relu"), (6, "gelu"), (7, "silu")])
def test_gemm_activation_backward_epilogue(act, name):
    torch.manual_seed(5)
    M, N, K = 384, 1024, 256
    dy = torch.randn(M, K, device=DEV).bfloat16()
    w = (torch.randn(K, N, device=DEV) / 16).bfloat16()     # dgrad: dh = dy @ w  (w stored [K_red, N])
    aux = torch.randn(M, N, device=DEV).bfloat16()
    out = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    ops.gemm(dy, w, out, b_mn_major=True, aux=aux, act=act)
    _status_ok()
    dh = dy.float() @ w.float()
    x = aux.float().requires_grad_(True)
    f = {"relu": torch.relu, "gelu": torch.nn.functional.gelu, "silu": torch.nn.functional.silu}[name]
    f(x).sum().backward()
    assert _rel_err(out, dh * x.grad) < 1.5e-2


@pytest.mark.parametrize("split_k", [0, 1, 4])
def test_gemm_wgrad_fp32_accumulate_split_k(split_k):
    torch.manual_seed(6)
    tokens, n_out, k_in = 4000, 1024, 1024
    dy = torch.randn(tokens, n_out, device=DEV).bfloat16()
    x = torch.randn(tokens, k_in, device=DEV).bfloat16()
    acc = torch.ones(n_out, k_in, device=DEV)
    ops.gemm(dy, x, acc, a_mn_major=True, b_mn_major=True, accumulate=True, allow_split_k=True, split_k=split_k)
    _status_ok()
    want = dy.float().t() @ x.float() + 1.0
    assert _rel_err(acc, want) < 5e-3


@pytest.mark.parametrize("tokens,n_out,k_in", [(8192, 3072, 1024), (8000, 4096, 1024), (5000, 1280, 768), (8192, 1024, 2048)])
@pytest.mark.parametrize("stream_k", [1, 0])
def test_gemm_wgrad_equal_runs_of_k_blocks(tokens, n_out, k_in, stream_k):
    """Weight gradients whose tiles do not fill the CTA pairs evenly are split into equal runs of k-blocks that may
    end inside a tile; the partial tiles meet in the fp32 output through reductions.  Same result either way."""
    torch.manual_seed(7)
    dy = torch.randn(tokens, n_out, device=DEV).bfloat16()
    x = torch.randn(tokens, k_in, device=DEV).bfloat16()
    acc = torch.full((n_out, k_in), 0.5, device=DEV)
    ops.ext().set_gemm_variant(40 + stream_k)
    try:
        ops.gemm(dy, x, acc, a_mn_major=True, b_mn_major=True, accumulate=True, allow_split_k=True)
    finally:
        ops.ext().set_gemm_variant(41)
    _status_ok()
    want = dy.float().t() @ x.float() + 0.5
    assert _rel_err(acc, want) < 5e-3


@pytest.mark.parametrize("M,N,K", [(256, 1024, 1024), (256, 1000, 512), (64, 4096, 1024), (256, 32000, 1024)])
def test_gemm_decode_shapes_bias_and_transposed_weight(M, N, K):
    """Few-row problems take 64-column tiles (many CTAs stream the weight matrix); bias epilogue, ragged N."""
    torch.manual_seed(0)
    a = torch.randn(M, K, device=DEV).bfloat16()
    w = torch.randn(N, K, device=DEV).bfloat16()
    bias = torch.randn(N, device=DEV).bfloat16()
    out = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    ops.gemm(a, w, out, bias=bias, act=1)
    torch.cuda.synchronize()
    _status_ok()
    want = torch.relu(a.float() @ w.float().t() + bias.float())
    assert _rel_err(out, want) < 1e-2
    wt = w.t().contiguous()                      # [K, N]: the same weights stored N-contiguous
    if N % 8 == 0:
        out2 = torch.empty_like(out)
        ops.gemm(a, wt, out2, b_mn_major=True, bias=bias, act=1)
        torch.cuda.synchronize()
        _status_ok()
        assert _rel_err(out2, want) < 1e-2


def test_gemm_sign_bit_mask_round_trip():
    """Forward epilogue writes one sign bit per output; the mask-backward epilogue applies it to another product."""
    torch.manual_seed(0)
    M, N, K = 300, 1000, 256
    a = torch.randn(M, K, device=DEV).bfloat16()
    w = torch.randn(N, K, device=DEV).bfloat16()
    out = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    bits = torch.zeros(M, (N + 31) // 32, dtype=torch.int32, device=DEV)
    ops.gemm(a, w, out, act=1, mask=bits)
    torch.cuda.synchronize()
    positive = out.float() > 0
    cols = torch.arange(N, device=DEV)
    got = ((bits[:, cols // 32] >> (cols % 32)) & 1).bool()
    assert torch.equal(got, positive)
    g = torch.randn(M, 64, device=DEV).bfloat16()
    w2 = torch.randn(N, 64, device=DEV).bfloat16()
    d = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    ops.gemm(g, w2, d, act=8, mask=bits, alpha=1.25)
    torch.cuda.synchronize()
    _status_ok()
    want = (g.float() @ w2.float().t()) * 1.25 * positive
    assert _rel_err(d, want) < 1e-2


@pytest.mark.parametrize("M,N,K", [(8192, 4096, 1024), (1000, 1024, 512), (300, 264, 256), (129, 64, 128)])
def test_gemm_column_sums_in_the_epilogue(M, N, K):
    """The sign-bit backward epilogue also adds the column sums of its bf16 output to an fp32 vector (bias gradient)."""
    torch.manual_seed(9)
    dy = torch.randn(M, K, device=DEV).bfloat16()
    w = (torch.randn(K, N, device=DEV) * 0.05).bfloat16()            # [K, N]: B read MN-major, as in the fc2 data gradient
    bits = torch.randint(-2 ** 31, 2 ** 31 - 1, (M, (N + 31) // 32), device=DEV, dtype=torch.int32)
    out = ops.empty_rows(M, N, DEV)
    gb = torch.full((N,), 0.25, device=DEV)
    ops.gemm(dy, w, out, b_mn_major=True, act=8, mask=bits, alpha=1.1, colsum=gb)
    _status_ok()
    ref = torch.empty_like(out)
    ops.gemm(dy, w, ref, b_mn_major=True, act=8, mask=bits, alpha=1.1)
    assert torch.equal(out, ref)
    want = ref.float().sum(0) + 0.25
    assert (gb - want).abs().max().item() <= 2e-3 * max(1.0, want.abs().max().item())


def test_sm_reserve_only_changes_the_grid():
    """SMs set aside for communication kernels: every launcher sizes its grid for the rest; results do not change."""
    torch.manual_seed(9)
    a = torch.randn(2048, 512, device=DEV).bfloat16()
    b = torch.randn(1024, 512, device=DEV).bfloat16()
    want = torch.empty(2048, 1024, device=DEV, dtype=torch.bfloat16)
    ops.gemm(a, b, want)
    try:
        ops.ext().set_sm_reserve(8)
        got = torch.empty_like(want)
        ops.gemm(a, b, got)
        x = torch.randn(4096, 1024, device=DEV).bfloat16()
        g = torch.ones(1024, device=DEV).bfloat16()
        y = ops.ext().layernorm_fwd(x, g, torch.zeros_like(g), 1e-5)[0] if hasattr(ops.ext(), "layernorm_fwd") else None
    finally:
        ops.ext().set_sm_reserve(0)
    _status_ok()
    assert torch.equal(got, want)
    if y is not None:
        assert torch.isfinite(y.float()).all()


@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (4, 1024, 1024), (16, 132, 72), (17, 512, 2048), (33, 3072, 1000), (64, 32000, 512),
                                   (65, 1000, 4096), (200, 1024, 1024), (257, 2048, 512), (512, 256, 256)])
def test_few_row_gemm(M, N, K, overlap):
    """Few-row products: 128-feature tiles, K cut over a cluster, every tile edge; strided activations, in-place residual."""
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, w, bias = rnd(M, K + 8)[:, :K], rnd(N, K) * K ** -0.5, rnd(N)
    out = ops.empty_rows(M, N, "cuda")
    res = rnd(M, N)
    acc = x.double() @ w.double().t() + bias.double()
    ops.ext().set_step_overlap(overlap)
    try:
        for act, fn in ((0, lambda t: t), (1, torch.relu), (2, torch.nn.functional.gelu), (3, torch.nn.functional.silu)):
            ops.gemm(x, w, out, bias=bias, act=act, allow_split_k=True)
            # one rounding to bf16 (2^-9) and 32-bit sums of K products of order K^-0.5
            assert torch.allclose(out.double(), fn(acc), rtol=2 ** -8, atol=2 ** -10), (act, (out.double() - fn(acc)).abs().max())
        y = ops.empty_rows(M, N, "cuda")
        y.copy_(res)
        ops.gemm(x, w, y, residual=y, allow_split_k=True)
        assert torch.allclose(y.double(), acc - bias.double() + res.double(), rtol=2 ** -8, atol=2 ** -10)
    finally:
        ops.ext().set_step_overlap(False)
    assert ops.check_status() == 0


@pytest.mark.parametrize("M,N,K", [(129, 64, 64), (200, 72, 128), (704, 256, 1024), (1000, 1032, 264), (1920, 512, 512), (2300, 520, 200), (3840, 512, 1000)])
def test_one_wave_tiles(M, N, K):
    """Products that fit a wave of narrow tiles, next to the same ones on the CTA-pair kernel: every epilogue of a training step, with the
    column sums from registers, ragged rows and columns, and weight gradients split over K."""
    e = ops.ext()
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, w, bias, res, dy = rnd(M, K), rnd(N, K) * K ** -0.5, rnd(N), rnd(M, N), rnd(M, N) * K ** -0.5
    got = {}
    for name, forced in (("auto", 0), ("pair", 256)):
        e.set_gemm_variant(0)
        out = {}
        n = lambda: torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
        ops.gemm(x, w, out.setdefault("plain", n()), force_bn=forced)
        out["bits"] = torch.zeros(M, (N + 31) // 32, device="cuda", dtype=torch.int32)
        ops.gemm(x, w, out.setdefault("fc1", n()), bias=bias, act=1, dropout_p=0.25, seed=3, stream_id=9, mask=out["bits"], force_bn=forced)
        ops.gemm(x, w, out.setdefault("pre_out", n()), bias=bias, act=2, preact=out.setdefault("pre", n()), force_bn=forced)
        ops.gemm(x, w, out.setdefault("res", n()), bias=bias, residual=res, dropout_p=0.25, seed=3, stream_id=10, force_bn=forced)
        ops.gemm(x, w, out.setdefault("act_bwd", n()), aux=res, act=6, force_bn=forced)
        cs = out["colsum"] = torch.ones(N, device="cuda")
        ops.gemm(x, w, out.setdefault("masked", n()), act=8, mask=out["bits"], alpha=1.25, colsum=cs, force_bn=forced)
        dw = out["dw"] = torch.ones(N, K, device="cuda")
        ops.gemm(dy, x, dw, a_mn_major=True, b_mn_major=True, accumulate=True, allow_split_k=True, force_bn=forced)
        got[name] = out
    assert ops.check_status() == 0
    for k in got["auto"]:
        a, b = got["auto"][k], got["pair"][k]
        if k == "colsum":       # 32-bit sums of M values of order 1 in another order
            want = 1 + got["auto"]["masked"].double().sum(0)
            assert (a.double() - want).abs().max() < 2 ** -20 * M + 1e-4 and (b.double() - want).abs().max() < 2 ** -20 * M + 1e-4
        elif k == "dw":
            want = 1 + dy.double().t() @ x.double()
            assert (a.double() - want).abs().max() < 2 ** -20 * M
        else:                   # one accumulator per element, its products in the same order
            assert torch.equal(a, b), k


def test_gelu_epilogues_over_the_whole_range():
    """GELU and its gradient against 64 bits for inputs from the lower tail to far above: every result within one bf16 rounding, plus
    the 1.2e-7 of the tail's fit where the result cancels (the gradient's zero near -0.75)."""
    n = 512
    x = torch.linspace(-12, 12, 256 * n, device="cuda").view(256, n).bfloat16()
    eye = torch.eye(n, device="cuda").bfloat16()
    out, ones = torch.empty(256, n, device="cuda", dtype=torch.bfloat16), torch.ones(256, n, device="cuda").bfloat16()
    xd = x.double()
    cdf, pdf = 0.5 * torch.erfc(-xd / 2 ** 0.5), torch.exp(-0.5 * xd * xd) / (2 * torch.pi) ** 0.5
    ops.gemm(x, eye, out, act=2)
    assert ((out.double() - xd * cdf).abs() <= 2 ** -8 * (xd * cdf).abs() + 1e-37).all()
    ops.gemm(ones, eye, out, aux=x, act=6)
    want = cdf + xd * pdf
    assert ((out.double() - want).abs() <= 2 ** -8 * want.abs() + 3e-7 * (cdf + (xd * pdf).abs())).all()


@pytest.mark.parametrize("M,N,K", [(5000, 2048, 512), (6100, 1600, 192), (9000, 1344, 64)])
def test_second_matrix_epilogues(M, N, K):
    """Activation gradients and stored pre-activations of many-wave products, whose second matrix goes through shared memory: ragged rows,
    a last column tile with work for half of the warps only; equal to the general epilogue, which reads and writes from the lanes."""
    e = ops.ext()
    g = torch.Generator(device="cuda").manual_seed(M + N)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, w, bias, aux = rnd(M, K), rnd(N, K) * K ** -0.5, rnd(N), rnd(M, N)
    got = []
    try:
        for variant in (30, 31):
            e.set_gemm_variant(variant)
            out = []
            for act in (5, 6, 7):
                for p in (0.0, 0.25):
                    out.append(torch.zeros(M, N, device="cuda", dtype=torch.bfloat16))
                    ops.gemm(x, w, out[-1], aux=aux, act=act, dropout_p=p, seed=3, stream_id=act)
            for act in (1, 2, 3):
                out += [torch.zeros(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
                ops.gemm(x, w, out[-2], bias=bias, act=act, preact=out[-1], dropout_p=0.25, seed=3, stream_id=act)
            got.append(out)
    finally:
        e.set_gemm_variant(30)
    assert ops.check_status() == 0
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("M,N,K", [(129, 64, 128), (200, 256, 256), (1000, 1032, 264), (2300, 512, 128)])
def test_column_sums_beside_every_operand(M, N, K):
    """Column sums with rows past the last tile, next to an aux operand, the sign bits and dropout, with the single-CTA kernel asked for
    and not: the product is the one without the sums, and a pre-activation beside them stays refused."""
    e = ops.ext()
    g = torch.Generator(device="cuda").manual_seed(M + N)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, w, aux = rnd(M, K), rnd(N, K) * K ** -0.5, rnd(M, N)
    bits = torch.randint(-2 ** 31, 2 ** 31 - 1, (M, (N + 31) // 32), device="cuda", generator=g).int()
    try:
        for variant in (0, 1):
            for more in (dict(act=8, mask=bits), dict(act=6, aux=aux), dict(act=5, aux=aux, dropout_p=0.25, seed=3, stream_id=1), dict(residual=aux)):
                e.set_gemm_variant(variant)
                out, cs = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16), torch.ones(N, device="cuda")
                ops.gemm(x, w, out, colsum=cs, **more)
                e.set_gemm_variant(0)
                want = torch.zeros_like(out)
                ops.gemm(x, w, want, force_bn=256, **more)
                assert torch.equal(out, want), more
                # 32-bit sums of M values of order 1
                assert (cs.double() - 1 - out.double().sum(0)).abs().max() < 2 ** -20 * M + 1e-4
            e.set_gemm_variant(variant)
            with pytest.raises(RuntimeError):
                ops.gemm(x, w, out, colsum=cs, act=2, preact=torch.zeros_like(out))
    finally:
        e.set_gemm_variant(0)
    assert ops.check_status() == 0


def test_gelu_in_32_bits_is_as_close_as_erff():
    """The epilogues' GELU and its gradient with 32-bit output against 64 bits, next to the formula with erff in 32 bits: no range of the input is
    further off, and the lower tail keeps its relative accuracy."""
    n, rows = 256, 288
    x = (torch.arange(rows * n, device="cuda", dtype=torch.float64) - rows * n // 2) / 4096          # -9 to 9, at most 16 bits
    # as a sum of two bf16 numbers, which a product with two stacked identities adds exactly
    hi = x.bfloat16()
    lo = (x - hi.double()).bfloat16()
    assert torch.equal(x, hi.double() + lo.double())
    eye = torch.eye(n, device="cuda").bfloat16()
    out = torch.empty(rows, n, device="cuda")
    ops.gemm(torch.cat([hi.view(rows, n), lo.view(rows, n)], 1), torch.cat([eye, eye], 1), out, act=2)
    aux = torch.linspace(-9, 9, rows * n, device="cuda").bfloat16()
    grad = torch.empty(rows, n, device="cuda")
    ops.gemm(torch.ones(rows, n, device="cuda").bfloat16(), eye, grad, aux=aux.view(rows, n), act=6)
    normal = lambda t: 0.5 * torch.erfc(-t / 2 ** 0.5)
    bell = lambda t: torch.exp(-0.5 * t * t) / (2 * torch.pi) ** 0.5
    with_erff = lambda t: 0.5 * (1.0 + torch.erf(t * 2 ** -0.5))
    f, ad, af = x.float(), aux.double(), aux.float()
    for name, t, got, want, plain in (("value", x, out.view(-1), x * normal(x), f * with_erff(f)),
                                      ("gradient", ad, grad.view(-1), normal(ad) + ad * bell(ad), with_erff(af) + af * bell(af))):
        err, ref = (got.double() - want).abs(), (plain.double() - want).abs()
        for a, b in ((-9, -4), (-4, -2), (-2, -1.25), (-1.25, -0.5), (-0.5, 0.5), (0.5, 1.25), (1.25, 3), (3, 9)):
            at = (t >= a) & (t < b)
            rms, ref_rms = err[at].square().mean().sqrt(), ref[at].square().mean().sqrt()
            assert rms <= 1.05 * ref_rms, (name, a, b, float(rms), float(ref_rms))
            assert err[at].max() <= 2.0 ** -23 * max(1.0, b), (name, a, b, float(err[at].max()))     # two ulps of a result in [0.5, 1), or of x itself
        low = (t > -8.5) & (t < -2)
        assert (err[low] <= 4e-6 * want[low].abs()).all()
    assert ops.check_status() == 0


@pytest.mark.parametrize("M,N,K", [(200, 72, 128), (704, 1024, 256), (1000, 520, 264), (1920, 512, 512), (3840, 512, 1000)])
def test_one_wave_tiles_of_data_gradients(M, N, K):
    """The same narrow tiles with the weight as the [K, N] operand of a data gradient: plain, with the sign bits and their column sums, with an
    activation gradient.  One accumulator per element, its products in the order of the CTA-pair kernel."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    dy, w, aux = rnd(M, K), rnd(K, N) * K ** -0.5, rnd(M, N)
    bits = torch.randint(-2 ** 31, 2 ** 31 - 1, (M, (N + 31) // 32), device="cuda", generator=g).int()
    got = []
    for forced in (0, 256):
        out = [torch.zeros(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(4)]
        ops.gemm(dy, w, out[0], b_mn_major=True, force_bn=forced)
        ops.gemm(dy, w, out[1], b_mn_major=True, act=8, mask=bits, alpha=1.25, colsum=torch.zeros(N, device="cuda"), force_bn=forced)
        ops.gemm(dy, w, out[2], b_mn_major=True, act=6, aux=aux, force_bn=forced)
        ops.gemm(dy, w, out[3], b_mn_major=True, act=7, aux=aux, dropout_p=0.25, seed=3, stream_id=2, force_bn=forced)
        got.append(out)
    assert ops.check_status() == 0
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("M,N,K", [(4, 128, 64), (200, 256, 128), (700, 512, 256), (5000, 1024, 64)])
@pytest.mark.parametrize("off", [1, 4])
def test_epilogue_operands_off_their_boundary(M, N, K, off):
    """Residual, bias, aux operand and pre-activation that start inside a 16-byte unit: the results of aligned copies."""
    g = torch.Generator(device="cuda").manual_seed(M + off)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, w = rnd(M, K), rnd(N, K) * K ** -0.5
    res, bias, pre = rnd(M, N + 8)[:, off:off + N], rnd(N + 8)[off:off + N], torch.zeros(M * N + 8, device="cuda").bfloat16()[off:off + M * N].view(M, N)
    new = lambda: torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
    for kw in (dict(residual=res), dict(bias=bias), dict(bias=bias, act=2), dict(aux=res, act=6), dict(aux=res, act=5, dropout_p=0.25, seed=3, stream_id=1),
               dict(bias=bias, act=1, preact=pre, dropout_p=0.25, seed=3, stream_id=1)):
        for split in (False, True):
            a, b = new(), new()
            ops.gemm(x, w, a, allow_split_k=split, **kw)
            whole = {k: v.clone() if torch.is_tensor(v) else v for k, v in kw.items()}
            ops.gemm(x, w, b, **whole)
            assert torch.allclose(a.float(), b.float(), rtol=2 ** -7, atol=2 ** -9) if split else torch.equal(a, b), list(kw)
            if "preact" in kw:
                assert torch.equal(kw["preact"], whole["preact"])
    assert ops.check_status() == 0


@pytest.mark.parametrize("T,O,I", [(4439, 1256, 896), (3835, 1128, 848), (5020, 1320, 152), (4850, 536, 752), (1920, 512, 512), (704, 256, 1024), (5632, 1024, 1024)])
def test_weight_gradients_are_no_further_off_than_the_pair_kernels(T, O, I):
    """32-bit sums over thousands of rows: narrow tiles may not add up longer chains than the kernel that they stand in for."""
    ops.ext().set_gemm_variant(0)
    g = torch.Generator(device="cuda").manual_seed(T)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    dy, x = rnd(T, O), rnd(T, I)
    want = dy.double().t() @ x.double()
    err = []
    for forced in (0, 256):
        dw = torch.zeros(O, I, device="cuda")
        ops.gemm(dy, x, dw, a_mn_major=True, b_mn_major=True, accumulate=True, allow_split_k=True, force_bn=forced)
        err.append(float((dw.double() - want).square().mean().sqrt()))
    assert err[0] <= 1.1 * err[1], err          # a million values each: the two figures are known to a part in a hundred


def test_first_product_of_a_thread_inside_a_capture():
    """A thread whose first product is a captured one, on operands that no descriptor has been made for yet."""
    import threading
    g = torch.Generator(device="cuda").manual_seed(2)
    x, w = torch.randn(200, 512, device="cuda", generator=g).bfloat16(), torch.randn(256, 512, device="cuda", generator=g).bfloat16()
    want, out = torch.empty(200, 256, device="cuda").bfloat16(), torch.empty(200, 256, device="cuda").bfloat16()
    ops.gemm(x.clone(), w.clone(), want)             # the kernel is loaded
    graph, errors = torch.cuda.CUDAGraph(), []

    def capture():
        try:
            torch.cuda.synchronize()
            with torch.cuda.graph(graph, stream=torch.cuda.Stream(), capture_error_mode="thread_local"):
                ops.gemm(x, w, out)
        except Exception as exc:
            errors.append(exc)
    t = threading.Thread(target=capture)
    t.start()
    t.join(60)
    assert not errors, errors
    graph.replay()
    assert torch.equal(out, want)


@pytest.mark.parametrize("M,N,K", [(1, 64, 4096), (129, 264, 5001), (300, 512, 8000), (512, 1024, 4100), (900, 8, 20000)])
def test_long_sums_of_small_outputs(M, N, K):
    """Generator data gradients whose sum over the vocabulary is cut over the GPU: one rounding to bf16 of a 32-bit sum."""
    g = torch.Generator(device="cuda").manual_seed(K)
    dz = ops.empty_rows(M, K, torch.device("cuda"))
    dz.copy_(torch.randn(M, K, device="cuda", generator=g))
    w = torch.randn(K, N, device="cuda", generator=g).bfloat16()
    out = ops._long_sum_gemm(dz, w)
    want, size = dz.double() @ w.double(), dz.double().abs() @ w.double().abs()
    assert ((out.double() - want).abs() <= 2 ** -8 * want.abs() + K ** 0.5 * 2 ** -22 * size).all()
    assert ops.check_status() == 0


@pytest.mark.parametrize("M,N,K", [(906, 256, 8000), (400, 1024, 30011), (100, 512, 4100), (130, 64, 60000)])
def test_long_sums_repeat(M, N, K):
    """The parts of a long sum meet in one order: the same bits every time, whatever else keeps the GPU busy."""
    g = torch.Generator(device="cuda").manual_seed(K)
    dz = ops.empty_rows(M, K, torch.device("cuda"))
    dz.copy_(torch.randn(M, K, device="cuda", generator=g))
    w = torch.randn(K, N, device="cuda", generator=g).bfloat16()
    want, side = ops._long_sum_gemm(dz, w), torch.cuda.Stream()
    for i in range(12):
        with torch.cuda.stream(side):
            busy = torch.randn(1 << (14 + i % 6), device="cuda").sort()
        assert torch.equal(ops._long_sum_gemm(dz, w), want)
    torch.cuda.synchronize()
    assert ops.check_status() == 0


@pytest.mark.parametrize("M,N,K", [(129, 4744, 72), (129, 9544, 64), (257, 6400, 136), (300, 12288, 64), (512, 9984, 64), (512, 12003, 200),
                                   (100, 20000, 80), (256, 51865, 64)])
@pytest.mark.parametrize("epilogue", ["plain", "residual", "gelu"])
def test_wide_outputs_of_few_rows(M, N, K, epilogue):
    """Up to 512 rows on either side of every line between the tile widths and the CTA pairs: one rounding to bf16 of a 32-bit sum, and the
    sum itself the same whatever the tiles are."""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w, b = rnd(M, K).bfloat16(), (rnd(N, K) * K ** -0.5).bfloat16(), rnd(N).bfloat16()
    kw, want = {}, x.double() @ w.double().T
    size = x.double().abs() @ w.double().abs().T + 1
    if epilogue != "plain":
        kw["bias"], want, size = b, want + b.double(), size + b.double().abs()
    if epilogue == "residual":
        kw["residual"] = ops.empty_rows(M, N, x.device)
        kw["residual"].copy_(rnd(M, N))
        want, size = want + kw["residual"].double(), size + kw["residual"].double().abs()
    if epilogue == "gelu":
        kw["act"], want = 2, torch.nn.functional.gelu(want)
    outs = []
    try:
        for variant in (0, 1):
            ops.ext().set_gemm_variant(variant)
            outs.append(ops.empty_rows(M, N, x.device))
            ops.gemm(x, w, outs[-1], **kw)
    finally:
        ops.ext().set_gemm_variant(0)
    assert ((outs[0].double() - want).abs() <= 2 ** -8 * want.abs() + K ** 0.5 * 2 ** -22 * size).all()
    assert torch.equal(*outs)
    assert ops.check_status() == 0


@pytest.mark.parametrize("M,N,K", [(256, 38150, 520), (256, 38150, 512), (130, 28500, 1032), (130, 28500, 1024), (130, 28300, 1032), (512, 14336, 64), (512, 13824, 64),
                                   (400, 14273, 64)])
@pytest.mark.parametrize("epilogue", ["plain", "residual"])
def test_wide_outputs_beyond_one_wave_of_pairs(M, N, K, epilogue):
    """Either side of the lines between 256 columns of one CTA and CTA pairs: widths of whole tiles and others, one and a half waves and two."""
    test_wide_outputs_of_few_rows(M, N, K, epilogue)


@pytest.mark.parametrize("M,N,K", [(30, 1024, 9000), (128, 4104, 5000), (400, 1000, 30011), (2304, 1024, 4160), (1, 8, 4096)])
def test_long_sums_in_wide_tiles_and_pairs(M, N, K):
    """Parts of 256 columns from one CTA and from pairs, ragged widths, and two parts as well as many."""
    test_long_sums_of_small_outputs(M, N, K)

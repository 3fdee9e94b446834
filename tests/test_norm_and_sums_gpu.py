"""LayerNorm, column sums and the optimizer's wide accesses at the edges of their shapes, against 64 bits."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,H", [(1, 8), (7, 264), (33, 384), (2500, 512), (9, 520), (300, 1024)])
def test_layer_norm(rows, H):
    from prometorch_b200.ops.fused_ops import layer_norm
    g = torch.Generator(device="cuda").manual_seed(rows + H)
    x = (torch.randn(rows, H, device="cuda", generator=g) * 2 + 5).bfloat16().requires_grad_()
    w = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).bfloat16().requires_grad_()
    b = torch.randn(H, device="cuda", generator=g).bfloat16().requires_grad_()
    dy = torch.randn(rows, H, device="cuda", generator=g).bfloat16()
    y = layer_norm(x, w, b)
    got = torch.autograd.grad(y, (x, w, b), dy)
    r = [t.detach().double().requires_grad_() for t in (x, w, b)]
    ry = F.layer_norm(r[0], (H,), r[1], r[2])
    want = torch.autograd.grad(ry, r, dy.double())
    # one rounding to bf16 (2^-8 of a value); in fp32 the sums of a row (2^-23 of terms up to 12 in size, H of them) and of a column
    assert bool(((y.double() - ry).abs() <= 2 ** -8 * ry.abs() + 1e-4).all())
    for a, c in zip(got, want):
        assert bool(((a.double() - c).abs() <= 2 ** -8 * c.abs() + 1e-4 * (1 + c.abs().max())).all())


def test_layer_norm_module_keeps_the_native_op_for_small_inputs():
    """Below ``LARGE`` values the kernel costs the host more than it saves the GPU."""
    from prometorch_b200.nn.fused import FusedLayerNorm
    m = FusedLayerNorm(512, device="cuda", dtype=torch.bfloat16)
    rows = FusedLayerNorm.LARGE // 512
    small, large = (torch.randn(n, 512, device="cuda", dtype=torch.bfloat16, requires_grad=True) for n in (rows - 1, rows))
    assert m(small).grad_fn.name() == "NativeLayerNormBackward0" and "_LayerNorm" in m(large).grad_fn.name()
    ref = F.layer_norm(large.double(), (512,))
    assert bool(((m(large).double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-4).all())          # one rounding to bf16 over fp32 sums


def test_layer_norm_and_column_sum_differentiate_twice():
    """Under ``create_graph`` and in function transforms the values are those of torch's op, derivatives of the gradients among them."""
    from prometorch_b200.nn.fused import FusedLayerNorm
    from prometorch_b200.ops.fused_ops import column_sum
    g = torch.Generator(device="cuda").manual_seed(3)
    x, dy, u = (torch.randn(5, 64, device="cuda", generator=g).bfloat16().requires_grad_() for _ in range(3))
    m = FusedLayerNorm(64, device="cuda", dtype=torch.bfloat16)
    m.LARGE = 0
    with torch.no_grad():
        m.weight.copy_(1 + 0.1 * torch.randn(64, device="cuda", generator=g))
        m.bias.copy_(torch.randn(64, device="cuda", generator=g))
    def second(x, dy, w, b):
        dx, dw, db = torch.autograd.grad(F.layer_norm(x, (64,), w, b) if x.dtype == torch.float64 else m(x), (x, w, b), dy, create_graph=True)
        return torch.autograd.grad((dx * u.to(dx.dtype)).sum() + (dw * dw).sum() + (db * db).sum(), (x, dy, w))
    got = second(x, dy, m.weight, m.bias)
    want = second(*(t.detach().double().requires_grad_() for t in (x, dy, m.weight, m.bias)))
    for a, b in zip(got, want):              # a handful of roundings to bf16 (2^-9 each, relative to the largest terms)
        assert float((a.double() - b).norm() / b.norm()) < 2e-2
    c, = torch.autograd.grad(column_sum(dy).float().square().sum(), dy)
    assert float((c.double() - 2 * dy.detach().double().sum(0)).norm() / c.double().norm()) < 1e-2
    plain = F.layer_norm(x, (64,), m.weight, m.bias)
    assert torch.allclose(torch.func.vmap(m)(x[:, None])[:, 0].float(), plain.float(), atol=2e-2)
    _, jvp = torch.func.jvp(m, (x.detach(),), (u.detach(),))
    _, ref = torch.func.jvp(lambda t: F.layer_norm(t, (64,), m.weight, m.bias), (x.detach(),), (u.detach(),))
    assert torch.equal(jvp, ref)


@pytest.mark.parametrize("rows,N", [(1, 8), (65, 264), (8193, 1152), (300, 2056)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("pitch", [0, 8])
def test_column_sum(rows, N, dtype, pitch):
    from prometorch_b200.ops.fused_ops import column_sum
    x = torch.randn(rows, N + pitch, device="cuda", generator=torch.Generator(device="cuda").manual_seed(rows)).to(dtype)[:, :N]
    want = x.double().sum(0)
    eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -22
    assert bool(((column_sum(x).double() - want).abs() <= eps * want.abs() + 2 ** -20 * rows ** 0.5 * 4).all())


@pytest.mark.parametrize("n,off", [(1, 0), (4095, 0), (4099, 0), (65539, 0), (70000, 1)])
def test_optimizer_wide_and_narrow(n, off):
    """Sizes that end between quads and chunks, and tensors that start between 16-byte pieces: the same update either way."""
    from prometorch_b200.optim import AdamW
    g = torch.Generator(device="cuda").manual_seed(n)
    def make(first):
        buf = torch.zeros(n + 4, device="cuda")
        p = torch.nn.Parameter(buf[first:first + n], requires_grad=False)
        return p
    start, grad = torch.randn(n, device="cuda", generator=g), torch.randn(n, device="cuda", generator=g).bfloat16()
    p = make(off)
    with torch.no_grad():
        p.copy_(start)
    low = torch.zeros(n + 1, device="cuda", dtype=torch.bfloat16)[off:off + n]
    opt = AdamW([p], lr=1e-2, betas=(0.9, 0.95), weight_decay=0.1, fused=True)
    opt.set_grad_source(p, grad)
    opt.attach_lowp(p, low)
    w, m, v = start.double(), torch.zeros(n, device="cuda", dtype=torch.float64), torch.zeros(n, device="cuda", dtype=torch.float64)
    for t in (1, 2):
        opt.step()
        m, v = 0.9 * m + 0.1 * grad.double(), 0.95 * v + 0.05 * grad.double().square()
        w = w * (1 - 1e-3) - 1e-2 * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.95 ** t)).sqrt() + 1e-8)
    # fp32 arithmetic of a few operations on values up to 5: 2^-20
    assert float((p.double() - w).abs().max()) < 5 * 2 ** -20 and torch.equal(low, p.detach().bfloat16())


@pytest.mark.parametrize("rows,H", [(1, 1032), (3, 2048), (700, 2040), (1, 2056), (601, 4096), (5, 4088)])
@pytest.mark.parametrize("resid", [False, True])
def test_rms_norm_backward_wide_rows(rows, H, resid):
    """Two and four 16-byte pieces a thread, the last ones partly past the row; one row (half of a CTA idle) and more rows than CTAs take at once."""
    from prometorch_b200.ops.fused_ops import add_rms_norm, rms_norm
    g = torch.Generator(device="cuda").manual_seed(rows + H)
    x = torch.randn(rows, H, device="cuda", generator=g).bfloat16().requires_grad_()
    r = torch.randn(rows, H, device="cuda", generator=g).bfloat16().requires_grad_()
    w = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).bfloat16().requires_grad_()
    dy, dh = (torch.randn(rows, H, device="cuda", generator=g).bfloat16() for _ in range(2))
    if resid:
        y, h = add_rms_norm(x, r, w)
        got = torch.autograd.grad((y, h), (x, w), (dy, dh))
        v = h.detach().double().requires_grad_()
    else:
        got = torch.autograd.grad(rms_norm(x, w), (x, w), dy)
        v = x.detach().double().requires_grad_()
    wd = w.detach().double().requires_grad_()
    ref = v * torch.rsqrt(v.square().mean(-1, keepdim=True) + 1e-6) * wd
    want = list(torch.autograd.grad(ref, (v, wd), dy.double()))
    if resid:
        want[0] = want[0] + dh.double()
    # one rounding to bf16 over fp32 sums of up to 4096 terms (2^-23 each)
    for a, b in zip(got, want):
        assert bool(((a.double() - b).abs() <= 2 ** -8 * b.abs() + 1e-4 * (1 + b.abs().max())).all())

"""Wide-access variants of the element-wise kernels at the sizes where they can go wrong, against the tensor-op forms."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,Hk,D,n", [(1, 1, 16, 1), (3, 1, 48, 65), (16, 4, 128, 33), (40, 40, 64, 130), (5, 5, 8, 7)])
def test_paged_rope_write_rows(H, Hk, D, n):
    """Head sizes of one and more 16-byte pieces a half (48: three), and 8, which stays with the element-wise kernel: the same pages and rows."""
    from prometorch_b200.ops import paged as P
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(H * 100 + n)
    table = torch.randperm(8, device=dev, generator=g)[:4].int().view(1, 4).contiguous()
    cos, sin = P.rope_tables(256, D, 10000.0, dev)
    qkv = torch.randn(n, (H + 2 * Hk) * D, device=dev, generator=g).bfloat16()
    pos, req = torch.arange(n, dtype=torch.int32, device=dev) + 3, torch.zeros(n, dtype=torch.int32, device=dev)
    kp = torch.zeros(8, Hk, P.PAGE, D, device=dev, dtype=torch.bfloat16)
    vp = torch.zeros_like(kp)
    kr, vr, qr = kp.float().cpu(), vp.float().cpu(), qkv.float().cpu()
    want = P.paged_rope_write(qr, H, Hk, D, pos.cpu(), req.cpu(), table.cpu(), cos.cpu(), sin.cpu(), kr, vr, want_k=True)
    k = P.paged_rope_write(qkv, H, Hk, D, pos, req, table, cos, sin, kp, vp, want_k=True)
    P.check_status(dev)
    # one rounding to bf16 (2^-9 of a value) over the fp32 result; rotation mixes two values of the pair
    for a, b in ((k, want), (qkv[:, :H * D], qr[:, :H * D]), (kp, kr)):
        assert float((a.float().cpu() - b).abs().max()) <= 2 ** -8 * float(b.abs().max())
    assert torch.equal(vp.float().cpu(), vr)


@pytest.mark.parametrize("kind", ["Q4_K", "Q6_K"])
@pytest.mark.parametrize("rows,cols", [(1, 256), (15, 512), (16, 256), (17, 2560), (24, 768), (300, 1024)])
def test_dequant_tiles_of_16_rows(kind, rows, cols):
    """Rows that end inside a half of eight, one block and several: every value is the file's, rounded once."""
    from prometorch_b200 import _native as N
    from prometorch_b200.io import gguf_quant as Q
    from prometorch_b200.io.gguf_model import pack_weight
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    qt = Q.GGMLType[kind]
    raw = Q.quantize(torch.randn(rows, cols, device="cuda", generator=g) * 0.02, qt)
    pw = pack_weight(raw, qt, cols, "cuda", layout=1)
    out = torch.full((rows + 1, cols), 7.0, dtype=torch.bfloat16, device="cuda")
    N.check(N.lib().ptb_dequant_weight(pw.data.data_ptr(), pw.qtype, 1, rows, cols, out.data_ptr(), torch.cuda.current_stream().cuda_stream), "dequant")
    want = Q.dequantize(raw, qt, cols).float()
    # half a step of bf16 (2^-9 of the value), and the fp32 rounding of a difference of two products of the size of the row's largest
    assert bool(((out[:rows].float() - want).abs() <= want.abs() * 2 ** -8 + 2 ** -21 * want.abs().max()).all())
    assert bool((out[rows] == 7).all())


@pytest.mark.parametrize("V,rows", [(1, 3), (8, 1), (65, 33), (520, 7)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("up", [1.0, -2.5])
def test_cross_entropy_gradient_of_the_mean(V, rows, dtype, up):
    """Odd widths (padded rows), ignored rows, and an upstream gradient that is not one."""
    from prometorch_b200.ops.fused_ops import cross_entropy
    g = torch.Generator(device="cuda").manual_seed(V + rows)
    x = (torch.randn(rows, V, device="cuda", generator=g) * 2).to(dtype).requires_grad_()
    t = torch.randint(0, V, (rows,), device="cuda", generator=g)
    if rows > 2:
        t[1] = -100
    (cross_entropy(x, t) * up).backward()
    r = x.detach().double().requires_grad_()
    (F.cross_entropy(r, t, ignore_index=-100) * up).backward()
    # up to two roundings of the stored type, and the fast exponential's error (2^-21 of the largest logit)
    eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -19
    assert float((x.grad.double() - r.grad).abs().max()) <= 2 * eps * abs(up) / max(1, int((t >= 0).sum()))


@pytest.mark.parametrize("V", [512, 33])
@pytest.mark.parametrize("up", [1.0, 0.25])
@pytest.mark.parametrize("inplace", [False, True])
def test_cross_entropy_second_backward_is_refused(V, up, inplace):
    """The gradient is scaled in place, so a second pass over the same graph would scale it twice."""
    from prometorch_b200.ops.fused_ops import cross_entropy
    x = torch.randn(9, V, device="cuda", generator=torch.Generator(device="cuda").manual_seed(V)).bfloat16().requires_grad_()
    loss = cross_entropy(x * 1.0, torch.arange(9, device="cuda"), inplace_grad=inplace) * up
    loss.backward(retain_graph=True)
    first = x.grad.clone()
    with pytest.raises(RuntimeError, match="inplace"):
        loss.backward()
    assert torch.equal(x.grad, first)


@pytest.mark.parametrize("kinds", [("Q4_K", "Q4_K", "Q6_K"), ("Q6_K", "Q4_K"), ("Q4_K", "Q8_0", "Q6_K"), ("Q6_K",)])
@pytest.mark.parametrize("rows", [(40, 8, 24), (16, 1, 7)])
@pytest.mark.parametrize("layout", [0, 1])
def test_dequant_stacked(kinds, rows, layout):
    """Several matrices into one stack: the same rows as one by one, whatever their types, also when a type has no wide form."""
    from prometorch_b200 import _native as N
    from prometorch_b200.io import gguf_quant as Q
    from prometorch_b200.io.gguf_model import pack_weight
    import ctypes as C
    if layout == 0 and "Q8_0" in kinds:
        pytest.skip("Q8_0 is streamed in tiles only")
    cols, st = 768, torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(sum(rows))
    pws = [pack_weight(Q.quantize(torch.randn(r, cols, device="cuda", generator=g), Q.GGMLType[k]), Q.GGMLType[k], cols, "cuda", layout=layout)
           for r, k in zip(rows, kinds)]
    n, total = len(pws), sum(pw.rows for pw in pws)
    out = torch.full((total + 1, cols), 7.0, dtype=torch.bfloat16, device="cuda")
    N.check(N.lib().ptb_dequant_weights((C.c_void_p * n)(*[p.data.data_ptr() for p in pws]), (C.c_int * n)(*[p.qtype for p in pws]),
                                        (C.c_int * n)(*[p.rows for p in pws]), n, layout, cols, out.data_ptr(), st), "dequant")
    at = 0
    for p in pws:
        one = torch.empty(p.rows, cols, dtype=torch.bfloat16, device="cuda")
        N.check(N.lib().ptb_dequant_weight(p.data.data_ptr(), p.qtype, layout, p.rows, cols, one.data_ptr(), st), "dequant")
        assert torch.equal(out[at:at + p.rows], one)
        at += p.rows
    assert bool((out[total] == 7).all())


@pytest.mark.parametrize("T,H,Hk,D,pos0", [(1, 1, 1, 64, 0), (7, 3, 1, 64, 5), (33, 4, 2, 128, 0), (5, 2, 2, 128, 59)])
@pytest.mark.parametrize("neox", [True, False])
@pytest.mark.parametrize("norm,add_one", [(True, False), (True, True), (False, False)])
def test_prompt_heads(T, H, Hk, D, pos0, neox, norm, add_one):
    from prometorch_b200 import _native as N
    from prometorch_b200.ops import fused_ops as K
    from prometorch_b200.ops.paged import rope_tables
    S, per = 64, H + 2 * Hk
    g = torch.Generator(device="cuda").manual_seed(T * D)
    x = torch.randn(T, per, D, device="cuda", generator=g).bfloat16()
    w = [torch.randn(D, device="cuda", generator=g) * 0.1 + (0 if add_one else 1) if norm else None for _ in range(2)]
    cos, sin = rope_tables(S, D, 10000.0, "cuda")
    kc, vc = (torch.zeros(Hk, S, D, dtype=torch.float16, device="cuda") for _ in range(2))
    want = x.double()
    if norm:
        r = want * torch.rsqrt(want.square().mean(-1, keepdim=True) + 1e-6)
        want = torch.cat([r[:, :H] * (w[0].double() + add_one), r[:, H:H + Hk] * (w[1].double() + add_one), want[:, H + Hk:]], 1)
    qk = K.rope(want[None, :, :H + Hk].cpu(), cos.cpu().double(), sin.cpu().double(), neox, pos0)[0].cuda()
    got = x.clone()
    N.check(N.lib().ptb_prompt_heads(got.data_ptr(), T, H, Hk, D, N.ptr(w[0]), N.ptr(w[1]), int(add_one), 1e-6, cos.data_ptr(), sin.data_ptr(), int(neox), pos0,
                                     kc.data_ptr(), vc.data_ptr(), S, torch.cuda.current_stream().cuda_stream), "prompt_heads")
    # one rounding: half a step of bf16 (eight significant bits: 2^-8 of a value at most) or fp16 (eleven: 2^-11), and fp32 arithmetic on values
    # of the size of the head's largest
    slack = 2 ** -20 * float(qk.abs().max())
    assert bool(((got[:, :H + Hk].double() - qk).abs() <= 2 ** -8 * qk.abs() + slack).all())
    assert torch.equal(got[:, H + Hk:], x[:, H + Hk:])
    assert bool(((kc[:, pos0:pos0 + T].permute(1, 0, 2).double() - qk[:, H:]).abs() <= 2 ** -11 * qk[:, H:].abs() + 2 ** -24 + slack).all())
    assert torch.equal(vc[:, pos0:pos0 + T].permute(1, 0, 2).float(), x[:, H + Hk:].half().float())
    assert not bool(kc[:, :pos0].any()) and not bool(kc[:, pos0 + T:].any())

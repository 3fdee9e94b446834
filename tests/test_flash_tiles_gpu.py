"""FlashAttention at the edges of its tiles, against plain softmax attention in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


# pairs of heads (even groups) and pairs of row blocks (odd groups); one row, the last block empty, full and ragged; keys that start before
# the queries, and queries that see none; a second tile past the end
SHAPES = [(1, 1, 1, 2, 1, 64, True, 0), (1, 127, 127, 2, 2, 128, True, 0), (2, 129, 129, 4, 2, 128, True, 0), (1, 257, 257, 3, 3, 64, True, 0),
          (2, 256, 384, 6, 2, 64, False, 0), (1, 130, 70, 8, 1, 128, False, 0), (1, 40, 300, 2, 1, 128, True, 260), (1, 200, 64, 3, 1, 128, True, -100),
          (1, 640, 640, 5, 5, 128, True, 0)]


def _one_tile(B, Tq, H, Hk):
    from prometorch_b200 import _native as N
    return bool(N.lib().ptb_flash_attn_one_tile(B, Tq, H, Hk, torch.cuda.get_device_properties(0).multi_processor_count))


@pytest.mark.parametrize("B,Tq,Tk,H,Hk,D,causal,off", SHAPES)
@pytest.mark.parametrize("scale", [None, 3.0])
@pytest.mark.parametrize("full", [False, True])
def test_forward_tiles(B, Tq, Tk, H, Hk, D, causal, off, scale, full):
    """``scale`` 3: maxima that keep growing from block to block, so that outputs are scaled on the way.  ``full``: as many entries as give every
    SM a tile and more, which takes the kernel with two tiles a CTA; fewer take the one with one, as do rows whose second tile would be empty."""
    from prometorch_b200.ops.attention import attention_reference, flash_attention
    if full:
        B = -(-160 // (-(-Tq // 128) * H))
    assert _one_tile(B, Tq, H, Hk) == (not full or (Tq <= 128 and (H // Hk) % 2 == 1))
    g = torch.Generator(device="cuda").manual_seed(Tq + Tk)
    q, k, v = (torch.randn(B, t, h, D, device="cuda", generator=g).bfloat16() for t, h in ((Tq, H), (Tk, Hk), (Tk, Hk)))
    if scale:
        k = k * torch.linspace(0.1, 1, Tk, device="cuda").bfloat16()[None, :, None, None]
    o, lse = flash_attention(q, k, v, causal=causal, q_offset=off, scale=scale, return_lse=True)
    ro, rl = attention_reference(q.double(), k.double(), v.double(), causal, off, scale)
    seen = torch.isfinite(rl)
    # weights and outputs are rounded to bf16 once each (2^-9, uniform: 2^-9 / sqrt(3) rms, and fewer than 128 terms dominate a row)
    assert _rel(o, torch.nan_to_num(ro)) < 4e-3
    # fp32 sums of 128-term products: 2^-22 of the largest score
    assert float((lse.double() - rl)[seen].abs().max()) < 1e-4 * max(1.0, float(rl[seen].abs().max()))
    assert bool((lse[~seen] == float("-inf")).all())


@pytest.mark.parametrize("lens,H,Hk,D", [([1], 1, 1, 64), ([5, 128, 1, 300, 129], 8, 2, 128), ([256, 31, 257], 3, 3, 64), ([127, 64], 4, 4, 128)])
@pytest.mark.parametrize("packed", [True, False])
def test_packed_sequences(lens, H, Hk, D, packed):
    """One launch over sequences side by side, from a packed projection's columns or from tensors of their own; what is not finite in one stays in it."""
    from prometorch_b200.ops.attention import attention_reference, flash_attention_varlen
    g = torch.Generator(device="cuda").manual_seed(sum(lens))
    offs = [0]
    for n in lens:
        offs.append(offs[-1] + n)
    x = torch.randn(offs[-1], H + 2 * Hk, D, device="cuda", generator=g).bfloat16()
    if len(lens) > 2:
        x[offs[1]:offs[2]] = float("inf")
    q, k, v = x[:, :H], x[:, H:H + Hk], x[:, H + Hk:]
    if not packed:
        q, k, v = q.contiguous(), k.contiguous(), v.contiguous()
    o = flash_attention_varlen(q, k, v, offs, torch.tensor(offs, dtype=torch.int32, device="cuda"))
    for i, (a, b) in enumerate(zip(offs, offs[1:])):
        if len(lens) > 2 and i == 1:
            continue
        want = attention_reference(q[None, a:b].double(), k[None, a:b].double(), v[None, a:b].double(), True)[0][0]
        assert _rel(o[a:b], want) < 4e-3, i


@pytest.mark.parametrize("B,Tq,Tk,H,Hk,D,causal,off", SHAPES)
def test_backward_tiles(B, Tq, Tk, H, Hk, D, causal, off):
    from prometorch_b200.ops.attention import attention_reference, flash_attention
    g = torch.Generator(device="cuda").manual_seed(Tq * Tk)
    q, k, v = (torch.randn(B, t, h, D, device="cuda", generator=g).bfloat16().requires_grad_() for t, h in ((Tq, H), (Tk, Hk), (Tk, Hk)))
    do = torch.randn(B, Tq, H, D, device="cuda", generator=g).bfloat16()
    r = [t.detach().double().requires_grad_() for t in (q, k, v)]
    skip = max(0, -off) if causal else 0          # rows that see no key: no gradient
    ro = attention_reference(r[0][:, skip:], r[1], r[2], causal, off + skip)[0]
    got = torch.autograd.grad(flash_attention(q, k, v, causal=causal, q_offset=off), (q, k, v), do)
    want = torch.autograd.grad(ro, r, do[:, skip:].double())
    for a, b in zip(got, want):
        # P, dS and the results rounded to bf16 once each, delta from an output rounded to bf16; a single key has no gradient but rounding
        assert float((a.double() - b).norm()) < 6e-3 * float(b.norm()) + 2 ** -9 * float(do.norm())


@pytest.mark.parametrize("Tq,Tk,causal", [(129, 129, True), (130, 70, False), (1, 257, False)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("entries", [2, 40])
def test_entries_of_a_batch_stay_apart(Tq, Tk, causal, D, entries):
    """Ragged last blocks lie over the next entry's rows: what is not finite there reaches neither outputs nor gradients of the entry before."""
    from prometorch_b200.ops.attention import flash_attention
    g = torch.Generator(device="cuda").manual_seed(Tq + Tk)
    one = [torch.randn(1, t, h, D, device="cuda", generator=g).bfloat16() for t, h in ((Tq, 4), (Tk, 2), (Tk, 2), (Tq, 4))]

    def run(x):
        q, k, v = (t.clone().requires_grad_() for t in x[:3])
        o = flash_attention(q, k, v, causal=causal)
        return [o.detach(), *torch.autograd.grad(o, (q, k, v), x[3])]
    want = run(one)
    for bad in (float("inf"), float("nan")):
        got = run([torch.cat([t, torch.full_like(t, bad)] * (entries // 2)) for t in one])
        for a, b in zip(got, want):             # the order in which key blocks are added to dQ is free
            assert bool(torch.isfinite(a[::2]).all()) and _rel(a[::2], b.double().expand_as(a[::2])) < 1e-3


@pytest.mark.parametrize("peak", [1.0, 3.0])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("H", [2, 24])
def test_forward_error_is_that_of_exact_maxima(peak, D, H):
    """Weights are rounded to bf16 under the running maximum of each block: no further from 64 bits than the same roundings in 64-bit arithmetic."""
    from prometorch_b200.ops.attention import flash_attention
    T, two = 1025, 1.4426950408889634
    assert _one_tile(1, T, H, H) == (H == 2)
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v = ((torch.randn(T, H, D, device="cuda", generator=g) * s).bfloat16() for s in (peak, 1, 1))
    o = flash_attention(q[None], k[None], v[None], causal=True)[0]
    s = torch.einsum("qhd,khd->hqk", q.double(), k.double()) * D ** -0.5 * two
    s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    vd = v.double().transpose(0, 1)
    want = torch.softmax(s / two, -1) @ vd
    m, total, acc = s[..., :1], 0.0, 0.0
    for j in range(0, T, 128):
        grown = torch.maximum(m, s[..., j:j + 128].amax(-1, keepdim=True))
        p = torch.exp2(s[..., j:j + 128] - grown)
        alpha, m = torch.exp2(m - grown), grown
        total, acc = total * alpha + p.sum(-1, keepdim=True), acc * alpha + p.bfloat16().double() @ vd[:, j:j + 128]
    # what is left is the arithmetic in 32 bits, a hundredth of a bf16 rounding
    assert _rel(o.transpose(0, 1), want) <= 1.01 * _rel((acc / total).bfloat16(), want)

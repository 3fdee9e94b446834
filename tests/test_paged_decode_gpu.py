"""Attention over pages with the tokens dealt to warps and the splits merged in a cluster, against the fp32 form."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G", [1, 2, 4, 8])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("nsplit", [1, 2, 7, 8, 16, 17])
def test_decode_splits(G, D, nsplit):
    """Lengths of one token, around a group (8 or 16 tokens) and a page, more splits than groups; rows of q that start between 16-byte pieces; what
    lies in a page behind the last token is not read into the result."""
    from prometorch_b200.ops import paged as P
    dev, Hk = "cuda", 2
    H, lens = Hk * G, [1, 7, 17, 64, 65, 300]
    g = torch.Generator(device=dev).manual_seed(G * D + nsplit)
    kp = torch.randn(40, Hk, P.PAGE, D, device=dev, generator=g).bfloat16()
    vp = torch.randn(40, Hk, P.PAGE, D, device=dev, generator=g).bfloat16()
    table = torch.zeros(len(lens), 6, dtype=torch.int32)
    perm, at = torch.randperm(40).int(), 0
    for b, n in enumerate(lens):
        k = -(-n // P.PAGE)
        table[b, :k] = perm[at:at + k]
        at += k
        if n % P.PAGE:
            kp[table[b, k - 1], :, n % P.PAGE:] = float("nan")
            vp[table[b, k - 1], :, n % P.PAGE:] = float("inf")
    rows = torch.randn(len(lens), H * D + 3, device=dev, generator=g).bfloat16()
    lens_d, table_d = torch.tensor(lens, dtype=torch.int32, device=dev), table.to(dev)
    for q in (rows[:, :H * D].contiguous(), rows[:, 1:1 + H * D]):
        want = P.paged_attention_reference(q.float().cpu(), H, Hk, D, torch.tensor(lens), table, kp.float().cpu(), vp.float().cpu())
        got = P.paged_attention_decode(q, H, Hk, D, lens_d, table_d, kp, vp, nsplit=nsplit)
        P.check_status(dev)
        # fp32 throughout, one rounding of the result to bf16 (2^-8 of a value) and the exponentials' 2^-21 of up to 300 weights that sum to one
        assert bool(((got.float().cpu() - want).abs() <= 2 ** -8 * want.abs() + 1e-4).all())


@pytest.mark.parametrize("D", [64, 128])
def test_decode_values_between_16_byte_pieces(D):
    """A pool of values that starts four bytes into its storage gives the same result as an aligned one."""
    from prometorch_b200.ops import paged as P
    g = torch.Generator(device="cuda").manual_seed(D)
    kp, vp = (torch.randn(3, 2, P.PAGE, D, device="cuda", generator=g).bfloat16() for _ in range(2))
    off = torch.empty(vp.numel() + 2, dtype=torch.bfloat16, device="cuda")[2:].view_as(vp).copy_(vp)
    q, table = torch.randn(1, 4 * D, device="cuda", generator=g).bfloat16(), torch.tensor([[2, 0, 1]], dtype=torch.int32, device="cuda")
    lens = torch.tensor([150], dtype=torch.int32, device="cuda")
    assert off.data_ptr() % 16 == 4
    assert torch.equal(P.paged_attention_decode(q, 4, 2, D, lens, table, kp, off, nsplit=2), P.paged_attention_decode(q, 4, 2, D, lens, table, kp, vp, nsplit=2))

"""The GEMM on pairs of SMs, whole tiles and tiles cut along K, against the product in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one row, column and k-block past a tile; fewer columns than a tile; several waves; a last wave that is cut (long K), all of it and some of it
@pytest.mark.parametrize("M,N,K,cut", [(6408, 2056, 72, False), (19200, 520, 200, False), (20000, 136, 520, False), (264, 392, 16392, True), (1160, 1032, 8200, True),
                                       (2568, 2056, 8192, True), (200, 8192, 8192, True)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_pair_gemm(M, N, K, cut, a_mn, b_mn):
    from prometorch_b200 import _native as NL
    from prometorch_b200.ops import gemm as G
    assert NL.lib().ptb_gemm_on_pairs(M, N, K, 148, 1) and (NL.lib().ptb_gemm_work_floats(M, N, K, 148) > 0) == cut
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn(*((K, M) if a_mn else (M, K)), device="cuda", generator=g).bfloat16()
    b = torch.randn(*((K, N) if b_mn else (N, K)), device="cuda", generator=g).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g)
    want = (a.double().T if a_mn else a.double()) @ (b.double() if b_mn else b.double().T)
    size = K ** 0.5                                                                # an element's standard deviation
    out = G.gemm_bf16(a, b, a_mn=a_mn, b_mn=b_mn)
    assert bool(((out.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-4 * size).all())            # one rounding to bf16 over fp32 sums
    acc = torch.ones(M, N, device="cuda")
    G.gemm_bf16(a, b, a_mn=a_mn, b_mn=b_mn, out=acc, bias=bias, accumulate=True)
    assert float((acc.double() - (want + bias + 1)).abs().max()) <= 1e-4 * size                       # fp32 sums of K exact products, in pieces
    act = G.gemm_bf16(a, b, a_mn=a_mn, b_mn=b_mn, bias=bias, relu2=True)
    ref = (want + bias).clamp_min(0).square()
    assert bool(((act.double() - ref).abs() <= 2 ** -8 * ref + 1e-3 * size * ref.sqrt() + 1e-6 * K).all())
    G.check_status()


@pytest.mark.parametrize("M,N,K,n_sm,work", [(2568, 2056, 1032, 148, False), (2568, 2056, 8192, 148, False), (520, 776, 2056, 6, False), (1160, 1032, 2056, 20, False),
                                             (1160, 1032, 2056, 20, True), (1160, 1032, 2056, 7, True), (1160, 1032, 2056, 2, False)])
def test_pair_gemm_on_fewer_sms_and_without_workspace(M, N, K, n_sm, work):
    """The caller's count of SMs bounds the pairs; without a workspace (or with one too small) tiles stay whole."""
    from prometorch_b200 import _native as NL
    from prometorch_b200.ops import gemm as G
    L, st = NL.lib(), torch.cuda.current_stream().cuda_stream
    floats = L.ptb_gemm_work_floats(M, N, K, n_sm) if work else 0
    assert L.ptb_gemm_on_pairs(M, N, K, n_sm, int(work)) and (floats > 0) == work
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, b = (torch.randn(r, K, device="cuda", generator=g).bfloat16() for r in (M, N))
    want = a.double() @ b.double().T
    status = G._status(a.device).data_ptr()

    def product(room):
        out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
        wk = torch.empty(max(1, room), device="cuda")
        NL.check(L.ptb_gemm_bf16_ws(a.data_ptr(), K, 0, b.data_ptr(), K, 0, out.data_ptr(), N, M, N, K, None, 0, wk.data_ptr() if room else None, room, status, n_sm, st))
        return out
    plain = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    NL.check(L.ptb_gemm_bf16(a.data_ptr(), K, 0, b.data_ptr(), K, 0, plain.data_ptr(), N, M, N, K, None, 0, status, n_sm, st))
    for out in (plain, product(floats), product(max(0, floats - 1))):
        assert bool(((out.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-4 * K ** 0.5).all())        # one rounding to bf16 over fp32 sums
    G.check_status()

"""LayerNorm, column sums and the optimizer's wide accesses at the edges of their shapes, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


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

"""The natively launched layers of a prompt against the same layers launched one by one (the path of models with biases or norms behind the sublayers)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,hidden,inter", [(8, 2, 512, 1024), (4, 4, 256, 768)])
@pytest.mark.parametrize("T", [1, 9, 64, 65, 128, 129, 300])
def test_native_and_python_launches_agree(tmp_path, monkeypatch, heads, kv_heads, hidden, inter, T):
    """Prompts of one token, around the tile widths of the decode-sized products and past them; with and without the logits of every position."""
    from prometorch_b200.io.config import tiny_qwen3_config
    from prometorch_b200.io.gguf_model import GGUFModel
    from prometorch_b200.io.synthetic import write_synthetic_gguf
    from prometorch_b200.ops import gemm as G
    path = str(tmp_path / "m.gguf")
    write_synthetic_gguf(path, tiny_qwen3_config(layers=2, hidden=hidden, heads=heads, kv_heads=kv_heads, inter=inter, vocab=512), seed=T)
    ids = [(7 * i + 3) % 512 for i in range(T + 1)]

    def outputs():
        m = GGUFModel(path, device="cuda:0", max_seq=320, want_logits=True)
        every = m.prefill(ids[:T], return_logits=True).clone()
        m.prefill(ids[:T])
        m.forward_decode(ids[T], T)
        m.check_status()
        nxt = m.logits_view().clone()
        m.close()
        return every, nxt
    got = outputs()
    monkeypatch.setattr(G, "_SPLITK", False)             # also: the ordinary products in place of the decode-sized ones
    want = outputs()
    for a, b in zip(got, want):
        # two layers in bf16: the products' order of summation and the gate's rounding differ
        assert float((a - b).norm() / b.norm()) < 2e-2

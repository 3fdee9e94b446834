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


def _with_biases(monkeypatch):
    """Files written from here on have biases on q, k and v."""
    from prometorch_b200.io import synthetic
    from prometorch_b200.io.gguf_quant import GGMLType

    class Writer(synthetic.GGUFWriter):
        def add_tensor(self, name, shape, qtype, data):
            super().add_tensor(name, shape, qtype, data)
            if name.endswith(("attn_q.weight", "attn_k.weight", "attn_v.weight")):
                g = torch.Generator().manual_seed(len(name) + shape[0])
                super().add_tensor(name[:-len("weight")] + "bias", shape[:1], GGMLType.F32, torch.randn(shape[0], generator=g).view(torch.uint8))
    monkeypatch.setattr(synthetic, "GGUFWriter", Writer)


@pytest.mark.parametrize("kind,T", [("wide", 300), ("wide", 70), ("biases", 9), ("biases", 200), ("post-norms", 9), ("post-norms", 200)])
def test_prompt_logits_match_dense_layers(tmp_path, monkeypatch, kind, T):
    """Every position's logits against dense fp32 layers over the file's dequantised weights, in one pass and continued on top of the cache.  ``wide``: the native
    launches, with a product whose tiles are cut along K; biases and norms behind the sublayers: the launches from Python."""
    from prometorch_b200 import _native as N
    from prometorch_b200.io.config import tiny_gemma3_config, tiny_qwen3_config
    from prometorch_b200.io.gguf_model import GGUFModel
    from prometorch_b200.io.synthetic import write_synthetic_gguf
    from prometorch_b200.models.gguf_oracle import OracleModel
    path = str(tmp_path / "m.gguf")
    if kind == "biases":
        _with_biases(monkeypatch)
    cfg = tiny_gemma3_config(layers=2, window=0) if kind == "post-norms" else \
        tiny_qwen3_config(layers=2, hidden=1024 if kind == "wide" else 512, heads=8, kv_heads=2, inter=8192 if kind == "wide" else 1024, vocab=512)
    write_synthetic_gguf(path, cfg, seed=T, device="cuda", std=0.05)
    m = GGUFModel(path, device="cuda:0", max_seq=320, want_logits=True)
    assert (m.layers[0]["q"].bias is not None) == (kind == "biases") and (m.layers[0]["post_attn_norm"] is not None) == (kind == "post-norms")
    if kind == "wide" and T > 128:
        assert N.lib().ptb_gemm_work_floats(T, cfg.hidden_size, cfg.intermediate_size, 148) > 0
    ids = [(7 * i + 3) % 512 for i in range(T)]
    want = OracleModel(path, device="cuda", max_seq=320).forward(ids)
    first = T // 2
    whole = m.prefill(ids, return_logits=True).clone()
    m.prefill(ids[:first])
    rest = m.prefill(ids[first:], pos0=first, return_logits=True)
    for got, ref in ((whole, want), (rest, want[first:])):
        # the same fp32 layers with weights, activations and attention weights rounded to bf16 where the prompt pass rounds them, evaluated on the CPU for
        # these shapes and lengths, are 0.0134 to 0.0167 from the oracle
        assert float((got - ref).norm() / ref.norm()) < 2e-2
    m.check_status()
    m.close()

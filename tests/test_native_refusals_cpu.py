"""Operands that a kernel of the native library could not read are refused on the host, before any launch."""
import ctypes as C

import pytest

BASE = 1 << 20          # an aligned address; nothing is read from it


def _lib():
    from prometorch_b200 import _native as N
    import prometorch_b200.ops.attention  # noqa: F401  (its prototypes)
    return N.lib()


def _refused(rc):
    return rc == -1 and _lib().ptb_last_error().decode()


@pytest.mark.parametrize("off_o,off_do,off_dq", [(4, 0, 0), (0, 2, 0), (0, 8, 0), (0, 0, 4)])
@pytest.mark.parametrize("D", [64, 128])
def test_flash_attention_delta_needs_aligned_rows(off_o, off_do, off_dq, D):
    L = _lib()
    vp = C.c_void_p
    L.ptb_flash_attn_delta.argtypes = [vp, vp, vp, C.c_int, C.c_int, C.c_int, C.c_int, vp, vp]
    assert "16-byte aligned" in _refused(L.ptb_flash_attn_delta(BASE + off_o, BASE + off_do, BASE, 1, 8, 2, D, BASE + off_dq, None))
    if not off_dq:      # the backward that takes no buffer to clear
        assert "16-byte aligned" in _refused(L.ptb_flash_attn_bwd(BASE, BASE, BASE, BASE + off_o, BASE + off_do, BASE, BASE, BASE, BASE, BASE, 0, 1, 8, 8, 2, 2, D, 1,
                                                                  1.0, 0, None))


@pytest.mark.parametrize("which", range(7))
def test_prompt_heads_needs_aligned_operands(which):
    """Pairs of values are read together: the projection, both norms, the tables and the caches."""
    L = _lib()
    a = [BASE + (4 if i == which else 0) for i in range(7)]
    assert "8-byte aligned" in _refused(L.ptb_prompt_heads(a[0], 3, 2, 1, 64, a[1], a[2], 0, 1e-6, a[3], a[4], 1, 0, a[5], a[6], 8, None))


@pytest.mark.parametrize("off_k,off_v", [(8, 0), (0, 2)])
def test_paged_attention_needs_aligned_pools(off_k, off_v):
    """Keys are read in 16-byte pieces, values that start between them in 4-byte ones."""
    import prometorch_b200.ops.paged  # noqa: F401
    L = _lib()
    assert "aligned pool" in _refused(L.ptb_paged_attn_decode(BASE, 128, BASE, 1, 2, 1, 64, BASE, BASE, 4, 4, BASE + off_k, BASE + off_v, 1.0, None, 1, BASE, None))


def test_flash_attention_output_has_to_be_aligned():
    L = _lib()
    assert "16-byte aligned" in _refused(L.ptb_flash_attn_varlen_fwd(BASE, 256, BASE, 256, BASE, 256, BASE + 8, BASE, 1, 4, 4, 2, 2, 64, 1, 1.0, BASE, None))

"""What the attention backward launcher refuses, it refuses on the host before anything else happens: the same answer comes
back on a machine without a GPU, where every later step fails with another error."""
import pytest

ARGS = ["qkv", "out", "dout", "lse", "dqkv", "dq_acc", "delta"]


@pytest.mark.parametrize("name,offset", [("dout", 8), ("dout", 2), ("out", 4), ("out", 2), ("qkv", 8), ("dqkv", 8),
                                         ("dq_acc", 4), ("dq_acc", 8), ("delta", 4), ("delta", 8)])
def test_attention_backward_refuses_addresses_its_kernels_cannot_read(name, offset):
    from meshslice_b200 import _native
    p = {n: 1 << 20 for n in ARGS}
    p[name] += offset
    with pytest.raises(RuntimeError, match="invalid argument"):
        _native.load().attention_bwd(*(p[n] for n in ARGS), 1, 128, 1, 1, 0.1, 1 << 20, 0)


def test_attention_takes_any_qkv_that_can_be_viewed_per_head():
    """Column slices and a trailing dimension of one, as the plain form takes them."""
    import torch

    from meshslice_b200.ops import functional as F
    batch, seq, heads, D = 2, 8, 3, 16
    g = torch.Generator().manual_seed(0)
    wide = torch.randn(batch * seq, heads * 3 * D + 40, generator=g)
    qkv = wide[:, 24:24 + heads * 3 * D]
    dout = torch.randn(batch * seq, heads * D, generator=g)
    want, lse = F.attention_fwd(qkv.contiguous(), batch, seq, heads, True)
    dwant = F.attention_bwd(dout, qkv.contiguous(), want, lse, batch, seq, heads, True)
    for form in (qkv, qkv.contiguous()[:, :, None]):
        out, l2 = F.attention_fwd(form, batch, seq, heads, True)
        assert torch.allclose(out, want) and torch.allclose(l2, lse)
        assert torch.allclose(F.attention_bwd(dout, form, out, l2, batch, seq, heads, True), dwant)

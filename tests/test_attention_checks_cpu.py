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

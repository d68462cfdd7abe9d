"""What the one-CTA form of two products refuses, it refuses on the host before its first launch: the same answer comes back on a
machine without a GPU, where a launch fails with another error."""
import pytest

BASE = 1 << 20


def _call(pre, out):
    from meshslice_b200 import _native
    first = (256, 128, 64, BASE, 256, 1, BASE, 128, 1, BASE, 128, 1, 1)
    second = (64, 256, 128, BASE, 128, 0, BASE, 128, 0, out, 256, 0, 0)
    _native.load().gemm_pair(*first, *second, 148, BASE, 0, pre)


@pytest.mark.parametrize("pre,out", [(BASE + 6, BASE), (BASE + 8, BASE), (BASE, BASE + 2), (BASE, BASE + 8)])
def test_one_cta_pair_refuses_addresses_the_derivative_cannot_read(pre, out, monkeypatch):
    monkeypatch.setenv("MSB_TWO_CTA", "0")
    with pytest.raises(RuntimeError, match="16-byte aligned"):
        _call(pre, out)

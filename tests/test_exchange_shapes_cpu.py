"""Launch shapes of the kernels that take part in a row exchange (every CTA counts one arrival on every peer)."""
import pytest


@pytest.mark.parametrize("rows", [1, 147, 1184, 1185, 4096, 32768, 1 << 20])
def test_arrivals_of_an_exchange_stay_few(rows):
    from meshslice_b200 import _native
    C = _native.load()
    assert 1 <= C.ce_grid(rows) <= min(rows, 148 * 8)
    for cols in (8, 256, 512, 1024, 1544, 2048, 4096, 8192, 16384):
        assert 1 <= C.ln_grid(0, rows, cols) <= min(rows, 148 * 16)
        assert 1 <= C.ln_grid(1, rows, cols) <= min(rows, 148 * 4)

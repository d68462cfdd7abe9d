"""The exponential that the attention's backward kernel evaluates on the FMA pipe, restated in fp32 from the constants in its source."""
import re
from pathlib import Path

import numpy as np

SOURCE = Path(__file__).resolve().parent.parent / "meshslice_b200" / "csrc" / "ops" / "attention.cu"


def _exp2_fma(x):
    body = re.search(r"float exp2_fma\(float x\) \{(.*?)\n\}", SOURCE.read_text(), re.S).group(1)
    first = np.float32(re.search(r"float p = ([0-9.e+-]+)f;", body).group(1))
    coefs = [np.float32(c) for c in re.findall(r"p = fmaf\(p, f, ([0-9.e+-]+)f\);", body)]
    assert len(coefs) == 5
    x = np.asarray(x, np.float32)
    t = np.where(np.isnan(x), x, np.maximum(x, np.float32(-125)))
    r = t + np.float32(12582912)
    f = t - (r - np.float32(12582912))
    p = np.full_like(f, first)
    for c in coefs:                        # one rounding per step: the product of two fp32 is exact in fp64
        p = (p.astype(np.float64) * f + np.float64(c)).astype(np.float32)
    scale = ((r.view(np.int32) << 23) + 0x3F800000).astype(np.int32).view(np.float32)
    return p * scale


def test_exp2_polynomial_is_as_accurate_as_the_instruction_beside_it():
    """Relative error against 64 bits at most 2^-22, that of ex2.approx, over the range that the kernel's probabilities come from
    (their exponents are at most about 0) and up to 126; below -125 it stays at 2^-125, and NaN stays NaN."""
    g = np.random.default_rng(0)
    x = np.concatenate([g.uniform(-125, 0, 1 << 20), g.uniform(-2, 2, 1 << 20), g.uniform(0, 126, 1 << 18),
                        np.arange(-125, 127), np.arange(-124.5, 126)]).astype(np.float32)
    want = np.exp2(x.astype(np.float64))
    assert np.max(np.abs(_exp2_fma(x) / want - 1)) <= 2.0 ** -22
    low = _exp2_fma(np.array([-125.0, -125.5, -126, -1000, -1e30, -np.inf], np.float32))
    assert np.all(np.abs(low / 2.0 ** -125 - 1) <= 2.0 ** -22)
    assert np.isnan(_exp2_fma(np.array([np.nan], np.float32))[0])

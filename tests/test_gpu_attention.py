"""tcgen05 flash attention forward / backward against the plain PyTorch fp32 formulation."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(qkv, batch, seq, heads, causal, dout):
    D = 128
    x = qkv.float().clone().requires_grad_(True)
    t = x.view(batch, seq, heads, 3, D)
    q, k, v = (t[:, :, :, i].permute(0, 2, 1, 3) for i in range(3))
    s = q @ k.transpose(-1, -2) / math.sqrt(D)
    if causal:
        s = s.masked_fill(torch.ones(seq, seq, dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    lse = torch.logsumexp(s, -1)
    o = (torch.softmax(s, -1) @ v).permute(0, 2, 1, 3).reshape(batch * seq, heads * D)
    o.backward(dout.float())
    return o.detach(), lse.detach(), x.grad


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("shape", [(1, 128, 1), (2, 256, 2), (2, 512, 3), (1, 2048, 2)])
def test_attention_fwd_bwd(shape, causal):
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    batch, seq, heads = shape
    g = torch.Generator(device="cuda").manual_seed(seq + heads)
    qkv = torch.randn(batch * seq, heads * 3 * 128, device="cuda", generator=g).bfloat16()
    dout = torch.randn(batch * seq, heads * 128, device="cuda", generator=g).bfloat16()
    out, lse = F.attention_fwd(qkv, batch, seq, heads, causal)
    _native.check_status()
    o_ref, lse_ref, dqkv_ref = _ref(qkv, batch, seq, heads, causal, dout)
    assert (out.float() - o_ref).abs().max().item() < 0.03
    assert (lse - lse_ref).abs().max().item() < 0.02
    dqkv = F.attention_bwd(dout, qkv, out, lse, batch, seq, heads, causal)
    _native.check_status()
    err = (dqkv.float() - dqkv_ref).abs().max().item()
    rel = ((dqkv.float() - dqkv_ref).norm() / dqkv_ref.norm()).item()
    assert err < 0.15 and rel < 2e-2, (err, rel)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("shape", [(5, 384, 61), (2, 1280, 40), (37, 128, 4), (149, 128, 1)])
def test_attention_items(shape, causal):
    """More items than SMs (running CTAs take the rest over), an odd number of tiles (an item of one tile), and the
    two sides of the rule that gives a forward CTA one or two tiles.  P and the result are rounded to bf16 (2^-9 each,
    of values that are averages of |v| <= 5.5): 0.022, and 1e-3 for the fp32 sums and exponentials.  Gradients: three
    such roundings (P or dS, an operand, the result) of random sign, 2^-9 / sqrt(3) each, and four times that."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    batch, seq, heads = shape
    g = torch.Generator(device="cuda").manual_seed(batch)
    qkv = torch.randn(batch * seq, heads * 3 * 128, device="cuda", generator=g).bfloat16()
    dout = torch.randn(batch * seq, heads * 128, device="cuda", generator=g).bfloat16()
    out, lse = F.attention_fwd(qkv, batch, seq, heads, causal)
    dqkv = F.attention_bwd(dout, qkv, out, lse, batch, seq, heads, causal)
    _native.check_status()
    ref, lse_ref, dref = _ref(qkv, batch, seq, heads, causal, dout)
    assert (out.float() - ref).abs().max().item() < 0.023
    assert (lse - lse_ref).abs().max().item() < 0.02
    assert ((dqkv.float() - dref).norm() / dref.norm()).item() < 4 * 2 ** -9


def test_attention_backward_takes_out_on_an_8_byte_boundary():
    """`out` is only read with plain loads: a tensor that starts 8 bytes off gives the same gradient."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    batch, seq, heads = 2, 256, 3
    g = torch.Generator(device="cuda").manual_seed(11)
    qkv = torch.randn(batch * seq, heads * 3 * 128, device="cuda", generator=g).bfloat16()
    dout = torch.randn(batch * seq, heads * 128, device="cuda", generator=g).bfloat16()
    out, lse = F.attention_fwd(qkv, batch, seq, heads, True)
    moved = torch.empty(out.numel() + 4, dtype=out.dtype, device="cuda")[4:].view_as(out).copy_(out)
    assert moved.data_ptr() % 16 == 8
    a = F.attention_bwd(dout, qkv, out, lse, batch, seq, heads, True)
    b = F.attention_bwd(dout, qkv, moved, lse, batch, seq, heads, True)
    _native.check_status()
    assert torch.equal(a, b)


def test_attention_backward_refuses_dout_off_a_16_byte_boundary():
    """The refusal comes from the host; the same call on an aligned copy works afterwards."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    batch, seq, heads = 1, 128, 2
    qkv = torch.randn(batch * seq, heads * 3 * 128, device="cuda").bfloat16()
    out, lse = F.attention_fwd(qkv, batch, seq, heads, True)
    dout = torch.randn(out.numel() + 4, device="cuda").bfloat16()[4:].view_as(out)
    assert dout.data_ptr() % 16 == 8
    with pytest.raises(RuntimeError, match="invalid argument"):
        F.attention_bwd(dout, qkv, out, lse, batch, seq, heads, True)
    dqkv = F.attention_bwd(dout.clone(), qkv, out, lse, batch, seq, heads, True)
    torch.cuda.synchronize()
    _native.check_status()
    _, _, dref = _ref(qkv, batch, seq, heads, True, dout)
    assert ((dqkv.float() - dref).norm() / dref.norm()).item() < 4 * 2 ** -9


@pytest.mark.parametrize("causal", [False, True])
def test_attention_on_strided_tensors(causal):
    """qkv, out and dout as column slices of wider tensors and a transposed lse: the same bits as on contiguous copies."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    batch, seq, heads = 2, 256, 3
    g = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda cols: torch.randn(batch * seq, cols, device="cuda", generator=g).bfloat16()
    cut = lambda t, n: t[:, 24:24 + n]
    qkv, dout = cut(rand(heads * 384 + 64), heads * 384), cut(rand(heads * 128 + 64), heads * 128)
    assert not qkv.is_contiguous()
    out, lse = F.attention_fwd(qkv, batch, seq, heads, causal)
    want, want_lse = F.attention_fwd(qkv.contiguous(), batch, seq, heads, causal)
    assert torch.equal(out, want) and torch.equal(lse, want_lse)
    strided_out = cut(torch.zeros(batch * seq, heads * 128 + 64, device="cuda").bfloat16(), heads * 128).copy_(out)
    strided_lse = lse.transpose(1, 2).contiguous().transpose(1, 2)
    assert not strided_out.is_contiguous() and not strided_lse.is_contiguous()
    got = F.attention_bwd(dout, qkv, strided_out, strided_lse, batch, seq, heads, causal)
    assert torch.equal(got, F.attention_bwd(dout.contiguous(), qkv.contiguous(), want, want_lse, batch, seq, heads, causal))
    _native.check_status()


def test_attention_large_scores_exercise_rescaling():
    """Scores that grow along the keys force the running maximum (and O) to be rescaled."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    batch, seq, heads = 1, 512, 1
    qkv = torch.randn(batch * seq, 3 * 128, device="cuda").bfloat16()
    ramp = torch.linspace(0.2, 3.0, seq, device="cuda")[:, None]
    qkv[:, 128:256] = (qkv[:, :128].float().mean(0, keepdim=True) * ramp * 4).bfloat16()
    dout = torch.randn(batch * seq, 128, device="cuda").bfloat16()
    out, lse = F.attention_fwd(qkv, batch, seq, heads, False)
    _native.check_status()
    o_ref, lse_ref, _ = _ref(qkv, batch, seq, heads, False, dout)
    assert (out.float() - o_ref).abs().max().item() < 0.05
    assert (lse - lse_ref).abs().max().item() < 0.05


def test_attention_backward_is_bit_identical_from_run_to_run():
    """dQ, dK and dV are accumulated in tensor memory by the CTA that owns them, never added to
    global memory from several CTAs: the same inputs give the same bits."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    batch, seq, heads = 2, 1024, 4
    g = torch.Generator(device="cuda").manual_seed(5)
    qkv = torch.randn(batch * seq, heads * 3 * 128, device="cuda", generator=g).bfloat16()
    dout = torch.randn(batch * seq, heads * 128, device="cuda", generator=g).bfloat16()
    out, lse = F.attention_fwd(qkv, batch, seq, heads, True)
    a = F.attention_bwd(dout, qkv, out, lse, batch, seq, heads, True).clone()
    b = F.attention_bwd(dout, qkv, out, lse, batch, seq, heads, True)
    _native.check_status()
    assert torch.equal(a, b)


@pytest.mark.parametrize("causal", [False, True])
def test_attention_backward_of_vanishing_probabilities_and_nan(causal):
    """Scores up to 400 apart: most probabilities are below 2^-126 (the polynomial's exponent is clamped there), one per row
    is not.  The oracle's are zero there, the kernel's at most 2^-125, which changes nothing in bf16.  A NaN in one head's
    dout and one in the other's qkv show where the oracle has them, whatever pipe computes the exponential."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    batch, seq, heads = 1, 384, 3
    g = torch.Generator(device="cuda").manual_seed(9)
    qkv = torch.randn(batch * seq, heads * 3 * 128, device="cuda", generator=g).bfloat16()
    for h in range(heads):
        qkv[:, h * 384:h * 384 + 256] *= 4.0
    dout = torch.randn(batch * seq, heads * 128, device="cuda", generator=g).bfloat16()
    out, lse = F.attention_fwd(qkv, batch, seq, heads, causal)
    dqkv = F.attention_bwd(dout, qkv, out, lse, batch, seq, heads, causal)
    _native.check_status()
    _, _, dref = _ref(qkv, batch, seq, heads, causal, dout)
    assert ((dqkv.float() - dref).norm() / dref.norm()).item() < 8 * 2 ** -9   # probabilities near 0 or 1: P - delta cancels
    dout[200, 5] = float("nan")                 # head 0
    qkv[130, 384 + 128 + 7] = float("nan")      # a key of head 1
    out, lse = F.attention_fwd(qkv, batch, seq, heads, causal)
    dqkv = F.attention_bwd(dout, qkv, out, lse, batch, seq, heads, causal)
    _native.check_status()
    _, _, dref = _ref(qkv, batch, seq, heads, causal, dout)
    rows = slice(200, 256) if causal else slice(0, seq)   # queries whose row holds a NaN
    assert torch.isnan(dqkv[200, :128]).all() and torch.isnan(dref[200, :128]).all()
    assert torch.isnan(dqkv[rows, 384:512]).all() and torch.isnan(dref[rows, 384:512]).all()
    clean = slice(768, 1152)
    assert torch.isfinite(dqkv[:, clean]).all()
    assert ((dqkv[:, clean].float() - dref[:, clean]).norm() / dref[:, clean].norm()).item() < 8 * 2 ** -9


@pytest.mark.parametrize("shape", [(1, 128, 1), (3, 640, 5), (2, 1024, 24)])
def test_attention_backward_launches_in_order(shape):
    """The three launches of a call overlap; what comes before and after them in the stream does not.  Calls follow one
    another on the same buffers, inputs are overwritten right behind a call and the result is copied right behind it: the
    same bits as a call by itself.  Items: fewer than SMs in both kernels together, about as many, more."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    batch, seq, heads = shape
    g = torch.Generator(device="cuda").manual_seed(3)
    sets = []
    for _ in range(3):
        qkv = torch.randn(batch * seq, heads * 3 * 128, device="cuda", generator=g).bfloat16()
        dout = torch.randn(batch * seq, heads * 128, device="cuda", generator=g).bfloat16()
        out, lse = F.attention_fwd(qkv, batch, seq, heads, True)
        torch.cuda.synchronize()
        want = F.attention_bwd(dout, qkv, out, lse, batch, seq, heads, True)
        torch.cuda.synchronize()
        sets.append((qkv, dout, out, lse, want.clone()))
    work = [torch.empty_like(t) for t in sets[0][:4]]
    got = []
    for i in range(24):
        for w, t in zip(work, sets[i % 3]):
            w.copy_(t)
        got.append(F.attention_bwd(work[1], work[0], work[2], work[3], batch, seq, heads, True).clone())
        for w in work:
            w.fill_(float("nan"))
    _native.check_status()
    for i, t in enumerate(got):
        assert torch.equal(t, sets[i % 3][4]), i


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("shape", [(1, 128, 1), (2, 1152, 8), (7, 2688, 1), (37, 512, 1), (148, 128, 1)])
def test_attention_backward_of_both_kinds_in_one_launch(shape, causal):
    """Up to as many items as SMs, dK / dV and dQ are one launch, whose CTAs change from one kind to the other (items of one to
    21 blocks, ring stages left at every phase); the same sequences twice are two launches.  Bits do not depend on it."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    batch, seq, heads = shape
    g = torch.Generator(device="cuda").manual_seed(seq)
    qkv = torch.randn(batch * seq, heads * 3 * 128, device="cuda", generator=g).bfloat16()
    dout = torch.randn(batch * seq, heads * 128, device="cuda", generator=g).bfloat16()
    copies = 149 // (batch * heads * (seq // 128)) + 1
    out, lse = F.attention_fwd(qkv, batch, seq, heads, causal)
    dqkv = F.attention_bwd(dout, qkv, out, lse, batch, seq, heads, causal)
    many = lambda t: torch.cat([t] * copies)
    want = F.attention_bwd(many(dout), many(qkv), many(out), many(lse), copies * batch, seq, heads, causal)
    _native.check_status()
    assert torch.isfinite(dqkv).all() and torch.equal(want, many(dqkv))

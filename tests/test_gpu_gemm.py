"""tcgen05 GEMM kernel against a plain PyTorch fp32 reference of the same product."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b, layout):
    a32, b32 = a.float(), b.float()
    if layout == "nn":
        return a32 @ b32
    if layout == "nt":
        return a32 @ b32.t()
    return a32.t() @ b32


def _operands(M, N, K, layout, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    sa = (M, K) if layout != "tn" else (K, M)
    sb = (K, N) if layout != "nt" else (N, K)
    a = torch.randn(sa, device="cuda", generator=g).bfloat16()
    b = torch.randn(sb, device="cuda", generator=g).bfloat16()
    return a, b


def _check(out, ref, K):
    err = (out.float() - ref).abs().max().item()
    tol = 0.02 * (K ** 0.5) + 1e-2
    assert err < tol, f"max abs err {err} > {tol}"
    rel = (out.float() - ref).norm() / ref.norm()
    assert rel < 1e-2, f"relative error {rel}"


@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("shape", [(128, 256, 64), (256, 512, 256), (384, 768, 1024), (200, 264, 72),
                                   (1024, 1024, 4096)])
def test_gemm_matches_fp32_reference(layout, shape):
    from meshslice_b200 import _native
    from meshslice_b200.ops.gemm import gemm
    M, N, K = shape
    a, b = _operands(M, N, K, layout)
    out = gemm(a, b, layout)
    _native.check_status()
    _check(out, _ref(a, b, layout), K)


def test_gemm_fp32_out_and_accumulate():
    from meshslice_b200 import _native
    from meshslice_b200.ops.gemm import gemm
    a, b = _operands(256, 512, 320, "nt")
    out = torch.ones(256, 512, device="cuda", dtype=torch.float32)
    gemm(a, b, "nt", out=out, accumulate=True)
    _native.check_status()
    _check(out, _ref(a, b, "nt") + 1.0, 320)
    outb = torch.ones(256, 512, device="cuda", dtype=torch.bfloat16)
    gemm(a, b, "nt", out=outb, accumulate=True)
    _native.check_status()
    _check(outb, _ref(a, b, "nt") + 1.0, 320)


def test_gemm_bias_gelu_epilogue():
    from meshslice_b200 import _native
    from meshslice_b200.ops.gemm import gemm
    a, b = _operands(256, 512, 256, "nn")
    a = a * 0.1
    bias = torch.randn(512, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5)).bfloat16()
    pre = torch.empty(256, 512, device="cuda", dtype=torch.bfloat16)
    out = gemm(a, b, "nn", bias=bias, act="gelu", pre_act=pre)
    _native.check_status()
    h = _ref(a, b, "nn") + bias.float()
    _check(pre, h, 256)
    ref = torch.nn.functional.gelu(h, approximate="tanh")   # the kernel applies GeLU to the fp32 sum
    assert ((out.float() - ref).abs() <= 0.03 + 0.01 * ref.abs()).all()


# Tile orders: panels of sixteen blocks along M (more than one, the last one short) and along N, panels of eight with an odd
# number of k-blocks whose last one is short.
@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("shape", [(4360, 2056, 136), (2056, 8456, 136), (8456, 1288, 4168), (4360, 4616, 4104)])
def test_gemm_tile_orders(layout, shape):
    from meshslice_b200 import _native
    from meshslice_b200.ops.gemm import gemm
    M, N, K = shape
    a, b = _operands(M, N, K, layout, seed=11)
    out = gemm(a, b, layout)
    acc = torch.ones(M, N, device="cuda", dtype=torch.float32)
    gemm(a, b, layout, out=acc, accumulate=True)
    _native.check_status()
    ref = _ref(a, b, layout)
    _check(out, ref, K)
    _check(acc, ref + 1.0, K)


def test_gemm_many_tiles_persistent_schedule():
    """More tiles than SMs, so every CTA walks several tiles and both TMEM accumulators."""
    from meshslice_b200 import _native
    from meshslice_b200.ops.gemm import gemm
    a, b = _operands(4096, 4096, 512, "nt", seed=3)
    out = gemm(a, b, "nt")
    _native.check_status()
    _check(out, _ref(a, b, "nt"), 512)


@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("shape", [(8, 8, 8), (264, 136, 72), (1400, 1032, 200), (2344, 2056, 136), (2304, 4672, 64)])
def test_gemm_output_boxes(layout, shape):
    """Every way an output leaves the kernel, on both sides of the rule for the tile width, with boxes of 32 rows x 64 or 32 columns cut at both edges and guard rows and columns around C:
    bf16, fp32, fp32 added to, bf16 added to, and GeLU with its pre-activation.  Products of bf16 values are summed in
    fp32 (K^0.5 * 2^-22 of the operands' scale at most), bf16 results are rounded once (2^-9)."""
    from meshslice_b200 import _native
    from meshslice_b200.ops.gemm import gemm
    M, N, K = shape
    a, b = _operands(M, N, K, layout, seed=M + N)
    sa, sb = (a.double().t() if layout == "tn" else a.double()), (b.double().t() if layout == "nt" else b.double())
    ref = sa @ sb

    def guarded(dtype, fill):
        full = torch.full((M + 2, N + 16), fill, device="cuda", dtype=dtype)
        return full, full[1:-1, 8:-8]

    def intact(full, fill):
        return bool((full[0] == fill).all() and (full[-1] == fill).all() and (full[:, :8] == fill).all()
                    and (full[:, -8:] == fill).all())

    scale = ref.abs().max().item() + 3.0
    for dtype, acc, tol in ((torch.bfloat16, False, 2 ** -8), (torch.float32, False, 1e-5), (torch.float32, True, 1e-5),
                            (torch.bfloat16, True, 2 ** -8)):
        full, out = guarded(dtype, 3.0)
        gemm(a, b, layout, out=out, accumulate=acc)
        _native.check_status()
        assert intact(full, 3.0), (dtype, acc)
        assert (out.double() - ref - (3.0 if acc else 0.0)).abs().max().item() <= tol * scale, (dtype, acc)
    full, out = guarded(torch.bfloat16, 3.0)
    fullp, pre = guarded(torch.bfloat16, 3.0)
    gemm(a, b, layout, out=out, act="gelu", pre_act=pre)
    _native.check_status()
    assert intact(full, 3.0) and intact(fullp, 3.0)
    assert (pre.double() - ref).abs().max().item() <= 2 ** -8 * scale
    g = torch.nn.functional.gelu(ref, approximate="tanh")
    assert ((out.double() - g).abs() <= 2 ** -8 * g.abs() + 2e-3 * ref.abs() + 1e-3).all()


@pytest.mark.parametrize("shape", [(20000, 24, 72), (20000, 8, 64), (15300, 536, 136), (10200, 288, 64)])
def test_gemm_gelu_fp32_output_with_half_a_box_left(shape):
    """fp32 result and bf16 pre-activation with 1 to 32 columns in the last group of 64 (the second fp32 box is left out
    there), several tiles per CTA: what one tile leaves in its staging must not meet the next one's.  Bounds as above."""
    from meshslice_b200 import _native
    from meshslice_b200.ops.gemm import gemm
    M, N, K = shape
    a, b = _operands(M, N, K, "nt", seed=N)
    ref = a.double() @ b.double().t()
    scale = ref.abs().max().item()
    g = torch.nn.functional.gelu(ref, approximate="tanh")
    for _ in range(3):
        pre = torch.full((M, N), 3.0, device="cuda", dtype=torch.bfloat16)
        out = gemm(a, b, "nt", out_dtype=torch.float32, act="gelu", pre_act=pre)
        _native.check_status()
        assert (pre.double() - ref).abs().max().item() <= 2 ** -8 * scale
        assert ((out.double() - g).abs() <= 2e-3 * ref.abs() + 1e-3).all()


@pytest.mark.parametrize("two_cta", [True, False])
@pytest.mark.parametrize("offset", [1, 2, 4, 6])
def test_gemm_output_may_start_at_any_element(offset, two_cta):
    """C and C_pre off a 16-byte boundary (TMA cannot address them): every kind of output, whole and cut groups of 32
    columns, guard values before and behind.  Bounds as in test_gemm_output_boxes."""
    from meshslice_b200 import _native
    from meshslice_b200.ops.gemm import gemm
    M, N, K = 264, 328, 72
    a, b = _operands(M, N, K, "nt", seed=offset)
    ref = a.double() @ b.double().t()
    scale = ref.abs().max().item() + 3.0

    def placed(dtype):
        flat = torch.full((M * N + 32,), 3.0, device="cuda", dtype=dtype)
        return flat, flat[8 + offset:8 + offset + M * N].view(M, N)

    def intact(flat):
        return bool((flat[:8 + offset] == 3.0).all() and (flat[8 + offset + M * N:] == 3.0).all())

    for dtype, acc, tol in ((torch.bfloat16, False, 2 ** -8), (torch.float32, False, 1e-5), (torch.float32, True, 1e-5),
                            (torch.bfloat16, True, 2 ** -8)):
        flat, out = placed(dtype)
        gemm(a, b, "nt", out=out, accumulate=acc, two_cta=two_cta)
        _native.check_status()
        assert intact(flat), (dtype, acc)
        assert (out.double() - ref - (3.0 if acc else 0.0)).abs().max().item() <= tol * scale, (dtype, acc)
    g = torch.nn.functional.gelu(ref, approximate="tanh")
    for where in ("both", "pre"):
        flat, out = placed(torch.bfloat16)
        if where == "pre":
            out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
        flatp, pre = placed(torch.bfloat16)
        gemm(a, b, "nt", out=out, act="gelu", pre_act=pre, two_cta=two_cta)
        _native.check_status()
        assert intact(flat) and intact(flatp)
        assert (pre.double() - ref).abs().max().item() <= 2 ** -8 * scale
        assert ((out.double() - g).abs() <= 2 ** -8 * g.abs() + 2e-3 * ref.abs() + 1e-3).all()


def test_gemm_fp32_accumulation_keeps_subnormals():
    """The adds that the copy engine does are those of fp32 without flushing: exact for subnormal operands and results."""
    from meshslice_b200 import _native
    from meshslice_b200.ops.gemm import gemm
    M, N, K = 256, 256, 64
    before = torch.tensor([0.0, 1e-40, -1e-40, 2.0 ** -149, 2.0 ** -126, -(2.0 ** -126), 1.0, 2.0 ** -130])
    before = before.repeat(M, N // 8)
    for ea, eb in ((-70, -70), (-75, -70), (-66, -66), (-64, -60)):      # products 2^-134, 2^-139, 2^-126, 2^-118
        a = torch.full((M, K), 2.0 ** ea, device="cuda").bfloat16()
        b = torch.full((N, K), 2.0 ** eb, device="cuda").bfloat16()
        b[::2] *= -1
        alone = gemm(a, b, "nt", out_dtype=torch.float32).cpu()
        out = before.cuda()
        gemm(a, b, "nt", out=out, accumulate=True)
        _native.check_status()
        assert alone[0, 1].item() == 64 * 2.0 ** (ea + eb)
        assert torch.equal(out.cpu(), (before.double() + alone.double()).float())


# Shapes (tokens, d_in, d_out) of the two gradients in one launch: fewer tiles than CTA pairs in both (narrow tiles), ragged
# edges and rows whose pitch is no multiple of 128 bytes, one problem longer than a wave, one with a single short k-block,
# a panel order of its own in each.
@pytest.mark.parametrize("dataflow", ["os", "ls", "rs"])
@pytest.mark.parametrize("shape", [(512, 512, 1536), (1992, 1032, 4104), (264, 5128, 72), (8, 264, 520), (4360, 2048, 3080)])
def test_gemm_pair_is_both_products(shape, dataflow):
    """Against the fp32 reference of each product, and bit for bit from run to run."""
    from meshslice_b200 import _native
    from meshslice_b200.ops.gemm import gemm_pair
    t, i, o = shape
    g = torch.Generator(device="cuda").manual_seed(t)
    rand = lambda *s: torch.randn(s, device="cuda", generator=g).bfloat16()
    x, dy, w = rand(t, i), rand(t, o), rand(o, i) if dataflow == "ls" else rand(i, o)
    if dataflow == "rs":
        x = rand(i, t)              # transposed input: y = x^T w, dw = x dy, dx = w dy^T
    first = {"os": (x, dy, "tn"), "ls": (dy, x, "tn"), "rs": (x, dy, "nn")}[dataflow]
    second = {"os": (dy, w, "nt"), "ls": (dy, w, "nn"), "rs": (w, dy, "nt")}[dataflow]
    got = []
    for _ in range(2):
        grad = torch.ones(w.shape, device="cuda", dtype=torch.float32)
        dw, dx = gemm_pair(*first, grad, True, *second)
        assert dw is grad
        got.append((dw, dx))
    _native.check_status()
    _check(got[0][0], _ref(*first) + 1.0, first[0].shape[0] if first[2] == "tn" else first[0].shape[1])
    _check(got[0][1], _ref(*second), second[0].shape[1])
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("K", [1032, 4104, 8192])
def test_gemm_rows_do_not_depend_on_the_tiles_around_them(K, layout):
    """A result's bits follow from its row of A and its column of B: more tiles than CTA pairs, the same rows in a product of one
    block of them, and the same product as either of two in a launch."""
    from meshslice_b200 import _native
    from meshslice_b200.ops.gemm import gemm, gemm_pair
    M, N = 5128, 4616
    a, b = _operands(M, N, K, layout, seed=K)
    whole = gemm(a, b, layout)
    for i in (0, 256, 2048, 5120):
        part = gemm(a[:, i:i + 256].contiguous() if layout == "tn" else a[i:i + 256], b, layout)
        assert torch.equal(part, whole[i:i + 256]), i
    x, y = _operands(1288, 1032, 4168, "nn")
    want = gemm(x, y, "nn")
    for first, second in (((a, b, layout), (x, y, "nn")), ((x, y, "nn"), (a, b, layout))):
        outs = gemm_pair(*first, torch.empty(first[0].shape[0 if first[2] != "tn" else 1], (first[1].shape[1] if first[2] != "nt" else first[1].shape[0]),
                                             device="cuda", dtype=torch.bfloat16), False, *second)
        _native.check_status()
        assert all(torch.equal(got, whole if f[0] is a else want) for got, f in zip(outs, (first, second)))


def test_gemm_pair_refuses_what_gemm_refuses():
    from meshslice_b200.ops.gemm import gemm_pair
    a, b = _operands(128, 256, 64, "nn")
    out = torch.zeros(128, 256, device="cuda")
    with pytest.raises(ValueError):
        gemm_pair(a, b, "nn", None, True, a, b, "nn")
    with pytest.raises(ValueError):
        gemm_pair(a, b, "nn", out, True, a, b, "nt")
    with pytest.raises(ValueError):
        gemm_pair(a, b.float(), "nn", out, True, a, b, "nn")
    with pytest.raises(RuntimeError):
        gemm_pair(a[:, :60], b[:60, 4:252], "nn", None, False, a, b, "nn")   # 8 bytes off the alignment


# (tokens, width, ffn): narrow and wide tiles, edges inside a group of 32 columns and of 32 rows, more tiles than CTA pairs
@pytest.mark.parametrize("dataflow", ["os", "ls"])
@pytest.mark.parametrize("shape", [(256, 128, 512), (1000, 264, 1048), (2056, 512, 8200)])
@pytest.mark.parametrize("offset", [0, 3])
def test_gemm_pair_times_gelu_derivative(shape, dataflow, offset):
    """dx * GeLU'(pre) in the epilogue against fp32: one bf16 rounding of the result (2^-9 of it) and the sum's fp32 error.
    `offset`: the pre-activation starts so many elements off a 16-byte boundary.  Infinite and NaN pre-activations give what
    the stand-alone kernel gives."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    from meshslice_b200.ops.gemm import gemm_pair
    t, d, f = shape
    g = torch.Generator(device="cuda").manual_seed(f)
    rand = lambda *s: torch.randn(s, device="cuda", generator=g).bfloat16()
    x, dy, w = rand(t, f), rand(t, d), rand(*((d, f) if dataflow == "ls" else (f, d)))
    pre = (rand(t * f + offset) * 2)[offset:].view(t, f)
    assert pre.data_ptr() % 16 == 2 * offset
    first, layout = ((dy, x, "tn"), "nn") if dataflow == "ls" else ((x, dy, "tn"), "nt")
    both = lambda p: gemm_pair(*first, torch.zeros(w.shape, device="cuda"), True, dy, w, layout, gelu_pre=p)
    dw, got = both(pre)
    plain = _ref(dy, w, layout)
    xr = pre.float().requires_grad_(True)
    torch.nn.functional.gelu(xr, approximate="tanh").backward(plain)
    _native.check_status()
    assert ((got.float() - xr.grad).norm() / xr.grad.norm()).item() < 2 ** -9
    _check(dw, _ref(*first), t)
    odd = pre.clone()                # starts on a 16-byte boundary, which the stand-alone kernel needs
    odd[5, :40:8] = torch.tensor([float("inf"), -float("inf"), float("nan"), 1e20, -1e20], device="cuda").bfloat16()
    got, want = both(odd)[1], F.gelu_bwd(both(None)[1], odd)
    _native.check_status()
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.isnan(want[5]).any()
    ok = ~torch.isnan(want)
    assert ((got[ok].float() - want[ok].float()).norm() / want[ok].float().norm()).item() < 2 ** -8


@pytest.mark.parametrize("offset", [0, 3])
def test_gemm_pair_times_gelu_derivative_with_the_one_cta_kernel(offset, monkeypatch):
    """MSB_TWO_CTA=0: the products one by one and the derivative by the stand-alone kernel, which reads 16 bytes at a time: a
    pre-activation that starts elsewhere gives the same bits.  Two bf16 roundings of the result (2^-9 each)."""
    from meshslice_b200 import _native
    from meshslice_b200.ops.gemm import gemm_pair
    monkeypatch.setenv("MSB_TWO_CTA", "0")
    t, d, f = 264, 136, 520
    g = torch.Generator(device="cuda").manual_seed(f)
    rand = lambda *s: torch.randn(s, device="cuda", generator=g).bfloat16()
    x, dy, w, pre = rand(t, f), rand(t, d), rand(f, d), rand(t, f) * 2
    moved = torch.empty(t * f + offset, device="cuda", dtype=torch.bfloat16)[offset:].view(t, f).copy_(pre)
    assert moved.data_ptr() % 16 == 2 * offset
    both = lambda p: gemm_pair(x, dy, "tn", torch.zeros(w.shape, device="cuda"), True, dy, w, "nt", gelu_pre=p)
    got, want = both(moved), both(pre)
    _native.check_status()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    xr = pre.float().requires_grad_(True)
    torch.nn.functional.gelu(xr, approximate="tanh").backward(_ref(dy, w, "nt"))
    assert ((got[1].float() - xr.grad).norm() / xr.grad.norm()).item() < 2 ** -8

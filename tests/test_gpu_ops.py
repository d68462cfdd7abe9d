"""Memory-bound kernels against plain PyTorch fp32 references."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _C():
    from meshslice_b200 import _native
    return _native.load(), _native.stream_ptr()


# Whole rows take the row kernels forward and, where the second look at dy and h is the faster one, backward.  The ring and the
# vectors per thread of the kernels behind them: test_layernorm_two_passes_of_wide_shards, test_layernorm_persistent_backward_in_one_pass.
@pytest.mark.parametrize("residual", [True, False])
@pytest.mark.parametrize("cols,rows", [(8, 1), (264, 5000), (2048, 9001), (2056, 1300), (4096, 1187), (8192, 600), (8200, 333),
                                       (12288, 450), (12296, 301), (16384, 300)])
def test_layernorm_row_ring(cols, rows, residual):
    """Every number of vectors per thread of both kernels, with fewer and with more rows than a CTA's ring holds, and
    dgamma / dbeta on a 4-byte boundary (their 16-byte atomics need a check).  Row results are rounded to bf16 once (2^-8
    of the value at most, with its fp32 statistics 2^-7 is safe); column sums are fp32 over ``rows`` values."""
    from meshslice_b200.ops import functional as F
    g = torch.Generator(device="cuda").manual_seed(cols + rows)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, res, dy, dres = mk(rows, cols), mk(rows, cols), mk(rows, cols), mk(rows, cols)
    gamma, beta = mk(cols), mk(cols)
    h, y, mr = F.ln_full(x, res if residual else None, gamma, beta, 1e-5)
    sums = torch.zeros(2 * cols + 2, device="cuda")
    dg, db = sums[1:cols + 1], sums[cols + 1:2 * cols + 1]
    dx = F.ln_bwd_full(dy, h, gamma, mr, dg, db, dres if residual else None)
    torch.cuda.synchronize()
    hh = (x.float() + res.float() if residual else x.float())
    assert torch.equal(h, hh.bfloat16())
    hd = h.double().requires_grad_(True)
    gd, bd = gamma.double().requires_grad_(True), beta.double().requires_grad_(True)
    ref = torch.nn.functional.layer_norm(hd, (cols,), gd, bd, 1e-5)
    ref.backward(dy.double())
    want = hd.grad + dres.double() if residual else hd.grad
    close = lambda a, b: ((a.double() - b).abs() <= 2 ** -7 * b.abs() + 2 ** -7 * b.abs().mean()).all()
    assert close(y, ref.detach()) and close(dx, want)
    assert (dg.double() - gd.grad).abs().max() <= 1e-5 * rows ** 0.5 * 30 and (db.double() - bd.grad).abs().max() <= 1e-5 * rows ** 0.5 * 30
    assert sums[0] == 0 and sums[-1] == 0


@pytest.mark.parametrize("residual", [True, False])
@pytest.mark.parametrize("cols,rows", [(8, 1), (256, 1025), (264, 1027), (1544, 1), (1544, 257), (1800, 1500), (2048, 256), (2048, 1030),
                                       (2056, 1025), (3080, 130), (4096, 300), (5128, 1024), (6152, 130), (8192, 128), (8200, 40),
                                       (16384, 33)])
def test_layernorm_of_whole_rows(cols, rows, residual):
    """One, four and eight warps per row at the edges of the rule (a vector more than a warp's registers take, few rows, the last
    CTA partly empty, the last vector in one lane), without affine parameters, and the backward pass without their gradients
    where the persistent kernel would otherwise run.  One bf16 rounding (2^-8 of the value, 2^-7 with the statistics)."""
    from meshslice_b200.ops import functional as F
    g = torch.Generator(device="cuda").manual_seed(cols * 7 + rows)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, res, dy, dres = mk(rows, cols) + 1, mk(rows, cols), mk(rows, cols), mk(rows, cols)
    h, y, mr = F.ln_full(x, res if residual else None, None, None, 1e-5)
    dx = F.ln_bwd_full(dy, h, None, mr, None, None, dres if residual else None)
    gamma = mk(cols)
    dxg = F.ln_bwd_full(dy, h, gamma, mr, None, None, dres if residual else None)
    torch.cuda.synchronize()
    assert torch.equal(h, (x.float() + res.float()).bfloat16() if residual else x)
    close = lambda a, b: ((a.double() - b).abs() <= 2 ** -7 * b.abs() + 2 ** -7 * b.abs().mean()).all()
    for got, scale in ((dx, None), (dxg, gamma.double())):
        hd = h.double().requires_grad_(True)
        ref = torch.nn.functional.layer_norm(hd, (cols,), scale, None, 1e-5)
        ref.backward(dy.double())
        assert close(got, hd.grad + dres.double() if residual else hd.grad)
        if scale is None:
            assert close(y, ref.detach())
    # rows with an infinity or a NaN are NaN, the others are not touched
    bad = x.clone()
    bad[0, 0], bad[rows // 2, cols - 1] = float("inf"), float("nan")
    hb, yb, mb = F.ln_full(bad, res if residual else None, None, None, 1e-5)
    keep = torch.ones(rows, dtype=torch.bool, device="cuda")
    keep[0] = keep[rows // 2] = False
    assert torch.isnan(yb[~keep]).any(1).all() and torch.equal(yb[keep], y[keep]) and torch.equal(mb[keep], mr[keep])


# Every size here is on the near side of the rule; test_layernorm_persistent_backward_in_one_pass has the far one.
@pytest.mark.parametrize("residual", [True, False])
@pytest.mark.parametrize("cols,rows", [(8, 1), (40, 3000), (264, 129), (1544, 127), (1800, 4099), (2048, 513), (2056, 1025), (3080, 4100),
                                       (6152, 33), (16384, 20), (1024, 31500), (4096, 3052)])
def test_layernorm_parameter_gradients(cols, rows, residual):
    """Column sums from a second look at the rows (last block of 32 columns partly empty, fewer rows than a step, several slices)
    and, in the last sizes with a residual, either side of the rule.  They are added to what is there; fp32 sums of ``rows``
    products of normal values: 1e-5 sqrt(rows) times thirty."""
    from meshslice_b200.ops import functional as F
    g = torch.Generator(device="cuda").manual_seed(cols * 3 + rows)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    h, dy, dres, gamma = mk(rows, cols) + 1, mk(rows, cols), mk(rows, cols), mk(cols)
    _, _, mr = F.ln_full(h, None, None, None, 1e-5)
    sums = torch.ones(2 * cols + 2, device="cuda")
    dg, db = sums[1:cols + 1], sums[cols + 1:2 * cols + 1]
    dx = F.ln_bwd_full(dy, h, gamma, mr, dg, db, dres if residual else None)
    only = torch.zeros(cols, device="cuda")
    assert torch.equal(F.ln_bwd_full(dy, h, gamma, mr, only, None, dres if residual else None), dx)
    torch.cuda.synchronize()
    hd, gd, bd = h.double().requires_grad_(True), gamma.double().requires_grad_(True), torch.zeros(cols, device="cuda", dtype=torch.double).requires_grad_(True)
    torch.nn.functional.layer_norm(hd, (cols,), gd, bd, 1e-5).backward(dy.double())
    want = hd.grad + dres.double() if residual else hd.grad
    assert ((dx.double() - want).abs() <= 2 ** -7 * want.abs() + 2 ** -7 * want.abs().mean()).all()
    tol = 3e-4 * rows ** 0.5
    assert (dg.double() - 1 - gd.grad).abs().max() <= tol and (db.double() - 1 - bd.grad).abs().max() <= tol
    assert (only.double() - gd.grad).abs().max() <= tol
    assert sums[0] == 1 and sums[-1] == 1


# The ring is the two-pass kernel's; in one pass both sizes take the row kernel, whose bits do not depend on the number of rows here.
@pytest.mark.parametrize("residual", [True, False])
@pytest.mark.parametrize("cols", [264, 1024, 2048])
def test_layernorm_forward_with_and_without_the_ring(cols, residual):
    """A call that moves more than 80 MiB takes the row ring, one of a sixteenth of its rows (8 to 80 MiB) does not: the same
    threads add the same vectors, so the results agree bit for bit, in one pass and in two (statistics, then rows)."""
    from meshslice_b200.ops import functional as F
    rows = 4 * (100 * 2 ** 20 // (2 * cols * 4))
    if not residual:
        rows *= 2
    g = torch.Generator(device="cuda").manual_seed(cols)
    x = torch.randn(rows, cols, device="cuda", generator=g).bfloat16()
    res = torch.randn(rows, cols, device="cuda", generator=g).bfloat16() if residual else None
    gamma, beta = (torch.randn(cols, device="cuda", generator=g).bfloat16() for _ in range(2))
    whole = F.ln_full(x, res, gamma, beta, 1e-5)
    h, stats = F.ln_stats(x, res)
    two = F.ln_apply(h, stats, gamma, beta, cols, 1e-5)
    q = rows // 16
    for i in (0, 7 * q, rows - q):
        cut = lambda t: None if t is None else t[i:i + q]
        part = F.ln_full(cut(x), cut(res), gamma, beta, 1e-5)
        assert all(torch.equal(p, cut(w)) for p, w in zip(part, whole))
        hp, sp = F.ln_stats(cut(x), cut(res))
        assert torch.equal(hp, cut(h)) and torch.equal(sp, cut(stats))
        assert all(torch.equal(p, cut(w)) for p, w in zip(F.ln_apply(hp, sp, gamma, beta, cols, 1e-5), two))


# Several rows per CTA and a row per CTA of the persistent kernel: test_layernorm_persistent_backward_in_one_pass; these sizes take
# the row kernels but for the widest.
@pytest.mark.parametrize("cols,rows", [(1024, 301), (768, 43), (64, 1000), (2048, 300), (4096, 300), (12288, 300)])
def test_layernorm_fwd_bwd_single_pass(cols, rows):
    """Widths up to 2048 run several rows per CTA in the backward kernel (row counts that leave the last CTA
    partly empty included); wider rows one row per CTA with one, two or four vectors per thread."""
    C, st = _C()
    x = torch.randn(rows, cols, device="cuda").bfloat16()
    res = torch.randn(rows, cols, device="cuda").bfloat16()
    gamma = (1 + 0.1 * torch.randn(cols, device="cuda")).bfloat16()
    beta = (0.1 * torch.randn(cols, device="cuda")).bfloat16()
    h = torch.empty_like(x)
    y = torch.empty_like(x)
    mr = torch.empty(rows, 2, device="cuda")
    C.ln_fwd(0, x.data_ptr(), res.data_ptr(), h.data_ptr(), y.data_ptr(), gamma.data_ptr(), beta.data_ptr(),
             0, mr.data_ptr(), rows, cols, cols, 1e-5, st)
    h_ref = (x.float() + res.float())
    assert (h.float() - h_ref).abs().max() < 0.05
    hh = h.float().requires_grad_(True)
    g32, b32 = gamma.float().requires_grad_(True), beta.float().requires_grad_(True)
    y_ref = torch.nn.functional.layer_norm(hh, (cols,), g32, b32, 1e-5)
    assert (y.float() - y_ref).abs().max() < 0.05
    dy = torch.randn(rows, cols, device="cuda").bfloat16()
    dres = torch.randn(rows, cols, device="cuda").bfloat16()
    y_ref.backward(dy.float())
    dx = torch.empty_like(x)
    dg = torch.zeros(cols, device="cuda")
    db = torch.zeros(cols, device="cuda")
    C.ln_bwd(0, dy.data_ptr(), h.data_ptr(), gamma.data_ptr(), mr.data_ptr(), dres.data_ptr(), dx.data_ptr(),
             0, dg.data_ptr(), db.data_ptr(), rows, cols, cols, st)
    torch.cuda.synchronize()
    assert (dx.float() - (hh.grad + dres.float())).abs().max() < 0.06
    assert (dg - g32.grad).abs().max() < 0.05 * rows ** 0.5
    assert (db - b32.grad).abs().max() < 0.05 * rows ** 0.5


def test_layernorm_two_pass_equals_single_pass():
    """The column-sharded path: partial statistics per shard, summed, then applied."""
    C, st = _C()
    rows, cols, parts = 64, 2048, 4
    x = torch.randn(rows, cols, device="cuda").bfloat16()
    gamma = torch.ones(cols, device="cuda").bfloat16()
    y_full = torch.empty_like(x)
    mr = torch.empty(rows, 2, device="cuda")
    C.ln_fwd(0, x.data_ptr(), 0, 0, y_full.data_ptr(), gamma.data_ptr(), 0, 0, mr.data_ptr(), rows, cols, cols, 1e-5, st)
    w = cols // parts
    shards = [x[:, i * w:(i + 1) * w].contiguous() for i in range(parts)]
    stats = [torch.empty(rows, 2, device="cuda") for _ in range(parts)]
    for s, t in zip(shards, stats):
        C.ln_fwd(1, s.data_ptr(), 0, 0, 0, 0, 0, t.data_ptr(), 0, rows, w, cols, 1e-5, st)
    total = sum(stats)
    outs = []
    for i, s in enumerate(shards):
        y = torch.empty_like(s)
        g = gamma[i * w:(i + 1) * w].contiguous()
        C.ln_fwd(2, s.data_ptr(), 0, 0, y.data_ptr(), g.data_ptr(), 0, total.data_ptr(), mr.data_ptr(), rows, w, cols, 1e-5, st)
        outs.append(y)
    torch.cuda.synchronize()
    assert (torch.cat(outs, 1).float() - y_full.float()).abs().max() < 0.02


@pytest.mark.parametrize("affine", [True, False])
def test_layernorm_backward_two_pass_equals_single_pass(affine):
    """Backward of the column-sharded path (partial dot products per shard, summed, then applied) against the
    single-pass kernel on the whole row and against autograd in fp32."""
    C, st = _C()
    rows, cols, parts = 97, 4096, 4
    hbuf = torch.randn(rows, cols, device="cuda").bfloat16()
    dy = torch.randn(rows, cols, device="cuda").bfloat16()
    dres = torch.randn(rows, cols, device="cuda").bfloat16()
    gamma = (1.0 + 0.1 * torch.randn(cols, device="cuda")).bfloat16() if affine else None
    gp = gamma.data_ptr() if affine else 0
    mean = hbuf.float().mean(1)
    rstd = (hbuf.float().var(1, unbiased=False) + 1e-5).rsqrt()
    mr = torch.stack([mean, rstd], 1).contiguous()
    dx_full = torch.empty_like(hbuf)
    dg_full = torch.zeros(cols, device="cuda")
    db_full = torch.zeros(cols, device="cuda")
    C.ln_bwd(0, dy.data_ptr(), hbuf.data_ptr(), gp, mr.data_ptr(), dres.data_ptr(), dx_full.data_ptr(), 0,
             dg_full.data_ptr() if affine else 0, db_full.data_ptr() if affine else 0, rows, cols, cols, st)
    w = cols // parts
    # the shards stay referenced until the kernels have run (only raw pointers are passed)
    cut = lambda t: [t[:, i * w:(i + 1) * w].contiguous() for i in range(parts)]
    dys, hs, drs = cut(dy), cut(hbuf), cut(dres)
    gs = [gamma[i * w:(i + 1) * w].contiguous() for i in range(parts)] if affine else [None] * parts
    stats, dgs, dbs = [], [], []
    for i in range(parts):
        t = torch.empty(rows, 2, device="cuda")
        dg = torch.zeros(w, device="cuda")
        db = torch.zeros(w, device="cuda")
        C.ln_bwd(1, dys[i].data_ptr(), hs[i].data_ptr(), gs[i].data_ptr() if affine else 0, mr.data_ptr(), 0, 0,
                 t.data_ptr(), dg.data_ptr() if affine else 0, db.data_ptr() if affine else 0, rows, w, cols, st)
        stats.append(t); dgs.append(dg); dbs.append(db)
    total = sum(stats)
    outs = []
    for i in range(parts):
        dx = torch.empty(rows, w, device="cuda", dtype=torch.bfloat16)
        C.ln_bwd(2, dys[i].data_ptr(), hs[i].data_ptr(), gs[i].data_ptr() if affine else 0, mr.data_ptr(),
                 drs[i].data_ptr(), dx.data_ptr(), total.data_ptr(), 0, 0, rows, w, cols, st)
        outs.append(dx)
    torch.cuda.synchronize()
    assert (torch.cat(outs, 1).float() - dx_full.float()).abs().max() < 0.04
    hh = hbuf.float().requires_grad_(True)
    g32 = gamma.float().requires_grad_(True) if affine else None
    torch.nn.functional.layer_norm(hh, (cols,), g32, None, 1e-5).backward(dy.float())
    assert (dx_full.float() - (hh.grad + dres.float())).abs().max() < 0.06
    if affine:
        assert (torch.cat(dgs) - dg_full).abs().max() < 1e-2
        assert (dg_full - g32.grad).abs().max() < 0.05 * rows ** 0.5
        assert (torch.cat(dbs) - dy.float().sum(0)).abs().max() < 1e-2


def test_gelu_fwd_bwd():
    C, st = _C()
    x = torch.randn(1 << 16, device="cuda").bfloat16()
    dy = torch.randn(1 << 16, device="cuda").bfloat16()
    y = torch.empty_like(x)
    dx = torch.empty_like(x)
    C.gelu_fwd(x.data_ptr(), y.data_ptr(), x.numel(), st)
    C.gelu_bwd(dy.data_ptr(), x.data_ptr(), dx.data_ptr(), x.numel(), st)
    x32 = x.float().requires_grad_(True)
    ref = torch.nn.functional.gelu(x32, approximate="tanh")
    ref.backward(dy.float())
    assert (y.float() - ref).abs().max() < 0.02
    assert (dx.float() - x32.grad).abs().max() < 0.03


def test_adamw_matches_torch():
    C, st = _C()
    n = 4096 * 3
    p32 = torch.randn(n, device="cuda")
    g = torch.randn(n, device="cuda").bfloat16()
    p = p32.bfloat16()
    master = p32.clone()
    m = torch.zeros(n, device="cuda")
    v = torch.zeros(n, device="cuda")
    ref = p32.clone().requires_grad_(True)
    opt = torch.optim.AdamW([ref], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    for step in range(1, 4):
        ref.grad = g.float()
        opt.step()
        C.adamw_step(p.data_ptr(), master.data_ptr(), m.data_ptr(), v.data_ptr(), g.data_ptr(), 0, n, 1e-2,
                     0.9, 0.95, 1e-8, 0.1, 1 - 0.9 ** step, 1 - 0.95 ** step, 0, st)
    torch.cuda.synchronize()
    assert (master - ref.detach()).abs().max() < 1e-4
    assert (p.float() - ref.detach()).abs().max() < 0.02


@pytest.mark.parametrize("cols,offset,vocab", [(8, 0, 5), (2048, 0, 2041), (8192, 0, 8192), (10240, 2048, 9999), (51200, 0, 50257),
                                               (64, 128, 100)])
def test_cross_entropy_row_statistics(cols, offset, vocab):
    """One pass over a row: rows that raise the maximum late, masked columns (-inf), a lone finite value, nothing but -inf,
    +inf, NaN and magnitudes of 1e4, against 64 bits.  The maximum is exact; the sum is fp32 over at most 51200 terms of
    at most 1 whose exponentials carry 2^-21 of the argument's rounding each: 1e-4 relative."""
    from meshslice_b200.ops import functional as F
    g = torch.Generator(device="cuda").manual_seed(cols)
    n = max(0, min(cols, vocab - offset))
    x = torch.randn(12, cols, device="cuda", generator=g)
    if n:
        x[1] += torch.linspace(0, 30, cols, device="cuda")
        x[2, ::2] = float("-inf")
        x[3] = float("-inf"); x[3, n - 1] = -7.0
        x[4] = float("-inf")
        x[5, n // 2] = float("inf")
        x[6, n // 3] = float("nan")
        x[7] *= 1e4
        x[8] = -1e4
        x[9, : n - 1] = float("-inf")
        x[10] = float("-inf"); x[10, 0] = float("nan")
    x = x.bfloat16()
    t = torch.full((12,), offset + max(0, n - 1), device="cuda")
    mx, se, tl = F.ce_partial(x, t, offset, vocab)
    torch.cuda.synchronize()
    if n == 0:
        assert (mx == float("-inf")).all() and (se == 0).all() and (tl == 0).all()
        return
    d = x[:, :n].double()
    assert torch.equal(tl, x[:, n - 1].float())
    for r in range(12):
        row = d[r]
        want_m = row[~row.isnan()].max() if (~row.isnan()).any() else torch.tensor(float("-inf"))
        assert mx[r].item() == want_m.item(), r
        want = torch.exp(row - want_m).sum().item()
        if want != want:
            assert se[r].item() != se[r].item(), r
        else:
            assert abs(se[r].item() - want) <= 1e-4 * want, (r, se[r].item(), want)


def test_cross_entropy_vocab_parallel():
    C, st = _C()
    rows, vocab, parts = 96, 1000, 4
    vpad = 1024
    w = vpad // parts
    logits = (3 * torch.randn(rows, vpad, device="cuda")).bfloat16()
    tgt = torch.randint(0, vocab, (rows,), device="cuda")
    ref_l = logits.float()[:, :vocab].clone().requires_grad_(True)
    loss_ref = torch.nn.functional.cross_entropy(ref_l, tgt, reduction="mean")
    loss_ref.backward()
    mx, se, tl = [], [], []
    shards = [logits[:, i * w:(i + 1) * w].contiguous() for i in range(parts)]
    for i, s in enumerate(shards):
        a, b, c = (torch.empty(rows, device="cuda") for _ in range(3))
        C.ce_partial(s.data_ptr(), w, tgt.data_ptr(), rows, w, i * w, vocab, a.data_ptr(), b.data_ptr(), c.data_ptr(), st)
        mx.append(a); se.append(b); tl.append(c)
    gmax = torch.stack(mx).max(0).values
    gsum = sum(s * torch.exp(m - gmax) for s, m in zip(se, mx))
    tlog = sum(tl)
    loss = (torch.log(gsum) + gmax - tlog).mean()
    assert abs(loss.item() - loss_ref.item()) < 2e-3
    for i, s in enumerate(shards):
        C.ce_grad(s.data_ptr(), w, tgt.data_ptr(), rows, w, i * w, vocab, gmax.data_ptr(), gsum.data_ptr(), 1.0 / rows, st)
    torch.cuda.synchronize()
    grad = torch.cat(shards, 1).float()
    assert (grad[:, :vocab] - ref_l.grad).abs().max() < 2e-4
    assert grad[:, vocab:].abs().max() == 0


@pytest.mark.parametrize("cols", [8, 1032, 4096, 4104, 9224])
def test_embedding_lookup_widths(cols):
    """Rows of one vector, of a batch of vectors per thread and of a little more: the sum of two bf16, rounded once."""
    from meshslice_b200.ops import functional as F
    g = torch.Generator(device="cuda").manual_seed(cols)
    tok, pos = (torch.randn(n, cols, device="cuda", generator=g).bfloat16() for n in (50, 24))
    ids = torch.randint(0, 50, (72,), device="cuda", generator=g)
    out = F.embedding_fwd(ids, tok, pos, 24)
    assert torch.equal(out, (tok[ids].float() + pos.repeat(3, 1).float()).bfloat16())


def test_embedding_fwd_bwd():
    C, st = _C()
    vocab, seq, nb, cols = 500, 16, 4, 256
    tok = torch.randint(0, vocab, (nb * seq,), device="cuda")
    te = torch.randn(vocab, cols, device="cuda").bfloat16()
    pe = torch.randn(seq, cols, device="cuda").bfloat16()
    out = torch.empty(nb * seq, cols, device="cuda", dtype=torch.bfloat16)
    C.embedding_fwd(tok.data_ptr(), te.data_ptr(), pe.data_ptr(), out.data_ptr(), nb * seq, seq, cols, st)
    ref = te.float()[tok] + pe.float().repeat(nb, 1)
    assert (out.float() - ref).abs().max() < 0.05
    dout = torch.randn(nb * seq, cols, device="cuda").bfloat16()
    dt = torch.zeros(vocab, cols, device="cuda")
    dp = torch.zeros(seq, cols, device="cuda")
    C.embedding_bwd(tok.data_ptr(), dout.data_ptr(), dt.data_ptr(), dp.data_ptr(), nb * seq, seq, cols, st)
    torch.cuda.synchronize()
    dt_ref = torch.zeros(vocab, cols, device="cuda").index_add_(0, tok, dout.float())
    dp_ref = dout.float().view(nb, seq, cols).sum(0)
    assert (dt - dt_ref).abs().max() < 1e-3
    assert (dp - dp_ref).abs().max() < 1e-3


def test_sumsq():
    C, st = _C()
    x = torch.randn(1 << 18, device="cuda").bfloat16()
    out = torch.zeros(1, device="cuda")
    C.sumsq(x.data_ptr(), 0, x.numel(), out.data_ptr(), st)
    torch.cuda.synchronize()
    assert abs(out.item() - (x.float() ** 2).sum().item()) / out.item() < 1e-4


def _emulated_exchange(n, rows, grid):
    """Descriptors of one row exchange among n emulated ranks that all live on this GPU: rank q's slot area and
    arrival counter are plain tensors.  The caller runs every rank's producer before any consumer, so no kernel
    waits for one that has not run; the consumers' waits are then satisfied on entry."""
    from meshslice_b200 import _native
    width = 4
    stride = rows * width
    slots = [torch.zeros(n * stride, device="cuda") for _ in range(n)]
    counters = [torch.zeros(16, dtype=torch.int32, device="cuda") for _ in range(n)]
    descs = []
    for q in range(n):
        descs.append(dict(n=n, me=q, dst=[slots[p].data_ptr() + q * stride * 4 for p in range(n)],
                          slots=slots[q].data_ptr(), stride=stride,
                          counter=[counters[p].data_ptr() for p in range(n)], my_counter=counters[q].data_ptr(),
                          target=(n - 1) * grid, timeout_ns=50_000_000, status=_native.status().dev))
    return descs, (slots, counters)


@pytest.mark.parametrize("n,w,rows", [(4, 1024, 203), (2, 4096, 64), (2, 256, 1000)])
def test_layernorm_row_exchange_emulated_ranks(n, w, rows):
    """LayerNorm forward and backward over a feature dimension split among n ranks, the partial row sums travelling
    through the in-kernel exchange (slots + arrival counters), against the single-device kernels on the whole rows.
    Narrow shards take the several-rows-per-CTA form of the backward kernel."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    C, st = _C()
    cols = n * w
    cut = lambda t: [t[:, q * w:(q + 1) * w].contiguous() for q in range(n)]
    x = torch.randn(rows, cols, device="cuda").bfloat16()
    res = torch.randn(rows, cols, device="cuda").bfloat16()
    gamma = (1 + 0.1 * torch.randn(cols, device="cuda")).bfloat16()
    beta = (0.1 * torch.randn(cols, device="cuda")).bfloat16()
    h_ref, y_ref, mr_ref = F.ln_full(x, res, gamma, beta, 1e-5)
    xs, rs = cut(x), cut(res)
    gs = [gamma[q * w:(q + 1) * w].contiguous() for q in range(n)]
    bs = [beta[q * w:(q + 1) * w].contiguous() for q in range(n)]
    descs, keep = _emulated_exchange(n, rows, C.ln_grid(0, rows, w))
    hs = [F.ln_stats(xs[q], rs[q], exch=descs[q])[0] for q in range(n)]
    outs = [F.ln_apply(hs[q], None, gs[q], bs[q], cols, 1e-5, exch=descs[q]) for q in range(n)]
    _native.check_status()
    assert torch.equal(torch.cat(hs, 1), h_ref)
    assert (torch.cat([o[0] for o in outs], 1).float() - y_ref.float()).abs().max() < 0.02
    for q in range(n):
        assert (outs[q][1] - mr_ref).abs().max() < 1e-3
    # backward
    dy = torch.randn(rows, cols, device="cuda").bfloat16()
    dres = torch.randn(rows, cols, device="cuda").bfloat16()
    dg_ref = torch.zeros(cols, device="cuda")
    db_ref = torch.zeros(cols, device="cuda")
    dx_ref = F.ln_bwd_full(dy, h_ref, gamma, mr_ref, dg_ref, db_ref, dres)
    dys, drs = cut(dy), cut(dres)
    dgs = [torch.zeros(w, device="cuda") for _ in range(n)]
    dbs = [torch.zeros(w, device="cuda") for _ in range(n)]
    descs, keep2 = _emulated_exchange(n, rows, C.ln_grid(1, rows, w))
    for q in range(n):
        F.ln_bwd_stats(dys[q], hs[q], gs[q], mr_ref, dgs[q], dbs[q], exch=descs[q])
    dxs = [F.ln_bwd_apply(dys[q], hs[q], gs[q], mr_ref, None, cols, drs[q], exch=descs[q]) for q in range(n)]
    _native.check_status()
    assert (torch.cat(dxs, 1).float() - dx_ref.float()).abs().max() < 0.04
    assert (torch.cat(dgs) - dg_ref).abs().max() < 1e-2 * rows ** 0.5
    assert (torch.cat(dbs) - db_ref).abs().max() < 1e-2 * rows ** 0.5
    # every rank's counter has seen exactly the other ranks' CTAs
    for q in range(n):
        assert int(keep2[1][q][0]) == (n - 1) * C.ln_grid(1, rows, w)


def test_layernorm_exchange_gives_up_when_nothing_arrives():
    """The consumers' waits run out (50 ms), with rows of theirs already on the way: a status, and the next call works."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    rows, w = 300, 1024
    x = torch.randn(rows, w, device="cuda").bfloat16()
    gamma, beta = torch.ones(w, device="cuda").bfloat16(), torch.zeros(w, device="cuda").bfloat16()
    h, y, mr = F.ln_full(x, None, gamma, beta, 1e-5)
    descs, keep = _emulated_exchange(2, rows, 300)
    F.ln_apply(x, None, gamma, beta, 2 * w, 1e-5, exch=descs[0])
    with pytest.raises(_native.KernelStatusError):
        _native.check_status()
    F.ln_bwd_apply(x, x, gamma, mr, None, 2 * w, None, exch=descs[1])
    with pytest.raises(_native.KernelStatusError):
        _native.check_status()
    assert torch.equal(F.ln_full(x, None, gamma, beta, 1e-5)[1], y)
    _native.check_status()


@pytest.mark.parametrize("rows", [1, 741, 5000])
def test_cross_entropy_row_exchange_emulated_ranks(rows):
    """Loss and gradient over a vocabulary split between two ranks, every producer before any consumer, with more rows than
    the exchange has CTAs; the counters see exactly the CTAs that the host was told.  A relative error e of the sum (1e-4, see
    the row-statistics test) is an absolute one of its logarithm, whatever the size of the loss; gradients are rounded to
    bf16 once."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    C, st = _C()
    n, w, vocab = 2, 512, 1000
    g = torch.Generator(device="cuda").manual_seed(rows)
    logits = (3 * torch.randn(rows, n * w, device="cuda", generator=g)).bfloat16()
    tgt = torch.randint(0, vocab, (rows,), device="cuda", generator=g)
    parts = [logits[:, q * w:(q + 1) * w].clone(memory_format=torch.contiguous_format) for q in range(n)]   # updated in place
    descs, keep = _emulated_exchange(n, rows, C.ce_grid(rows))
    for q in range(n):
        F.ce_partial(parts[q], tgt, q * w, vocab, exch=descs[q])
    losses = [F.ce_grad_exchanged_(parts[q], tgt, q * w, vocab, 1.0, descs[q]) for q in range(n)]
    _native.check_status()
    x = logits[:, :vocab].double().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(x, tgt, reduction="none")
    ref.sum().backward()
    got = torch.cat(parts, 1).double()
    errors = [(l.double() - ref).abs().max().item() for l in losses]
    assert max(errors) < 1e-4, (errors, ref.abs().max().item())
    assert ((got[:, :vocab] - x.grad).abs() <= 2 ** -8 * x.grad.abs() + 1e-4).all() and (got[:, vocab:] == 0).all()
    for q in range(n):
        assert int(keep[1][q][0]) == (n - 1) * C.ce_grid(rows)


@pytest.mark.parametrize("sq", [(0.0, 0.0), (9.0, 16.0), (0.09, 0.16), (float("inf"), 1.0), (float("nan"), 1.0)])
def test_clip_scale(sq):
    """Norm and clipping factor as the optimizer's CPU path computes them (three fp32 roundings: 2^-21)."""
    C, st = _C()
    t = torch.tensor(sq, device="cuda")
    out = torch.zeros(2, device="cuda")
    C.clip_scale(t.data_ptr(), 2, 1.0, out.data_ptr(), out.data_ptr() + 4, st)
    norm = torch.sqrt(t.cpu().sum())
    want = torch.stack([norm, torch.clamp(1.0 / (norm + 1e-6), max=1.0)])
    assert torch.allclose(out.cpu(), want, rtol=2 ** -21, atol=0, equal_nan=True)


def test_cross_entropy_gradient_returns_the_row_loss():
    """One launch for gradient and loss: the gradient is that of ce_grad_ bit for bit, the loss log(sum) + max - target."""
    from meshslice_b200.ops import functional as F
    x = (3 * torch.randn(5, 4096, device="cuda")).bfloat16()
    t = torch.tensor([0, 7, 8, 3990, 1234], device="cuda")
    mx, se, tl = F.ce_partial(x, t, 0, 3991)
    a, b = x.clone(), x.clone()
    F.ce_grad_(a, t, 0, 3991, mx, se, 0.2)
    loss = F.ce_grad_loss_(b, t, 0, 3991, mx, se, tl, 0.2)
    ref = torch.nn.functional.cross_entropy(x[:, :3991].double(), t, reduction="none")
    assert torch.equal(a, b)
    assert (loss.double() - ref).abs().max() < 1e-4


@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("n", [4, 148 * 32 * 256 * 4, 148 * 32 * 256 * 16 + 12, 30000004])
def test_sumsq_steps(n, fp32):
    """One vector, less than a step of four vectors per thread, a whole one and a remainder: fp32 sums over at most a few hundred
    values per thread, then over threads (1e-5 relative)."""
    C, st = _C()
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, device="cuda", generator=g)
    x = x if fp32 else x.bfloat16()
    out = torch.zeros(1, device="cuda")
    C.sumsq(x.data_ptr(), 1 if fp32 else 0, n, out.data_ptr(), st)
    torch.cuda.synchronize()
    want = x.double().square().sum().item()
    assert abs(out.item() - want) <= 1e-5 * want


@pytest.mark.parametrize("rows,d", [(64, 128), (512, 512), (2056, 1032)])
def test_dependent_launches_stay_in_order(rows, d):
    """A chain of kernels that set up while the one before ends, on buffers that the next turn overwrites: the bits of the same
    chain with a synchronisation after every call (fewer blocks than SMs, about as many, more)."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    from meshslice_b200.ops.gemm import gemm, gemm_pair
    g = torch.Generator(device="cuda").manual_seed(rows)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    inputs = [(mk(rows, d), mk(rows, d)) for _ in range(3)]
    w, gamma, beta = mk(d, d) * 0.1, mk(d), mk(d)
    targets = torch.randint(0, d, (rows,), device="cuda", generator=g)
    x, r, buf = torch.empty_like(inputs[0][0]), torch.empty_like(inputs[0][0]), torch.empty(rows, d, device="cuda").bfloat16()

    def turn(i, sync):
        done = torch.cuda.synchronize if sync else (lambda: None)
        x.copy_(inputs[i][0]); r.copy_(inputs[i][1]); done()
        h, y, mr = F.ln_full(x, r, gamma, beta, 1e-5); done()
        gemm(y, w, "nn", out=buf); done()
        z = F.add(F.gelu(buf), h); done()
        mx, se, tl = F.ce_partial(z, targets, 0, d); done()
        loss = F.ce_grad_loss_(z, targets, 0, d, mx, se, tl, 1.0 / rows); done()
        dw = torch.zeros(d, d, device="cuda"); done()
        _, dx = gemm_pair(y, z, "tn", dw, True, z, w, "nt", gelu_pre=buf); done()
        dx = F.ln_bwd_full(dx, h, gamma, mr, None, None, z); done()
        out = [t.clone() for t in (loss, dw, dx, buf)]
        buf.fill_(float("nan")); x.fill_(float("nan")); r.fill_(float("nan")); done()
        return out

    want = [turn(i, True) for i in range(3)]
    got = [turn(i % 3, False) for i in range(18)]
    torch.cuda.synchronize()
    _native.check_status()
    for i, out in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(out, want[i % 3])), i


@pytest.mark.parametrize("rows,cols,vocab", [(3, 8, 5), (5, 2048, 1000), (300, 1024, 1024), (7, 16392, 16385), (9, 51200, 50257),
                                             (2, 102400, 102391), (2, 102408, 102401)])
def test_cross_entropy_of_whole_rows(rows, cols, vocab):
    """Loss and gradient in one launch (the last size, a vector too wide for it, in two): against 64 bits, and rows of -inf, with an
    infinity or a NaN as the two-launch form gives them.  fp32 sums of ``vocab`` exponentials: 1e-6 relative, 2e-6 in the loss;
    the gradient is rounded to bf16 once (2^-9, 2^-8 with the sum)."""
    from meshslice_b200.ops import functional as F
    g = torch.Generator(device="cuda").manual_seed(cols)
    x = (2 * torch.randn(rows, cols, device="cuda", generator=g)).bfloat16()
    t = torch.randint(0, vocab, (rows,), device="cuda", generator=g)
    t[0] = vocab - 1
    ref = x.double()
    ref[:, vocab:] = float("-inf")
    want = torch.softmax(ref, 1)
    want[torch.arange(rows), t] -= 1
    want_loss = torch.logsumexp(ref, 1) - ref.gather(1, t[:, None])[:, 0]
    got = x.clone()
    loss = F.ce_loss_grad_(got, t, vocab, 0.25)
    torch.cuda.synchronize()
    assert ((loss.double() - want_loss).abs() <= 4e-6 * (1 + want_loss.abs())).all()
    assert ((got.double() - 0.25 * want).abs() <= 2 ** -8 * 0.25 * want.abs() + 1e-30).all()
    assert (got[:, vocab:] == 0).all()
    total = F.sum_over(loss, 2)
    assert total.shape == () and abs(total.item() - 0.5 * loss.double().sum().item()) <= 1e-5 * abs(total.item())
    odd = x.clone()
    odd[0] = float("-inf")
    odd[1, 3] = float("inf")
    odd[rows - 1, vocab - 1] = float("nan")
    odd[0, vocab:] = 7.0
    a, b = odd.clone(), odd.clone()
    la = F.ce_loss_grad_(a, t, vocab, 0.25)
    lb = F.ce_grad_loss_(b, t, 0, vocab, *F.ce_partial(b, t, 0, vocab), 0.25)
    assert torch.equal(torch.isnan(la), torch.isnan(lb)) and torch.equal(torch.isnan(a), torch.isnan(b))
    assert torch.equal(torch.isinf(la), torch.isinf(lb))


def test_a_refused_launch_leaves_no_error_for_the_next_call():
    """No rows are a launch of no blocks, which the host refuses.  The next call, launched plainly and so asking for the last
    error behind it, is not answered with that of the one before."""
    from meshslice_b200.ops import functional as F
    x = torch.randn(64, 4096, device="cuda").bfloat16()
    t = torch.zeros(0, dtype=torch.int64, device="cuda")
    want = F.ln_stats(x, None)[1]
    for _ in range(2):
        with pytest.raises(RuntimeError, match="ce_partial"):
            F.ce_partial(x[:0], t, 0, 4096)
        assert torch.equal(F.ln_stats(x, None)[1], want)


@pytest.mark.parametrize("over", ["dy", "h"])
@pytest.mark.parametrize("cols,rows", [(264, 4099), (2048, 4099), (4096, 3000)])
def test_layernorm_backward_over_its_own_inputs(cols, rows, over):
    """dx written over dy or h, as row by row it may be: the parameters' gradients are those of the inputs that were there.
    Rows agree bit for bit with a dx of its own or, from another kernel, within a bf16 rounding; column sums are fp32 over
    ``rows`` values."""
    C, st = _C()
    g = torch.Generator(device="cuda").manual_seed(rows)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    dy, h, gamma = mk(rows, cols), mk(rows, cols), mk(cols)
    mr = torch.stack([h.float().mean(1), (h.float().var(1, unbiased=False) + 1e-5).rsqrt()], 1).contiguous()

    def run(d, hh, out):
        dg, db = torch.zeros(cols, device="cuda"), torch.zeros(cols, device="cuda")
        C.ln_bwd(0, d.data_ptr(), hh.data_ptr(), gamma.data_ptr(), mr.data_ptr(), 0, out.data_ptr(), 0, dg.data_ptr(), db.data_ptr(),
                 rows, cols, cols, st)
        torch.cuda.synchronize()
        return out, dg, db

    want = run(dy, h, torch.empty_like(dy))
    for _ in range(3):
        d, hh = dy.clone(), h.clone()
        got = run(d, hh, d if over == "dy" else hh)
        assert ((got[0].float() - want[0].float()).abs() <= 2 ** -7 * want[0].float().abs() + 2 ** -7 * want[0].float().abs().mean()).all()
        for a, b in zip(got[1:], want[1:]):
            assert (a - b).abs().max() <= 3e-4 * rows ** 0.5


def _steps(F, x, r, gamma, w, targets, rows, d):
    """Dependent launches of every kind: LayerNorm, product, elementwise, loss, both gradients, attention."""
    from meshslice_b200.ops.gemm import gemm, gemm_pair
    h, y, mr = F.ln_full(x, r, gamma, None, 1e-5)
    buf = gemm(y, w, "nn")
    z = F.add(F.gelu(buf), h)
    loss = F.sum_over(F.ce_loss_grad_(z, targets, d, 1.0 / rows), rows)
    dw = torch.zeros(d, d, device="cuda")
    _, dx = gemm_pair(y, z, "tn", dw, True, z, w, "nt", gelu_pre=buf)
    dx = F.ln_bwd_full(dx, h, gamma, mr, None, None, z)
    qkv = torch.cat([x, y, dx], 1)
    out, lse = F.attention_fwd(qkv, 1, rows, d // 128, True)
    return [loss, dw, dx, out, F.attention_bwd(dx, qkv, out, lse, 1, rows, d // 128, True)]


def _step_inputs(rows, d):
    g = torch.Generator(device="cuda").manual_seed(rows + d)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    targets = torch.randint(0, d, (rows,), device="cuda", generator=g)
    return [(mk(rows, d), mk(rows, d)) for _ in range(3)], mk(d), mk(d, d) / d ** 0.5, targets


@pytest.mark.parametrize("rows,d", [(128, 128), (1024, 512)])
def test_dependent_launches_behind_an_event_of_another_stream(rows, d):
    """The first launch of a stream comes right behind its wait for an event of another one, which is still writing the inputs (a
    large product in front of the copy), and the other stream overwrites them right behind an event of this one: the same bits
    as with a synchronisation between all of it."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    inputs, gamma, w, targets = _step_inputs(rows, d)
    want = [[t.clone() for t in _steps(F, x, r, gamma, w, targets, rows, d)] for x, r in inputs]
    torch.cuda.synchronize()
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    x, r = torch.zeros_like(inputs[0][0]), torch.zeros_like(inputs[0][1])
    busy = torch.randn(4096, 4096, device="cuda")
    torch.cuda.synchronize()
    got = []
    for i in range(9):
        with torch.cuda.stream(one):
            torch.mm(busy, busy)
            x.copy_(inputs[i % 3][0])
            r.copy_(inputs[i % 3][1])
            ready = one.record_event()
        with torch.cuda.stream(two):
            two.wait_event(ready)
            got.append([t.clone() for t in _steps(F, x, r, gamma, w, targets, rows, d)])
            done = two.record_event()
        with torch.cuda.stream(one):
            one.wait_event(done)
            x.fill_(float("nan"))
            r.fill_(float("nan"))
    torch.cuda.synchronize()
    _native.check_status()
    for i, out in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(out, want[i % 3])), i


@pytest.mark.parametrize("rows,d", [(128, 128), (1024, 512)])
def test_dependent_launches_in_a_captured_graph(rows, d):
    """The same steps captured and replayed on new inputs in the same buffers: the bits of the calls themselves."""
    from meshslice_b200 import _native
    from meshslice_b200.ops import functional as F
    inputs, gamma, w, targets = _step_inputs(rows, d)
    want = [[t.clone() for t in _steps(F, x, r, gamma, w, targets, rows, d)] for x, r in inputs]
    torch.cuda.synchronize()
    x, r = inputs[0][0].clone(), inputs[0][1].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = _steps(F, x, r, gamma, w, targets, rows, d)
    for i in range(9):
        x.copy_(inputs[i % 3][0])
        r.copy_(inputs[i % 3][1])
        graph.replay()
        got = [t.clone() for t in out]
        assert all(torch.equal(a, b) for a, b in zip(got, want[i % 3])), i
    _native.check_status()


@pytest.mark.parametrize("cols,rows,residual", [(264, 125000, True), (1024, 33000, True), (2048, 16500, True), (4096, 3300, True),
                                                (4096, 4300, False), (3080, 4200, True), (12288, 1500, True)])
def test_layernorm_persistent_backward_in_one_pass(cols, rows, residual):
    """Calls beyond the rule for the second look: the persistent kernel with several rows per CTA (widths up to 2048, the last CTA
    partly empty) and with a row each, with the parameters' gradients, which it adds to what is there.  Rows are rounded to bf16
    once (2^-8 of the value, 2^-7 with the statistics); fp32 sums of ``rows`` products of normal values: 1e-5 sqrt(rows) times
    thirty."""
    from meshslice_b200.ops import functional as F
    g = torch.Generator(device="cuda").manual_seed(cols + rows)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    h, dy, dres, gamma = mk(rows, cols) + 1, mk(rows, cols), mk(rows, cols), mk(cols)
    _, _, mr = F.ln_full(h, None, None, None, 1e-5)
    dg, db = torch.ones(cols, device="cuda"), torch.ones(cols, device="cuda")
    dx = F.ln_bwd_full(dy, h, gamma, mr, dg, db, dres if residual else None)
    torch.cuda.synchronize()
    hd, gd, bd = h.double().requires_grad_(True), gamma.double().requires_grad_(True), torch.zeros(cols, device="cuda", dtype=torch.double).requires_grad_(True)
    torch.nn.functional.layer_norm(hd, (cols,), gd, bd, 1e-5).backward(dy.double())
    want = hd.grad + dres.double() if residual else hd.grad
    assert ((dx.double() - want).abs() <= 2 ** -7 * want.abs() + 2 ** -7 * want.abs().mean()).all()
    tol = 3e-4 * rows ** 0.5
    assert (dg.double() - 1 - gd.grad).abs().max() <= tol and (db.double() - 1 - bd.grad).abs().max() <= tol


@pytest.mark.parametrize("residual", [True, False])
@pytest.mark.parametrize("cols,rows", [(2048, 9001), (2056, 1300), (4096, 1187), (4104, 700), (8192, 600), (8200, 333), (16384, 300)])
def test_layernorm_two_passes_of_wide_shards(cols, rows, residual):
    """Every number of vectors per thread of the two-pass forward kernel (shards of up to 16384 columns), with fewer and with more
    rows than a CTA's ring holds: statistics in fp32 over ``cols`` values (1e-5 of the sum of their sizes), rows rounded to
    bf16 once (2^-8 of the value, 2^-7 with the statistics)."""
    from meshslice_b200.ops import functional as F
    g = torch.Generator(device="cuda").manual_seed(cols + rows)
    mk = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, res, gamma, beta = mk(rows, cols), mk(rows, cols), mk(cols), mk(cols)
    h, stats = F.ln_stats(x, res if residual else None)
    y, mr = F.ln_apply(h, stats, gamma, beta, cols, 1e-5)
    torch.cuda.synchronize()
    assert torch.equal(h, (x.float() + res.float()).bfloat16() if residual else x)
    hd = h.double()
    want = torch.stack([hd.sum(1), (hd * hd).sum(1)], 1)
    assert ((stats.double() - want).abs() <= 1e-5 * torch.stack([hd.abs().sum(1), want[:, 1]], 1)).all()
    ref = torch.nn.functional.layer_norm(hd, (cols,), gamma.double(), beta.double(), 1e-5)
    assert ((y.double() - ref).abs() <= 2 ** -7 * ref.abs() + 2 ** -7 * ref.abs().mean()).all()
    assert (mr[:, 0].double() - hd.mean(1)).abs().max() <= 1e-5 and ((mr[:, 1].double() - (hd.var(1, unbiased=False) + 1e-5).rsqrt()).abs() <= 1e-5).all()

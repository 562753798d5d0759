"""sm_100a kernels vs the fp32 PyTorch statements of the same ops."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _K():
    from kareus_b200.kernels import cuda as KC
    return KC


def _rel(a, b):
    return ((a.float() - b.float()).norm() / (b.float().norm() + 1e-12)).item()


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 512), (384, 640, 3072), (1000, 328, 200),
                                   (4096, 3072, 1024), (130, 72, 136),
                                   # long-K problems with more than one wave of 256x256 tiles
                                   (4096, 4096, 4096), (4500, 4096, 2304)])
@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, False), (True, True)])
def test_gemm_layouts(M, N, K, ta, tb):
    KC = _K()
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + K)
    a = torch.randn((K, M) if ta else (M, K), device="cuda", generator=g).bfloat16()
    b = torch.randn((N, K) if tb else (K, N), device="cuda", generator=g).bfloat16()
    if (a.shape[1] % 8) or (b.shape[1] % 8):
        pytest.skip("row stride not a multiple of 16 bytes")
    c = KC.gemm(a, b, trans_a=ta, trans_b=tb)
    KC.check_status()
    A = a.float().t() if ta else a.float()
    B = b.float().t() if tb else b.float()
    want = A @ B
    assert c.shape == want.shape
    assert _rel(c, want) < 1e-2
    # fp32 output with accumulation
    acc = torch.randn(M, N, device="cuda", generator=g)
    want2 = acc + want
    if N % 4 == 0:
        KC.gemm(a, b, trans_a=ta, trans_b=tb, accumulate=acc)
        KC.check_status()
        assert _rel(acc, want2) < 2e-3


@pytest.mark.parametrize("bn", [64, 128, 192, 256])
@pytest.mark.parametrize("M,N,K", [(8, 8, 8), (136, 72, 64), (257, 264, 400), (600, 520, 136), (2000, 1096, 720)])
@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, False), (True, True)])
def test_two_sm_gemm_tile_edges(bn, M, N, K, ta, tb):
    """Every tile width of the two-SM kernel at the edges of its tiles (256 rows, bn columns, 64-deep steps, parts
    of less than a tile included).  bf16 results are within one rounding of the fp32 product (2^-9 relative, as a
    norm), fp32 sums within fp32 accumulation of exact bf16 products."""
    import ctypes
    KC = _K()
    L = KC.lib()
    L.kb_gemm_force_width.argtypes = [ctypes.c_int]
    L.kb_gemm_force_width.restype = None
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + K)
    a = torch.randn((K, (M + 7) // 8 * 8) if ta else (M, K), device="cuda", generator=g).bfloat16()
    a = a[:, :M] if ta else a
    b = torch.randn((N, K) if tb else (K, N), device="cuda", generator=g).bfloat16()
    want = (a.double().t() if ta else a.double()) @ (b.double().t() if tb else b.double())
    acc = torch.randn(M, N, device="cuda", generator=g)
    want_acc = acc.double() + want
    try:
        L.kb_gemm_force_width(bn)
        c = KC.gemm(a, b, trans_a=ta, trans_b=tb)
        f = KC.gemm(a, b, trans_a=ta, trans_b=tb, out_dtype=torch.float32)
        KC.gemm(a, b, trans_a=ta, trans_b=tb, accumulate=acc)
        KC.check_status()
    finally:
        L.kb_gemm_force_width(0)
    assert _rel(c, want.float()) < 2 ** -8
    assert _rel(f, want.float()) < 1e-5 and _rel(acc, want_acc.float()) < 1e-5


@pytest.mark.parametrize("tile,ks", [(128, 2), (128, 3), (128, 7), (256, 2), (256, 5)])
@pytest.mark.parametrize("n_out,n_in,tokens", [(640, 3072, 4096), (3072, 384, 2048), (1024, 1024, 8192),
                                               (520, 776, 4096)])
def test_weight_gradient_split_k(tile, ks, n_out, n_in, tokens):
    """dW += dYᵀ·X with the K (token) loop split over several CTAs per tile: every part adds its partial
    sum with vector reductions.  Forced splits and what the library picks itself against fp32."""
    import ctypes
    KC = _K()
    L = KC.lib()
    L.kb_gemm_accum_force.argtypes = [ctypes.c_int, ctypes.c_int]
    L.kb_gemm_accum_force.restype = None
    g = torch.Generator(device="cuda").manual_seed(tile + ks + n_out)
    dy = torch.randn(tokens, n_out, device="cuda", generator=g).bfloat16()
    x = torch.randn(tokens, n_in, device="cuda", generator=g).bfloat16()
    start = torch.randn(n_out, n_in, device="cuda", generator=g)
    want = start + dy.float().t() @ x.float()
    try:
        L.kb_gemm_accum_force(tile, ks)
        acc = start.clone()
        KC.gemm(dy, x, trans_a=True, trans_b=False, accumulate=acc)
        KC.check_status()
        assert _rel(acc, want) < 2e-3
    finally:
        L.kb_gemm_accum_force(0, 0)
    acc = start.clone()
    KC.gemm(dy, x, trans_a=True, trans_b=False, accumulate=acc)
    KC.check_status()
    assert _rel(acc, want) < 2e-3


@pytest.mark.parametrize("n_out,n_in,tokens", [(640, 1026, 4096), (1000, 1001, 2048), (136, 33, 3000), (264, 130, 520), (2000, 4099, 700)])
def test_weight_gradient_odd_rows(n_out, n_in, tokens):
    """Gradients whose rows TMA cannot store, at the edges of 32-column groups and 128-row tiles, with and without a K split."""
    KC = _K()
    g = torch.Generator(device="cuda").manual_seed(n_in)
    dy = torch.randn(tokens, n_out, device="cuda", generator=g).bfloat16()
    x = torch.randn(tokens, (n_in + 7) // 8 * 8, device="cuda", generator=g).bfloat16()[:, :n_in]
    want = dy.double().t() @ x.double()
    buf = torch.full((n_out * n_in + 64,), 2.0, device="cuda")
    acc = buf[:n_out * n_in].view(n_out, n_in)
    KC.gemm(dy, x, trans_a=True, trans_b=False, accumulate=acc)
    f = KC.gemm(dy, x, trans_a=True, trans_b=False, out_dtype=torch.float32)
    KC.check_status()
    # fp32 sums of exact bf16 products
    assert _rel(acc, (want + 2).float()) < 1e-5 and _rel(f, want.float()) < 1e-5
    assert (buf[n_out * n_in:] == 2).all()


# full waves of tiles and some left over; forced splits of all tiles with ragged edges and uneven parts
@pytest.mark.parametrize("n_out,n_in,tokens,ks", [(5120, 3072, 8192, 0), (2048, 3072, 8192, 0), (3072, 8192, 4096, 0),
                                                  (2304, 2056, 1104, 2), (2304, 2056, 1104, 5), (3000, 2060, 520, 3)])
def test_weight_gradient_repeats_bitwise(n_out, n_in, tokens, ks):
    """Outputs of more tiles than SMs: the parts of a K split are added in order, the same operands give the same bits."""
    import ctypes
    KC = _K()
    L = KC.lib()
    L.kb_gemm_accum_force.argtypes = [ctypes.c_int, ctypes.c_int]
    L.kb_gemm_accum_force.restype = None
    g = torch.Generator(device="cuda").manual_seed(n_out)
    dy = torch.randn(tokens, n_out, device="cuda", generator=g).bfloat16()
    x = torch.randn(tokens, (n_in + 7) // 8 * 8, device="cuda", generator=g).bfloat16()[:, :n_in]
    start = torch.randn(n_out, n_in, device="cuda", generator=g)
    try:
        L.kb_gemm_accum_force(256, ks)
        assert L.kb_gemm_accum_scratch_floats(n_out, n_in, tokens, 0) > 0          # the tiles are split
        runs = [KC.gemm(dy, x, trans_a=True, trans_b=False, accumulate=start.clone()) for _ in range(8)]
        KC.check_status()
    finally:
        L.kb_gemm_accum_force(0, 0)
    # fp32 sums of exact bf16 products
    assert _rel(runs[0], (start.double() + dy.double().t() @ x.double()).float()) < 1e-5
    assert all(torch.equal(r, runs[0]) for r in runs[1:])


def test_gemm_sm_limit_and_views():
    KC = _K()
    a = torch.randn(512, 1024, device="cuda").bfloat16()
    w = torch.randn(768, 1024, device="cuda").bfloat16()
    full = KC.gemm(a, w)
    few = KC.gemm(a, w, num_sms=7)
    KC.check_status()
    torch.testing.assert_close(full, few)
    big = torch.randn(512, 2048, device="cuda").bfloat16()
    view = big[:, 512:1536]                       # strided rows
    got = KC.gemm(view, w)
    assert _rel(got, view.float() @ w.float().t()) < 1e-2


# rows whose length allows 16-byte stores and rows whose length does not, from an aligned base and from 1, 2 or 4 elements on
@pytest.mark.parametrize("off", [0, 1, 2, 4])
@pytest.mark.parametrize("M,N,K", [(130, 256, 200), (300, 328, 136), (129, 250, 72), (257, 33, 64)])
def test_gemm_output_base_alignment(off, M, N, K):
    KC = _K()
    from kareus_b200.kernels import ref
    g = torch.Generator(device="cuda").manual_seed(M + N + off)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = torch.randn(N, K, device="cuda", generator=g).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g).bfloat16()
    want = a.double() @ w.double().t()

    def place(dtype):
        buf = torch.full((M * N + off + 8,), 3.0, device="cuda", dtype=dtype)
        return buf, buf[off:off + M * N].view(M, N)

    # bf16 results within one rounding (2^-9 relative, as a norm), fp32 sums within fp32 accumulation of exact products
    for dtype, tol in ((torch.bfloat16, 2 ** -8), (torch.float32, 1e-5)):
        for kw, expect in (({}, want), ({"bias": bias, "activation": "gelu"}, ref.bias_act(want, bias.double(), "gelu"))):
            buf, out = place(dtype)
            KC.gemm(a, w, out=out, **kw)
            KC.check_status()
            assert _rel(out, expect.float()) < tol
            assert (buf[:off] == 3).all() and (buf[off + M * N:] == 3).all()
    buf, acc = place(torch.float32)
    KC.gemm(a, w, accumulate=acc)
    KC.check_status()
    assert _rel(acc, (want + 3).float()) < 1e-5
    assert (buf[:off] == 3).all() and (buf[off + M * N:] == 3).all()


@pytest.mark.parametrize("rows,H", [(64, 3072), (1000, 512), (33, 8192), (257, 128), (16, 4096)])
def test_rmsnorm(rows, H):
    KC = _K()
    from kareus_b200.kernels import ref
    x = torch.randn(rows, H, device="cuda").bfloat16()
    w = (1 + 0.1 * torch.randn(H, device="cuda")).bfloat16()
    dy = torch.randn(rows, H, device="cuda").bfloat16()
    y, rstd = KC.rmsnorm_fwd(x, w, 1e-5)
    yr, rr = ref.rmsnorm_fwd(x.float(), w.float(), 1e-5)
    assert _rel(y, yr) < 5e-3 and _rel(rstd, rr) < 1e-5
    dx, dw = KC.rmsnorm_bwd(dy, x, rstd, w)
    dxr, dwr = ref.rmsnorm_bwd(dy.float(), x.float(), rr, w.float())
    assert _rel(dx, dxr) < 5e-3 and _rel(dw, dwr) < 5e-3


@pytest.mark.parametrize("rows,H,width", [(257, 128, 640), (64, 1024, 1536)])
def test_rmsnorm_of_rows_inside_a_wider_buffer(rows, H, width):
    """Keys of a packed QKV buffer: rows of H elements whose stride is the packed width."""
    KC = _K()
    from kareus_b200.kernels import ref
    x = torch.randn(rows, width, device="cuda").bfloat16()[:, 128:128 + H]
    dy = torch.randn(rows, width, device="cuda").bfloat16()[:, :H]
    w = (1 + 0.1 * torch.randn(H, device="cuda")).bfloat16()
    y, rstd = KC.rmsnorm_fwd(x, w, 1e-6)
    yr, rr = ref.rmsnorm_fwd(x.float(), w.float(), 1e-6)
    assert _rel(y, yr) < 5e-3 and _rel(rstd, rr) < 1e-5
    dx, dw = KC.rmsnorm_bwd(dy, x, rstd, w)
    dxr, dwr = ref.rmsnorm_bwd(dy.float(), x.float(), rr, w.float())
    assert _rel(dx, dxr) < 5e-3 and _rel(dw, dwr) < 5e-3


def test_rope_strided_views_and_inverse():
    KC = _K()
    from kareus_b200.kernels import ref
    s, b, g, rep, d = 96, 2, 2, 3, 128
    base = torch.randn(s, b, g, (rep + 2) * d, device="cuda").bfloat16()
    orig = base.clone()
    q = base[..., : rep * d].unflatten(-1, (rep, d))
    k = base[..., rep * d:(rep + 1) * d]
    fr = ref.rope_table(s, d, 500000.0, device="cuda")
    want_q = ref.rope_apply(orig[..., : rep * d].unflatten(-1, (rep, d)).float(), fr)
    want_k = ref.rope_apply(orig[..., rep * d:(rep + 1) * d].float(), fr)
    KC.rope_inplace(q, k, fr)
    assert _rel(q, want_q) < 5e-3 and _rel(k, want_k) < 5e-3
    torch.testing.assert_close(base[..., (rep + 1) * d:], orig[..., (rep + 1) * d:])   # v untouched
    KC.rope_inplace(q, k, fr, inverse=True)
    assert _rel(base, orig) < 1e-2


def test_swiglu_dropout_add():
    KC = _K()
    from kareus_b200.kernels import ref
    x = torch.randn(300, 2 * 1024, device="cuda").bfloat16()
    dy = torch.randn(300, 1024, device="cuda").bfloat16()
    assert _rel(KC.swiglu_fwd(x), ref.swiglu_fwd(x.float())) < 5e-3
    assert _rel(KC.swiglu_bwd(dy, x), ref.swiglu_bwd(dy.float(), x.float())) < 5e-3
    # values bounded away from zero: the masks below are read off the outputs as "!= 0", and a normal
    # sample is exactly 0.0 once in a few hundred runs of this size
    a = (torch.rand(64, 3072, device="cuda") + 0.5).bfloat16()
    r = -(torch.rand(64, 3072, device="cuda") + 0.5).bfloat16()
    assert _rel(KC.dropout_add_fwd(a, r, 0.0, 0), a.float() + r.float()) < 5e-3
    assert _rel(KC.add(a, r), a.float() + r.float()) < 5e-3
    y = KC.dropout_add_fwd(a, torch.zeros_like(a), 0.25, 77)
    keep = (y != 0).float().mean().item()
    assert abs(keep - 0.75) < 0.02
    kept = y != 0
    assert _rel(y[kept], a.float()[kept] / 0.75) < 5e-3
    dx, dres = KC.dropout_add_bwd(r, 0.25, 77)
    torch.testing.assert_close((dx != 0), kept | False, msg="backward must regenerate the forward mask")
    assert dres is r or torch.equal(dres, r)


def test_embedding_and_cross_entropy():
    KC = _K()
    from kareus_b200.kernels import ref
    V, H, T = 1000, 256, 500
    w = torch.randn(V, H, device="cuda").bfloat16()
    tok = torch.randint(0, 2 * V, (50, 10), device="cuda")
    out = KC.embedding_fwd(tok, w, 500)
    torch.testing.assert_close(out, ref.embedding_fwd(tok, w, 500))
    gw = torch.zeros(V, H, device="cuda")
    gw_ref = torch.zeros(V, H, device="cuda")
    d = torch.randn(50, 10, H, device="cuda").bfloat16()
    KC.embedding_bwd(d, tok, gw, 500)
    ref.embedding_bwd(d, tok, gw_ref, 500)
    assert _rel(gw, gw_ref) < 1e-3
    logits = (3 * torch.randn(T, 16032, device="cuda")).bfloat16()
    tgt = torch.randint(0, 2 * 16032, (T,), device="cuda")
    m, s, t = KC.cross_entropy_local_stats(logits, tgt, 16032)
    mr, sr, tr = ref.cross_entropy_local_stats(logits, tgt, 16032)
    torch.testing.assert_close(m, mr)
    assert _rel(s, sr) < 1e-4 and _rel(t, tr) < 1e-6
    sc = torch.rand(T, device="cuda")
    want = ref.cross_entropy_finish(logits.clone().float(), tgt, 16032, mr, sr, sc)
    got = KC.cross_entropy_finish(logits.clone(), tgt, 16032, m, s, sc)
    assert _rel(got, want) < 1e-2


def test_adamw_and_sumsq():
    KC = _K()
    from kareus_b200.kernels import ref
    n = 1000003
    g = torch.randn(n, device="cuda")
    master = torch.randn(n, device="cuda")
    m = torch.zeros(n, device="cuda"); v = torch.zeros(n, device="cuda")
    p = master.bfloat16()
    mr, vr, wr = m.clone(), v.clone(), master.clone()
    for step in (1, 2):
        KC.adamw_step(p, g, m, v, master, 1e-3, 0.9, 0.98, 1e-8, 0.01, step, 0.5)
        ref.adamw_step(wr, g, mr, vr, wr, 1e-3, 0.9, 0.98, 1e-8, 0.01, step, 0.5)
    assert _rel(master, wr) < 1e-5 and _rel(m, mr) < 1e-5 and _rel(v, vr) < 1e-5
    assert _rel(p, wr) < 5e-3
    assert abs(KC.sumsq(g).item() / g.double().pow(2).sum().item() - 1) < 1e-4
    assert abs(KC.sumsq(p).item() / p.double().pow(2).sum().item() - 1) < 1e-3


@pytest.mark.parametrize("total", [0.0, 1e-14, 0.81, 1.0, 6.25, 1e30, float("inf"), float("nan")])
@pytest.mark.parametrize("clip", [1.0, 0.3])
def test_clip_scale_matches_torch_statements(total, clip):
    """Norm and clipping factor in one launch against the statements it replaces; one rounding each in fp32."""
    KC = _K()
    t = torch.tensor(total, device="cuda")
    norm, scale = KC.clip_scale(t, clip)
    want = t.sqrt()
    torch.testing.assert_close(norm, want, rtol=2e-7, atol=0, equal_nan=True)
    torch.testing.assert_close(scale, torch.clamp(clip / (want + 1e-6), max=1.0).reshape(1), rtol=5e-7, atol=0, equal_nan=True)


def test_bounded_wait_reports_timeout_status():
    """A status word records an expired wait and the context stays usable (host-side check of the
    status plumbing; no kernel is made to hang)."""
    KC = _K()
    w = KC.status_word("cuda")
    w.fill_(5)
    with pytest.raises(KC.KernelError):
        KC.check_status()
    KC.check_status()      # reset by the failed check
    assert torch.ones(4, device="cuda").sum().item() == 4


@pytest.mark.parametrize("s,b,g,rep", [(256, 1, 1, 1), (512, 2, 2, 3), (1000, 1, 1, 3), (4096, 1, 1, 2)])
def test_flash_attention_forward(s, b, g, rep):
    KC = _K()
    from kareus_b200.kernels import attention_cuda, ref
    if not attention_cuda.have_native():
        pytest.skip("native attention kernel not built")
    d = 128
    packed = torch.randn(s, b, g, (rep + 2) * d, device="cuda").bfloat16()
    q = packed[..., : rep * d].unflatten(-1, (rep, d))
    k = packed[..., rep * d:(rep + 1) * d]
    v = packed[..., (rep + 1) * d:]
    out, lse = attention_cuda.forward(q, k, v, d ** -0.5, True, 0, None)
    KC.check_status()
    want, lse_w = ref.attention_fwd(q.float(), k.float(), v.float(), d ** -0.5, True)
    assert _rel(out, want) < 1e-2
    torch.testing.assert_close(lse, lse_w, rtol=1e-3, atol=1e-3)


def test_flash_attention_forward_offsets():
    """Context-parallel style masks: query chunk at an offset against a key prefix."""
    KC = _K()
    from kareus_b200.kernels import attention_cuda, ref
    if not attention_cuda.have_native():
        pytest.skip("native attention kernel not built")
    d, c = 128, 192
    q = torch.randn(c, 2, 2, 2, d, device="cuda").bfloat16()
    k = torch.randn(4 * c, 2, 2, d, device="cuda").bfloat16()
    v = torch.randn(4 * c, 2, 2, d, device="cuda").bfloat16()
    for cid in (0, 2, 3):
        out, lse = attention_cuda.forward(q, k, v, d ** -0.5, True, cid * c, (cid + 1) * c)
        KC.check_status()
        want, lse_w = ref.attention_fwd(q.float(), k.float(), v.float(), d ** -0.5, True, cid * c, (cid + 1) * c)
        assert _rel(out, want) < 1e-2
        torch.testing.assert_close(lse, lse_w, rtol=1e-3, atol=1e-3)


@pytest.mark.parametrize("s,b,g,rep", [(256, 1, 1, 1), (512, 2, 2, 3), (1000, 1, 1, 3)])
def test_flash_attention_backward(s, b, g, rep):
    KC = _K()
    from kareus_b200.kernels import attention_cuda, ref
    if not (attention_cuda.have_native() and hasattr(KC.lib(), "kb_flash_attn_bwd")):
        pytest.skip("native attention backward not built")
    d = 128
    packed = torch.randn(s, b, g, (rep + 2) * d, device="cuda").bfloat16()
    q = packed[..., : rep * d].unflatten(-1, (rep, d))
    k = packed[..., rep * d:(rep + 1) * d]
    v = packed[..., (rep + 1) * d:]
    out, lse = attention_cuda.forward(q, k, v, d ** -0.5, True, 0, None)
    do = torch.randn_like(out)
    gbase = torch.full((s, b, g, (rep + 2) * d), float("nan"), device="cuda", dtype=torch.bfloat16)
    dq = gbase[..., : rep * d].unflatten(-1, (rep, d))
    dk = gbase[..., rep * d:(rep + 1) * d]
    dv = gbase[..., (rep + 1) * d:]
    attention_cuda.backward(do, q, k, v, out, lse, d ** -0.5, True, 0, None, (dq, dk, dv))
    KC.check_status()
    o_ref, lse_ref = ref.attention_fwd(q.float(), k.float(), v.float(), d ** -0.5, True)
    wq, wk, wv = ref.attention_bwd(do.float(), q.float(), k.float(), v.float(), o_ref, lse_ref, d ** -0.5, True)
    assert not torch.isnan(gbase.float()).any()
    assert _rel(dq, wq) < 2e-2 and _rel(dk, wk) < 2e-2 and _rel(dv, wv) < 2e-2


def test_flash_attention_backward_offsets():
    KC = _K()
    from kareus_b200.kernels import attention_cuda, ref
    if not (attention_cuda.have_native() and hasattr(KC.lib(), "kb_flash_attn_bwd")):
        pytest.skip("native attention backward not built")
    d, c = 128, 192
    q = torch.randn(c, 2, 2, 2, d, device="cuda").bfloat16()
    k = torch.randn(4 * c, 2, 2, d, device="cuda").bfloat16()
    v = torch.randn(4 * c, 2, 2, d, device="cuda").bfloat16()
    for cid in (0, 2):
        out, lse = attention_cuda.forward(q, k, v, d ** -0.5, True, cid * c, (cid + 1) * c)
        do = torch.randn_like(out)
        dq, dk, dv = attention_cuda.backward(do, q, k, v, out, lse, d ** -0.5, True, cid * c, (cid + 1) * c)
        KC.check_status()
        o_ref, lse_ref = ref.attention_fwd(q.float(), k.float(), v.float(), d ** -0.5, True, cid * c, (cid + 1) * c)
        wq, wk, wv = ref.attention_bwd(do.float(), q.float(), k.float(), v.float(), o_ref, lse_ref, d ** -0.5, True,
                                       cid * c, (cid + 1) * c)
        assert _rel(dq, wq) < 2e-2 and _rel(dk, wk) < 2e-2 and _rel(dv, wv) < 2e-2
        assert dk[(cid + 1) * c:].abs().max().item() == 0


# query tiles go in pairs once single tiles no longer fit the chip in one wave (148 SMs): an odd number of tiles, fewer
# rows than a tile, one row, a last tile of one row, and pairs whose halves see different numbers of key tiles
@pytest.mark.parametrize("sq,skv,b,g,rep,off,causal",
                         [(1, 1, 3, 2, 2, 0, True), (1, 1, 50, 2, 2, 0, True), (127, 127, 40, 2, 2, 0, True),
                          (129, 129, 20, 2, 3, 0, True), (641, 641, 9, 2, 3, 0, True), (1000, 1000, 4, 2, 3, 0, True),
                          (385, 1025, 12, 1, 4, 640, True), (385, 300, 12, 1, 4, 640, True), (300, 200, 20, 1, 4, -150, True),
                          (260, 131, 16, 2, 2, 0, False)])
def test_flash_attention_tile_pairs(sq, skv, b, g, rep, off, causal):
    KC = _K()
    from kareus_b200.kernels import attention_cuda, ref
    d = 128
    q = torch.randn(sq, b, g, rep, d, device="cuda").bfloat16()
    k = torch.randn(skv, b, g, d, device="cuda").bfloat16()
    v = torch.randn(skv, b, g, d, device="cuda").bfloat16()
    out, lse = attention_cuda.forward(q, k, v, d ** -0.5, causal, off, None)
    do = torch.randn_like(out)
    dq, dk, dv = attention_cuda.backward(do, q, k, v, out, lse, d ** -0.5, causal, off, None)
    KC.check_status()
    o_ref, lse_ref = ref.attention_fwd(q.float(), k.float(), v.float(), d ** -0.5, causal, off)
    wq, wk, wv = ref.attention_bwd(do.float(), q.float(), k.float(), v.float(), o_ref,
                                   lse_ref.masked_fill(lse_ref == float("-inf"), 0.0), d ** -0.5, causal, off)
    torch.testing.assert_close(lse, lse_ref, rtol=1e-3, atol=1e-3)
    # P and dS are rounded to bf16 (2^-9 each) and so are the results: below 1e-2 of the tensor.  One key leaves
    # dS = P (dP - delta) = 0 up to rounding, so dq and dk are compared with the size of their terms there.
    assert _rel(out, o_ref) < 1e-2 and _rel(dv, wv) < 1e-2
    if skv > 1:
        assert _rel(dq, wq) < 2e-2 and _rel(dk, wk) < 2e-2
    else:
        assert dq.abs().max() < 0.5 and dk.abs().max() < 2.0


@pytest.mark.parametrize("s,b,g,rep", [(459, 2, 2, 2), (640, 8, 4, 3)])
def test_flash_attention_backward_rounds_scaled_ds(s, b, g, rep):
    """dS carries the softmax scale (not a power of two) when it is rounded to bf16.  The same roundings in fp64: what is left
    is P and dS that fall on the other side of a rounding because of fp32 (1e-6 of the exponent, so about one in 2000) and the
    final rounding of sums that differ by that (one in 40, 2^-8 each): 6e-4 as a norm.  Rounding dS before the scale is 3e-3 away."""
    KC = _K()
    from kareus_b200.kernels import attention_cuda
    d = 128
    scale = d ** -0.5
    gen = torch.Generator(device="cuda").manual_seed(s)
    rnd = lambda *sh: torch.randn(*sh, device="cuda", generator=gen).bfloat16()
    q, k, v, do = rnd(s, b, g, rep, d), rnd(s, b, g, d), rnd(s, b, g, d), rnd(s, b, g * rep, d)
    out, lse = attention_cuda.forward(q, k, v, scale)
    dq, dk, dv = attention_cuda.backward(do, q, k, v, out, lse, scale)
    KC.check_status()
    q6, k6, v6, do6, o6 = (t.double() for t in (q, k, v, do.view(q.shape), out.view(q.shape)))
    hidden = torch.ones(s, s, device="cuda", dtype=torch.bool).triu(1)
    p = (torch.einsum("sbgrd,tbgd->bgrst", q6, k6) * scale - lse.double().view(b, g, rep, s, 1)).exp().masked_fill(hidden, 0)
    p = p.bfloat16().double()
    ds = p * (torch.einsum("sbgrd,tbgd->bgrst", do6, v6) - torch.einsum("sbgrd,sbgrd->bgrs", do6, o6)[..., None]) * scale
    ds = ds.bfloat16().double()
    assert _rel(dq, torch.einsum("bgrst,tbgd->sbgrd", ds, k6).bfloat16()) < 1.2e-3
    assert _rel(dk, torch.einsum("bgrst,sbgrd->tbgd", ds, q6).bfloat16()) < 1.2e-3
    assert _rel(dv, torch.einsum("bgrst,sbgrd->tbgd", p, do6).bfloat16()) < 1.2e-3


def test_flash_attention_backward_output_alignment():
    """The forward output may start on any 8-byte boundary; a gradient that TMA cannot read is refused."""
    KC = _K()
    from kareus_b200.kernels import attention_cuda
    s, b, g, rep, d = 200, 2, 2, 2, 128
    q = torch.randn(s, b, g, rep, d, device="cuda").bfloat16()
    k, v = torch.randn(2, s, b, g, d, device="cuda").bfloat16()
    out, lse = attention_cuda.forward(q, k, v, d ** -0.5)
    do = torch.randn_like(out)
    want = attention_cuda.backward(do, q, k, v, out, lse, d ** -0.5)
    moved = torch.empty(out.numel() + 4, device="cuda", dtype=out.dtype)[4:].view(out.shape).copy_(out)
    assert moved.data_ptr() % 16 == 8
    got = attention_cuda.backward(do, q, k, v, moved, lse, d ** -0.5)
    KC.check_status()
    # the same operands; dQ, dK and dV are summed in fp32 in an order that may differ, then rounded once (2^-9)
    for a, w in zip(got, want):
        assert _rel(a, w) < 2 ** -8
    do_moved = torch.empty(out.numel() + 4, device="cuda", dtype=out.dtype)[4:].view(out.shape).copy_(do)
    with pytest.raises(KC.KernelError):
        attention_cuda.backward(do_moved, q, k, v, out, lse, d ** -0.5)
    assert torch.ones(4, device="cuda").sum().item() == 4


# one query tile per CTA, whose even and odd key tiles go to different warps: one, two, three and many key tiles, shares of
# unequal length, a share whose keys are all hidden from some rows, query tiles that see nothing, no causal mask
@pytest.mark.parametrize("sq,skv,b,g,rep,off,causal",
                         [(1, 1, 1, 1, 1, 0, True), (128, 128, 2, 1, 2, 0, True), (129, 129, 1, 2, 3, 0, True),
                          (77, 260, 2, 1, 1, 183, True), (130, 384, 1, 1, 2, 254, True), (256, 512, 1, 2, 2, 127, True),
                          (200, 1500, 1, 1, 4, 1300, True), (384, 300, 1, 1, 2, -200, True), (100, 385, 3, 1, 2, 0, False),
                          (1111, 1111, 1, 2, 2, 0, True)])
def test_flash_attention_shared_query_tile(sq, skv, b, g, rep, off, causal):
    assert (sq + 127) // 128 * b * g * rep <= _K().sm_count()
    test_flash_attention_tile_pairs(sq, skv, b, g, rep, off, causal)


def test_flash_attention_shared_query_tile_keeps_nan():
    """A NaN score reaches its row's output whichever share of the keys it lies in, and no other row."""
    KC = _K()
    from kareus_b200.kernels import attention_cuda
    s, d = 300, 128
    q, v = torch.randn(s, 1, 1, 1, d, device="cuda").bfloat16(), torch.randn(s, 1, 1, d, device="cuda").bfloat16()
    k = torch.randn(s, 1, 1, d, device="cuda").bfloat16()
    for row in (0, 130, 299):
        bad = q.clone()
        bad[row, ..., 5] = float("nan")
        out, _ = attention_cuda.forward(bad, k, v, d ** -0.5)
        KC.check_status()
        nan = out.isnan().all(-1).flatten()
        assert nan[row] and nan.sum() == 1 and out.isnan().sum() == d


def test_gelu_geglu_kernels():
    from kareus_b200.engine.context import OpContext
    from kareus_b200.ops.activations import GegluOp, GeluOp, gelu_grad_ref, gelu_ref
    for op, width in ((GeluOp(), 1024), (GegluOp(), 2048)):
        x = torch.randn(200, width, device="cuda").bfloat16()
        ctx = OpContext()
        (y,) = op.forward(ctx, x)
        ctx2 = OpContext()
        (yr,) = op.forward(ctx2, x.float())
        assert _rel(y, yr) < 5e-3
        g = torch.randn_like(y)
        (dx,) = op.backward(ctx, g)
        (dxr,) = op.backward(ctx2, g.float())
        assert _rel(dx, dxr) < 5e-3


def test_layernorm_and_bias_kernels():
    from kareus_b200.engine.context import OpContext
    from kareus_b200.ops.extras import BiasOp, LayerNormOp
    for rows, H in ((300, 1024), (64, 3072)):
        x = torch.randn(rows, H, device="cuda").bfloat16()
        g = torch.randn(rows, H, device="cuda").bfloat16()
        ln = LayerNormOp(H, dtype=torch.bfloat16, device="cuda")
        ref = LayerNormOp(H, dtype=torch.float32, device="cuda")
        with torch.no_grad():
            ln.weight.mul_(1.25); ln.bias.add_(0.5); ref.weight.mul_(1.25); ref.bias.add_(0.5)
        c1, c2 = OpContext(), OpContext()
        (y,) = ln.forward(c1, x)
        (yr,) = ref.forward(c2, x.float())
        assert _rel(y, yr) < 5e-3
        (dx,) = ln.backward(c1, g)
        (dxr,) = ref.backward(c2, g.float())
        assert _rel(dx, dxr) < 1e-2
        assert _rel(ln.weight.main_grad, ref.weight.main_grad) < 1e-2 and _rel(ln.bias.main_grad, ref.bias.main_grad) < 1e-2
        b = BiasOp(H, dtype=torch.bfloat16, device="cuda")
        with torch.no_grad():
            b.bias.add_(0.75)
        (z,) = b.forward(OpContext(), x)
        assert _rel(z, x.float() + 0.75) < 5e-3
        b.backward(OpContext(), g)
        assert _rel(b.bias.main_grad, g.float().sum(0)) < 1e-2


@pytest.mark.parametrize("cp,c", [(2, 128), (2, 256), (4, 128)])
def test_chunked_attention_matches_reference(cp, c, b=2):
    """Context-parallel attention in one launch: K/V chunks in several buffers (here: local tensors that
    stand for the ranks' shards), two query chunks with their own positions, dK/dV scattered per chunk
    into a rank-ordered buffer.  Every rank's view is checked against the fp32 statement of the math."""
    from kareus_b200.kernels import attention_bwd_native, attention_native, ref
    from kareus_b200.parallel.ring_attention import chunk_owner, chunk_table
    KC = _K()
    g, rep, d = 2, 3, 128
    gen = torch.Generator(device="cuda").manual_seed(11 * cp + c)
    packed = [torch.randn(2 * c, b, g, (rep + 2) * d, device="cuda", generator=gen).bfloat16() for _ in range(cp)]
    qs = [p[..., : rep * d].unflatten(-1, (rep, d)) for p in packed]
    sources = [(p[..., rep * d:(rep + 1) * d], p[..., (rep + 1) * d:]) for p in packed]
    table = chunk_table(cp, c)
    dk_base = [r * 4 * c + half * c for r, half in (chunk_owner(j, cp) for j in range(2 * cp))]
    dv_base = [x + 2 * c for x in dk_base]
    f32 = [(k.float(), v.float()) for k, v in sources]
    for rank in range(cp):
        q = qs[rank]
        qpos = [rank * c, (2 * cp - 1 - rank) * c]
        out, lse = attention_native.forward_chunked(q, sources, table, c, qpos, d ** -0.5)
        KC.check_status()
        want, lse_w = ref.attention_fwd_chunked(q.float(), f32, table, c, qpos, d ** -0.5)
        assert _rel(out, want.reshape(out.shape)) < 2e-2, ("fwd", rank)
        torch.testing.assert_close(lse, lse_w.reshape(lse.shape), rtol=1e-2, atol=2e-2)
        do = torch.randn(out.shape, device="cuda", generator=gen).bfloat16()
        dq = torch.empty_like(q)
        dkv = torch.full((cp * 4 * c, b, g, d), float("nan"), device="cuda", dtype=torch.bfloat16)
        attention_bwd_native.backward_chunked(do, q, sources, table, c, qpos, out, lse, d ** -0.5, dq, dkv, dk_base,
                                              dv_base)
        KC.check_status()
        wq, wk, wv = ref.attention_bwd_chunked(do.float(), q.float(), f32, table, c, qpos, want, lse_w, d ** -0.5)
        assert _rel(dq, wq.reshape(dq.shape)) < 3e-2, ("dq", rank)
        assert not torch.isnan(dkv.float()).any()            # every row of the collective's input was written
        for j in range(2 * cp):
            assert _rel(dkv[dk_base[j]:dk_base[j] + c], wk[j * c:(j + 1) * c]) < 3e-2 or \
                wk[j * c:(j + 1) * c].abs().max() == 0, ("dk", rank, j)
            assert _rel(dkv[dv_base[j]:dv_base[j] + c], wv[j * c:(j + 1) * c]) < 3e-2 or \
                wv[j * c:(j + 1) * c].abs().max() == 0, ("dv", rank, j)
            if wk[j * c:(j + 1) * c].abs().max() == 0:      # chunk no local query can see: exact zeros
                assert dkv[dk_base[j]:dk_base[j] + c].abs().max() == 0


# more than 148 query tiles, so that they go in pairs: both chunks in one pair, and a middle pair of three tiles per chunk
@pytest.mark.parametrize("cp,c,b", [(2, 128, 13), (2, 384, 6)])
def test_chunked_attention_tile_pairs(cp, c, b):
    assert 2 * c // 128 * 6 * b > _K().sm_count()
    test_chunked_attention_matches_reference(cp, c, b)


# enough (batch, group) pairs that the backward gives all query heads of a group to one CTA, which writes dK/dV itself
def test_attention_backward_merged_heads():
    test_chunked_attention_matches_reference(2, 128, b=10)
    test_flash_attention_backward(640, 8, 4, 3)
    test_flash_attention_backward(300, 20, 3, 1)


@pytest.mark.parametrize("M,N,K", [(256, 384, 512), (1000, 328, 200), (4096, 4096, 2048)])
@pytest.mark.parametrize("activation", [None, "gelu"])
def test_gemm_bias_activation_epilogue(M, N, K, activation):
    """Bias and GELU applied to the accumulator inside the GEMM kernel."""
    KC = _K()
    from kareus_b200.kernels import ref
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g).bfloat16()
    got = KC.gemm(a, w, bias=bias, activation=activation)
    KC.check_status()
    want = ref.bias_act(a.float() @ w.float().t(), bias.float(), activation)
    assert _rel(got, want) < 1e-2
    only_act = KC.gemm(a, w, activation=activation)
    assert _rel(only_act, ref.bias_act(a.float() @ w.float().t(), None, activation)) < 1e-2


# a warp per row from 148 * 40 rows on; 4, 8, 12 or 16 vectors a lane, last vectors of a row missing in some lanes
@pytest.mark.parametrize("rows,H", [(5919, 1032), (5920, 512), (5923, 1032), (5950, 2056), (5921, 3072), (5927, 4088), (5920, 4096),
                                    (5920, 4104)])
def test_rmsnorm_forward_rows(rows, H):
    KC = _K()
    from kareus_b200.kernels import ref
    x, w = torch.randn(rows, H, device="cuda").bfloat16(), torch.randn(H, device="cuda").bfloat16()
    y, rstd = KC.rmsnorm_fwd(x, w, 1e-5)
    want, rstd_w = ref.rmsnorm_fwd(x.double(), w.double(), 1e-5)
    assert _rel(y, want) < 3e-3 and _rel(rstd, rstd_w) < 1e-5            # bf16 rounding of the result: 2^-9


@pytest.mark.parametrize("s,b,g,rep,d", [(1, 1, 1, 1, 128), (37, 3, 2, 3, 128), (5, 2, 8, 2, 64), (9, 1, 3, 1, 256), (7, 2, 2, 2, 8),
                                         (6, 2, 2, 2, 96)])
def test_rmsnorm_heads_views(s, b, g, rep, d):
    KC = _K()
    from kareus_b200.kernels import ref
    packed = torch.randn(s, b, g, (rep + 2) * d, device="cuda").bfloat16()
    q = packed[..., : rep * d].unflatten(-1, (rep, d))
    w = torch.randn(d, device="cuda").bfloat16()
    for x in (q, packed[..., rep * d:(rep + 1) * d], q.permute(1, 0, 3, 2, 4), q.contiguous(), packed[..., d:2 * d].expand(s, b, g, d)):
        y, rstd = KC.rmsnorm_fwd_heads(x, w, 1e-6)
        want, rstd_w = ref.rmsnorm_fwd(x.reshape(-1, d).double(), w.double(), 1e-6)
        assert y.shape == x.shape and y.is_contiguous()
        assert _rel(y.reshape(-1, d), want) < 3e-3 and _rel(rstd, rstd_w) < 1e-5


@pytest.mark.parametrize("rows,V", [(3, 8), (5, 16376), (2, 16384), (4, 16392), (3, 50264), (2, 4096), (3, 4000), (2, 4104),
                                    (9, 50257), (9, 1003), (3, 5)])
def test_cross_entropy_vector_groups(rows, V):
    """Rows around multiples of the two vectors a thread takes at once, with hidden logits."""
    KC = _K()
    logits = (4 * torch.randn(rows, V, device="cuda")).bfloat16()
    logits[0, : V // 2] = float("-inf")
    tgt = torch.randint(0, V, (rows,), device="cuda")
    tgt[0], tgt[-1] = V - 1, V - 2
    m, se, tl = KC.cross_entropy_local_stats(logits, tgt, 0)
    x = logits.double()
    assert torch.equal(m.double(), x.max(-1).values)
    assert _rel(m.double() + se.double().log() - tl.double(), x.logsumexp(-1) - x.gather(1, tgt[:, None])[:, 0]) < 1e-5
    sc = torch.rand(rows, device="cuda")
    want = (x.softmax(-1) - torch.nn.functional.one_hot(tgt, V)) * sc.double()[:, None]
    KC.cross_entropy_finish(logits, tgt, 0, m, se, sc)
    assert _rel(logits, want) < 4e-3


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,Kd", [(300, 1093, 64), (5000, 1093, 1040), (300, 9, 136), (129, 65, 64), (300, 3, 64), (257, 1030, 520)])
def test_gemm_leaves_the_columns_behind_its_output_alone(M, N, Kd, dtype):
    KC = _K()
    a, b = torch.randn(M, Kd, device="cuda").bfloat16(), torch.randn(N, Kd, device="cuda").bfloat16()
    wide = torch.full((M, (N + 7) // 8 * 8 + 8), 7.0, device="cuda", dtype=dtype)
    KC.gemm(a, b, out=wide[:, :N])
    assert bool((wide[:, N:] == 7.0).all())
    assert _rel(wide[:, :N], a.double() @ b.double().t()) < (2e-3 if dtype == torch.bfloat16 else 1e-5)


@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, False)])
@pytest.mark.parametrize("M,N,Kd,ks,bn", [(1, 8, 1024, 4, 64), (130, 200, 1032, 2, 128), (300, 1000, 1344, 5, 256), (72, 328, 4104, 7, 192),
                                          (5000, 1096, 1040, 3, 256)])
def test_bf16_outputs_in_parts_of_k(M, N, Kd, ks, bn, ta, tb):
    """Rows, columns and steps that fill no tile and no part; whole tiles before split ones in the last shape."""
    import kareus_b200.kernels as KK
    KC = _K()
    a, b = torch.randn(*((Kd, M) if ta else (M, Kd)), device="cuda").bfloat16(), torch.randn(*((N, Kd) if tb else (Kd, N)), device="cuda").bfloat16()
    if ta and M % 8:
        a = torch.cat([a, a.new_zeros(Kd, 8 - M % 8)], 1)[:, :M]
    want = (a.double().t() if ta else a.double()) @ (b.double().t() if tb else b.double())
    try:
        KC.lib().kb_gemm_parts_force(1, 0)
        one = _rel(KK.gemm(a, b, trans_a=ta, trans_b=tb), want)
        KC.lib().kb_gemm_parts_force(ks, bn)
        assert KC.lib().kb_gemm_scratch_floats(M, N, Kd, 0 if tb else 1, 0) > 0
        got = [KK.gemm(a, b, trans_a=ta, trans_b=tb) for _ in range(3)]
        odd = torch.zeros(M, N + 8, device="cuda", dtype=torch.bfloat16)          # rows of a wider output
        got.append(KC.gemm(a, b, trans_a=ta, trans_b=tb, out=odd[:, :N]))
        if tb:                                                                    # a length that is no multiple of a vector
            got.append(KC.gemm(a, b, out=torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)))
            KC.gemm(a, b[:N - 3], out=odd[:, :N - 3])
    finally:
        KC.lib().kb_gemm_parts_force(0, 0)
    torch.cuda.synchronize()
    KC.check_status()
    assert not odd[:, N:].any() and torch.equal(odd[:, :N], got[0])
    for g in got:
        assert torch.equal(g, got[0]) and _rel(g, want) < 1.01 * one
    assert KC.lib().kb_gemm_scratch_floats(M, N, 64, 0, 0) == 0


@pytest.mark.parametrize("M,N,Kd", [(1, 8, 64), (130, 1000, 72), (300, 2048, 520), (257, 16392, 128), (513, 4104, 1032), (128, 64, 8)])
def test_logits_with_row_statistics(M, N, Kd):
    """Statistics from the epilogue of the product against those of the product, with and without storing it."""
    import kareus_b200.kernels as KK
    KC = _K()
    x, w = torch.randn(M, Kd, device="cuda").bfloat16(), (torch.randn(N, Kd, device="cuda") / Kd ** 0.5).bfloat16()
    start = 40
    tgt = torch.randint(0, N + 2 * start, (M,), device="cuda")
    tgt[0], tgt[-1] = start, start + N - 1
    weight = torch.rand(M, device="cuda")
    logits, m, se, tl, loss = KK.linear_cross_entropy_stats(x, w, tgt, start, weight=weight)
    torch.cuda.synchronize()
    KC.check_status()
    assert _rel(logits, KC.gemm(x, w)) < 2e-3              # another order of summation moves some bf16 roundings
    mr, sr, tr = KC.cross_entropy_local_stats(logits, tgt, start)
    assert torch.equal(m, mr) and torch.equal(tl, tr)
    assert _rel(se.double(), (logits.double() - m.double()[:, None]).exp().sum(-1)) < 2e-6
    want = ((m.double() + se.double().log() - tl.double()) * weight.double()).sum()
    assert abs(loss.double() - want) < 1e-5 * ((m.double() + se.double().log() - tl.double()).abs() * weight.double()).sum()
    none, m2, se2, tl2, no_loss = KK.linear_cross_entropy_stats(x, w, tgt, start, store=False)
    assert none is None and no_loss is None
    assert torch.equal(m, m2) and torch.equal(se, se2) and torch.equal(tl, tl2)
    x[0] = float("nan")
    _, m, se, _, _ = KK.linear_cross_entropy_stats(x, w, tgt, start, store=False)
    assert se[0].isnan() and (M == 1 or not se[1:].isnan().any())


@pytest.mark.parametrize("M,N,Kd", [(2003, 16392, 64), (5001, 2056, 136)])
def test_row_statistics_alone_over_many_tiles(M, N, Kd):
    """Many tiles for each pair of SMs and no product to store: nothing but the statistics stands between two reads of TMEM, and
    rows, columns and targets inside and outside of a tile part the lanes of a warp."""
    import kareus_b200.kernels as KK
    KC = _K()
    x, w = torch.randn(M, Kd, device="cuda").bfloat16(), (torch.randn(N, Kd, device="cuda") / Kd ** 0.5).bfloat16()
    tgt = torch.randint(-N // 2, 2 * N, (M,), device="cuda")
    logits, m, se, tl, _ = KK.linear_cross_entropy_stats(x, w, tgt, 0)
    for _ in range(5):
        none, m2, se2, tl2, _ = KK.linear_cross_entropy_stats(x, w, tgt, 0, store=False)
        assert none is None and torch.equal(m, m2) and torch.equal(se, se2) and torch.equal(tl, tl2)
    torch.cuda.synchronize()
    KC.check_status()
    mr, _, tr = KC.cross_entropy_local_stats(logits, tgt, 0)
    assert torch.equal(m, mr) and torch.equal(tl, tr)


@pytest.mark.parametrize("M,F,Kd", [(1, 8, 8), (130, 72, 64), (257, 200, 520), (513, 1000, 1032), (128, 128, 64), (300, 328, 72)])
def test_swiglu_in_gemm_epilogues(M, F, Kd):
    """Against the two kernels of its own: the same roundings, so errors against 64 bits as large as theirs."""
    import kareus_b200.kernels as KK
    from kareus_b200.kernels import ref
    KC = _K()
    x, w1 = torch.randn(M, Kd, device="cuda").bfloat16(), (3 * torch.randn(2 * F, Kd, device="cuda") / Kd ** 0.5).bfloat16()
    dy, w2 = torch.randn(M, Kd, device="cuda").bfloat16(), (torch.randn(Kd, F, device="cuda") / Kd ** 0.5).bfloat16()
    x[-1] *= 40                                           # activations far out on both sides
    try:
        KC.lib().kb_gemm_swiglu_force(1)
        y, h = KK.linear_swiglu(x, w1)
        none, h2 = KK.linear_swiglu(x, w1, store=False)
        dx = KK.linear_swiglu_dgrad(dy, w2, y)
    finally:
        KC.lib().kb_gemm_swiglu_force(0)
    torch.cuda.synchronize()
    KC.check_status()
    assert none is None and torch.equal(h, h2)
    assert _rel(y, KC.gemm(x, w1)) < 2e-3                 # another order of summation moves some bf16 roundings
    want = ref.swiglu_fwd(y.double())
    assert _rel(h, want) < 1.01 * _rel(KC.swiglu_fwd(y), want) + 1e-7
    dh = KC.gemm(dy, w2, trans_b=False)
    sep, want = KC.swiglu_bwd(dh, y), ref.swiglu_bwd((dy.double() @ w2.double()), y.double())
    assert _rel(dx, want) < 1.02 * _rel(sep, want) + 1e-7


@pytest.mark.parametrize("H", [8, 1032, 3072])
def test_embedding_backward_vectors(H):
    KC = _K()
    tok = torch.randint(0, 50, (3, 41), device="cuda")
    dout = torch.randn(3, 41, H, device="cuda").bfloat16()
    for gw in (torch.zeros(30, H, device="cuda"), torch.zeros(30 * H + 1, device="cuda")[1:].view(30, H)):
        KC.embedding_bwd(dout, tok, gw, 10)
        keep = (tok >= 10) & (tok < 40)
        want = torch.zeros(30, H, device="cuda", dtype=torch.float64).index_add_(0, tok[keep] - 10, dout[keep].double())
        assert _rel(gw, want) < 1e-6
    x, s = torch.randn(5, H, device="cuda").bfloat16(), torch.tensor(0.3333, device="cuda")
    assert torch.equal(KC.scale(x, s), x * s.to(x.dtype))

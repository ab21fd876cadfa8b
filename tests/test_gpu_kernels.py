"""Raw sm_100a kernels against plain PyTorch fp32 references (GPU tier).

Covers the tcgen05 GEMM in all four operand-major combinations, the fused tile-resident
NS5 kernel, the optimizer multi-tensor kernels, the HBM-bound model kernels and flash
attention forward/backward.  Mirrors the role of the reference's
tests/integration/test_kernels.py (kernels vs pure torch at bf16 tolerance).
"""

import math
import struct

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ext():
    from himuon_b200._ext import ext

    return ext()


def _assert_status_clean():
    assert _ext().status(True) == 0, "a bounded device wait ran out (status word set)"


def _close(out, ref, atol, rtol):
    out = out.float()
    ref = ref.float()
    err = (out - ref).abs()
    tol = atol + rtol * ref.abs()
    # Every element is checked.  A few per hundred thousand may exceed the tolerance (rounding of a value that sits on
    # a bf16 boundary), none may exceed it four-fold, and no single row or column may collect the outliers: a wrong
    # boundary row or tile edge fails even when it is a vanishing share of the matrix.
    over = err > tol
    bad = over.float().mean().item()
    assert bad <= 1e-5, f"{bad:.4%} elements out of tolerance; max err {err.max().item():.4g}, ref max {ref.abs().max().item():.4g}"
    worst = (err / tol).max().item()
    assert worst <= 4.0, f"an element is {worst:.1f}x outside the tolerance (max err {err.max().item():.4g})"
    if over.dim() >= 2 and over.any():
        per_row = over.reshape(-1, over.shape[-1]).float().mean(dim=1).max().item()
        per_col = over.reshape(-1, over.shape[-2], over.shape[-1]).float().mean(dim=1).max().item()
        assert per_row <= 0.02 and per_col <= 0.02, f"outliers concentrate in one row/column ({per_row:.2%} / {per_col:.2%})"


@pytest.mark.parametrize("trans_a,trans_b", [(False, True), (False, False), (True, False), (True, True)])
@pytest.mark.parametrize("shape", [(256, 512, 384), (128, 128, 64), (200, 328, 136), (1024, 2560, 1024), (520, 776, 2304),
                                   (2048, 2560, 4096)])
def test_gemm_majors(trans_a, trans_b, shape):
    M, N, K = shape
    torch.manual_seed(0)
    a = torch.randn((K, M) if trans_a else (M, K), device="cuda", dtype=torch.bfloat16)
    b = torch.randn((N, K) if trans_b else (K, N), device="cuda", dtype=torch.bfloat16)
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    _ext().gemm(a, b, out, None, trans_a, trans_b, 1.0, 0.0, False, 0)
    ref = (a.float().t() if trans_a else a.float()) @ (b.float().t() if trans_b else b.float())
    torch.cuda.synchronize()
    _assert_status_clean()
    _close(out, ref, atol=0.25, rtol=2e-2)


def test_gemm_batched_epilogue_and_fp32_accumulate():
    torch.manual_seed(1)
    B, M, N, K = 5, 256, 320, 192
    a = torch.randn(B, M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(B, N, K, device="cuda", dtype=torch.bfloat16)
    aux = torch.randn(B, M, N, device="cuda", dtype=torch.bfloat16)
    out = torch.empty_like(aux)
    _ext().gemm(a, b, out, aux, False, True, 0.5, -1.5, False, 0)
    ref = 0.5 * torch.bmm(a.float(), b.float().transpose(1, 2)) - 1.5 * aux.float()
    _close(out, ref, atol=0.25, rtol=2e-2)
    # fp32 output accumulating into itself (weight-gradient accumulation)
    acc = torch.randn(B, M, N, device="cuda", dtype=torch.float32)
    ref2 = acc.clone() + torch.bmm(a.float(), b.float().transpose(1, 2))
    _ext().gemm(a, b, acc, acc, False, True, 1.0, 1.0, False, 0)
    torch.cuda.synchronize()
    _assert_status_clean()
    _close(acc, ref2, atol=1e-2, rtol=1e-3)


@pytest.mark.parametrize("M,N,K", [(2048, 2560, 2560), (2000, 2560, 9728), (2560, 2304, 2048), (11520, 2560, 4096)])
def test_gemm_pair_split_tail(M, N, K):
    """Shapes whose last wave of 256x256 tiles is mostly idle: the tail tiles are cut along K, summed in an fp32
    scratch by TMA reductions and finished by a second kernel.  Run twice (the scratch must come back zeroed), with
    the aux epilogue and with fp32 accumulation into the output."""
    torch.manual_seed(2)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    aux = torch.randn(M, N, device="cuda", dtype=torch.bfloat16)
    ref = a.float() @ b.float().t()
    for _ in range(2):
        out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
        _ext().gemm(a, b, out, None, False, True, 1.0, 0.0, False, 0)
        _close(out, ref, atol=0.3, rtol=2e-2)
        out2 = torch.empty_like(out)
        _ext().gemm(a, b, out2, aux, False, True, 0.5, -1.5, False, 0)
        _close(out2, 0.5 * ref - 1.5 * aux.float(), atol=0.3, rtol=2e-2)
    acc = torch.randn(M, N, device="cuda", dtype=torch.float32)
    ref2 = acc + ref
    _ext().gemm(a, b, acc, acc, False, True, 1.0, 1.0, False, 0)
    torch.cuda.synchronize()
    _assert_status_clean()
    _close(acc, ref2, atol=2e-2, rtol=1e-3)


@pytest.mark.parametrize("M,N,K", [(2048, 2560, 2048), (4096, 2560, 2048), (2560, 9728, 2048), (2304, 2560, 4096),
                                   (19456, 2560, 2048)])
def test_gemm_pair_stream_k_accumulate(M, N, K):
    """fp32 `C += A^T B` (the weight-gradient GEMM) on shapes whose tile count does not fill the last wave: the work is
    dealt out as contiguous (tile, k-block) ranges and every partial tile is added into C by TMA reductions."""
    torch.manual_seed(3)
    a = torch.randn(K, M, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(K, N, device="cuda", dtype=torch.bfloat16)
    acc = torch.randn(M, N, device="cuda", dtype=torch.float32)
    ref = acc.clone()
    prod = a.float().t() @ b.float()
    for i in range(2):
        _ext().gemm(a, b, acc, acc, True, False, 1.0, 1.0, False, 0)
        ref += prod
        _close(acc, ref, atol=2e-2, rtol=1e-3)
    torch.cuda.synchronize()
    _assert_status_clean()
    # bf16 accumulator (the banks' gradient buffers): every partial is rounded to bf16 and added in bf16
    acc16 = torch.randn(M, N, device="cuda", dtype=torch.float32).mul_(30).bfloat16()
    ref16 = acc16.float()
    for i in range(2):
        _ext().gemm(a, b, acc16, acc16, True, False, 1.0, 1.0, False, 0)
        ref16 = (ref16 + prod).bfloat16().float()
    torch.cuda.synchronize()
    _assert_status_clean()
    _close(acc16, ref16, atol=2.0, rtol=2e-2)


def _ns_ref(x, steps=5):
    a, b, c = 3.4445, -4.7750, 2.0315
    X = x.float()
    X = X / (X.norm(dim=(-2, -1), keepdim=True) + 1e-7)
    X = X.bfloat16().float()
    for _ in range(steps):
        A = (X @ X.transpose(-2, -1)).bfloat16().float()
        Bm = (c * (A @ A) + b * A).bfloat16().float()
        X = ((Bm @ X).bfloat16().float() + a * X).bfloat16().float()
    return X


def _well_conditioned(B, m, n, seed=0):
    g = torch.Generator(device="cpu").manual_seed(seed)
    x = torch.randn(B, m, n, generator=g)
    U, _, Vh = torch.linalg.svd(x, full_matrices=False)
    s = torch.linspace(0.8, 1.2, min(m, n))
    return (U * s) @ Vh


@pytest.mark.parametrize("m,n", [(128, 128), (64, 128), (64, 256), (32, 64), (128, 256)])
def test_ns5_fused(m, n):
    x = _well_conditioned(37, m, n).cuda().bfloat16()
    out = torch.empty_like(x)
    _ext().ns5_fused(x, out, 5, 1e-7)
    torch.cuda.synchronize()
    _assert_status_clean()
    _close(out, _ns_ref(x), atol=4e-2, rtol=4e-2)
    # an all-zero (padding) tile stays exactly zero
    z = torch.zeros(3, m, n, device="cuda", dtype=torch.bfloat16)
    oz = torch.empty_like(z)
    _ext().ns5_fused(z, oz, 5, 1e-7)
    assert oz.abs().max().item() == 0.0


def test_ns_normalize():
    x = torch.randn(9, 256, 512, device="cuda", dtype=torch.bfloat16)
    x[3].zero_()
    ref = x.float() / (x.float().norm(dim=(1, 2), keepdim=True) + 1e-7)
    _ext().ns_normalize(x, 9, 256 * 512, 1e-7)
    _close(x, ref, atol=1e-4, rtol=1e-2)
    assert x[3].abs().max().item() == 0.0


def test_momentum_tile_and_untile_apply():
    e = _ext()
    torch.manual_seed(0)
    Th = Tw = 128
    shapes = [(256, 384), (200, 300), (64, 64)]
    mu, lr, wd = 0.95, 0.02, 0.1
    grads = [torch.randn(s, device="cuda", dtype=torch.bfloat16) for s in shapes]
    moms = [torch.randn(s, device="cuda", dtype=torch.bfloat16) * 0.1 for s in shapes]
    params = [torch.randn(s, device="cuda", dtype=torch.bfloat16) for s in shapes]
    moms_ref = [m.clone() for m in moms]
    params_ref = [p.clone() for p in params]
    sz = e.sizeof_entries()
    assert sz[0] == 104 and sz[1] == 48 and sz[2] == 56
    mom_tab, app_tab = b"", b""
    tile_base, unit = 0, 0
    metas = []
    for g, m, p in zip(grads, moms, params):
        h, w = g.shape
        R, C = math.ceil(h / Th), math.ceil(w / Tw)
        mom_tab += struct.pack("<8QQq6i", g.data_ptr(), 0, 0, 0, 0, 0, 0, 0, m.data_ptr(), tile_base, h, w, R, C, unit, g.stride(0))
        app_tab += struct.pack("<Qq6ifi", p.data_ptr(), tile_base, h, w, R, C, unit, 0, 0.2 * math.sqrt(max(Th, Tw)), p.stride(0))
        metas.append((tile_base, R, C))
        tile_base += R * C
        unit += e.momentum_tile_units(R, C, Th)
    mom_dev = torch.frombuffer(bytearray(mom_tab), dtype=torch.uint8).cuda()
    app_dev = torch.frombuffer(bytearray(app_tab), dtype=torch.uint8).cuda()
    tiles = torch.full((tile_base, Th, Tw), 7.0, device="cuda", dtype=torch.bfloat16)
    e.momentum_tile(mom_dev, len(shapes), unit, Th, Tw, tiles, mu, True, 1.0, 1, False)
    for g, m_ref, m, (tb, R, C) in zip(grads, moms_ref, moms, metas):
        buf = m_ref.mul(mu).add(g)
        nes = g.add(buf, alpha=mu)
        _close(m, buf, atol=1e-2, rtol=1e-2)
        h, w = g.shape
        padded = torch.zeros(R * Th, C * Tw, device="cuda", dtype=torch.bfloat16)
        padded[:h, :w] = nes
        ref_tiles = padded.view(R, Th, C, Tw).permute(0, 2, 1, 3).reshape(R * C, Th, Tw)
        _close(tiles[tb:tb + R * C], ref_tiles, atol=2e-2, rtol=1e-2)
    hyper = torch.tensor([lr, wd], device="cuda", dtype=torch.float32)
    e.untile_apply(app_dev, len(shapes), unit, Th, Tw, tiles, hyper, False)
    for p_ref, p, (tb, R, C) in zip(params_ref, params, metas):
        h, w = p.shape
        u = tiles[tb:tb + R * C].view(R, C, Th, Tw).permute(0, 2, 1, 3).reshape(R * Th, C * Tw)[:h, :w]
        ref = p_ref.float() * (1 - lr * wd) - lr * 0.2 * math.sqrt(128) * u.float()
        _close(p, ref, atol=2e-2, rtol=1e-2)


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_adamw_multi(mode):
    e = _ext()
    torch.manual_seed(0)
    sizes = [5000, 17, 4096 * 3]
    lr, wd, b1, b2, eps = 1e-2, 0.1, 0.9, 0.95, 1e-8
    ps = [torch.randn(n, device="cuda") for n in sizes]
    gs = [torch.randn(n, device="cuda") for n in sizes]
    ms = [torch.zeros(n, device="cuda") for n in sizes]
    vs = [torch.zeros(n, device="cuda") for n in sizes]
    ref_p = [p.clone() for p in ps]
    tab, unit = b"", 0
    for p, g, m, v in zip(ps, gs, ms, vs):
        tab += struct.pack("<4Qqq2i", p.data_ptr(), g.data_ptr(), m.data_ptr(), v.data_ptr(), p.numel(), unit, 0, 0)
        unit += (p.numel() + 4095) // 4096
    dev = torch.frombuffer(bytearray(tab), dtype=torch.uint8).cuda()
    hyper = torch.tensor([lr, wd, b1, b2, eps, 0, 0, 0], device="cuda", dtype=torch.float32)
    step = torch.zeros((), device="cuda", dtype=torch.float32)
    rm = [torch.zeros_like(p) for p in ps]
    rv = [torch.zeros_like(p) for p in ps]
    for t in range(1, 4):
        e.adamw_multi(dev, len(sizes), unit, hyper, step, mode, True, True)
        e.adamw_step_advance(step)
        bc1, bc2 = 1 - b1 ** t, 1 - b2 ** t
        for p, g, m, v in zip(ref_p, gs, rm, rv):
            m.lerp_(g, 1 - b1)
            v.lerp_(g * g, 1 - b2)
            if mode == 0:
                u = (m / bc1) / (v.sqrt() / math.sqrt(bc2) + eps)
                p.mul_(1 - lr * wd).sub_(lr * u)
            elif mode == 1:
                u = m / (eps + v.sqrt())
                p.mul_(1 - lr * wd).sub_(u * (lr / (bc1 / math.sqrt(bc2))))
            else:
                p.sub_(m / (v.sqrt() + eps) * (lr * math.sqrt(bc2) / bc1))
                p.sub_(p * (lr * wd))
    assert step.item() == 3.0
    for p, r in zip(ps, ref_p):
        _close(p, r, atol=1e-5, rtol=1e-4)


def test_rmsnorm_fwd_bwd():
    e = _ext()
    torch.manual_seed(0)
    rows, cols = 777, 2560
    x = torch.randn(rows, cols, device="cuda", dtype=torch.bfloat16)
    w = (1 + 0.1 * torch.randn(cols, device="cuda")).bfloat16()
    dy = torch.randn(rows, cols, device="cuda", dtype=torch.bfloat16)
    y = torch.empty_like(x)
    rstd = torch.empty(rows, device="cuda")
    e.rmsnorm_fwd(x, w, y, rstd, 1e-6)
    xr = x.float().requires_grad_(True)
    wr = w.float().requires_grad_(True)
    yr = xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-6) * wr
    yr.backward(dy.float())
    _close(y, yr, atol=2e-2, rtol=2e-2)
    dx = torch.empty_like(x)
    dw = torch.zeros(cols, device="cuda")
    e.rmsnorm_bwd(dy, x, w, rstd, dx, dw)
    _close(dx, xr.grad, atol=2e-2, rtol=2e-2)
    _close(dw, wr.grad, atol=0.3, rtol=2e-2)


def _rope_table(S, theta=1e6, D=128):
    inv = 1.0 / (theta ** (torch.arange(0, D, 2, dtype=torch.float32) / D))
    ang = torch.arange(S, dtype=torch.float32)[:, None] * inv[None, :]
    return torch.stack([ang.cos(), ang.sin()], dim=-1).contiguous()  # (S, 64, 2)


def test_add_rmsnorm_fwd_bwd():
    """Fused residual add + RMSNorm: both outputs and the joined gradient against plain PyTorch in fp32."""
    from himuon_b200 import ops

    torch.manual_seed(5)
    T, H = 300, 2560
    x = torch.randn(T, H, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    d = torch.randn(T, H, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (1 + 0.1 * torch.randn(H, device="cuda")).bfloat16().requires_grad_(True)
    h, y = ops.add_rmsnorm(x, d, w, 1e-6)
    gh = torch.randn_like(h)
    gy = torch.randn_like(y)
    gx, gd, gw = torch.autograd.grad((h, y), (x, d, w), (gh, gy))
    xr, dr, wr = x.detach().float().requires_grad_(True), d.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    # value rounded to bf16 like the kernel's h, gradient of the plain sum
    hr = (xr + dr) + ((xr + dr).bfloat16().float() - (xr + dr)).detach()
    yr = hr * torch.rsqrt(hr.pow(2).mean(-1, keepdim=True) + 1e-6) * wr
    rgx, rgd, rgw = torch.autograd.grad((hr, yr), (xr, dr, wr), (gh.float(), gy.float()), retain_graph=True)
    _close(h, hr.detach(), atol=1e-2, rtol=1e-2)
    _close(y, yr.detach(), atol=3e-2, rtol=2e-2)
    _close(gx, rgx, atol=5e-2, rtol=3e-2)
    assert gd.data_ptr() == gx.data_ptr()                    # one gradient tensor serves both inputs
    _close(gw, rgw, atol=0.5, rtol=3e-2)
    # only the normalised output used (final norm of the model)
    h2, y2 = ops.add_rmsnorm(x, d, w, 1e-6)
    gx2, = torch.autograd.grad(y2, x, gy)
    rgx2, = torch.autograd.grad(yr, xr, gy.float())
    _close(gx2, rgx2, atol=5e-2, rtol=3e-2)


@pytest.mark.parametrize("use_norm", [True, False])
def test_headnorm_rope(use_norm):
    e = _ext()
    torch.manual_seed(0)
    B, S, H, D = 2, 96, 4, 128
    x = torch.randn(B * S, H * D, device="cuda", dtype=torch.bfloat16)
    w = (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16()
    dy = torch.randn_like(x)
    cs = _rope_table(S).cuda()
    y = torch.empty_like(x)
    rstd = torch.empty(B * S * H, device="cuda")
    e.headnorm_rope_fwd(x, w if use_norm else None, y, rstd if use_norm else None, cs, H, S, 1e-6)
    xr = x.float().view(B, S, H, D).requires_grad_(True)
    wr = w.float().requires_grad_(True)
    xn = xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-6) * wr if use_norm else xr
    cos = torch.cat([cs[..., 0], cs[..., 0]], -1)[None, :, None, :]
    sin = torch.cat([cs[..., 1], cs[..., 1]], -1)[None, :, None, :]
    rot = torch.cat([-xn[..., D // 2:], xn[..., :D // 2]], -1)
    yr = xn * cos + rot * sin
    yr.backward(dy.float().view(B, S, H, D))
    _close(y, yr.reshape(B * S, H * D), atol=3e-2, rtol=2e-2)
    dx = torch.empty_like(x)
    dw = torch.zeros(D, device="cuda")
    e.headnorm_rope_bwd(dy, x if use_norm else None, w if use_norm else None, rstd if use_norm else None, dx,
                        dw if use_norm else None, cs, H, S)
    _close(dx, xr.grad.reshape(B * S, H * D), atol=3e-2, rtol=2e-2)
    if use_norm:
        _close(dw, wr.grad, atol=0.3, rtol=2e-2)


def test_swiglu_embedding_ce():
    e = _ext()
    torch.manual_seed(0)
    T, I = 300, 1024
    g = torch.randn(T, I, device="cuda", dtype=torch.bfloat16)
    u = torch.randn(T, I, device="cuda", dtype=torch.bfloat16)
    d = torch.randn(T, I, device="cuda", dtype=torch.bfloat16)
    out = torch.empty_like(g)
    e.swiglu_fwd(g, u, out)
    gr, ur = g.float().requires_grad_(True), u.float().requires_grad_(True)
    ref = torch.nn.functional.silu(gr) * ur
    ref.backward(d.float())
    _close(out, ref, atol=2e-2, rtol=2e-2)
    dg, du = torch.empty_like(g), torch.empty_like(g)
    e.swiglu_bwd(d, g, u, dg, du)
    _close(dg, gr.grad, atol=3e-2, rtol=2e-2)
    _close(du, ur.grad, atol=3e-2, rtol=2e-2)

    V, H = 1000, 256
    table = torch.randn(V, H, device="cuda", dtype=torch.bfloat16)
    ids = torch.randint(0, V, (T,), device="cuda")
    emb = torch.empty(T, H, device="cuda", dtype=torch.bfloat16)
    e.embedding_fwd(ids, table, emb)
    assert torch.equal(emb, table[ids])
    dt = torch.zeros(V, H, device="cuda", dtype=torch.float32)
    demb = torch.randn(T, H, device="cuda", dtype=torch.bfloat16)
    e.embedding_bwd(ids, demb, dt)
    ref_dt = torch.zeros(V, H, device="cuda").index_add_(0, ids, demb.float())
    _close(dt, ref_dt, atol=1e-3, rtol=1e-3)

    vocab = 5000
    logits = (torch.randn(T, vocab, device="cuda") * 3).bfloat16()
    labels = torch.randint(0, vocab, (T,), device="cuda")
    labels[::7] = -100
    lr_ = logits.float().requires_grad_(True)
    loss_ref = torch.nn.functional.cross_entropy(lr_, labels, ignore_index=-100, reduction="sum")
    loss_ref.backward()
    loss = torch.zeros((), device="cuda")
    cnt = torch.zeros((), device="cuda")
    work = logits.clone()
    e.cross_entropy(work, labels, loss, cnt, None, 1.0, None, -100)
    assert cnt.item() == (labels != -100).sum().item()
    assert abs(loss.item() - loss_ref.item()) / loss_ref.item() < 2e-3
    _close(work, lr_.grad, atol=2e-3, rtol=2e-2)


def _attn_ref(q, k, v, scale):
    B, S, Hq, D = q.shape
    Hkv = k.shape[2]
    kk = k.repeat_interleave(Hq // Hkv, dim=2)
    vv = v.repeat_interleave(Hq // Hkv, dim=2)
    s = torch.einsum("bqhd,bkhd->bhqk", q, kk) * scale
    mask = torch.ones(S, S, device=q.device, dtype=torch.bool).tril()
    s = s.masked_fill(~mask, float("-inf"))
    p = s.softmax(-1)
    return torch.einsum("bhqk,bkhd->bqhd", p, vv)


@pytest.mark.parametrize("B,S,Hq,Hkv", [(1, 128, 2, 1), (2, 384, 4, 2), (1, 200, 2, 2), (1, 1024, 8, 2)])
def test_flash_attention_fwd_bwd(B, S, Hq, Hkv):
    e = _ext()
    torch.manual_seed(0)
    D = 128
    scale = 1.0 / math.sqrt(D)
    q = torch.randn(B * S, Hq * D, device="cuda", dtype=torch.bfloat16)
    k = torch.randn(B * S, Hkv * D, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(B * S, Hkv * D, device="cuda", dtype=torch.bfloat16)
    o = torch.empty_like(q)
    lse = torch.empty(B * Hq * S, device="cuda")
    e.flash_attn_fwd(q, k, v, o, lse, B, S, Hq, Hkv, scale)
    torch.cuda.synchronize()
    _assert_status_clean()
    qr = q.float().view(B, S, Hq, D).requires_grad_(True)
    kr = k.float().view(B, S, Hkv, D).requires_grad_(True)
    vr = v.float().view(B, S, Hkv, D).requires_grad_(True)
    ref = _attn_ref(qr, kr, vr, scale)
    _close(o, ref.reshape(B * S, Hq * D), atol=2e-2, rtol=2e-2)
    do = torch.randn_like(q)
    ref.backward(do.float().view(B, S, Hq, D))
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    delta = torch.empty(B * Hq * S, device="cuda")
    e.flash_attn_bwd(do, q, k, v, o, lse, dq, dk, dv, delta, torch.empty(2, B * S, Hq * 128, device='cuda', dtype=torch.bfloat16) if Hq > Hkv else None, B, S, Hq, Hkv, scale)
    torch.cuda.synchronize()
    _assert_status_clean()
    _close(dq, qr.grad.reshape(B * S, Hq * D), atol=3e-2, rtol=3e-2)
    _close(dk, kr.grad.reshape(B * S, Hkv * D), atol=3e-2, rtol=3e-2)
    _close(dv, vr.grad.reshape(B * S, Hkv * D), atol=3e-2, rtol=3e-2)


@pytest.mark.parametrize("D", [8, 56, 64, 72, 96, 120])
@pytest.mark.parametrize("B,S,Hq,Hkv", [(1, 128, 2, 1), (2, 256, 4, 4), (1, 200, 4, 2)])
def test_attention_narrow_heads(D, B, S, Hq, Hkv):
    """Heads narrower than the kernels' 64- and 128-column tiles, from contiguous, sliced and misaligned operands."""
    from himuon_b200 import ops

    torch.manual_seed(1)
    wide = torch.randn(B * S, (Hq + 2 * Hkv) * D, device="cuda", dtype=torch.bfloat16)
    # column slices of one projection output, the last one with rows that start off the 16-byte grid
    odd = torch.randn(B * S, Hkv * D + 1, device="cuda", dtype=torch.bfloat16)[:, 1:]
    q, k, v = wide[:, : Hq * D], wide[:, Hq * D: (Hq + Hkv) * D], odd
    leaves = [t.detach().clone().requires_grad_(True) for t in (q, k, v)]
    views = [q.detach().requires_grad_(True), k.detach().requires_grad_(True), v.detach().requires_grad_(True)]
    do = torch.randn(B * S, Hq * D, device="cuda", dtype=torch.bfloat16)
    for ins in (leaves, views):
        o = ops.attention(*ins, B, S, Hq, Hkv, D)
        o.backward(do)
        ref_in = [t.detach().float().reshape(B, S, h, D).requires_grad_(True) for t, h in zip(ins, (Hq, Hkv, Hkv))]
        ref = _attn_ref(*ref_in, 1.0 / math.sqrt(D))
        ref.backward(do.float().view(B, S, Hq, D))
        _assert_status_clean()
        # as for 128-wide heads: bf16 probabilities and score gradients, summed over at most 256 positions
        _close(o, ref.reshape(B * S, Hq * D), atol=2e-2, rtol=2e-2)
        for t, r in zip(ins, ref_in):
            _close(t.grad, r.grad.reshape(t.shape), atol=3e-2, rtol=3e-2)


@pytest.mark.parametrize("D", [40, 64, 96, 128])
@pytest.mark.parametrize("S", [1, 33, 64, 65, 128, 129, 192, 193])
def test_attention_of_a_prefix_has_the_same_bits(S, D):
    """A causal row does not see what follows it: the first S rows of 256 are those of the prefix alone, whatever rows the
    prefix's last tile holds (its epilogue depends on them)."""
    e = _ext()
    torch.manual_seed(S + D)
    H, whole = 3, 256
    q, k, v = (torch.randn(whole, H * D, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    outs = []
    for n in (whole, S):
        o, lse = torch.full((n + 1, H * D), 7.0, device="cuda", dtype=torch.bfloat16), torch.empty(H, n, device="cuda")
        e.flash_attn_fwd(q[:n], k[:n], v[:n], o, lse, 1, n, H, H, D ** -0.5)
        assert (o[n] == 7.0).all()                         # nothing past the last row
        outs.append((o[:S], lse[:, :S]))
    _assert_status_clean()
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("D", [8, 40, 64, 72, 128])
@pytest.mark.parametrize("B,S,Hq,Hkv", [(1, 1, 1, 1), (2, 64, 2, 2), (1, 129, 4, 2), (2, 333, 2, 1)])
def test_attention_backward_sums_delta_in_column_order(D, B, S, Hq, Hkv):
    """delta = sum of o * dO over a head: pairs of columns, each rounded once, added first to last in fp32.  The score gradients
    are rounded to bf16 after it is subtracted, so its last bit shows in dQ and dK: the order is part of the result."""
    e = _ext()
    torch.manual_seed(3)
    bf = dict(device="cuda", dtype=torch.bfloat16)
    q, k, v, do = (torch.randn(B * S, h * D, **bf) for h in (Hq, Hkv, Hkv, Hq))
    o, dq, dk, dv = torch.empty_like(q), torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    lse, delta = torch.empty(B * Hq * S, device="cuda"), torch.full((B * Hq * S,), float("nan"), device="cuda")
    part = torch.empty(2, B * S, Hq * D, **bf) if Hq != Hkv else None
    e.flash_attn_fwd(q, k, v, o, lse, B, S, Hq, Hkv, D ** -0.5)
    e.flash_attn_bwd(do, q, k, v, o, lse, dq, dk, dv, delta, part, B, S, Hq, Hkv, D ** -0.5)
    _assert_status_clean()
    term = (o.float() * do.float()).view(B, S, Hq, D // 2, 2).sum(-1)      # products of two bf16 values are exact in fp32
    want = torch.zeros(B, S, Hq, device="cuda")
    for c in range(D // 2):
        want = want + term[..., c]
    assert torch.equal(delta.view(B, Hq, S), want.transpose(1, 2))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("tokens,H", [(1, 2), (37, 3), (74, 4), (37, 6), (1998, 8), (999, 10), (2047, 4), (2048, 4), (4096, 4),
                                      (1279, 2), (1280, 2), (2560, 2)])
def test_head_norm_rope_heads_taken_together_match_one_by_one(tokens, H, D):
    """The kernels take up to four heads of a token per pass; a head's values have the same bits as when it is the only one."""
    from himuon_b200.ops import reference as ref

    e = _ext()
    torch.manual_seed(5)
    S = 37 if tokens % 37 == 0 else 1
    x, dy = (torch.randn(tokens, H, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    w = (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16()
    cs = ref.rope_tables(S, D, 1e4, device="cuda")

    def run(x, dy, heads):
        y, dx, rstd, dw = torch.empty_like(x), torch.empty_like(x), torch.empty(tokens, heads, device="cuda"), torch.zeros(D, device="cuda")
        e.headnorm_rope_fwd(x, w, y, rstd, cs, heads, S, 1e-6)
        e.headnorm_rope_bwd(dy, x, w, rstd, dx, dw, cs, heads, S)
        return y, dx, rstd, dw

    y, dx, rstd, dw = run(x.view(tokens, H * D), dy.view(tokens, H * D), H)
    alone = [run(x[:, h].contiguous(), dy[:, h].contiguous(), 1) for h in range(H)]
    assert torch.equal(y.view(tokens, H, D), torch.stack([a[0] for a in alone], 1))
    assert torch.equal(dx.view(tokens, H, D), torch.stack([a[1] for a in alone], 1))
    assert torch.equal(rstd, torch.cat([a[2] for a in alone], 1))
    # fp32 sums of tokens * H terms in another order: 2^-24 times the number of additions times the sum of magnitudes bounds it;
    # terms here are below 32, and the order of the atomics varies from run to run
    torch.testing.assert_close(dw, torch.stack([a[3] for a in alone]).sum(0), atol=32 * tokens * H * 2.0 ** -24 * 64, rtol=1e-4)


def test_head_norm_rope_takes_heads_together_only_where_the_chip_stays_busy():
    """Few vectors go one by one: a pass of four heads would only make their one round of blocks longer."""
    rule = _ext().headnorm_heads_per_pass
    for D, lanes in ((64, 8), (128, 16)):
        four, two = 512 * 256 // lanes, 160 * 256 // lanes          # vectors
        assert [rule(t // 4, 4, D, False) for t in (4, 1024, two - 4, two, four - 4, four, 1 << 20)] == [1, 1, 1, 2, 2, 4, 4]
        assert [rule(t // 2, 2, D, False) for t in (2, two - 2, two, 1 << 20)] == [1, 1, 2, 2]
        assert rule(1 << 20, 3, D, False) == 1
    assert [rule(t, 4, 128, True) for t in (16, 1024, 2048, 1 << 18)] == [1, 2, 4, 4]
    assert rule(1 << 18, 4, 64, True) == 1


@pytest.mark.parametrize("use_norm", [True, False])
@pytest.mark.parametrize("aligned", [True, False])
def test_head_norm_rope_64(use_norm, aligned):
    """64-wide heads: the kernel (16-byte aligned rows) and the PyTorch path (any other layout) agree with fp32."""
    from himuon_b200 import ops
    from himuon_b200.ops import reference as ref

    torch.manual_seed(2)
    B, S, H, D = 3, 37, 5, 64
    base = torch.randn(B * S, H * D + 8, device="cuda", dtype=torch.bfloat16)
    x = (base[:, 8:] if aligned else base[:, 1: 1 + H * D]).detach().requires_grad_(True)
    w = (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16().requires_grad_(True) if use_norm else None
    cs = ref.rope_tables(S, D, 1e4, device="cuda")
    dy = torch.randn(B * S, H * D, device="cuda", dtype=torch.bfloat16)
    before = ops.launch_count()
    y = ops.head_norm_rope(x, w, cs, H, S, D, 1e-6)
    assert (ops.launch_count() > before) == aligned
    y.backward(dy)
    xr = x.detach().float().requires_grad_(True)
    wr = w.detach().float().requires_grad_(True) if use_norm else None
    h = xr.view(B, S, H, D)
    yr = ref.apply_rope(ref.rmsnorm(h, wr, 1e-6) if use_norm else h, cs).reshape(B * S, H * D)
    yr.backward(dy.float())
    _close(y, yr, atol=3e-2, rtol=2e-2)
    _close(x.grad, xr.grad, atol=3e-2, rtol=2e-2)
    if use_norm:
        _close(w.grad, wr.grad, atol=0.3, rtol=2e-2)


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("tile", [128, 132])
def test_fp32_momentum_tile_and_untile_apply(tile, offset):
    """fp32 matrices: 16-byte rows, ragged widths, strided and misaligned tensors give the element-wise result."""
    e = _ext()
    torch.manual_seed(0)
    Th = Tw = tile
    mu, lr, wd, scale = 0.95, 0.02, 0.1, 2.0
    shapes = [(256, 384), (200, 301), (65, 64), (131, 132)]

    def make(h, w, pitch):      # rows `pitch` elements apart, first element `offset` elements past an aligned address
        return torch.randn(h * pitch + 4, device="cuda")[offset:].as_strided((h, w), (pitch, 1))

    grads = [make(h, w, w + 4) for h, w in shapes]
    moms = [make(h, w, w) for h, w in shapes]
    params = [make(h, w, w + 4) for h, w in shapes]
    moms_ref, params_ref = [m.clone() for m in moms], [p.clone() for p in params]
    mom_tab, app_tab, tile_base, unit, metas = b"", b"", 0, 0, []
    for g, m, p in zip(grads, moms, params):
        h, w = g.shape
        R, C = math.ceil(h / Th), math.ceil(w / Tw)
        mom_tab += struct.pack("<8QQq6i", g.data_ptr(), 0, 0, 0, 0, 0, 0, 0, m.data_ptr(), tile_base, h, w, R, C, unit, g.stride(0))
        app_tab += struct.pack("<Qq6ifi", p.data_ptr(), tile_base, h, w, R, C, unit, 0, scale, p.stride(0))
        metas.append((tile_base, R, C))
        tile_base += R * C
        unit += e.momentum_tile_units(R, C, Th)
    mom_dev = torch.frombuffer(bytearray(mom_tab), dtype=torch.uint8).cuda()
    app_dev = torch.frombuffer(bytearray(app_tab), dtype=torch.uint8).cuda()
    tiles = torch.full((tile_base, Th, Tw), 7.0, device="cuda", dtype=torch.bfloat16)
    e.momentum_tile(mom_dev, len(shapes), unit, Th, Tw, tiles, mu, True, 1.0, 1, True)
    hyper = torch.tensor([lr, wd], device="cuda", dtype=torch.float32)
    e.untile_apply(app_dev, len(shapes), unit, Th, Tw, tiles, hyper, True)
    for g, m_ref, m, p_ref, p, (tb, R, C) in zip(grads, moms_ref, moms, params_ref, params, metas):
        h, w = g.shape
        buf = m_ref * mu + g
        # two roundings of fp32 (values up to ~5): 5 * 2^-22 and the multiply-add contraction either way
        _close(m, buf, atol=3e-6, rtol=1e-6)
        padded = torch.zeros(R * Th, C * Tw, device="cuda")
        padded[:h, :w] = g + mu * buf
        got = tiles[tb:tb + R * C].view(R, C, Th, Tw).permute(0, 2, 1, 3).reshape(R * Th, C * Tw).float()
        _close(got, padded, atol=1e-5, rtol=2 ** -8)       # stored in bf16
        assert got[h:].abs().sum() == 0 and got[:, w:].abs().sum() == 0
        _close(p, p_ref * (1 - lr * wd) - lr * scale * got[:h, :w], atol=3e-6, rtol=1e-6)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,S,Hq,Hkv", [(1, 1, 1, 1), (2, 63, 2, 1), (1, 65, 2, 2), (2, 192, 4, 2), (1, 255, 4, 1), (1, 777, 2, 1)])
def test_attention_ragged_lengths(D, B, S, Hq, Hkv):
    """Sequence lengths around the 64- and 128-position blocks of the backward kernels."""
    from himuon_b200 import ops

    torch.manual_seed(3)
    ins = [torch.randn(B * S, h * D, device="cuda", dtype=torch.bfloat16, requires_grad=True) for h in (Hq, Hkv, Hkv)]
    o = ops.attention(*ins, B, S, Hq, Hkv, D)
    do = torch.randn_like(o)
    o.backward(do)
    ref_in = [t.detach().float().view(B, S, h, D).requires_grad_(True) for t, h in zip(ins, (Hq, Hkv, Hkv))]
    ref = _attn_ref(*ref_in, 1.0 / math.sqrt(D))
    ref.backward(do.float().view(B, S, Hq, D))
    _assert_status_clean()
    # bounds of test_flash_attention_fwd_bwd, which covers the same sums up to 1024 positions
    _close(o, ref.reshape(B * S, Hq * D), atol=2e-2, rtol=2e-2)
    for t, r in zip(ins, ref_in):
        _close(t.grad, r.grad.reshape(t.shape), atol=3e-2, rtol=3e-2)


@pytest.mark.parametrize("B,m,n", [(3, 256, 256), (1, 512, 512), (2, 264, 1000), (1, 1024, 3072), (2, 8, 8192)])
@pytest.mark.parametrize("out_of_place", [False, True])
def test_ns_normalize_cluster(B, m, n, out_of_place):
    """Tiles split over a cluster: whole slices, a ragged last one, slices longer than the registers hold, zero tiles."""
    torch.manual_seed(0)
    x = torch.randn(B + 1, m, n, device="cuda", dtype=torch.bfloat16)
    x[B].zero_()
    ref = x.float() / (x.double().norm(dim=(1, 2), keepdim=True).float() + 1e-7)
    out = torch.full_like(x, 5.0) if out_of_place else None
    src = x.clone()
    _ext().ns_normalize(x, B + 1, m * n, 1e-7, out)
    # half a bf16 ulp is 2^-8 of the value; the rest covers fp32 sums of up to 3 Mi squares in 8 * 1024 chains
    _close(out if out_of_place else x, ref, atol=1e-9, rtol=2 ** -7.9)
    assert not out_of_place or torch.equal(x, src)


@pytest.mark.parametrize("M,N,K,batch", [(512, 512, 512, 160), (336, 504, 504, 3), (264, 1000, 72, 2), (384, 256, 2048, 1),
                                         (1024, 3072, 1024, 4), (640, 640, 256, 5)])
@pytest.mark.parametrize("mode", ["aux", "aux_broadcast", "add", "fp32", "sym"])
def test_gemm_kernel_choice(M, N, K, batch, mode):
    """Both kernels, all tile widths and every epilogue form, on whole and ragged tiles."""
    from himuon_b200 import ops

    torch.manual_seed(0)
    dt = torch.float32 if mode == "fp32" else torch.bfloat16
    a = torch.randn(batch, M, K, device="cuda", dtype=torch.bfloat16)
    if mode == "sym":
        out = torch.full((batch, M, M), 9.0, device="cuda", dtype=dt)
        ops.gemm(a, a, trans_b=True, out=out, symmetric=True)
        ref = a.float() @ a.float().transpose(1, 2)
        assert torch.equal(out, out.transpose(1, 2))
    else:
        b = torch.randn(batch, K, N, device="cuda", dtype=torch.bfloat16)
        ref = a.float() @ b.float()
        out = torch.full((batch, M, N), 9.0, device="cuda", dtype=dt)
        if mode == "aux":
            x = torch.randn(batch, M, N, device="cuda", dtype=dt)
            ops.gemm(a, b, out=out, aux=x, alpha=0.5, beta=-2.0)
            ref = 0.5 * ref - 2.0 * x.float()
        elif mode == "aux_broadcast":
            x = torch.randn(1, 1, N, device="cuda", dtype=dt).expand(batch, M, N)
            ops.gemm(a, b, out=out, aux=x, beta=1.5)
            ref = ref + 1.5 * x.float()
        elif mode == "add":
            ref = ref + out.float()
            ops.gemm(a, b, out=out, aux=out, beta=1.0)
        else:
            x = torch.randn(batch, M, N, device="cuda")
            ops.gemm(a, b, out=out, aux=x, beta=0.5)
            ref = ref + 0.5 * x
    torch.cuda.synchronize()
    _assert_status_clean()
    # fp32 sums of K products (about sqrt(K)); half a bf16 ulp is 2^-8, twice that where partial sums are added into C
    tol = 1e-5 if dt == torch.float32 else 2 ** -7
    _close(out, ref, atol=tol * math.sqrt(K), rtol=tol)


@pytest.mark.parametrize("B,m,n", [(1, 64, 64), (500, 64, 64), (500, 40, 64), (5, 128, 192), (450, 120, 128)])
def test_ns5_fused_warp_splits(B, m, n):
    """Four and eight warps per tile, more tiles than fit the chip at once, short tiles."""
    torch.manual_seed(0)
    U, _, Vh = torch.linalg.svd(torch.randn(B, m, n), full_matrices=False)
    x = ((U * torch.linspace(0.8, 1.2, m)) @ Vh).cuda().bfloat16()
    out = torch.empty_like(x)
    _ext().ns5_fused(x, out, 5, 1e-7)
    torch.cuda.synchronize()
    _assert_status_clean()
    _close(out, _ns_ref(x), atol=4e-2, rtol=4e-2)      # the bounds of the test above: five bf16 iterations


@pytest.mark.parametrize("D,B,S,Hq,Hkv", [(128, 2, 1280, 16, 8), (128, 1, 1118, 24, 8), (64, 2, 1280, 32, 8), (128, 6, 129, 8, 8)])
def test_attention_forward_waits_for_its_last_product(D, B, S, Hq, Hkv):
    """The output is read when the last P V product is complete: whole 32-row groups miss their last KV blocks otherwise,
    in other places on every run."""
    e = _ext()
    torch.manual_seed(4)
    q, k, v = (torch.randn(B * S, h * D, device="cuda", dtype=torch.bfloat16) for h in (Hq, Hkv, Hkv))
    scale = 1.0 / math.sqrt(D)
    runs = []
    for _ in range(8):
        o, lse = torch.empty_like(q), torch.empty(B * Hq * S, device="cuda")
        e.flash_attn_fwd(q, k, v, o, lse, B, S, Hq, Hkv, scale)
        runs.append(o)
    _assert_status_clean()
    ref = _attn_ref(q.float().view(B, S, Hq, D), k.float().view(B, S, Hkv, D), v.float().view(B, S, Hkv, D), scale)
    _close(runs[0], ref.reshape(B * S, Hq * D), atol=2e-2, rtol=2e-2)        # the bounds of test_flash_attention_fwd_bwd
    for o in runs[1:]:
        assert torch.equal(o, runs[0])


def _momentum_apply_case(dtype, Th, Tw, offset, n_src, tile_offset=0):
    """momentum_tile, then untile_apply, on matrices whose first element lies `offset` elements past an aligned address;
    the gradient is the sum of `n_src` buffers.  Returns (momentum, tiles as matrices, parameters) and their references."""
    e = _ext()
    torch.manual_seed(0)
    mu, lr, wd, scale, gscale = 0.95, 0.02, 0.1, 2.0, 1.0 / n_src
    esz = torch.empty(0, dtype=dtype).element_size()
    shapes = [(256, 384), (200, 304), (65, 301), (64, 64), (131, 132)]

    def make(h, w, pitch):
        flat = torch.randn(h * pitch + 16 // esz, device="cuda").to(dtype)
        return flat[offset:].as_strided((h, w), (pitch, 1))

    grads = [[make(h, w, w + 8) for _ in range(n_src)] for h, w in shapes]
    moms = [make(h, w, w) for h, w in shapes]
    params = [make(h, w, w + 8) for h, w in shapes]
    moms_ref, params_ref = [m.float().clone() for m in moms], [p.float().clone() for p in params]
    mom_tab, app_tab, tile_base, unit, metas = b"", b"", 0, 0, []
    for gs, m, p in zip(grads, moms, params):
        h, w = m.shape
        R, C = math.ceil(h / Th), math.ceil(w / Tw)
        ptrs = [g.data_ptr() for g in gs] + [0] * (8 - n_src)
        mom_tab += struct.pack("<8QQq6i", *ptrs, m.data_ptr(), tile_base, h, w, R, C, unit, gs[0].stride(0))
        app_tab += struct.pack("<Qq6ifi", p.data_ptr(), tile_base, h, w, R, C, unit, 0, scale, p.stride(0))
        metas.append((tile_base, R, C))
        tile_base += R * C
        unit += e.momentum_tile_units(R, C, Th)
    mom_dev = torch.frombuffer(bytearray(mom_tab), dtype=torch.uint8).cuda()
    app_dev = torch.frombuffer(bytearray(app_tab), dtype=torch.uint8).cuda()
    buf = torch.full((tile_base * Th * Tw + 8,), 7.0, device="cuda", dtype=torch.bfloat16)
    tiles = buf[tile_offset: tile_offset + tile_base * Th * Tw].view(tile_base, Th, Tw)
    fp32 = dtype == torch.float32
    e.momentum_tile(mom_dev, len(shapes), unit, Th, Tw, tiles, mu, True, gscale, n_src, fp32)
    hyper = torch.tensor([lr, wd], device="cuda", dtype=torch.float32)
    e.untile_apply(app_dev, len(shapes), unit, Th, Tw, tiles, hyper, fp32)
    torch.cuda.synchronize()
    rnd = (lambda t: t) if fp32 else (lambda t: t.bfloat16().float())
    out = []
    for gs, m_ref, m, p_ref, p, (tb, R, C) in zip(grads, moms_ref, moms, params_ref, params, metas):
        h, w = m.shape
        g = rnd(sum(x.float() for x in gs) * gscale)
        b = rnd(rnd(m_ref * mu) + g)
        got = tiles[tb:tb + R * C].view(R, C, Th, Tw).permute(0, 2, 1, 3).reshape(R * Th, C * Tw).float()
        assert got[h:].abs().sum() == 0 and got[:, w:].abs().sum() == 0
        out.append(((m, b), (got[:h, :w], rnd(g + mu * b)),
                    (p, rnd(p_ref * (1 - lr * wd)) - lr * scale * got[:h, :w])))
    return out


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("offset,tile_offset", [(0, 0), (1, 0), (2, 0), (0, 1), (0, 4)])
@pytest.mark.parametrize("n_src", [1, 3])
@pytest.mark.parametrize("Th,Tw", [(128, 128), (96, 136)])
def test_momentum_and_apply_at_any_address(dtype, offset, tile_offset, n_src, Th, Tw):
    """Parameters, gradients, momenta and tiles that start anywhere (views into flat buffers), and a gradient that is the
    sum of several buffers: the 16-byte and the element-wise path."""
    # one rounding of the storage type either way of the multiply-add: half a bf16 ulp is 2^-9 of the value, sums of three
    # fp32 values of up to ~5 round by 2^-22 * 5 each
    rtol, atol = (2 ** -7.9, 1e-6) if dtype == torch.bfloat16 else (1e-6, 4e-6)
    for mom, tile, param in _momentum_apply_case(dtype, Th, Tw, offset, n_src, tile_offset):
        _close(*mom, atol=atol, rtol=rtol)
        _close(*tile, atol=1e-5, rtol=2 ** -7.9)            # stored in bf16
        _close(*param, atol=atol, rtol=rtol)


@pytest.mark.parametrize("B,S,H", [(1, 1, 1), (3, 37, 5), (2, 1313, 10)])
def test_rope_64_rounds_as_pytorch_does(B, S, H):
    """Heads of 64 without a norm: the kernel and the PyTorch formulation (which takes every layout) give the same bits."""
    from himuon_b200 import ops
    from himuon_b200.ops import reference as ref

    torch.manual_seed(7)
    D = 64
    x = torch.randn(B * S, H * D, device="cuda", dtype=torch.bfloat16)
    dy = torch.randn_like(x)
    cs = ref.rope_tables(S, D, 1e4, device="cuda")
    xk, xr = x.clone().requires_grad_(True), x.clone().requires_grad_(True)
    before = ops.launch_count()
    yk = ops.head_norm_rope(xk, None, cs, H, S, D, 1e-6)
    assert ops.launch_count() == before + 1
    yr = ref.apply_rope(xr.view(B, S, H, D), cs).view(B * S, H * D)
    yk.backward(dy)
    yr.backward(dy)
    assert torch.equal(yk, yr) and torch.equal(xk.grad, xr.grad)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("offset", [0, 1])
def test_untile_apply_rounds_alike_on_every_path(dtype, offset):
    """The decayed parameter is rounded, then one fused multiply-add follows, on 16-byte and element-wise accesses."""
    e = _ext()
    torch.manual_seed(8)
    h, w, T = 256, 320, 64
    flat = torch.randn(h * w + 16, device="cuda").to(dtype)
    p = flat[offset: offset + h * w].view(h, w)
    p0 = p.clone()
    tiles = torch.randn(20, T, T, device="cuda", dtype=torch.bfloat16)
    tab = struct.pack("<Qq6ifi", p.data_ptr(), 0, h, w, 4, 5, 0, 0, 2.0, w)
    hyper = torch.tensor([0.02, 0.1], device="cuda")
    e.untile_apply(torch.frombuffer(bytearray(tab), dtype=torch.uint8).cuda(), 1, e.momentum_tile_units(4, 5, T), T, T, tiles,
                   hyper, dtype == torch.float32)
    u = tiles.view(4, 5, T, T).permute(0, 2, 1, 3).reshape(h, w).double()
    decay = (1 - hyper[0].double() * hyper[1].double()).float()
    # the sum of a product and an fp32 value is exact in 64 bits here up to a rounding 2^-29 times as likely to matter
    want = ((p0.float() * decay).to(dtype).double() - (hyper[0] * 2.0).double() * u).float().to(dtype)
    assert torch.equal(p, want), (p != want).sum().item()


@pytest.mark.parametrize("M,N,K", [(64, 72, 64), (256, 512, 2048)])
def test_gemm_aux_with_more_matrices_than_the_product(M, N, K):
    """A batched aux operand may have matrices to spare; one with too few is refused."""
    from himuon_b200 import ops

    torch.manual_seed(0)
    a = torch.randn(3, M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(3, K, N, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(5, M, N, device="cuda", dtype=torch.bfloat16)
    out = ops.gemm(a, b, aux=x, beta=1.0)
    assert torch.equal(out, ops.gemm(a, b, aux=x[:3].clone(), beta=1.0))
    with pytest.raises(RuntimeError):
        ops.gemm(a, b, aux=x[:2], beta=1.0)
    _assert_status_clean()


def test_attention_accepts_and_refuses_the_shapes_it_always_has():
    """Heads of 128: keys and values may have tokens to spare.  Narrower heads: also (tokens, heads, head_dim) operands, but
    no spare tokens.  A width that does not belong to head_dim is refused by both, and by the rotary op."""
    from himuon_b200 import ops
    from himuon_b200.ops import reference as ref

    torch.manual_seed(0)
    B, S, Hq, Hkv = 2, 96, 4, 2
    for D in (128, 64):
        q = torch.randn(B * S, Hq * D, device="cuda", dtype=torch.bfloat16, requires_grad=True)
        k, v = (torch.randn(B * S + 40, Hkv * D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        want = ops.attention(q, k[: B * S], v[: B * S], B, S, Hq, Hkv, D)
        (g_want,) = torch.autograd.grad(want.float().square().sum(), q)
        if D == 128:
            got = ops.attention(q, k, v, B, S, Hq, Hkv, D)
            assert torch.equal(got, want)
            assert torch.equal(torch.autograd.grad(got.float().square().sum(), q)[0], g_want)
        else:
            with pytest.raises(RuntimeError):
                ops.attention(q, k, v, B, S, Hq, Hkv, D)
            got = ops.attention(q.view(B * S, Hq, D), k[: B * S].view(B * S, Hkv, D), v[: B * S].view(B * S, Hkv, D), B, S, Hq, Hkv, D)
            assert torch.equal(got, want)
        with pytest.raises(RuntimeError):
            ops.attention(q, k[: B * S - 1], v[: B * S - 1], B, S, Hq, Hkv, D)
        other = 192 - D
        with pytest.raises(RuntimeError):
            ops.attention(q, k[: B * S], v[: B * S], B, S, Hq, Hkv, other)
        with pytest.raises(RuntimeError):
            ops.head_norm_rope(q, None, ref.rope_tables(S, 128, 1e4, device="cuda"), Hq, S, other, 1e-6)
    _assert_status_clean()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,S", [(2, 96), (1, 1)])
@pytest.mark.parametrize("form", ["offset", "pitch"])
def test_gradients_and_operands_at_any_address(D, B, S, form):
    """Incoming gradients (and operands of narrow heads) that are contiguous but start off the 16-byte grid, or whose row
    pitch is odd, also where one row makes them contiguous all the same."""
    from himuon_b200 import ops
    from himuon_b200.ops import reference as ref

    torch.manual_seed(0)
    Hq, Hkv, T = 4, 2, B * S

    def odd(t):
        if form == "offset":
            flat = torch.empty(t.numel() + 1, device="cuda", dtype=t.dtype)
            out = flat[1:].view(t.shape)
        else:
            out = torch.empty(t.shape[0] * (t.shape[1] + 1) + 8, device="cuda", dtype=t.dtype).as_strided(t.shape, (t.shape[1] + 1, 1))
        return out.copy_(t)

    q, k, v = (torch.randn(T, h * D, device="cuda", dtype=torch.bfloat16) for h in (Hq, Hkv, Hkv))
    do = torch.randn_like(q)
    cs = ref.rope_tables(S, D, 1e4, device="cuda")
    w = torch.ones(D, device="cuda", dtype=torch.bfloat16)

    def run(operands, grad):
        leaves = [t.detach().requires_grad_(True) for t in operands]
        o = ops.attention(*leaves, B, S, Hq, Hkv, D)
        o.backward(grad)
        x = q.clone().requires_grad_(True)
        y = ops.head_norm_rope(x, w, cs, Hq, S, D, 1e-6)
        y.backward(grad)
        return [o.detach(), y.detach(), x.grad] + [t.grad for t in leaves]

    want = run((q, k, v), do)
    got = run([odd(t) for t in (q, k, v)] if D < 128 else (q, k, v), odd(do))
    for a, b in zip(want, got):
        assert torch.equal(a, b)
    _assert_status_clean()


@pytest.mark.parametrize("trans_a,trans_b", [(False, True), (False, False), (True, False)])
@pytest.mark.parametrize("M,N,K,dtype", [(2176, 16400, 1024, torch.bfloat16), (2112, 16392, 1088, torch.bfloat16),
                                         (4096, 8200, 392, torch.float32), (520, 1023, 200, torch.bfloat16), (520, 777, 72, torch.float32)])
def test_gemm_with_the_longer_operand_ring(M, N, K, dtype, trans_a, trans_b):
    """Long plain products with many rounds of tiles, and outputs whose rows TMA cannot store: four stages, two slabs."""
    from himuon_b200 import ops

    torch.manual_seed(0)
    a = torch.randn((K, M) if trans_a else (M, K), device="cuda", dtype=torch.bfloat16)
    pad = -N % 8                                         # operand rows stay addressable where the output's are not
    b = torch.randn((N, K) if trans_b else (K, N + pad), device="cuda", dtype=torch.bfloat16)
    b = b if trans_b else b[:, :N]
    out = torch.full((M, N), 9.0, device="cuda", dtype=dtype)
    ops.gemm(a, b, trans_a=trans_a, trans_b=trans_b, out=out)
    torch.cuda.synchronize()
    _assert_status_clean()
    ref = (a.float().t() if trans_a else a.float()) @ (b.float().t() if trans_b else b.float())
    tol = 1e-5 if dtype == torch.float32 else 2 ** -8     # as in test_gemm_kernel_choice, rounded once
    _close(out, ref, atol=tol * math.sqrt(K), rtol=tol)


@pytest.mark.parametrize("M,N,K,batch", [(256, 333, 64, 3), (200, 257, 72, 2), (300, 515, 2048, 1), (130, 9, 64, 2), (64, 7, 64, 1),
                                         (513, 1021, 136, 30)])
@pytest.mark.parametrize("mode", ["plain", "aux", "fp32", "fp32_aux", "add"])
def test_gemm_writes_only_its_own_columns(M, N, K, batch, mode):
    """A column slice as output: row pitch on the 16-byte grid, width off it.  TMA stores whole 16-byte groups, so the last
    columns are written one by one and the neighbouring columns stay."""
    from himuon_b200 import ops

    torch.manual_seed(0)
    dt = torch.float32 if mode.startswith("fp32") else torch.bfloat16
    a = torch.randn(batch, M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(batch, K, (N + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, :, :N]
    buf = torch.full((batch, M, (N + 7) // 8 * 8 + 8), 9.0, device="cuda", dtype=dt)
    out = buf[:, :, :N]
    x = torch.randn(batch, M, buf.shape[2], device="cuda", dtype=dt)[:, :, :N] if "aux" in mode else out if mode == "add" else None
    ref = a.float() @ b.float() + (1.5 * x.float() if x is not None else 0.0)
    ops.gemm(a, b, out=out, aux=x, beta=1.5 if x is not None else 0.0)
    torch.cuda.synchronize()
    _assert_status_clean()
    assert (buf[:, :, N:] == 9.0).all(), "columns of the neighbour were written"
    tol = 1e-5 if dt == torch.float32 else 2 ** -7
    _close(out, ref, atol=tol * math.sqrt(K), rtol=tol)


@pytest.mark.parametrize("m", [139, 333, 515])
def test_symmetric_gemm_writes_only_its_own_columns(m):
    from himuon_b200 import ops

    torch.manual_seed(0)
    x = torch.randn(2, m, 96, device="cuda", dtype=torch.bfloat16)
    buf = torch.full((2, m, (m + 7) // 8 * 8), 9.0, device="cuda", dtype=torch.bfloat16)
    ops.gemm(x, x, trans_b=True, out=buf[:, :, :m], symmetric=True)
    _assert_status_clean()
    assert (buf[:, :, m:] == 9.0).all() and torch.equal(buf[:, :, :m], buf[:, :, :m].transpose(1, 2))
    _close(buf[:, :, :m], x.float() @ x.float().transpose(1, 2), atol=2 ** -8 * math.sqrt(96), rtol=2 ** -8)


@pytest.mark.parametrize("N", [136, 160, 192])
@pytest.mark.parametrize("batch", [1, 400])
@pytest.mark.parametrize("mode", ["plain", "aux", "fp32", "fp32_aux"])
def test_gemm_192_wide_tiles(N, batch, mode):
    """Outputs of 129 to 192 columns: three bf16 slabs a tile, so that the two epilogue groups swap parity from tile to tile
    (400 matrices of two row blocks: every CTA walks several)."""
    from himuon_b200 import ops

    torch.manual_seed(0)
    M, K = 200, 136
    dt = torch.float32 if mode.startswith("fp32") else torch.bfloat16
    a = torch.randn(batch, M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(batch, K, N, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(batch, M, N, device="cuda", dtype=dt) if "aux" in mode else None
    out = torch.full((batch, M, N), 9.0, device="cuda", dtype=dt)
    ops.gemm(a, b, out=out, aux=x, alpha=0.5, beta=-2.0 if x is not None else 0.0)
    torch.cuda.synchronize()
    _assert_status_clean()
    ref = 0.5 * (a.float() @ b.float()) - (2.0 * x.float() if x is not None else 0.0)
    tol = 1e-5 if dt == torch.float32 else 2 ** -7        # as in test_gemm_kernel_choice
    _close(out, ref, atol=tol * math.sqrt(K), rtol=tol)


@pytest.mark.parametrize("M,N,K,batch", [(130, 129, 64, 3), (256, 191, 200, 1), (300, 333, 264, 40), (136, 513, 72, 2), (4, 1, 8, 3)])
@pytest.mark.parametrize("mode", ["plain", "aux", "round_acc", "strided", "fp32", "fp32_aux"])
def test_gemm_outputs_that_tma_cannot_store(M, N, K, batch, mode):
    """Output rows off the 16-byte grid leave by plain stores from both epilogue groups; nothing around them is written."""
    from himuon_b200 import ops

    torch.manual_seed(0)
    dt = torch.float32 if mode.startswith("fp32") else torch.bfloat16
    a = torch.randn(batch, M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(batch, N, K, device="cuda", dtype=torch.bfloat16)
    gap = 3 if mode == "strided" else 0
    buf = torch.full((batch, M, N + gap), 9.0, device="cuda", dtype=dt)
    out = buf[:, :, :N]
    x = torch.randn(batch, M, N, device="cuda", dtype=dt) if mode in ("aux", "round_acc", "fp32_aux") else None
    ops.gemm(a, b, trans_b=True, out=out, aux=x, alpha=0.5, beta=1.5 if x is not None else 0.0, round_acc=mode == "round_acc")
    torch.cuda.synchronize()
    _assert_status_clean()
    ref = 0.5 * (a.float() @ b.float().transpose(1, 2))
    if mode == "round_acc":
        ref = ref.bfloat16().float()
    if x is not None:
        ref = ref + 1.5 * x.float()
    assert (buf[:, :, N:] == 9.0).all()
    tol = 1e-5 if dt == torch.float32 else 2 ** -7
    _close(out, ref, atol=tol * math.sqrt(K), rtol=tol)


@pytest.mark.parametrize("use_norm", [True, False])
def test_head_norm_rope_64_differentiates_twice(use_norm):
    """create_graph=True on the 64-wide op: gradients of gradients follow the fp32 formulation."""
    from himuon_b200 import ops
    from himuon_b200.ops import reference as ref

    torch.manual_seed(3)
    B, S, H, D = 2, 9, 3, 64
    cs = ref.rope_tables(S, D, 1e4, device="cuda")
    x0 = torch.randn(B * S, H * D, device="cuda", dtype=torch.bfloat16)
    w0 = (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16() if use_norm else None
    c = torch.randn(B * S, H * D, device="cuda", dtype=torch.bfloat16)

    def second(fn, x, w):
        leaves = [x] if w is None else [x, w]
        y = fn(x, w)
        grads = torch.autograd.grad((y.float() ** 3 * c.float()).sum(), leaves, create_graph=True)
        return torch.autograd.grad(sum((g.float() ** 2).sum() for g in grads), leaves)

    got = second(lambda x, w: ops.head_norm_rope(x, w, cs, H, S, D, 1e-6), x0.clone().requires_grad_(True),
                 None if w0 is None else w0.clone().requires_grad_(True))

    def plain(x, w):
        h = x.view(B, S, H, D)
        return ref.apply_rope(ref.rmsnorm(h, w, 1e-6) if use_norm else h, cs).reshape(B * S, H * D)

    want = second(plain, x0.float().requires_grad_(True), None if w0 is None else w0.float().requires_grad_(True))
    for g, r in zip(got, want):
        # bf16 intermediates (2^-9 each, about a dozen of them) through two backward passes
        assert float((g.float() - r).norm() / r.norm()) < 12 * 2 ** -8


def test_head_norm_rope_64_under_transforms():
    """vmap and forward-mode tangents, for which the autograd function has no rules, take the PyTorch formulation."""
    import warnings

    from himuon_b200 import ops
    from himuon_b200.ops import reference as ref

    torch.manual_seed(4)
    B, S, H, D = 2, 9, 3, 64
    cs = ref.rope_tables(S, D, 1e4, device="cuda")
    x = torch.randn(4, B * S, H * D, device="cuda", dtype=torch.bfloat16)
    want = torch.stack([ref.apply_rope(t.view(B, S, H, D), cs).reshape(B * S, H * D) for t in x])
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        got = torch.vmap(lambda t: ops.head_norm_rope(t, None, cs, H, S, D, 1e-6))(x)
        assert torch.equal(got, want)
        with torch.autograd.forward_ad.dual_level():
            dual = torch.autograd.forward_ad.make_dual(x[0], x[1])
            y, tangent = torch.autograd.forward_ad.unpack_dual(ops.head_norm_rope(dual, None, cs, H, S, D, 1e-6))
    assert torch.equal(y, want[0]) and torch.equal(tangent, want[1])      # the rotation is linear


def _three_gemm_iteration(x, steps):
    """The products of the Newton-Schulz iteration one GEMM at a time, on a scaled bf16 batch."""
    from himuon_b200.ops import gemm, ns

    for _ in range(steps):
        wide = x.shape[1] <= x.shape[2]
        a = gemm(x, x, trans_b=True) if wide else gemm(x, x, trans_a=True)
        b = gemm(a, a, trans_b=True, alpha=ns.C_COEF, beta=ns.B_COEF, aux=a)
        x = gemm(b, x, alpha=1.0, beta=ns.A_COEF, aux=x, round_acc=True) if wide else \
            gemm(x, b, alpha=1.0, beta=ns.A_COEF, aux=x, round_acc=True)
    return x


# One block and two of the short side, one to eight of the long one, wide and tall, sides at and beside the edges of the 64 and
# 256 wide blocks; plans with one, two and four pairs per matrix (by the number of matrices), several rounds of matrices per
# pair, interleaved ones, and ragged last rounds.
@pytest.mark.parametrize("shape,steps", [
    ((1, 256, 256), 5), ((3, 16, 264), 5), ((2, 512, 512), 5), ((19, 512, 512), 2), ((40, 512, 512), 5), ((75, 512, 504), 3),
    ((5, 264, 1000), 5), ((5, 1000, 264), 5), ((100, 264, 1000), 2), ((20, 136, 2040), 5), ((20, 2040, 136), 4),
    ((90, 336, 504), 5), ((90, 504, 336), 5), ((230, 256, 200), 5), ((331, 200, 256), 5), ((77, 24, 320), 5), ((250, 320, 24), 5),
    ((80, 192, 328), 6), ((8, 448, 520), 5), ((8, 64, 8), 5)])
def test_ns_pair_kernel_matches_the_gemms_bit_for_bit(shape, steps):
    from himuon_b200.ops import ns, reference

    g = torch.Generator("cuda").manual_seed(sum(shape))
    x = torch.randn(shape, device="cuda", dtype=torch.bfloat16, generator=g)
    assert _ext().ns_pair_plan(x) is not None
    scaled = torch.empty_like(x)
    _ext().ns_normalize(x, shape[0], shape[1] * shape[2], ns.EPS, scaled)
    out = ns.ns_inplace_cuda(scaled.clone(), steps, normalize=False)
    again = ns.ns_inplace_cuda(torch.full_like(x, float("nan")), steps, source=x)     # out of place, from unscaled values
    _assert_status_clean()
    assert torch.equal(out, _three_gemm_iteration(scaled, steps))
    assert torch.equal(out, again)
    # against the PyTorch path on fp32 copies of one matrix: five bf16 iterations leave 1-2 % (2-norm)
    ref = reference.newton_schulz(x[-1].float().cpu(), steps=steps)
    assert (out[-1].float().cpu() - ref).norm() <= 0.03 * ref.norm()


def test_ns_pair_plan_declines_rounds_that_do_not_pay():
    """Matrices beyond the pairs take whole rounds; the lines lie between shapes measured slower and faster than the GEMMs."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the shapes are those of 74 CTA pairs")

    def taken(b, m, n):
        return _ext().ns_pair_plan(torch.empty(b, m, n, device="cuda", dtype=torch.bfloat16)) is not None

    for shape in [(160, 16, 512), (230, 128, 264), (80, 128, 768), (160, 128, 768), (80, 16, 1024), (300, 16, 264), (200, 264, 128),
                  (150, 640, 128), (80, 264, 768), (80, 384, 1024), (150, 264, 1024), (1, 512, 1024), (4, 384, 1024), (75, 512, 1024)]:
        assert not taken(*shape), shape
    for shape in [(74, 16, 1024), (148, 16, 512), (100, 128, 768), (148, 1024, 16), (296, 512, 16), (296, 264, 64), (296, 256, 128), (296, 128, 200),
                  (80, 264, 512), (100, 384, 1024), (185, 264, 768), (92, 768, 264), (1, 264, 1024), (5, 512, 1024), (84, 512, 1024),
                  (75, 448, 768), (592, 256, 256), (80, 192, 2048)]:
        assert taken(*shape), shape


def test_ns_pair_kernel_keeps_a_bad_matrix_to_itself():
    from himuon_b200.ops import ns

    x = torch.randn(9, 256, 256, device="cuda", dtype=torch.bfloat16)
    good = ns.newton_schulz(x)
    for bad in (float("nan"), float("inf")):
        y = x.clone()
        y[4, 17, 33] = bad
        out = ns.newton_schulz(y)
        assert out[4].isnan().all()
        assert torch.equal(torch.cat([out[:4], out[5:]]), torch.cat([good[:4], good[5:]]))
    x[4] = 0
    assert (ns.newton_schulz(x)[4] == 0).all()
    _assert_status_clean()


# Reductions of 512 to 2047, plain and with every epilogue form, ragged rows and columns, every operand-major combination: the plain
# products run on CTA pairs, the others on either kernel (test_pair_gemm_rule has the line between them).
@pytest.mark.parametrize("M,N,K,batch", [(1281, 2048, 512, 1), (2056, 1288, 1096, 1), (328, 520, 2040, 8), (2560, 2560, 640, 1)])
@pytest.mark.parametrize("trans_a,trans_b", [(False, True), (False, False), (True, True), (True, False)])
@pytest.mark.parametrize("mode", ["plain", "aux", "add", "fp32"])
def test_pair_gemm_on_short_reductions(M, N, K, batch, trans_a, trans_b, mode):
    from himuon_b200 import ops

    if trans_a and M % 8:
        M += 8 - M % 8                                     # the rows of a transposed operand are 16-byte aligned
    g = torch.Generator("cuda").manual_seed(M + N + K)
    a = torch.randn(batch, *((K, M) if trans_a else (M, K)), device="cuda", dtype=torch.bfloat16, generator=g)
    b = torch.randn(batch, *((N, K) if trans_b else (K, N)), device="cuda", dtype=torch.bfloat16, generator=g)
    ref = (a.float().mT if trans_a else a.float()) @ (b.float().mT if trans_b else b.float())
    out = torch.randn(batch, M, N, device="cuda", generator=g).to(torch.float32 if mode == "fp32" else torch.bfloat16)
    x = torch.randn(batch, M, N, device="cuda", generator=g).to(out.dtype)
    kw = dict(trans_a=trans_a, trans_b=trans_b, out=out)
    atol = 4e-4 if mode == "fp32" else 1e-2
    if mode == "plain":
        ops.gemm(a, b, **kw)
    elif mode == "add":
        ref = ref + out.float()
        ops.gemm(a, b, aux=out, beta=1.0, **kw)
    else:
        ops.gemm(a, b, aux=x, alpha=0.5, beta=-2.0, round_acc=mode == "aux", **kw)
        ref = 0.5 * ref
        if mode == "aux":                                  # the rounded accumulator: half an ulp of it, which the sum may cancel
            atol += 2 ** -9 * ref.abs().max().item()
        ref = ref - 2.0 * x.float()
    torch.cuda.synchronize()
    _assert_status_clean()
    # fp32 sums of K products of unit normals differ by some 2^-24 of sqrt(K) per term in any order; a bf16 result adds half
    # an ulp, 2^-9 of the value
    _close(out, ref, atol=atol, rtol=1e-5 if mode == "fp32" else 2 ** -8)


# mode, batch, M, N and the shortest reduction that goes to CTA pairs; 16 less does not.  One round of 128 x 256 tiles and
# several, matrices that barely overflow one row of tiles, ragged rows and columns.
_PAIR_LINES = [("plain", 1, 1281, 2048, 512), ("plain", 20, 136, 520, 512), ("plain", 80, 136, 200, 512),
               ("plain", 100, 264, 264, 512),
               ("aux", 1, 1281, 4104, 1280), ("aux", 8, 1000, 1032, 1024), ("add", 1, 1281, 4104, 1280), ("add", 8, 1000, 1032, 1024),
               ("fp32", 1, 1281, 4104, 1024), ("fp32", 8, 1000, 1032, 768), ("fp32 add", 8, 1000, 1032, 1536),
               ("add", 1, 1024, 3072, 648), ("fp32 add", 1, 1024, 3072, 1032)]


def _pair_case(mode, batch, M, N, K, trans_a=False, trans_b=True):
    g = torch.Generator("cuda").manual_seed(M + N + K)
    a = torch.randn(batch, *((K, M) if trans_a else (M, K)), device="cuda", dtype=torch.bfloat16, generator=g)
    b = torch.randn(batch, *((N, K) if trans_b else (K, N)), device="cuda", dtype=torch.bfloat16, generator=g)
    out = torch.randn(batch, M, N, device="cuda", generator=g).to(torch.float32 if "fp32" in mode else torch.bfloat16)
    aux = {"aux": lambda: torch.randn_like(out), "add": lambda: out, "fp32 add": lambda: out}.get(mode, lambda: None)()
    beta = 0.0 if aux is None else 1.0 if aux is out else -2.0
    return a, b, out, aux, trans_a, trans_b, 1.0 if beta == 1.0 else 0.5, beta, mode == "aux"


@pytest.mark.parametrize("mode,batch,M,N,K", _PAIR_LINES)
def test_pair_gemm_rule(mode, batch, M, N, K):
    from himuon_b200 import ops

    on_pairs = _ext().gemm_on_pairs
    assert on_pairs(*_pair_case(mode, batch, M, N, K)) and not on_pairs(*_pair_case(mode, batch, M, N, K - 16))
    assert on_pairs(*_pair_case(mode, batch, M, N, 2048))
    for trans_a, trans_b in ((False, True), (False, False), (True, True), (True, False)):
        if trans_a and M % 8:
            continue                                       # the rows of a transposed operand are 16-byte aligned
        a, b, out, aux, ta, tb, alpha, beta, round_acc = _pair_case(mode, batch, M, N, K, trans_a, trans_b)
        parts = []
        for r in range(0, M, 128):                         # rows of one tile at a time run on the one-CTA kernel
            rows = a[:, :, r:r + 128].contiguous() if ta else a[:, r:r + 128]
            part = out[:, r:r + 128].clone()
            x = None if aux is None else part if aux is out else aux[:, r:r + 128]
            assert not on_pairs(rows, b, part, x, ta, tb, alpha, beta, round_acc)
            parts.append(ops.gemm(rows, b, trans_a=ta, trans_b=tb, alpha=alpha, beta=beta, aux=x, out=part, round_acc=round_acc))
        ops.gemm(a, b, trans_a=ta, trans_b=tb, alpha=alpha, beta=beta, aux=aux, out=out, round_acc=round_acc)
        _assert_status_clean()
        assert torch.equal(out, torch.cat(parts, 1))       # the same products and sums, in the same order


def test_pair_gemm_declines_where_padding_or_few_tiles_cost_a_round():
    on_pairs = _ext().gemm_on_pairs
    for batch, M, N, K in ((1, 320, 12288, 1728), (1, 257, 12288, 640), (1, 777, 5120, 1024), (40, 320, 320, 1024), (12, 384, 384, 512),
                           (1, 320, 5120, 512), (10, 264, 264, 1536)):
        assert not on_pairs(*_pair_case("plain", batch, M, N, K))
    for mode in ("aux", "add", "fp32", "fp32 add"):          # one round of tiles, unless the operands' rows are off the sectors' grid
        assert not on_pairs(*_pair_case(mode, 1, 1024, 3072, 1536)) and on_pairs(*_pair_case(mode, 1, 1024, 3072, 1544))
        assert not on_pairs(*_pair_case(mode, 1, 1024, 3072, 1544, True, False))
    assert on_pairs(*_pair_case("plain", 1, 1024, 3072, 512))
    assert on_pairs(*_pair_case("plain", 100, 264, 264, 1024)) and not on_pairs(*_pair_case("plain", 100, 264, 264, 1024, True))

"""Newton-Schulz dispatcher.

``newton_schulz(G, steps)`` is the op behind ``HiMuon.newton_schulz`` and Muon's
``zeropower_via_newtonschulz5`` (reference: ``src/himuon/optimizers/himuon.py:263-284``,
``muon.py:13-44``).  On a CUDA device it runs

* the tile-resident fused kernel (one CTA per tile, operands in shared memory, accumulators
  in TMEM) for tiles with at most 128 rows and 64..256 columns,
* one launch that takes every matrix through all iterations on CTA pairs, intermediates in the
  L2, for short sides up to 512 (``csrc/ns_pair_sm100.cu``; ``ns_pair_plan`` has the exact line), and
* otherwise a batched three-GEMM iteration on the persistent tcgen05 GEMM with fused
  epilogues (``A = X X^T``; ``B = c A A + b A``; ``X = bf16(B X) + a X``; the two symmetric
  products compute only the tiles that touch the lower triangle and mirror them, as the
  reference's ``XXT`` / ``ba_plus_cAA`` kernels do), which handles any
  shape whose sides are multiples of 8, tall tiles included (no transpose copy: the GEMM
  reads either operand in either major).

Off-GPU the PyTorch reference with the same rounding points runs.
"""

from __future__ import annotations

import torch

from .. import _ext
from . import reference as ref
from . import _count, gemm

A_COEF, B_COEF, C_COEF = ref.NS_COEFFS
EPS = 1e-7


class NSWorkspace:
    """Reusable scratch of the Newton-Schulz paths (keeps addresses stable for CUDA graphs).  Matrices of one shape share a
    scratch: calls that may overlap, on two streams, need a workspace each unless their shapes differ."""

    def __init__(self):
        self.bufs: dict[tuple, tuple[torch.Tensor, torch.Tensor, torch.Tensor]] = {}
        self.flat: dict[tuple, torch.Tensor] = {}          # scratch of ns_pair
        self.captured: dict[int, torch.Tensor] = {}        # by address: those of `flat` that a CUDA graph may replay on

    def get(self, B: int, m: int, n: int, device) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
        k = min(m, n)
        key = (m, n, str(device))
        cur = self.bufs.get(key)
        if cur is None or cur[0].shape[0] < B:
            cur = (
                torch.empty(B, k, k, device=device, dtype=torch.bfloat16),
                torch.empty(B, k, k, device=device, dtype=torch.bfloat16),
                torch.empty(B, m, n, device=device, dtype=torch.bfloat16),
            )
            self.bufs[key] = cur
        return cur[0][:B], cur[1][:B], cur[2][:B]

    def scratch(self, nbytes: int, m: int, n: int, device) -> torch.Tensor:
        """At least `nbytes` for matrices of m x n.  A buffer that has become too small is given back, unless a graph holds it."""
        key = (m, n, str(device))
        cur = self.flat.get(key)
        if cur is None or cur.numel() < nbytes:
            cur = self.flat[key] = torch.empty(nbytes, device=device, dtype=torch.uint8)
        if torch.cuda.is_current_stream_capturing():
            self.captured[cur.data_ptr()] = cur
        return cur

    def clear(self):
        self.bufs.clear()
        self.flat.clear()
        self.captured.clear()


def fused_supported(m: int, n: int) -> bool:
    lo, hi = min(m, n), max(m, n)
    return lo >= 1 and lo <= 128 and hi % 64 == 0 and 64 <= hi <= 256


def ns_inplace_cuda(X: torch.Tensor, steps: int = 5, eps: float = EPS, workspace: NSWorkspace | None = None,
                    normalize: bool = True, source: torch.Tensor | None = None) -> torch.Tensor:
    """Orthogonalise a contiguous bf16 ``(B, m, n)`` CUDA buffer in place and return it.  With ``source`` (same shape and
    type) that tensor is read instead and left as it is: the first pass over the data, which scales every tile, writes to
    ``X`` or to scratch, so no copy is needed."""
    assert X.is_cuda and X.dtype == torch.bfloat16 and X.dim() == 3 and X.is_contiguous()
    e = _ext.ext()
    Bt, m, n = X.shape
    if Bt == 0:
        return X
    assert source is None or (normalize and source.shape == X.shape and source.dtype == X.dtype and source.is_contiguous())
    src = X if source is None else source
    if m <= n and e.ns5_fused_supported(m, n) and normalize:
        e.ns5_fused(src, X, int(steps), float(eps))
        _count()
        return X
    if m % 8 or n % 8:
        raise ValueError(f"newton_schulz on CUDA needs tile sides that are multiples of 8, got ({m}, {n})")
    ws = workspace or NSWorkspace()
    plan = e.ns_pair_plan(X) if steps >= 2 else None
    if plan is not None:
        pairs, interleaved, nbytes = plan
        if normalize:
            e.ns_normalize(src, Bt, m * n, float(eps), X)
            _count()
        e.ns_pair(X, X, ws.scratch(nbytes, m, n, X.device), int(steps), pairs, interleaved)
        _count()
        return X
    A, Bm, Y = ws.get(Bt, m, n, X.device)
    cur, nxt = X, Y
    if normalize:
        # With an odd number of iterations the normalised copy goes to the scratch buffer, so that the ping-pong ends
        # in X and no copy back is needed.
        if steps % 2 == 1:
            e.ns_normalize(src, Bt, m * n, float(eps), Y)
            cur, nxt = Y, X
        elif source is not None:
            e.ns_normalize(src, Bt, m * n, float(eps), X)
        else:
            e.ns_normalize(X, Bt, m * n, float(eps))
        _count()
    wide = m <= n
    for _ in range(steps):
        if wide:
            gemm(cur, cur, trans_b=True, out=A, symmetric=True)                   # A = X X^T        (m x m)
            gemm(A, A, trans_b=True, alpha=C_COEF, beta=B_COEF, aux=A, out=Bm, symmetric=True)  # B = c A A + b A
            gemm(Bm, cur, alpha=1.0, beta=A_COEF, aux=cur, out=nxt, round_acc=True)  # X' = B X + a X
        else:
            gemm(cur, cur, trans_a=True, out=A, symmetric=True)                   # A = X^T X        (n x n)
            gemm(A, A, trans_b=True, alpha=C_COEF, beta=B_COEF, aux=A, out=Bm, symmetric=True)
            gemm(cur, Bm, alpha=1.0, beta=A_COEF, aux=cur, out=nxt, round_acc=True)  # X' = X B + a X
        cur, nxt = nxt, cur
    if cur is not X:
        X.copy_(cur)
    return X


def newton_schulz(G: torch.Tensor, steps: int = 5, workspace: NSWorkspace | None = None) -> torch.Tensor:
    """Orthogonalise the last two dims of ``G`` (2-D or batched 3-D); returns ``G``'s dtype."""
    assert G.ndim >= 2
    if not G.is_cuda:
        return ref.newton_schulz(G, steps=steps)
    shape = G.shape
    X = G.reshape(-1, shape[-2], shape[-1])
    m, n = X.shape[-2:]
    # A result for a tensor that records its gradient stays attached to it, whatever its type, sides and address: that path
    # is made of PyTorch's own copies.
    attached = torch.is_grad_enabled() and G.requires_grad
    if (m % 8 or n % 8) and attached:
        padded = torch.nn.functional.pad(X.to(torch.bfloat16), (0, -n % 8, 0, -m % 8))
        out = ns_inplace_cuda(_pre_normalized(padded), steps, workspace=workspace, normalize=False)[:, :m, :n]
        return out.reshape(shape).to(G.dtype)
    if m % 8 or n % 8:
        # pad to the TMA granularity; zero rows/columns do not change the iteration
        if X.dtype not in (torch.bfloat16, torch.float32):
            X = X.to(torch.bfloat16)
        X = X.contiguous()
        out = torch.empty(X.shape, device=X.device, dtype=X.dtype)
        if X.numel():
            e = _ext.ext()
            pm, pn = -(-m // 8) * 8, -(-n // 8) * 8
            pad = torch.empty(X.shape[0], pm, pn, device=X.device, dtype=torch.bfloat16)
            e.ns_repad(X, pad)
            # the same bits as _pre_normalized: this norm adds the same fp32 squares in the same order, without the copy
            e.ns_repad(pad, pad, torch.linalg.vector_norm(pad, dim=(-2, -1), dtype=torch.float32), EPS)
            if e.ns5_fused_supported(pm, pn):
                e.ns5_fused(pad, pad, int(steps), EPS, False)
                _count()
            else:
                ns_inplace_cuda(pad, steps, workspace=workspace, normalize=False)
            e.ns_repad(pad, out)
            _count(3)
        return out.reshape(shape).to(G.dtype)
    Xb = X.to(torch.bfloat16)
    if not Xb.is_contiguous():
        out = ns_inplace_cuda(Xb.contiguous(), steps, workspace=workspace)
    elif Xb.data_ptr() != G.data_ptr():                    # a converted copy: ours to overwrite
        out = ns_inplace_cuda(Xb, steps, workspace=workspace)
    elif Xb.data_ptr() % 16 == 0 and not attached:         # G itself, which is only read
        out = ns_inplace_cuda(torch.empty_like(Xb), steps, workspace=workspace, source=Xb)
    else:
        out = ns_inplace_cuda(Xb.clone(), steps, workspace=workspace)
    return out.reshape(shape).to(G.dtype)


def _pre_normalized(X: torch.Tensor, eps: float = EPS) -> torch.Tensor:
    norm = X.float().norm(dim=(-2, -1), keepdim=True)
    return (X.float() / (norm + eps)).to(torch.bfloat16).contiguous()

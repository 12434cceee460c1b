"""Mixture-of-experts feed-forward on the sm_100a kernels: router GEMM (fp32 logits) ->
top-k routing -> expert-sorted permutation -> grouped tcgen05 GEMM (gate|up) -> SwiGLU ->
grouped GEMM (down) -> weighted combine. No host synchronisation anywhere: the number of
live tiles is read by the grouped GEMM from device memory.

Weights: ``w_router`` [E, d], ``w_gate_up`` [E, 2F, d] (gate rows then up rows per expert),
``w_down`` [E, d, F], all bf16. Matches the math of the tensor-runtime stages
``router_topk`` + ``grouped_swiglu_experts`` (reference ``torch_backend.py`` MoE stages and
``kernels.cu:12612-12862``).
"""
from __future__ import annotations

import ctypes
from ctypes import c_float, c_int, c_void_p

import torch

from . import _lib
from .gemm import gemm, gemm_grouped_k
from .infer import swiglu_forward

__all__ = ["MoEWorkspace", "moe_forward", "moe_reference", "moe_experts", "moe_experts_native_ok"]

GROUPED = 3


def _p(t):
    return c_void_p(0 if t is None else t.data_ptr())


def _st():
    return c_void_p(_lib.stream_ptr())


class MoEWorkspace:
    """Buffers for up to ``max_tokens`` tokens (worst-case padded row capacity)."""

    def __init__(self, max_tokens: int, n_experts: int, top_k: int, d_model: int, d_ff: int, device) -> None:
        cap = (max_tokens * top_k + n_experts * 127 + 127) // 128 * 128
        self.capacity_rows, self.max_tiles = cap, cap // 128
        i32 = dict(dtype=torch.int32, device=device)
        self.logits = torch.empty(max_tokens, n_experts, dtype=torch.float32, device=device)
        self.topk_idx = torch.empty(max_tokens, top_k, **i32)
        self.topk_w = torch.empty(max_tokens, top_k, dtype=torch.float32, device=device)
        self.counts = torch.zeros(n_experts, **i32)
        self.offsets = torch.zeros(n_experts + 1, **i32)
        self.cursor = torch.zeros(n_experts, **i32)
        self.tile_expert = torch.zeros(self.max_tiles, **i32)
        self.plan = torch.zeros(2, **i32)
        self.row_of = torch.empty(max_tokens * top_k, **i32)
        bf = dict(dtype=torch.bfloat16, device=device)
        self.xs = torch.zeros(cap, d_model, **bf)
        self.h = torch.empty(cap, 2 * d_ff, **bf)
        self.a = torch.empty(cap, d_ff, **bf)
        self.ys = torch.empty(cap, d_model, **bf)


def _grouped_gemm(a: torch.Tensor, w: torch.Tensor, out: torch.Tensor, ws: MoEWorkspace) -> None:
    from ..parallel.tp import GemmTpArgs
    E, N, K = w.shape
    args = GemmTpArgs()
    args.mode = GROUPED
    args.a, args.b, args.c = a.data_ptr(), w.data_ptr(), out.data_ptr()
    args.m, args.n, args.k = a.shape[0], N, K
    args.lda, args.ldb, args.ldc = a.stride(0), K, out.stride(0)
    args.tile_group, args.num_m_tiles_dev, args.groups = ws.tile_expert.data_ptr(), ws.plan.data_ptr(), E
    _lib.check(_lib.load().nfn_gemm_tp(ctypes.byref(args), _st()), "nfn_gemm_tp(grouped)")


def moe_forward(x: torch.Tensor, w_router: torch.Tensor, w_gate_up: torch.Tensor, w_down: torch.Tensor, top_k: int, ws: MoEWorkspace, *,
                score_fn: str = "softmax", norm_topk: bool = True, route_scale: float = 1.0, resid: torch.Tensor | None = None,
                out: torch.Tensor | None = None) -> torch.Tensor:
    """x bf16 [T, d] -> bf16 [T, d] (+ resid)."""
    T, d = x.shape
    E, F2, _ = w_gate_up.shape
    F = F2 // 2
    L = _lib.load()
    if E % 8:
        # the GEMM wants N in multiples of 8: pad the router with zero rows once (their logits are
        # never looked at - the routing kernel reads the first E columns only)
        key = (w_router.data_ptr(), w_router._version)
        if getattr(ws, "_router_key", None) != key:
            Ep = (E + 7) // 8 * 8
            ws._router_pad = torch.zeros(Ep, d, dtype=w_router.dtype, device=w_router.device)
            ws._router_pad[:E].copy_(w_router)
            ws._logits_pad = torch.empty(ws.logits.shape[0], Ep, dtype=torch.float32, device=w_router.device)
            ws._router_key = key
        gemm(x, ws._router_pad, out=ws._logits_pad[:T], out_dtype=torch.float32)
        logits = ws._logits_pad
    else:
        gemm(x, w_router, out=ws.logits[:T], out_dtype=torch.float32)
        logits = ws.logits
    ws.counts.zero_()
    _lib.check(L.nfn_moe_route(_p(logits), c_int(logits.stride(0)), c_int(T), c_int(E), c_int(top_k), c_int(1 if score_fn == "sigmoid" else 0),
                               c_int(int(norm_topk)), c_float(route_scale), _p(ws.topk_idx), _p(ws.topk_w), _p(ws.counts), _st()), "nfn_moe_route")
    _lib.check(L.nfn_moe_plan(_p(ws.counts), c_int(E), c_int(ws.max_tiles), _p(ws.offsets), _p(ws.cursor), _p(ws.tile_expert), _p(ws.plan), _st()),
               "nfn_moe_plan")
    _lib.check(L.nfn_moe_permute(_p(x), c_int(x.stride(0)), c_int(T), c_int(top_k), c_int(d), _p(ws.topk_idx), _p(ws.offsets), _p(ws.cursor),
                                 c_int(ws.capacity_rows), _p(ws.xs), _p(ws.row_of), _st()), "nfn_moe_permute")
    _grouped_gemm(ws.xs, w_gate_up, ws.h, ws)
    swiglu_forward(ws.h, F, out=ws.a)
    _grouped_gemm(ws.a, w_down, ws.ys, ws)
    out = torch.empty(T, d, dtype=torch.bfloat16, device=x.device) if out is None else out
    _lib.check(L.nfn_moe_combine(_p(ws.ys), c_int(d), c_int(T), c_int(top_k), _p(ws.row_of), _p(ws.topk_w), _p(resid),
                                 c_int(0 if resid is None else resid.stride(0)), _p(out), c_int(out.stride(0)), _st()), "nfn_moe_combine")
    return out


def moe_reference(x, w_router, w_gate_up, w_down, top_k: int, *, score_fn: str = "softmax", norm_topk: bool = True,
                  route_scale: float = 1.0, resid=None) -> torch.Tensor:
    """fp32 PyTorch oracle of ``moe_forward`` (dense loop over experts)."""
    xf = x.float()
    logits = xf @ w_router.float().T
    scores = torch.sigmoid(logits) if score_fn == "sigmoid" else torch.softmax(logits, -1)
    w, idx = scores.topk(top_k, dim=-1)
    if norm_topk:
        w = w / w.sum(-1, keepdim=True)
    w = w * route_scale
    F = w_gate_up.shape[1] // 2
    out = torch.zeros_like(xf)
    for e in range(w_gate_up.shape[0]):
        sel = (idx == e)
        rows = sel.any(-1).nonzero().flatten()
        if rows.numel() == 0:
            continue
        h = xf[rows] @ w_gate_up[e].float().T
        a = torch.nn.functional.silu(h[:, :F]) * h[:, F:]
        y = a @ w_down[e].float().T
        out[rows] += y * (w[rows] * sel[rows]).sum(-1, keepdim=True)
    return out + (resid.float() if resid is not None else 0)


# --------------------------------------------------------------------------- training path --
class _ExpertsArgs(ctypes.Structure):
    """nfn_moe_experts_args (csrc/kernels/nfn_kernels.h)."""
    _fields_ = [(n, c_void_p) for n in ("x", "w1", "w2", "w3", "weights", "indices", "out", "work")] + \
               [(n, c_int) for n in ("tokens", "d", "ff", "experts", "top", "capacity_rows", "save")] + \
               [(n, c_void_p) for n in ("dout", "scratch", "dx", "dw1", "dw2", "dw3", "dweights")]


def _dense(t: torch.Tensor) -> torch.Tensor:
    """Contiguous and 16-byte aligned, as the kernels' wide loads and tile copies want it."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _experts_lib():
    L = _lib.load()
    L.nfn_moe_experts_work_bytes.restype = L.nfn_moe_experts_scratch_bytes.restype = ctypes.c_longlong
    return L


class _MoEExpertsFn(torch.autograd.Function):
    """Dropless expert FFN with gradients. Inputs in the tensor-runtime layout: x [T, d] bf16,
    w1 / w3 [E, d, h] (gate / up), w2 [E, h, d], routing weights [T, k] (any float dtype) and
    indices [T, k] (int64). One native call per direction (``csrc/kernels/moe_experts.cu``): a stable
    sort of the rows by expert, grouped tcgen05 products on the weights as they are stored with
    SwiGLU and its derivative in their epilogues, weighted combine; routing weights get
    <expert output, upstream gradient>, the weight gradients of all experts come from grouped contractions.

    Reference counterparts: ``moe_swiglu_forward/backward`` (``kernels.cu:12612-12862``), which
    loop per token over its k experts with dense weights and no permutation."""

    @staticmethod
    def forward(ctx, x, w1, w2, w3, weights, indices):
        T, d = x.shape
        E, _, h = w1.shape
        k = indices.shape[-1]
        L = _experts_lib()
        x, d1, d2, d3 = _dense(x), _dense(w1), _dense(w2), _dense(w3)
        wt, idx = weights.to(torch.float32).contiguous(), indices.to(torch.int64).contiguous()
        a = _ExpertsArgs(x=x.data_ptr(), w1=d1.data_ptr(), w2=d2.data_ptr(), w3=d3.data_ptr(), weights=wt.data_ptr(), indices=idx.data_ptr(),
                         tokens=T, d=d, ff=h, experts=E, top=k, capacity_rows=(T * k + E * 127 + 127) // 128 * 128,
                         save=int(any(ctx.needs_input_grad)))
        work = torch.empty(L.nfn_moe_experts_work_bytes(ctypes.byref(a)), dtype=torch.uint8, device=x.device)
        out = torch.empty(T, d, dtype=torch.bfloat16, device=x.device)
        a.work, a.out = work.data_ptr(), out.data_ptr()
        _lib.check(L.nfn_moe_experts_forward(ctypes.byref(a), _st()), "nfn_moe_experts_forward")
        if a.save:
            ctx.save_for_backward(w1, w2, w3, wt)
            ctx.work, ctx.dims, ctx.w_dtype = work, (T, d, E, h, k, a.capacity_rows), weights.dtype
        return out

    @staticmethod
    def backward(ctx, dout):
        w1, w2, w3, wt = ctx.saved_tensors
        T, d, E, h, k, capacity = ctx.dims
        L, work = _experts_lib(), ctx.work
        dout, d1, d2, d3 = _dense(dout), _dense(w1), _dense(w2), _dense(w3)
        dx, dweights = torch.empty_like(dout), torch.empty_like(wt)
        dw1, dw2, dw3 = (torch.empty(w.shape, dtype=w.dtype, device=w.device) for w in (w1, w2, w3))
        a = _ExpertsArgs(w1=d1.data_ptr(), w2=d2.data_ptr(), w3=d3.data_ptr(), weights=wt.data_ptr(), work=work.data_ptr(),
                         tokens=T, d=d, ff=h, experts=E, top=k, capacity_rows=capacity, save=1, dout=dout.data_ptr(), dx=dx.data_ptr(),
                         dw1=dw1.data_ptr(), dw2=dw2.data_ptr(), dw3=dw3.data_ptr(), dweights=dweights.data_ptr())
        scratch = torch.empty(L.nfn_moe_experts_scratch_bytes(ctypes.byref(a)), dtype=torch.uint8, device=dout.device)
        a.scratch = scratch.data_ptr()
        _lib.check(L.nfn_moe_experts_backward(ctypes.byref(a), _st()), "nfn_moe_experts_backward")
        ctx.work = None
        return dx, dw1, dw2, dw3, dweights.to(ctx.w_dtype), None


class _MoEExpertsStagedFn(torch.autograd.Function):
    """The same for what the native call does not take: widths that are multiples of eight but not of 64 (its tiles walk whole 64-value blocks), more than
    eight experts per token (it keeps a token's rows in registers), no tokens. One kernel per stage on K-major copies of the weights: 7.0 ms at
    8192 tokens x 2048, 64 experts of 1024, top 8, where the native call takes 2.8."""

    @staticmethod
    def forward(ctx, x, w1, w2, w3, weights, indices):
        T, d = x.shape
        E, _, h = w1.shape
        k = indices.shape[-1]
        L = _lib.load()
        ws = MoEWorkspace(T, E, k, d, h, x.device)
        ws.topk_idx.copy_(indices)
        ws.topk_w.copy_(weights)
        ws.counts.copy_(torch.bincount(indices.reshape(-1), minlength=E))
        w_gu = torch.cat([w1.transpose(1, 2), w3.transpose(1, 2)], 1).contiguous()  # [E, 2h, d]
        w_dn = w2.transpose(1, 2).contiguous()                                     # [E, d, h]
        _lib.check(L.nfn_moe_plan(_p(ws.counts), c_int(E), c_int(ws.max_tiles), _p(ws.offsets), _p(ws.cursor), _p(ws.tile_expert), _p(ws.plan), _st()),
                   "nfn_moe_plan")
        _lib.check(L.nfn_moe_permute(_p(x), c_int(x.stride(0)), c_int(T), c_int(k), c_int(d), _p(ws.topk_idx), _p(ws.offsets), _p(ws.cursor),
                                     c_int(ws.capacity_rows), _p(ws.xs), _p(ws.row_of), _st()), "nfn_moe_permute")
        _grouped_gemm(ws.xs, w_gu, ws.h, ws)
        swiglu_forward(ws.h, h, out=ws.a)
        _grouped_gemm(ws.a, w_dn, ws.ys, ws)
        out = torch.empty(T, d, dtype=torch.bfloat16, device=x.device)
        _lib.check(L.nfn_moe_combine(_p(ws.ys), c_int(d), c_int(T), c_int(k), _p(ws.row_of), _p(ws.topk_w), _p(None), c_int(0), _p(out),
                                     c_int(out.stride(0)), _st()), "nfn_moe_combine")
        ctx.ws, ctx.dims = ws, (T, d, E, h, k)
        ctx.save_for_backward(w1, w2, w3)
        ctx.w_dtype = weights.dtype
        return out

    @staticmethod
    def backward(ctx, dout):
        from .infer import swiglu_backward
        w1, w2, w3 = ctx.saved_tensors
        ws, (T, d, E, h, k) = ctx.ws, ctx.dims
        dout = dout.contiguous()
        rows = ws.row_of.long()                                         # [T * k] sorted row of every (token, slot)
        # routing-weight gradient and the upstream gradient of every sorted row
        ys_tk = ws.ys[rows].view(T, k, d)
        d_w = torch.einsum("tkd,td->tk", ys_tk.float(), dout.float())
        dys = torch.zeros_like(ws.ys)
        dys[rows] = (dout[:, None, :].float() * ws.topk_w[:, :, None]).to(torch.bfloat16).view(T * k, d)
        # input gradients through the two grouped GEMMs (weights as stored are the [E, N, K] operands)
        da = torch.empty_like(ws.a)
        _grouped_gemm(dys, w2.contiguous(), da, ws)                     # [cap, h] = dys @ w2[e]^T
        dh = swiglu_backward(ws.h, da, h)                               # [cap, 2h]
        dxs = torch.empty_like(ws.xs)
        _grouped_gemm(dh, torch.cat([w1, w3], 2).contiguous(), dxs, ws)  # [cap, d] = dh @ [w1 | w3][e]^T
        dx = dxs[rows].view(T, k, d).float().sum(1).to(torch.bfloat16)
        # weight gradients of all experts: three grouped contractions over the plan's padded row segments (pad rows of xs and
        # dys are zero, those of a and dh are finite), no host read of the counts
        dw1, dw2, dw3 = torch.empty_like(w1), torch.empty_like(w2), torch.empty_like(w3)
        gemm_grouped_k(ws.xs, dh[:, :h], ws.offsets, dw1)               # [E, d, h] = xs^T dh_gate
        gemm_grouped_k(ws.xs, dh[:, h:], ws.offsets, dw3)
        gemm_grouped_k(ws.a, dys, ws.offsets, dw2)                      # [E, h, d] = a^T dys
        ctx.ws = None
        return dx, dw1, dw2, dw3, d_w.to(ctx.w_dtype), None


def moe_experts_native_ok(x: torch.Tensor, w1: torch.Tensor, w2: torch.Tensor, w3: torch.Tensor, indices: torch.Tensor) -> bool:
    E, d, h = w1.shape
    return (x.is_cuda and x.dtype == torch.bfloat16 and w1.dtype == w2.dtype == w3.dtype == torch.bfloat16 and _lib.available()
            and d % 64 == 0 and h % 64 == 0 and E <= 256 and indices.shape[-1] <= 8 and x.shape[0] > 0)


_WHOLE = frozenset((torch.uint8, torch.int8, torch.int16, torch.int32, torch.int64))


def _expert_operands(x, w1, w2, w3, weights, indices):
    """The routing weights as [T, k] and the indices as whole numbers, both on x's device. The kernels get addresses only, so whatever does not fit x and
    the others is refused here. Operands that lie as the kernels want them make no call into torch but reads of their fields: a short batch is bound by
    what the host does."""
    sx, s1, si = x.shape, w1.shape, indices.shape
    if len(sx) != 2 or len(s1) != 3 or len(si) not in (1, 2):
        raise RuntimeError(f"moe_experts: x {tuple(sx)}, w1 {tuple(s1)}, indices {tuple(si)}: need [T, d], [E, d, h], [T, k]")
    (T, d), (E, d1, h), k = sx, s1, si[-1]
    if d1 != d or w3.shape != s1 or w2.shape != (E, h, d):
        raise RuntimeError(f"moe_experts: w1 {tuple(s1)}, w3 {tuple(w3.shape)} must be [E, {d}, h], w2 {tuple(w2.shape)} [E, h, {d}]")
    if (si != (T, k) and (T != 1 or len(si) != 1)) or indices.dtype not in _WHOLE:
        raise RuntimeError(f"moe_experts: indices {tuple(si)} {indices.dtype}: need whole numbers, k for each of {T} tokens")
    bf = torch.bfloat16
    if not (x.dtype is bf and w1.dtype is bf and w2.dtype is bf and w3.dtype is bf):
        raise RuntimeError("moe_experts: x, w1, w2 and w3 must be bf16")
    device = x.device
    if not (w1.device == device and w2.device == device and w3.device == device):
        raise RuntimeError("moe_experts: w1, w2 and w3 must be on the device of x")
    if weights.shape != (T, k) or weights.device != device:
        weights = weights.to(device).expand(T, k)
    if len(si) != 2 or indices.device != device:
        indices = indices.to(device).reshape(T, k)
    return weights, indices


def moe_experts(x: torch.Tensor, w1: torch.Tensor, w2: torch.Tensor, w3: torch.Tensor, weights: torch.Tensor, indices: torch.Tensor) -> torch.Tensor:
    """Differentiable expert FFN on the native kernels (see ``_MoEExpertsFn``, ``_MoEExpertsStagedFn``). ``weights`` of one column, one row or one number are
    expanded; weights and indices may lie on the host."""
    weights, indices = _expert_operands(x, w1, w2, w3, weights, indices)
    if not x.is_cuda:
        raise RuntimeError("moe_experts: x must be on a CUDA device")
    (T, k), (_, d, h) = indices.shape, w1.shape
    native = T > 0 and 0 < k <= 8 and d % 64 == 0 and h % 64 == 0
    return (_MoEExpertsFn if native else _MoEExpertsStagedFn).apply(x.contiguous(), w1, w2, w3, weights, indices)

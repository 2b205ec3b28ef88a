"""Backward pass of the W8A8 LoRA linear (straight-through estimator).

The reference defines the operator as a `jax.custom_vjp` whose backward treats both quantisers as the
identity and the frozen base as its dequantised weight (`_quantized_lora_linear_bwd`,
skyrl/tx/kernels/quantized_lora.py:337-394):

    R  = s * (dy @ B^T)
    dx = dy @ deq(W)^T + R @ A^T          (dominant: an [M, N] x [N, K] contraction)
    dA = x^T @ R,   dB = s * (x @ A)^T @ dy,   ds = sum(dy * ((x @ A) @ B))

Here the dominant contraction runs on the same tcgen05 int8 path as the forward: the weight's
per-output-channel scale moves to the cotangent, g = dy * sw, each row of g is split into two int8 planes
(`skyrl_w8a8_grad_quant_sm100_v1`), and one GEMM over a TRANSPOSED packed copy of the codes multiplies both planes
with every weight tile it loads.  dx therefore equals the fp32 product to about 2^-15 relative (two planes), far
inside bf16's own rounding, at the cost of one bf16 GEMM, and `R @ A^T` rides the same launch as `s (x A) B` does in
the forward.  dA and dB contract x and dy with the two LoRA projections (the forward's, which it keeps, and the
cotangent's, which dx needs anyway) in one launch over the adapters' row ranges.

A training step takes the LoRA tables in the reference's layout, [A, K, r] and [A, r, N]: they change at every
optimizer step, so the forward lays them out for its kernels in one launch and the backward, whose operator is the
transposed one, reads them as they are.

`W8A8LoRALinearFunction` ties forward and backward together for `torch.autograd`, the counterpart of the
reference's `quantized_lora_linear.defvjp(...)` (quantized_lora.py:397).
"""

from __future__ import annotations

import ctypes as C
from dataclasses import dataclass

import torch

from . import _lib, ops
from .ops import EPI_LINEAR, LORA_RANK_PAD, Z_PARTS, PackedLoRA, PackedW8Weight


@dataclass(frozen=True)
class PackedW8Backward:
    """What the input gradient needs from a frozen weight: the codes packed with N as the contraction
    dimension and the forward scales as a column vector.  Built once per weight at load time."""

    wq_t: PackedW8Weight     # in_features = padded N of the forward weight, out_features = K, scales 1
    col_scale: torch.Tensor  # fp32 [padded N]: the forward weight's per-output-channel scales
    in_features: int         # K of the forward weight
    out_features: int        # N of the forward weight


def pack_weight_backward(weight) -> PackedW8Backward:
    """Forward weight (reference storage or packed) -> its backward companion."""
    w = ops._weight_of(weight)
    if w.group_size:
        raise ops.SkyrlKernelError("the backward path takes per-output-channel scales (one group over K)")
    k, npad = w.in_features, w.padded_out_features
    if k % 32:
        raise ValueError(f"the input gradient needs K to be a multiple of 32, got {k}")
    kb, _, blk = w.wq.shape
    codes_kn = w.wq.permute(0, 2, 1).reshape(kb * blk, npad)[:k].contiguous()   # [K, padded N]: rows = outputs of W^T
    ones = torch.ones((k,), dtype=torch.float32, device=w.wq.device)
    return PackedW8Backward(ops.pack_weight_nk(codes_kn, ones), w.sw.contiguous(), k, w.out_features)


def pack_lora_backward(lora_a: torch.Tensor, lora_b: torch.Tensor, lora_scaling, weight_bwd: PackedW8Backward) -> PackedLoRA:
    """LoRA tables of the transposed operator: "A" = B^T [A, N, r], "B" = A^T [A, r, K], same scaling, so that
    s (dy B^T) A^T is the forward LoRA expression of the transposed weight."""
    if lora_a.ndim == 2:
        lora_a, lora_b = lora_a[None], lora_b[None]
    return ops.pack_lora(lora_b.transpose(1, 2).contiguous(), lora_a.transpose(1, 2).contiguous(), lora_scaling,
                         in_features=weight_bwd.wq_t.in_features,
                         padded_out_features=weight_bwd.wq_t.padded_out_features)


def w8a8_lora_linear_input_grad(dy: torch.Tensor, weight_bwd: PackedW8Backward, lora_bwd: PackedLoRA | None = None,
                                adapter_ids=None, *, planes: int = 2, enabled: bool = False) -> torch.Tensor:
    """dx = dy @ deq(W)^T + s (dy @ B^T) @ A^T as bf16 [..., K] (quantized_lora.py:364-372)."""
    ops._validate_exact_bool("enabled", enabled)
    if not enabled:
        raise RuntimeError("the W8A8 backward kernel is disabled by default")
    if planes not in (1, 2):
        raise ValueError("planes must be 1 or 2")
    lib = _lib.load()
    wt = weight_bwd.wq_t
    n_logical, npad, k = weight_bwd.out_features, wt.in_features, wt.out_features
    dy2 = ops._pad_cols(ops._check_x(dy, n_logical), npad)
    m, dev = dy2.shape[0], dy2.device
    na = lora_bwd.num_adapters if lora_bwd is not None else 1
    ids = ops._check_ids(adapter_ids, m, lora_bwd)
    st = ops._status_word(dev)
    if planes == 2:
        a = _train_args(m, npad, k, n_logical, lora_bwd.rank if lora_bwd is not None else 0, na, st)
        a.dy, a.dy_row_stride = dy2.data_ptr(), dy2.stride(0)
        a.wq, a.sw = wt.wq.data_ptr(), weight_bwd.col_scale.data_ptr()
        if lora_bwd is not None:
            table = lora_bwd.b_rows if lora_bwd.b_rows is not None else lora_bwd.b
            a.lora_scaling = lora_bwd.scaling.data_ptr()
            a.bwd_a, a.bwd_a_rows, a.bwd_a_cols = lora_bwd.a.data_ptr(), lora_bwd.a.shape[1], lora_bwd.a.shape[2]
            a.bwd_b, a.bwd_b_slots = table.data_ptr(), table.shape[2]
        a.adapter_ids = ids.data_ptr() if ids is not None else None
        dx = torch.empty((m, k), dtype=torch.bfloat16, device=dev)
        a.dx = dx.data_ptr()
        _owner = _with_scratch(a, dev, True)
        _lib.check(lib.skyrl_w8a8_train_backward_sm100_v1(C.byref(a), ops._stream()), "train_backward (input gradient)")
        return dx.reshape(*dy.shape[:-1], k)
    # one plane: the int8 step of the cotangent stays visible in dx; same kernels as the forward
    perm, tiles, num = ops.prepare_routing(ids, m, na)
    row_map = perm if ids is not None else None
    max_tiles = tiles.shape[0]

    q = torch.empty((m, npad), dtype=torch.int8, device=dev)
    s = torch.empty((m,), dtype=torch.float32, device=dev)
    _lib.check(lib.skyrl_w8a8_grad_quant_sm100_v1(
        ops._ptr(dy2), dy2.stride(0), ops._ptr(weight_bwd.col_scale), ops._ptr(row_map), m, npad, ops._ptr(q), ops._ptr(s),
        None, None, ops._stream()), "grad_quant")

    z_parts = None
    if lora_bwd is not None:
        if ids is not None:
            _, _, ys = ops.rms_quant(dy2, row_map=perm, want_normalized=True)   # dy rows in adapter-sorted order
        else:
            ys = dy2.contiguous()
        z_parts = torch.empty((m, Z_PARTS, LORA_RANK_PAD), dtype=torch.bfloat16, device=dev)
        _lib.check(lib.skyrl_lora_a_proj_sm100_v1(ops._ptr(ys), m, npad, ops._ptr(lora_bwd.a), ops._ptr(lora_bwd.scaling),
                                                  na, lora_bwd.rank, ops._ptr(tiles), ops._ptr(num), max_tiles,
                                                  ops._ptr(z_parts), ops._ptr(st), ops._stream()), "lora_a_proj (backward)")

    dx = torch.empty((m, k), dtype=torch.bfloat16, device=dev)
    a = _lib.GemmArgs()
    a.struct_size = C.sizeof(_lib.GemmArgs)
    a.epilogue = EPI_LINEAR
    a.m, a.n, a.k = m, k, npad
    a.xq, a.sx, a.sw = q.data_ptr(), s.data_ptr(), wt.sw.data_ptr()
    a.wq = wt.wq.data_ptr()
    a.rank = lora_bwd.rank if lora_bwd is not None else 0
    a.num_adapters = na
    a.max_tiles = max_tiles
    if a.rank:
        a.z_parts, a.lora_b_packed = z_parts.data_ptr(), lora_bwd.b.data_ptr()
    a.tiles, a.num_tiles = tiles.data_ptr(), num.data_ptr()
    a.out_row_map = row_map.data_ptr() if row_map is not None else None
    a.out, a.out_row_stride = dx.data_ptr(), k
    a.status = st.data_ptr()
    _lib.check(lib.skyrl_w8a8_gemm_sm100_v1(C.byref(a), ops._stream()), "w8a8_gemm (input gradient)")
    return dx.reshape(*dy.shape[:-1], k)


def _train_args(m: int, n: int, k: int, n_logical: int, rank: int, adapters: int, status: torch.Tensor):
    a = _lib.TrainArgs()
    a.struct_size = C.sizeof(_lib.TrainArgs)
    a.m, a.n, a.k, a.n_logical, a.rank, a.num_adapters = m, n, k, n_logical, rank, adapters
    a.status = status.data_ptr()
    return a


def _with_scratch(a, device, backward: bool) -> torch.Tensor:
    """Gives `a` scratch of its own and returns its owner, which has to live until the call is enqueued."""
    a.workspace_bytes = _lib.load().skyrl_w8a8_train_workspace_bytes(a.m, a.n, a.k, a.rank, a.num_adapters, backward)
    owner, a.workspace = ops._scratch(device, a.workspace_bytes)
    return owner


def _mm_f32(a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
    """fp32 result of a @ b.  bf16 operands on a CUDA device multiply on the tensor cores (products of bf16 pairs are
    exact in the fp32 accumulator) without an fp32 copy of either operand; anything else takes the plain fp32 path."""
    if a.is_cuda and a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16:
        return torch.mm(a, b, out_dtype=torch.float32)
    return a.float() @ b.float()


def _split_bf16(t: torch.Tensor):
    """fp32 -> (hi, lo) bf16 with hi + lo == t to 2^-17 relative: keeps a small fp32 factor exact enough for a bf16
    tensor-core matmul against a large bf16 operand."""
    hi = t.to(torch.bfloat16)
    return hi, (t - hi.float()).to(torch.bfloat16)


def lora_parameter_grads(x: torch.Tensor, dy: torch.Tensor, lora_a: torch.Tensor, lora_b: torch.Tensor, lora_scaling,
                         adapter_ids=None):
    """(dA [A, K, r], dB [A, r, N], ds [A]) in fp32 (quantized_lora.py:374-389), rows grouped by adapter.

    Library matmuls.  Each gradient is a rank-r reduction over the rows: U = x A and R' = dy B^T are [M, r]; then
    dA = x^T (s R'), dB = s U^T dy and ds = sum(U * R') (the reference's sum(dy * (U B)) with the contraction over N
    done first).  On a CUDA device the large operands x and dy stay bf16: the small fp32 factors are split into two
    bf16 terms, so every product runs on the tensor cores with fp32 accumulation."""
    squeeze = lora_a.ndim == 2
    if squeeze:
        lora_a, lora_b = lora_a[None], lora_b[None]
    na, k, r = lora_a.shape
    n = lora_b.shape[2]
    x2 = x.reshape(-1, k)
    dy2 = dy.reshape(-1, n)
    m = x2.shape[0]
    scaling = torch.as_tensor(lora_scaling, dtype=torch.float32, device=x.device).reshape(-1)
    d_a = torch.zeros((na, k, r), dtype=torch.float32, device=x.device)
    d_b = torch.zeros((na, r, n), dtype=torch.float32, device=x.device)
    d_s = torch.zeros((na,), dtype=torch.float32, device=x.device)
    if adapter_ids is None:
        xs, gs, counts = x2, dy2, [m] + [0] * (na - 1)
    else:
        ids = adapter_ids.reshape(-1).to(torch.int64)
        order = torch.argsort(ids, stable=True)
        counts = torch.bincount(ids, minlength=na).tolist()
        xs, gs = x2[order], dy2[order]            # one gather; the adapters' rows are then contiguous slices
    fast = xs.is_cuda and xs.dtype == torch.bfloat16 and gs.dtype == torch.bfloat16
    start = 0
    for a, count in enumerate(counts):
        if count == 0:
            continue
        xa, ga = xs[start:start + count], gs[start:start + count]
        start += count
        inter = _mm_f32(xa, lora_a[a])                       # U  [Ma, r]
        low_unscaled = _mm_f32(ga, lora_b[a].t())            # R' [Ma, r]
        low = low_unscaled * scaling[a]
        if fast:
            low_hi, low_lo = _split_bf16(low)
            int_hi, int_lo = _split_bf16(inter)
            xat, gat = xa.t(), ga
            d_a[a] = _mm_f32(xat, low_hi) + _mm_f32(xat, low_lo)
            d_b[a] = (_mm_f32(int_hi.t(), gat) + _mm_f32(int_lo.t(), gat)) * scaling[a]
        else:
            d_a[a] = xa.float().t() @ low
            d_b[a] = (inter.t() @ ga.float()) * scaling[a]
        d_s[a] = (inter * low_unscaled).sum()
    if squeeze:
        return d_a[0], d_b[0], d_s[0]
    return d_a, d_b, d_s


class W8A8LoRALinearFunction(torch.autograd.Function):
    """y = w8a8_lora_linear(x, W, A, B, s, ids) with the reference's straight-through backward
    (quantized_lora.py:317-397).  The frozen weight receives no gradient."""

    @staticmethod
    def forward(ctx, x, lora_a, lora_b, lora_scaling, weight, weight_bwd, adapter_ids):
        w = ops._weight_of(weight)
        if w.group_size:
            raise ops.SkyrlKernelError("the backward path takes per-output-channel scales (one group over K)")
        k, npad, n = w.in_features, w.padded_out_features, w.out_features
        k_logical = weight.original_in_features if isinstance(weight, ops.GroupQuantizedWeight) else k
        x2 = ops._pad_cols(ops._check_x(x, k_logical), k)
        m, dev = x2.shape[0], x2.device
        a3, b3, scaling = _tables(lora_a, lora_b, lora_scaling, k, n)
        na, _, rank = a3.shape
        if adapter_ids is None and na != 1:
            raise ValueError("adapter_ids is required when the LoRA tables hold more than one adapter")
        ids = ops._check_ids(adapter_ids, m, None)
        lib = _lib.load()
        saved = torch.empty(lib.skyrl_w8a8_train_saved_bytes(m, na), dtype=torch.uint8, device=dev)
        y = torch.empty((m, npad), dtype=torch.bfloat16, device=dev)
        a = _train_args(m, npad, k, n, rank, na, ops._status_word(dev))
        a.x, a.x_row_stride = x2.data_ptr(), x2.stride(0)
        a.wq, a.sw = w.wq.data_ptr(), w.sw.data_ptr()
        a.lora_a, a.lora_b, a.lora_scaling = a3.data_ptr(), b3.data_ptr(), scaling.data_ptr()
        a.adapter_ids = ids.data_ptr() if ids is not None else None
        a.y = y.data_ptr()
        _with_saved(a, saved)
        _owner = _with_scratch(a, dev, False)
        _lib.check(lib.skyrl_w8a8_train_forward_sm100_v1(C.byref(a), ops._stream()), "train_forward")
        ctx.save_for_backward(x, lora_a, lora_b, lora_scaling, ids, saved)
        ctx.weight_bwd = weight_bwd
        return y[:, :n].reshape(*x.shape[:-1], n)

    @staticmethod
    def backward(ctx, dy):
        x, lora_a, lora_b, lora_scaling, ids, saved = ctx.saved_tensors
        wb = ctx.weight_bwd
        k, n, npad = wb.in_features, wb.out_features, wb.wq_t.in_features
        x2 = ops._pad_cols(x.reshape(-1, x.shape[-1]), k)
        dy2 = ops._pad_cols(ops._check_x(dy, n), npad)
        m, dev = dy2.shape[0], dy2.device
        a3, b3, scaling = _tables(lora_a, lora_b, lora_scaling, k, n)
        na, _, rank = a3.shape
        # the transposed operator's tables are B and A themselves, padded where a row is no multiple of 16 bytes
        table_b = a3 if rank % 8 == 0 else torch.nn.functional.pad(a3, (0, -rank % 8))
        table_a = b3 if n % 8 == 0 else torch.nn.functional.pad(b3, (0, -n % 8))
        d_a = torch.empty((na, k, rank), dtype=torch.bfloat16, device=dev)
        d_b = torch.empty((na, rank, n), dtype=torch.bfloat16, device=dev)
        dx = torch.empty((m, k), dtype=torch.bfloat16, device=dev) if ctx.needs_input_grad[0] else None
        a = _train_args(m, npad, k, n, rank, na, ops._status_word(dev))
        a.x, a.x_row_stride = x2.data_ptr(), x2.stride(0)
        a.dy, a.dy_row_stride = dy2.data_ptr(), dy2.stride(0)
        a.wq, a.sw = wb.wq_t.wq.data_ptr(), wb.col_scale.data_ptr()
        a.lora_scaling = scaling.data_ptr()
        a.adapter_ids = ids.data_ptr() if ids is not None else None
        a.bwd_a, a.bwd_a_rows, a.bwd_a_cols = table_a.data_ptr(), rank, table_a.shape[2]
        a.bwd_b, a.bwd_b_slots = table_b.data_ptr(), table_b.shape[2]
        a.dx = dx.data_ptr() if dx is not None else None
        a.da, a.db = d_a.data_ptr(), d_b.data_ptr()
        saved = _with_saved(a, saved)
        _owner = _with_scratch(a, dev, True)
        _lib.check(_lib.load().skyrl_w8a8_train_backward_sm100_v1(C.byref(a), ops._stream()), "train_backward")
        d_s = None
        if ctx.needs_input_grad[3]:   # rarely wanted (alpha / r is a constant): library matmuls
            d_s = lora_parameter_grads(x.detach(), dy.contiguous(), lora_a.detach(), lora_b.detach(), lora_scaling.detach(), ids)[2]
            d_s = d_s.reshape(lora_scaling.shape).to(lora_scaling.dtype)
        if lora_a.shape[-2] != k:   # a K that the packed weight rounds up to a multiple of 16
            d_a = d_a[:, :lora_a.shape[-2]]
        if dx is not None:
            dx = (dx if x.shape[-1] == k else dx[:, :x.shape[-1]]).reshape(x.shape)
        return (dx, d_a.reshape(lora_a.shape), d_b.reshape(lora_b.shape), d_s, None, None, None)


def _tables(lora_a, lora_b, lora_scaling, k: int, n: int):
    """LoRA tables in the reference's layout (one adapter as matrices, or a stack) as contiguous [A, K, r], [A, r, N], [A].
    K is the packed weight's, a multiple of 16: shorter tables are padded with zeros."""
    ops._require_cuda(lora_a, "lora_a")
    ops._require_cuda(lora_b, "lora_b")
    if lora_a.dtype != torch.bfloat16 or lora_b.dtype != torch.bfloat16:
        raise TypeError("LoRA A and B must both be BF16")
    if lora_a.ndim == 2 and lora_b.ndim == 2:
        lora_a, lora_b = lora_a[None], lora_b[None]
    if lora_a.ndim != 3 or lora_b.ndim != 3:
        raise ValueError("lora_a and lora_b must both be rank-two or both rank-three")
    na, ka, r = lora_a.shape
    if lora_b.shape[:2] != (na, r):
        raise ValueError(f"incompatible LoRA shapes: A={tuple(lora_a.shape)}, B={tuple(lora_b.shape)}")
    if not ka <= k < ka + 16 or lora_b.shape[2] != n:
        raise ValueError(f"LoRA tables of {ka} and {lora_b.shape[2]} features do not match the weight's {k} and {n}")
    if r > ops.MAX_LORA_RANK:
        raise ValueError(f"LoRA rank must not exceed {ops.MAX_LORA_RANK}, got {r}")
    scaling = lora_scaling.detach().reshape(-1)
    if scaling.dtype != torch.float32 or not scaling.is_cuda:
        scaling = scaling.to(device=lora_a.device, dtype=torch.float32)
    if scaling.numel() != na:
        raise ValueError(f"lora_scaling must have {na} entries, got {scaling.numel()}")
    lora_a = lora_a.detach()
    if ka != k:
        lora_a = torch.nn.functional.pad(lora_a, (0, 0, 0, k - ka))
    return _dense(lora_a), _dense(lora_b.detach()), scaling.contiguous()


def _dense(t: torch.Tensor) -> torch.Tensor:
    """Contiguous and 16-byte aligned, as tensor maps need it: a table may be a view into a flat parameter buffer."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.contiguous_format)


def _with_saved(a, saved: torch.Tensor) -> torch.Tensor:
    """Points `a` at the buffer the forward keeps.  Its layout starts at its first byte: between the passes it may have been
    moved (hooks on saved tensors take it to the host and back).  Returns the tensor that has to live until the call is
    enqueued."""
    saved = _dense(saved)
    a.saved, a.saved_bytes = saved.data_ptr(), saved.numel()
    return saved


def w8a8_lora_linear_trainable(x, weight, weight_bwd: PackedW8Backward, lora_a, lora_b, lora_scaling, adapter_ids=None):
    """Differentiable form of `ops.w8a8_lora_linear` (x, A, B and the scaling receive gradients)."""
    scaling = lora_scaling if isinstance(lora_scaling, torch.Tensor) else torch.as_tensor(
        lora_scaling, dtype=torch.float32, device=x.device)
    return W8A8LoRALinearFunction.apply(x, lora_a, lora_b, scaling, weight, weight_bwd, adapter_ids)

"""Python side of the sm_100a kernels: argument checks, output allocation, ctypes launches.

Every launcher validates shapes/strides/alignment on the host before the launch (the GPU pool has no
compute-sanitizer), launches on the current torch stream, and returns torch tensors.  A nonzero
return code from the native side raises.  ``check_status()`` reads the device status word that
bounded waits write when they give up.
"""

from __future__ import annotations

import ctypes
import os
from ctypes import c_int, c_longlong, c_void_p

import torch
from torch import Tensor

from . import _lib

launch_count = 0  # number of native kernel launches issued through this module (for benchmarks)

EPI_BIAS, EPI_RESIDUAL, EPI_ACCUM, EPI_OUT_F32 = 1, 2, 4, 8
EPI_GLU_GELU, EPI_GLU_SILU, EPI_BIAS_F32, EPI_NO_OUT, EPI_ACT_GELU, EPI_GATE = 16, 32, 64, 128, 256, 512

_status_ptr: dict[int, int] = {}


_call = _lib.entry


def _raw_stream() -> int:
    # the handle alone: building a Stream object for every launch took a sixth of a small training step's host time
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def _stream() -> c_void_p:
    return c_void_p(_raw_stream())


def _ptr(t: Tensor | None) -> int | None:
    return t.data_ptr() if t is not None else None


def _check(rc: int, what: str) -> None:
    if rc != 0:
        raise RuntimeError(f"native {what} failed with code {rc}")


def status_pointer() -> int:
    dev = torch.cuda.current_device()
    if dev not in _status_ptr:
        out = c_void_p(0)
        _check(_lib.load("elementwise").otb_status_alloc(ctypes.byref(out)), "status_alloc")
        _status_ptr[dev] = out.value
    return _status_ptr[dev]


def check_status(reset: bool = True) -> None:
    """Raises if any kernel reported a timed-out wait since the last check (synchronises)."""
    dev = torch.cuda.current_device()
    if dev not in _status_ptr:
        return
    torch.cuda.synchronize()
    buf = (ctypes.c_uint * 4)()
    _check(_lib.load("elementwise").otb_status_read(c_void_p(_status_ptr[dev]), buf, int(reset)), "status_read")
    if buf[0] != 0:
        raise RuntimeError(f"kernel wait timed out: kernel={buf[0] >> 16} stage={buf[0] & 0xffff} "
                           f"block={buf[1]} detail={buf[2]} reports={buf[3]}")


# --------------------------------------------------------------------------------------------- GEMM
SKINNY = os.environ.get("OPENTAU_B200_SKINNY_GEMM", "1") != "0"


def use_skinny(layout: str, M: int, N: int, accumulate: bool, bn: int, K: int = 0, gated: bool = True,
               end: str = "", no_grad: bool = True) -> bool:
    """``x @ W^T`` with few rows goes to the weight-streaming split-K kernel.  ``gated``: the product ends in a gated
    residual, which only that kernel fuses (the gate then multiplies the fp32 sum); ``end``: "act" or "glu" where it ends in an
    activation or a gated MLP's product; ``no_grad``: nothing is differentiated through it."""
    if not SKINNY or layout != "nt" or accumulate or bn:
        return False
    if gated:
        # the alternative rounds the sum to bf16 in front of the gate: every few-row product keeps the fusion, but for
        # more columns than the 128 x 256 tiles of the persistent kernel need to fill the chip.  Up to 640 rows where two CTAs
        # may share the sums of 64-row chunks: 400 x 1024 x 4096 20.6 -> 12.4 us with the norm behind it against the persistent
        # kernel and a gated residual of its own, 640 x 1280 x 2048 15.0 -> 12.0; without the room 600 x 2048 x 2048 16.3 -> 17.3
        return M <= 128 or (M <= 256 and N <= 8192) or (M <= 640 and N <= 2048 and -(-N // 128) * -(-M // 64) <= 148)
    if M <= 64 or (M <= 256 and N <= 2048 and K >= 3072):
        return True
    # a product that is differentiated keeps the persistent kernel and with it the order of its sums: few of a training pass are this small
    return no_grad and end != "glu" and M <= 768 and N <= 6144 and _few_row_wins(M, N, K, end)


def _few_row_wins(M: int, N: int, K: int, end: str) -> bool:
    """Products of 65 - 768 rows of an inference pass: up to one CTA of 128 columns x 64 rows to an SM, fewer where the sum is short."""
    tiles = -(-N // 128) * -(-M // 64)
    if end:
        # with an activation it wins on half as many tiles: 256 x 1024 x 1024 7.2 / 9.4 us (few-row / persistent kernel), 128 x 4304 x 1152
        # 8.7 / 10.1, 256 x 4304 x 1152 11.4 / 10.6; with a gated MLP's product on narrow ones alone (200 x 4096 x 1024 10.2 / 9.8)
        return tiles <= 74
    if tiles > 148 or K < 128:
        return False
    # The persistent kernel's cost is one round of tiles whatever their number; the few-row kernel's grows with the area, the less the
    # longer the sum that it splits.  us in a replayed graph with a norm in front and cold weights, few-row / persistent kernel: 100 x 1024 x
    # 1024 5.7 / 8.1, 333 x 2560 x 1024 8.8 / 9.8, 400 x 1024 x 4096 13.3 / 19.9, 450 x 2048 x 8192 28.5 / 34.8; on the line 256 x 3456 x
    # 1152 10.5 / 10.2 and 768 x 1152 x 1152 even, beyond it 512 x 2048 x 1152 11.1 / 10.0.  More than one round of 64-column tiles turns it
    # again: 400 x 2560 x 1024 9.5 / 10.4, 550 x 2048 x 2048 14.5 / 15.4.  Of 7437 random sizes up to 148 tiles, K 64 - 8192, the line takes
    # 5875 at 0.74 in the mean and loses more than a twentieth at 69 (outputs of 16 columns, up to 13 %); what it leaves is 1.02 in the
    # mean, sums below 128 1.00
    line = 48 if K < 256 else 60 if K < 512 else 82 if K < 1024 else 108 if K < 2048 else 112 if K < 4096 else 148
    return M * N <= line * 64 * 128 or (K >= 256 and -(-M // 128) * -(-N // 64) > 148)


class _SkinnyArgs(ctypes.Structure):
    """``OtbSkinnyArgs`` of ``csrc/gemm_skinny_tcgen05.cu``."""

    _fields_ = ([(n, c_void_p) for n in ("x", "w", "out", "bias", "residual", "out2", "gate", "mod_idx", "status")]
                + [(n, c_longlong) for n in ("ldx", "ldw", "ldo", "ldr", "ldo2", "gate_stride")]
                + [(n, c_int) for n in ("M", "N", "K", "rows_per_gate", "flags", "splits")])


def _skinny_launch(x: Tensor, w: Tensor, out: Tensor | None, M: int, N: int, K: int, flags: int, *, bias=None,
                   residual=None, ldr: int = 0, out2=None, ldo2: int = 0, gate=None, gate_stride: int = 0,
                   rows_per_gate: int = 1, mod_idx=None, splits: int = 0) -> None:
    global launch_count
    args = _SkinnyArgs(_ptr(x), _ptr(w), _ptr(out), _ptr(bias), _ptr(residual), _ptr(out2), _ptr(gate), _ptr(mod_idx),
                       status_pointer(), x.stride(0), w.stride(0), out.stride(0) if out is not None else N, ldr, ldo2,
                       gate_stride, M, N, K, rows_per_gate, flags, splits)
    _check(_call("gemm_skinny_tcgen05", "otb_gemm_skinny_bf16", "pp")(ctypes.byref(args), _raw_stream()),
           f"gemm_skinny[{M}x{N}x{K}]")
    launch_count += 1


def _operand(t: Tensor) -> Tensor:
    """A bf16 operand whose rows the TMA can load (16-byte aligned starts)."""
    assert t.dtype == torch.bfloat16, "gemm expects bf16 operands"
    return t.contiguous() if t.stride(-1) != 1 or (t.stride(0) % 8) or (t.data_ptr() % 16) else t


def gemm(a: Tensor, b: Tensor, layout: str, bias: Tensor | None = None, residual: Tensor | None = None,
         out: Tensor | None = None, accumulate: bool = False, out_dtype: torch.dtype | None = None,
         glu: str | None = None, glu_out: Tensor | None = None, store_out: bool = True, act: str | None = None,
         bn: int = 0, splits: int = 0, gate: Tensor | None = None, no_grad: bool = False) -> Tensor:
    """tcgen05 GEMM.  layout 'nt': a(M,K) b(N,K); 'nn': a(M,K) b(K,N); 'tn': a(K,M) b(K,N).  ``bn`` forces the column
    tile of the persistent kernel, ``splits`` (1, 2, 4, 8) forces the weight-streaming split-K kernel; ``no_grad`` as in
    ``use_skinny``."""
    global launch_count
    a, b = _operand(a), _operand(b)
    if layout == "nt":
        M, K = a.shape
        N, Kb = b.shape
        a_mn, b_mn = 0, 0
    elif layout == "nn":
        M, K = a.shape
        Kb, N = b.shape
        a_mn, b_mn = 0, 1
    elif layout == "tn":
        K, M = a.shape
        Kb, N = b.shape
        a_mn, b_mn = 1, 1
    else:
        raise ValueError(layout)
    if K != Kb:
        raise ValueError(f"inner dimensions differ: {tuple(a.shape)} x {tuple(b.shape)} ({layout})")
    if N % 8:
        raise ValueError(f"N={N} must be a multiple of 8")
    flags = 0
    odt = out_dtype or (out.dtype if out is not None else torch.bfloat16)
    if out is None and store_out:
        out = torch.empty(M, N, dtype=odt, device=a.device)
    if out is not None:
        if out.shape != (M, N) or out.stride(1) != 1 or out.stride(0) % 8 or out.data_ptr() % 16:
            raise ValueError("bad output tensor for gemm")
        if out.dtype == torch.float32:
            flags |= EPI_OUT_F32
        elif out.dtype != torch.bfloat16:
            raise ValueError("gemm output must be bf16 or fp32")
    else:
        flags |= EPI_NO_OUT
    if accumulate:
        flags |= EPI_ACCUM
    if bias is not None:
        if bias.numel() != N:
            raise ValueError("bias size")
        flags |= EPI_BIAS
        if bias.dtype == torch.float32:
            flags |= EPI_BIAS_F32
        elif bias.dtype != torch.bfloat16:
            raise ValueError("bias dtype")
        bias = bias.contiguous()
    if act == "gelu_tanh":
        flags |= EPI_ACT_GELU
    elif act is not None:
        raise ValueError(act)
    ldr = 0
    if residual is not None:
        if residual.shape != (M, N) or residual.dtype != torch.bfloat16 or residual.stride(1) != 1:
            raise ValueError("bad residual for gemm")
        flags |= EPI_RESIDUAL
        ldr = residual.stride(0)
    ldo2 = 0
    if glu is not None:
        flags |= EPI_GLU_GELU if glu == "gelu_tanh" else EPI_GLU_SILU
        if glu_out is None:
            glu_out = torch.empty(M, N // 2, dtype=torch.bfloat16, device=a.device)
        ldo2 = glu_out.stride(0)
    if splits and (layout != "nt" or accumulate):
        raise ValueError("the split-K kernel computes a @ b^T without accumulation")
    skinny = bool(splits) or use_skinny(layout, M, N, accumulate, bn, K, gate is not None,
                                       "glu" if glu is not None else "act" if act is not None else "", no_grad)
    g_stride, g_rows = 0, 1
    if gate is not None:
        # out = residual + gate * (a @ b^T): rows of N gates, one per `M / gate rows` consecutive output rows
        if not skinny or residual is None or gate.dim() != 2 or gate.shape[1] != N or gate.stride(1) != 1 \
                or gate.dtype != torch.bfloat16 or M % gate.shape[0]:
            raise ValueError("a gated residual epilogue needs the few-row kernel, a residual and (rows, N) bf16 gates")
        flags |= EPI_GATE
        g_stride, g_rows = gate.stride(0), M // gate.shape[0]
    if skinny:
        if residual is not None and (ldr % 4 or residual.data_ptr() % 8):
            residual = residual.contiguous()
            ldr = residual.stride(0)
        if gate is not None and (gate.stride(0) % 4 or gate.data_ptr() % 8):
            gate = gate.contiguous()
            g_stride = gate.stride(0)
        _skinny_launch(a, b, out, M, N, K, flags, bias=bias, residual=residual, ldr=ldr, out2=glu_out, ldo2=ldo2,
                       gate=gate, gate_stride=g_stride, rows_per_gate=g_rows, splits=splits)
        if glu is not None:
            return glu_out if not store_out else (out, glu_out)
        return out
    rc = _call("gemm_tcgen05", "otb_gemm_bf16", "pppiiillliipplpliipp")(
        _ptr(a), _ptr(b), _ptr(out), M, N, K, a.stride(0), b.stride(0), out.stride(0) if out is not None else N,
        a_mn, b_mn, _ptr(bias), _ptr(residual), ldr, _ptr(glu_out), ldo2, flags, bn, status_pointer(), _raw_stream())
    _check(rc, f"gemm[{layout} {M}x{N}x{K}]")
    launch_count += 1
    if glu is not None:
        return glu_out if not store_out else (out, glu_out)
    return out


# --------------------------------------------------------------------------------------------- few-row products
class RowNorm:
    """The RMS norm in front of a product: ``weight`` (plain norms, ``unit_offset`` adds 1) or ``mod`` rows of
    ``(scale | shift | gate)`` picked per row by ``idx`` (adaptive norms)."""

    __slots__ = ("eps", "weight", "unit_offset", "mod", "idx")

    def __init__(self, eps: float, weight: Tensor | None = None, unit_offset: bool = True, mod: Tensor | None = None,
                 idx: Tensor | None = None):
        self.eps, self.weight, self.unit_offset, self.mod, self.idx = eps, weight, unit_offset, mod, idx

    def apply(self, x2: Tensor) -> Tensor:
        """The norm as its own launch."""
        global launch_count
        R, H = x2.shape
        if x2.dtype != torch.bfloat16 or x2.stride(1) != 1 or (self.mod is not None and (
                self.mod.dtype != torch.bfloat16 or self.mod.stride(1) != 1 or self.mod.shape[1] != 3 * H)):
            raise ValueError("RowNorm takes bf16 rows and bf16 modulation rows")
        y = torch.empty(R, H, dtype=x2.dtype, device=x2.device)
        wt = self.weight.to(torch.bfloat16).contiguous() if self.weight is not None else None
        mode = 0 if wt is None else (1 if self.unit_offset else 2)
        _check(_call("elementwise", "otb_rms_fwd", "plpplippplifip")(
            _ptr(x2), x2.stride(0), _ptr(wt), _ptr(self.mod), self.mod.stride(0) if self.mod is not None else 0, 1,
            _ptr(self.idx), _ptr(y), 0, R, H, self.eps, mode, _raw_stream()), "rms_fwd")
        launch_count += 1
        return y

    @property
    def gate(self) -> Tensor | None:
        return self.mod[:, 2 * (self.mod.shape[1] // 3):] if self.mod is not None else None


def rows_linear(x: Tensor, w: Tensor, bias: Tensor | None = None, *, norm: RowNorm | None = None,
                residual: Tensor | None = None, gated_by: RowNorm | None = None, glu: str | None = None,
                out_f32: bool = False) -> Tensor:
    """``x @ w^T`` for the rows of an inference pass: ``x (R, K)`` dense bf16, optionally normalised first (``norm``),
    plus ``residual + gate * ...`` with the gate rows of the adaptive norm ``gated_by``, or the gated-MLP product
    (``glu``).  The norm is a launch of its own: folded into the product's staging warps it measured slower (12.7 us
    against 2.3 + 6.6 for 50 rows: the code that runs once per launch from a cold instruction cache outweighs the
    launch)."""
    global launch_count
    if norm is not None:
        x = norm.apply(x)
    x, w = _operand(x), _operand(w)
    R, K = x.shape
    N = w.shape[0]
    gate = gated_by.gate if gated_by is not None else None
    if w.shape[1] != K:
        raise ValueError(f"inner dimensions differ: {tuple(x.shape)} x {tuple(w.shape)}")
    if residual is not None and (residual.shape != (R, N) or residual.dtype != torch.bfloat16 or not residual.is_contiguous()):
        raise ValueError("bad residual for rows_linear")
    if gate is not None and (gate.shape[1] != N or gate.dtype != torch.bfloat16 or gate.stride(1) != 1 or residual is None):
        raise ValueError("bad gate for rows_linear")
    if bias is not None:
        if bias.numel() != N or bias.dtype not in (torch.bfloat16, torch.float32):
            raise ValueError("bad bias for rows_linear")
        bias = bias.contiguous()
    if not use_skinny("nt", R, N, False, 0, K, gate is not None, "glu" if glu is not None else ""):
        if gate is not None:
            y = gemm(x, w, "nt", bias=bias)
            out = torch.empty_like(y)
            _check(_call("elementwise", "otb_gated_residual", "ppplipplip")(
                _ptr(residual), _ptr(y), _ptr(gate), gate.stride(0), 1, _ptr(gated_by.idx), _ptr(out), R, N,
                _raw_stream()), "gated_residual")
            launch_count += 1
            return out
        if glu is not None:
            return gemm(x, w, "nt", glu=glu, store_out=False)
        return gemm(x, w, "nt", bias=bias, residual=residual, out_dtype=torch.float32 if out_f32 else None)
    flags, kw = 0, {}
    if bias is not None:
        flags |= EPI_BIAS | (EPI_BIAS_F32 if bias.dtype == torch.float32 else 0)
    if residual is not None:
        flags |= EPI_RESIDUAL
        kw.update(residual=residual, ldr=residual.stride(0))
    if gate is not None:
        flags |= EPI_GATE
        kw.update(gate=gate, gate_stride=gate.stride(0), mod_idx=gated_by.idx)
    if glu is not None:
        out = torch.empty(R, N // 2, dtype=torch.bfloat16, device=x.device)
        flags |= EPI_NO_OUT | (EPI_GLU_GELU if glu == "gelu_tanh" else EPI_GLU_SILU)
        _skinny_launch(x, w, None, R, N, K, flags, out2=out, ldo2=N // 2, **kw)
        return out
    out = torch.empty(R, N, dtype=torch.float32 if out_f32 else torch.bfloat16, device=x.device)
    _skinny_launch(x, w, out, R, N, K, flags | (EPI_OUT_F32 if out_f32 else 0), bias=bias, **kw)
    return out


# --------------------------------------------------------------------------------------------- norms
def _rows(x: Tensor) -> tuple[Tensor, int, int]:
    H = x.shape[-1]
    x2 = x.reshape(-1, H)
    if x2.stride(1) != 1 or x2.stride(0) % 8 or x2.data_ptr() % 16:
        x2 = x2.contiguous()
    return x2, x2.shape[0], H


def rms_fwd(x: Tensor, w: Tensor | None, eps: float, unit_offset: bool):
    global launch_count
    x2, R, H = _rows(x)
    y = torch.empty(R, H, dtype=x.dtype, device=x.device)
    rstd = torch.empty(R, dtype=torch.float32, device=x.device)
    mode = 0 if w is None else (1 if unit_offset else 2)
    wt = w.to(torch.bfloat16).contiguous() if w is not None else None
    _check(_call("elementwise", "otb_rms_fwd", "plpplippplifip")(
        _ptr(x2), x2.stride(0), _ptr(wt), 0, 0, 1, 0, _ptr(y), _ptr(rstd), R, H, eps, mode, _raw_stream()), "rms_fwd")
    launch_count += 1
    return y.view(x.shape), rstd


def _bwd_blocks(R: int) -> tuple[int, int]:
    rpb = max(1, (R + 591) // 592)
    return rpb, (R + rpb - 1) // rpb


def _dres_rows(dres: Tensor | None, R: int, H: int) -> Tensor | None:
    if dres is None:
        return None
    d = dres.reshape(R, H)
    return d if d.is_contiguous() else d.contiguous()


def rms_bwd(dy: Tensor, x: Tensor, w: Tensor | None, rstd: Tensor, unit_offset: bool, dres: Tensor | None = None):
    """``dres``: a gradient of the same shape as ``x`` that is added to ``dx`` inside the kernel."""
    global launch_count
    x2, R, H = _rows(x)
    dy2, _, _ = _rows(dy)
    if dy2.stride(0) != H:
        dy2 = dy2.contiguous()
    dx = torch.empty(R, H, dtype=x.dtype, device=x.device)
    mode = 0 if w is None else (1 if unit_offset else 2)
    rpb, nb = _bwd_blocks(R)
    partial = torch.empty(nb, H, dtype=torch.float32, device=x.device) if w is not None else None
    wt = w.to(torch.bfloat16).contiguous() if w is not None else None
    dr = _dres_rows(dres, R, H)
    _check(_call("elementwise", "otb_rms_bwd", "pplpplippppppliiip")(
        _ptr(dy2), _ptr(x2), x2.stride(0), _ptr(wt), 0, 0, 1, _ptr(rstd), _ptr(dx), _ptr(partial), 0, 0, _ptr(dr), R,
        H, mode, rpb, _raw_stream()), "rms_bwd")
    launch_count += 1
    dw = None
    if w is not None:
        dw = torch.empty(H, dtype=torch.bfloat16, device=x.device)
        _check(_call("elementwise", "otb_colsum_partials", "piipip")(
            _ptr(partial), nb, H, _ptr(dw), 0, _raw_stream()), "colsum")
        launch_count += 1
        dw = dw.to(w.dtype)
    return dx.view(x.shape), dw


def ada_rms_fwd(x: Tensor, mod: Tensor, eps: float):
    global launch_count
    B, S, H = x.shape
    x2, R, _ = _rows(x)
    mod2 = mod.reshape(-1, 3 * H)
    if mod2.stride(1) != 1 or mod2.stride(0) % 8 or mod2.data_ptr() % 16:
        mod2 = mod2.contiguous()
    rows_per_mod = S if mod.dim() == 2 else 1
    y = torch.empty(R, H, dtype=x.dtype, device=x.device)
    rstd = torch.empty(R, dtype=torch.float32, device=x.device)
    _check(_call("elementwise", "otb_rms_fwd", "plpplippplifip")(
        _ptr(x2), x2.stride(0), 0, _ptr(mod2), mod2.stride(0), rows_per_mod, 0, _ptr(y), _ptr(rstd), R, H, eps, 0,
        _raw_stream()),
           "ada_rms_fwd")
    launch_count += 1
    return y.view(x.shape), rstd


def ada_rms_bwd(dy: Tensor, x: Tensor, mod: Tensor, rstd: Tensor, dres: Tensor | None = None):
    global launch_count
    B, S, H = x.shape
    x2, R, _ = _rows(x)
    dy2 = dy.reshape(R, H).contiguous()
    mod2 = mod.reshape(-1, 3 * H)
    if mod2.stride(1) != 1 or mod2.stride(0) % 8 or mod2.data_ptr() % 16:
        mod2 = mod2.contiguous()
    rows_per_mod = S if mod.dim() == 2 else 1
    dx = torch.empty(R, H, dtype=x.dtype, device=x.device)
    dscale = torch.empty(R, H, dtype=x.dtype, device=x.device)
    dshift = torch.empty(R, H, dtype=x.dtype, device=x.device)
    _check(_call("elementwise", "otb_rms_bwd", "pplpplippppppliiip")(
        _ptr(dy2), _ptr(x2), x2.stride(0), 0, _ptr(mod2), mod2.stride(0), rows_per_mod, _ptr(rstd), _ptr(dx), 0,
        _ptr(dscale), _ptr(dshift), _ptr(_dres_rows(dres, R, H)), R, H, 0, 1, _raw_stream()), "ada_rms_bwd")
    launch_count += 1
    dscale, dshift = dscale.view(B, S, H), dshift.view(B, S, H)
    if mod.dim() == 2:
        dscale, dshift = dscale.float().sum(1).to(mod.dtype), dshift.float().sum(1).to(mod.dtype)
    return dx.view(x.shape), dscale, dshift


def ln_fwd(x: Tensor, w: Tensor, b: Tensor, eps: float):
    global launch_count
    x2, R, H = _rows(x)
    if x2.stride(0) != H:
        x2 = x2.contiguous()
    y = torch.empty(R, H, dtype=x.dtype, device=x.device)
    mean = torch.empty(R, dtype=torch.float32, device=x.device)
    rstd = torch.empty(R, dtype=torch.float32, device=x.device)
    # held until the launch is issued: a converted weight that died with its pointer would lend the bias its memory
    wt, bt = w.to(torch.bfloat16).contiguous(), b.to(torch.bfloat16).contiguous()
    _check(_call("elementwise", "otb_ln_fwd", "pppppplifp")(
        _ptr(x2), _ptr(wt), _ptr(bt), _ptr(y), _ptr(mean), _ptr(rstd), R, H, eps, _raw_stream()), "ln_fwd")
    launch_count += 1
    return y.view(x.shape), mean, rstd


def ln_bwd(dy: Tensor, x: Tensor, w: Tensor, mean: Tensor, rstd: Tensor):
    """-> ``dx`` (like x), ``dw``, ``db`` (like w).  One kernel for dx and the per-block weight / bias partials, two
    fixed-order column sums."""
    global launch_count
    x2, R, H = _rows(x)
    dy2, _, _ = _rows(dy)
    if x2.stride(0) != H:
        x2 = x2.contiguous()
    if dy2.stride(0) != H:
        dy2 = dy2.contiguous()
    dx = torch.empty(R, H, dtype=x.dtype, device=x.device)
    rpb, nb = _bwd_blocks(R)
    partial = torch.empty(2, nb, H, dtype=torch.float32, device=x.device)
    wt = w.to(torch.bfloat16).contiguous()
    _check(_call("elementwise", "otb_ln_bwd", "ppppppppliip")(
        _ptr(dy2), _ptr(x2), _ptr(wt), _ptr(mean), _ptr(rstd), _ptr(dx), _ptr(partial[0]), _ptr(partial[1]), R, H, rpb,
        _raw_stream()), "ln_bwd")
    out = torch.empty(2, H, dtype=torch.bfloat16, device=x.device)
    for k in range(2):
        _check(_call("elementwise", "otb_colsum_partials", "piipip")(
            _ptr(partial[k]), nb, H, _ptr(out[k]), 0, _raw_stream()), "colsum")
    launch_count += 3
    return dx.view(x.shape), out[0].to(w.dtype), out[1].to(w.dtype)


# --------------------------------------------------------------------------------------------- GLU / RoPE
_ACT = {"gelu_tanh": 0, "silu": 1}


def glu_fwd(gu: Tensor, act: str) -> Tensor:
    global launch_count
    gu2, M, I2 = _rows(gu)
    if gu2.stride(0) != I2:
        gu2 = gu2.contiguous()
    h = torch.empty(M, I2 // 2, dtype=gu.dtype, device=gu.device)
    _check(_call("elementwise", "otb_glu_fwd", "ppliip")(
        _ptr(gu2), _ptr(h), M, I2 // 2, _ACT[act], _raw_stream()), "glu_fwd")
    launch_count += 1
    return h.view(*gu.shape[:-1], I2 // 2)


def glu_bwd(gu: Tensor, dh: Tensor, act: str, inplace: bool = False) -> Tensor:
    global launch_count
    gu2, M, I2 = _rows(gu)
    if gu2.stride(0) != I2:
        gu2 = gu2.contiguous()
    dh2 = dh.reshape(M, I2 // 2).contiguous()
    dgu = gu2 if inplace else torch.empty_like(gu2)
    _check(_call("elementwise", "otb_glu_bwd", "pppliip")(
        _ptr(gu2), _ptr(dh2), _ptr(dgu), M, I2 // 2, _ACT[act], _raw_stream()), "glu_bwd")
    launch_count += 1
    return dgu.view(gu.shape)


def rope_fwd(x: Tensor, cos: Tensor, sin: Tensor, inverse: bool = False) -> Tensor:
    global launch_count
    B, S, H, D = x.shape
    if x.stride(3) != 1 or any(s % 8 for s in x.stride()[:3]) or x.data_ptr() % 16:
        x = x.contiguous()
    cos = cos.float().contiguous()
    sin = sin.float().contiguous()
    if cos.shape != (B, S, D // 2):
        cos = cos.expand(B, S, D // 2).contiguous()
        sin = sin.expand(B, S, D // 2).contiguous()
    y = torch.empty(B, S, H, D, dtype=x.dtype, device=x.device)
    _check(_call("elementwise", "otb_rope", "plllpppiiiiip")(
        _ptr(x), x.stride(0), x.stride(1), x.stride(2), _ptr(cos), _ptr(sin), _ptr(y), B, S, H, D, int(inverse),
        _raw_stream()), "rope")
    launch_count += 1
    return y


# --------------------------------------------------------------------------------------------- CE
CE_VOCAB_TILE = 16384      # vocabulary columns per pass of the tiled cross-entropy head


def _ce_tiles(V: int):
    return [(c0, min(V, c0 + CE_VOCAB_TILE)) for c0 in range(0, V, CE_VOCAB_TILE)]


def linear_ce_fwd(h: Tensor, w: Tensor, bias: Tensor | None, labels: Tensor):
    """Per-row cross entropy of ``h @ w.T + b`` and the fp32 log-sum-exp, one vocabulary tile at a time: the logits
    of a tile (rows x <= 16384, fp32) live only until the tile has been folded into the rows' running max / sum,
    so the 257 152-wide language-model head never needs its 8 GB of logits."""
    global launch_count
    R, V = h.shape[0], w.shape[0]
    labels = labels.contiguous()
    if V <= CE_VOCAB_TILE:
        logits = gemm(h, w, "nt", bias=bias, out_dtype=torch.float32)
        loss = torch.empty(R, dtype=torch.float32, device=h.device)
        lse = torch.empty(R, dtype=torch.float32, device=h.device)
        _check(_call("elementwise", "otb_ce_fwd", "pppplip")(
            _ptr(logits), _ptr(labels), _ptr(loss), _ptr(lse), R, V, _raw_stream()), "ce_fwd")
        launch_count += 1
        return loss, lse
    m = torch.full((R,), float("-inf"), dtype=torch.float32, device=h.device)
    s = torch.zeros(R, dtype=torch.float32, device=h.device)
    tgt = torch.zeros(R, dtype=torch.float32, device=h.device)
    for c0, c1 in _ce_tiles(V):
        logits = gemm(h, w[c0:c1], "nt", bias=bias[c0:c1] if bias is not None else None, out_dtype=torch.float32)
        _check(_call("train_elementwise", "otb_ce_tile_fwd", "ppllipppp")(
            _ptr(logits), _ptr(labels), c0, R, c1 - c0, _ptr(m), _ptr(s), _ptr(tgt), _raw_stream()), "ce_tile_fwd")
        launch_count += 1
        del logits
    lse = m + torch.log(s)
    return lse - tgt, lse


def linear_ce_bwd(dloss: Tensor, h: Tensor, w: Tensor, bias: Tensor | None, labels: Tensor, lse: Tensor,
                  dw_into: Tensor | None = None):
    """``(dh, dw, dbias)`` of :func:`linear_ce_fwd`, tile by tile: each tile's logits are recomputed, turned into
    ``(softmax - onehot) * dloss`` (bf16) and consumed by the two gradient products before the next tile starts.
    ``dw_into``: a ``(V, H)`` gradient buffer the weight gradient is ACCUMULATED into (then ``dw`` is None)."""
    global launch_count
    R, V = h.shape[0], w.shape[0]
    labels = labels.contiguous()
    dl32 = dloss.float().contiguous()
    tiles = _ce_tiles(V)
    dh32 = None
    dw = None if dw_into is not None else torch.empty_like(w)
    db = torch.empty(V, dtype=bias.dtype, device=h.device) if bias is not None else None
    for c0, c1 in tiles:
        wc = w[c0:c1]
        logits = gemm(h, wc, "nt", bias=bias[c0:c1] if bias is not None else None, out_dtype=torch.float32)
        dlogits = torch.empty(R, c1 - c0, dtype=torch.bfloat16, device=h.device)
        lab = labels if c0 == 0 else labels - c0          # a label outside the tile matches no column
        _check(_call("elementwise", "otb_ce_bwd", "ppppplip")(
            _ptr(logits), _ptr(lab), _ptr(lse), _ptr(dl32), _ptr(dlogits), R, c1 - c0, _raw_stream()), "ce_bwd")
        launch_count += 1
        del logits
        if len(tiles) == 1:
            dh = gemm(dlogits, wc, "nn")
        else:
            part = gemm(dlogits, wc, "nn", out_dtype=torch.float32)
            dh32 = part if dh32 is None else dh32.add_(part)
        if dw_into is not None:
            gemm(dlogits, h, "tn", out=dw_into[c0:c1], accumulate=True)
        else:
            gemm(dlogits, h, "tn", out=dw[c0:c1])
        if db is not None:
            db[c0:c1] = col_sum(dlogits).to(bias.dtype)
    if len(tiles) > 1:
        dh = dh32.to(h.dtype)
    return dh, dw, db


def col_sum(a: Tensor) -> Tensor:
    global launch_count
    a2, R, H = _rows(a)
    rpb = max(1, (R + 255) // 256)
    nb = (R + rpb - 1) // rpb
    partial = torch.empty(nb, H, dtype=torch.float32, device=a.device)
    _check(_call("elementwise", "otb_colsum_bf16", "plilpip")(
        _ptr(a2), R, H, a2.stride(0), _ptr(partial), rpb, _raw_stream()), "colsum_bf16")
    out = torch.empty(H, dtype=torch.bfloat16, device=a.device)
    _check(_call("elementwise", "otb_colsum_partials", "piipip")(
        _ptr(partial), nb, H, _ptr(out), 0, _raw_stream()), "colsum")
    launch_count += 2
    return out


# --------------------------------------------------------------------------------------------- optimizer
def sumsq_partials(g: Tensor, partial: Tensor) -> None:
    global launch_count
    _check(_call("elementwise", "otb_sumsq", "plipip")(
        _ptr(g), g.numel(), int(g.dtype == torch.bfloat16), _ptr(partial), partial.numel(), _raw_stream()), "sumsq")
    launch_count += 1


def clip_coef(partial: Tensor, grad_scale: float, max_norm: float, out: Tensor) -> None:
    global launch_count
    _check(_call("elementwise", "otb_clip_coef", "piffpp")(
        _ptr(partial), partial.numel(), grad_scale, max_norm, _ptr(out), _raw_stream()), "clip_coef")
    launch_count += 1


def adamw(p32: Tensor, g: Tensor, m: Tensor, v: Tensor, p16: Tensor | None, *, lr: float, beta1: float, beta2: float,
          eps: float, weight_decay: float, step: int, scale: Tensor | None = None) -> None:
    global launch_count
    n = p32.numel()
    assert g.numel() == n and m.numel() == n and v.numel() == n
    _check(_call("elementwise", "otb_adamw", "ppippplfffffffpp")(
        _ptr(p32), _ptr(g), int(g.dtype == torch.bfloat16), _ptr(m), _ptr(v), _ptr(p16), n, lr, beta1, beta2, eps,
        weight_decay, 1.0 - beta1 ** step, 1.0 - beta2 ** step, _ptr(scale), _raw_stream()), "adamw")
    launch_count += 1


# --------------------------------------------------------------------------------------------- images
def resize_with_pad(img: Tensor, width: int, height: int, pad_value: float = -1.0) -> Tensor:
    global launch_count
    N, C, Hin, Win = img.shape
    ratio = max(Win / width, Hin / height)
    rh, rw = int(Hin / ratio), int(Win / ratio)
    x = img.float().contiguous()
    out = torch.empty(N, C, height, width, dtype=torch.float32, device=img.device)
    _check(_call("elementwise", "otb_resize_pad", "ppiiiiiiifp")(
        _ptr(x), _ptr(out), N * C, Hin, Win, height, width, rh, rw, pad_value, _raw_stream()),
           "resize_pad")
    launch_count += 1
    return out


def gated_residual(x: Tensor, y: Tensor, gate: Tensor) -> Tensor:
    global launch_count
    B, S, H = x.shape
    x2, y2 = x.reshape(-1, H).contiguous(), y.reshape(-1, H).contiguous()
    g2 = gate.reshape(-1, H) if gate.stride(-1) == 1 else gate.reshape(-1, H).contiguous()
    if g2.stride(0) % 8 or g2.data_ptr() % 16:
        g2 = g2.contiguous()
    rows_per_gate = (B * S) // g2.shape[0]
    out = torch.empty_like(x2)
    _check(_call("elementwise", "otb_gated_residual", "ppplipplip")(
        _ptr(x2), _ptr(y2), _ptr(g2), g2.stride(0), rows_per_gate, 0, _ptr(out), B * S, H, _raw_stream()), "gated_residual")
    launch_count += 1
    return out.view(x.shape)


def qkv_post(qkv: Tensor, H: int, Hkv: int, D: int, q_norm, k_norm, cos: Tensor, sin: Tensor,
             k_dst: Tensor | None = None, v_dst: Tensor | None = None):
    global launch_count
    B, T, W = qkv.shape
    assert W == (H + 2 * Hkv) * D and qkv.dtype == torch.bfloat16
    if qkv.stride(-1) != 1 or qkv.stride(0) != T * qkv.stride(1):
        qkv = qkv.contiguous()
    cos = cos.float().contiguous()
    sin = sin.float().contiguous()
    if cos.shape != (B, T, D // 2):
        cos = cos.expand(B, T, D // 2).contiguous()
        sin = sin.expand(B, T, D // 2).contiguous()
    q = torch.empty(B, T, H, D, dtype=qkv.dtype, device=qkv.device)
    if k_dst is None:
        k_dst = torch.empty(B, T, Hkv, D, dtype=qkv.dtype, device=qkv.device)
        v_dst = torch.empty(B, T, Hkv, D, dtype=qkv.dtype, device=qkv.device)
    for t in (k_dst, v_dst):
        if t.shape != (B, T, Hkv, D) or t.stride(3) != 1 or t.stride(2) != D or t.dtype != qkv.dtype:
            raise ValueError("k / v destination must be (B,T,Hkv,D) with dense heads")
    norm = q_norm is not None
    qw = q_norm.weight.to(qkv.dtype) if norm else None
    kw = k_norm.weight.to(qkv.dtype) if norm else None
    _check(_call("elementwise", "otb_qkv_post", "plppfippppllplliiiiip")(
        _ptr(qkv), qkv.stride(1), _ptr(qw), _ptr(kw), q_norm.eps if norm else 0.0,
        int(q_norm.unit_offset) if norm else 0, _ptr(cos), _ptr(sin), _ptr(q), _ptr(k_dst), k_dst.stride(0),
        k_dst.stride(1), _ptr(v_dst), v_dst.stride(0), v_dst.stride(1), B, T, H, Hkv, D, _raw_stream()), "qkv_post")
    launch_count += 1
    return q, k_dst, v_dst


def patch_embed(pixels: Tensor, weight: Tensor, bias: Tensor, pos: Tensor, patch: int, out_dtype: torch.dtype) -> Tensor:
    """``pixels (B,C,H,W)`` fp32 / bf16, ``weight (N, C*p*p)``, ``bias (N)``, ``pos (gh*gw, N)`` all fp32 ->
    ``(B, gh*gw, N)`` in ``out_dtype``."""
    global launch_count
    B, C, H, W = pixels.shape
    N = weight.shape[0]
    if pixels.dtype not in (torch.float32, torch.bfloat16):
        pixels = pixels.float()
    pixels = pixels.contiguous()
    weight, bias, pos = weight.float().contiguous(), bias.float().contiguous(), pos.float().contiguous()
    out = torch.empty(B, (H // patch) * (W // patch), N, dtype=out_dtype, device=pixels.device)
    _check(_call("elementwise", "otb_patch_embed", "pippppiiiiiiip")(
        _ptr(pixels), int(pixels.dtype == torch.bfloat16), _ptr(weight), _ptr(bias), _ptr(pos), _ptr(out),
        int(out_dtype == torch.bfloat16), B, C, H, W, patch, N, _raw_stream()), "patch_embed")
    launch_count += 1
    return out


def time_embed(time: Tensor, dim: int, min_period: float, max_period: float, out_dtype: torch.dtype) -> Tensor:
    global launch_count
    t = time.float().contiguous()
    out = torch.empty(*t.shape, dim, dtype=out_dtype, device=t.device)
    _check(_call("elementwise", "otb_time_embed", "ppliffip")(
        _ptr(t), _ptr(out), t.numel(), dim, min_period, max_period, int(out_dtype == torch.bfloat16), _raw_stream()), "time_embed")
    launch_count += 1
    return out


def euler_step_(x: Tensor, v: Tensor, dt: float, frozen: Tensor | None = None, prefix: Tensor | None = None,
                x16: Tensor | None = None) -> Tensor:
    """In place: ``x += dt * v``; rows with ``frozen`` set take ``prefix`` instead.  ``x`` fp32 contiguous (B,T,D).
    ``x16``: a contiguous bf16 tensor of the same shape that receives a rounded copy."""
    global launch_count
    assert x.dtype == torch.float32 and x.is_contiguous() and v.shape == x.shape
    v = v.contiguous()
    fz = pf = None
    if frozen is not None and prefix is not None:
        fz = frozen.contiguous()
        fz = fz.view(torch.uint8) if fz.dtype == torch.bool else fz.to(torch.uint8)
        pf = prefix.float().contiguous()
    D = x.shape[-1]
    _check(_call("elementwise", "otb_euler_step", "ppifppplip")(
        _ptr(x), _ptr(v), int(v.dtype == torch.bfloat16), dt, _ptr(fz), _ptr(pf), _ptr(x16), x.numel() // D, D,
        _raw_stream()),
           "euler_step")
    launch_count += 1
    return x


def flow_interpolate(actions: Tensor, noise: Tensor, time: Tensor) -> tuple[Tensor, Tensor]:
    global launch_count
    a, n, t = actions.float().contiguous(), noise.float().contiguous(), time.float().contiguous()
    x_t, u_t = torch.empty_like(a), torch.empty_like(a)
    D = a.shape[-1]
    _check(_call("elementwise", "otb_flow_interpolate", "ppppplip")(
        _ptr(a), _ptr(n), _ptr(t), _ptr(x_t), _ptr(u_t), a.numel() // D, D, _raw_stream()),
           "flow_interpolate")
    launch_count += 1
    return x_t, u_t


# --------------------------------------------------------------------------------------------- attention
def attn_fwd(q, k, v, q_blk, k_blk, q_valid, k_valid, scale):
    from . import attention
    return attention.attn_fwd(q, k, v, q_blk, k_blk, q_valid, k_valid, scale)


def attn_bwd(do, q, k, v, o, lse, q_blk, k_blk, q_valid, k_valid, scale):
    from . import attention
    return attention.attn_bwd(do, q, k, v, o, lse, q_blk, k_blk, q_valid, k_valid, scale)


# --------------------------------------------------------------------------------------------- training elementwise
def dropout_residual_fwd(x: Tensor, y: Tensor, gate: Tensor | None, p: float, seed: int) -> Tensor:
    """``x + gate * dropout(y, p)`` for ``(B, T, H)`` bf16 tensors (``gate (B, 1 | T, H)`` or None), one pass; the keep
    mask comes from ``seed`` and is never stored."""
    global launch_count
    H = x.shape[-1]
    x2, y2 = x.reshape(-1, H), y.reshape(-1, H)
    x2 = x2 if x2.is_contiguous() else x2.contiguous()
    y2 = y2 if y2.is_contiguous() else y2.contiguous()
    rows = x2.shape[0]
    g2, stride, rpg = None, 0, 1
    if gate is not None:
        g2 = gate.reshape(-1, H)
        if g2.stride(1) != 1 or g2.stride(0) % 8 or g2.data_ptr() % 16:
            g2 = g2.contiguous()
        stride, rpg = g2.stride(0), rows // g2.shape[0]
    out = torch.empty_like(x2)
    _check(_call("train_elementwise", "otb_drop_res_fwd", "pppliplifup")(
        _ptr(x2), _ptr(y2), _ptr(g2), stride, rpg, _ptr(out), rows, H, p, seed, _raw_stream()), "drop_res_fwd")
    launch_count += 1
    return out.view(x.shape)


def dropout_residual_bwd(dout: Tensor, y: Tensor | None, gate: Tensor | None, p: float, seed: int):
    """Gradients of :func:`dropout_residual_fwd` w.r.t. ``y`` (and ``gate``, as fp32 ``(gate rows, H)``)."""
    global launch_count
    H = dout.shape[-1]
    d2 = dout.reshape(-1, H)
    d2 = d2 if d2.is_contiguous() else d2.contiguous()
    rows = d2.shape[0]
    g2, stride, rpg, dgate, y2 = None, 0, 1, None, None
    if gate is not None:
        g2 = gate.reshape(-1, H)
        if g2.stride(1) != 1 or g2.stride(0) % 8 or g2.data_ptr() % 16:
            g2 = g2.contiguous()
        stride, rpg = g2.stride(0), rows // g2.shape[0]
        dgate = torch.empty(g2.shape[0], H, dtype=torch.float32, device=dout.device)
        y2 = y.reshape(-1, H)
        y2 = y2 if y2.is_contiguous() else y2.contiguous()
    dy = torch.empty_like(d2)
    _check(_call("train_elementwise", "otb_drop_res_bwd", "ppplipplifup")(
        _ptr(d2), _ptr(y2), _ptr(g2), stride, rpg, _ptr(dy), _ptr(dgate), rows, H, p, seed, _raw_stream()), "drop_res_bwd")
    launch_count += 1
    return dy.view(dout.shape), dgate


def masked_mse_fwd(u: Tensor, v: Tensor, frozen: Tensor | None, pad: Tensor | None, real_dim: Tensor | None):
    """Per-sample ``(sum of squared differences, number of counted elements)`` of ``(B, T, D)`` fp32 tensors."""
    global launch_count
    B, T, D = u.shape
    sums = torch.empty(B, dtype=torch.float32, device=u.device)
    counts = torch.empty(B, dtype=torch.float32, device=u.device)
    _check(_call("train_elementwise", "otb_masked_mse_fwd", "pppppiiippp")(
        _ptr(u), _ptr(v), _ptr(frozen), _ptr(pad), _ptr(real_dim), B, T, D, _ptr(sums), _ptr(counts), _raw_stream()),
           "masked_mse_fwd")
    launch_count += 1
    return sums, counts


def masked_mse_bwd(u: Tensor, v: Tensor, frozen: Tensor | None, pad: Tensor | None, real_dim: Tensor | None,
                   coef: Tensor) -> Tensor:
    global launch_count
    B, T, D = u.shape
    dv = torch.empty_like(v)
    _check(_call("train_elementwise", "otb_masked_mse_bwd", "pppppiiippp")(
        _ptr(u), _ptr(v), _ptr(frozen), _ptr(pad), _ptr(real_dim), B, T, D, _ptr(coef), _ptr(dv), _raw_stream()),
           "masked_mse_bwd")
    launch_count += 1
    return dv


def embed_fwd(table: Tensor, ids: Tensor, scale: float) -> Tensor:
    global launch_count
    H = table.shape[1]
    flat = ids.reshape(-1).to(torch.int64).contiguous()
    out = torch.empty(flat.numel(), H, dtype=table.dtype, device=table.device)
    _check(_call("train_elementwise", "otb_embed_fwd", "ppplilfp")(
        _ptr(table), _ptr(flat), _ptr(out), flat.numel(), H, table.shape[0], scale, _raw_stream()),
           "embed_fwd")
    launch_count += 1
    return out.view(*ids.shape, H)


def embed_bwd(dout: Tensor, ids: Tensor, grad: Tensor, scale: float, padding_idx: int | None = None) -> None:
    """``grad[ids[i], :] += scale * dout[i, :]`` for a ``(V, H)`` bf16 or fp32 gradient table, deterministic (rows
    with the same id are summed in token order by one warp)."""
    global launch_count
    H = grad.shape[1]
    flat = ids.reshape(-1).to(torch.int64)
    sorted_ids, order = torch.sort(flat, stable=True)
    n = flat.numel()
    if n == 0:
        return
    d2 = dout.reshape(-1, H)
    d2 = d2 if d2.is_contiguous() else d2.contiguous()
    _check(_call("train_elementwise", "otb_embed_bwd", "ppplpiillfp")(
        _ptr(d2), _ptr(sorted_ids), _ptr(order), n, _ptr(grad), int(grad.dtype == torch.float32), H, grad.shape[0],
        -1 if padding_idx is None else padding_idx, scale, _raw_stream()),
        "embed_bwd")
    launch_count += 1


def pos_resample(table: Tensor, gh: int, gw: int) -> Tensor:
    """Bicubic resample of a square ``(g*g, d)`` fp32 position table to ``(gh*gw, d)``."""
    global launch_count
    import math
    g = int(math.isqrt(table.shape[0]))
    tab = table.detach().float().contiguous()
    out = torch.empty(gh * gw, tab.shape[1], dtype=torch.float32, device=tab.device)
    _check(_call("train_elementwise", "otb_pos_resample", "piipiip")(
        _ptr(tab), g, tab.shape[1], _ptr(out), gh, gw, _raw_stream()), "pos_resample")
    launch_count += 1
    return out


def seq_concat(a: Tensor, c: Tensor) -> Tensor:
    """``cat([a, c], dim=1)`` for bf16 ``(B, S, ...)`` tensors whose trailing dims are dense: one vectorised copy kernel
    (the library's batched concatenation moves these shapes at a tenth of the copy bandwidth)."""
    global launch_count
    B, S1, S2 = a.shape[0], a.shape[1], c.shape[1]
    E = a[0, 0].numel() if S1 else c[0, 0].numel()
    out = torch.empty(B, S1 + S2, *a.shape[2:], dtype=a.dtype, device=a.device)
    _check(_call("train_elementwise", "otb_seq_concat", "pllpllpliiip")(
        _ptr(a), a.stride(0), a.stride(1), _ptr(c), c.stride(0), c.stride(1), _ptr(out), B, S1, S2, E, _raw_stream()), "seq_concat")
    launch_count += 1
    return out


def zero_(t: Tensor) -> Tensor:
    """``t.zero_()`` for a dense CUDA tensor through the driver's memset (about twice the rate of the element-wise fill
    on multi-GB buffers); anything else falls back to ``t.zero_()``."""
    global launch_count
    if not (t.is_cuda and t.is_contiguous() and t.numel() > 0):
        return t.zero_()
    from ctypes import c_ulonglong
    _check(_call("train_elementwise", "otb_zero_bytes", "pup")(_ptr(t), t.numel() * t.element_size(), _raw_stream()),
           "zero_bytes")
    launch_count += 1
    return t


def seq_concat_supported(a: Tensor, c: Tensor) -> bool:
    if not (a.is_cuda and a.dtype == c.dtype == torch.bfloat16 and a.dim() == c.dim() >= 3):
        return False
    if a.shape[0] != c.shape[0] or a.shape[2:] != c.shape[2:] or a.shape[1] == 0 or c.shape[1] == 0:
        return False
    E = a[0, 0].numel()

    def rows_dense(t: Tensor) -> bool:
        exp = 1
        for size, stride in zip(reversed(t.shape[2:]), reversed(t.stride()[2:])):
            if size != 1 and stride != exp:
                return False
            exp *= size
        return t.stride(0) % 8 == 0 and t.stride(1) % 8 == 0 and t.data_ptr() % 16 == 0
    return E % 8 == 0 and rows_dense(a) and rows_dense(c)

"""ctypes launchers of the block-causal attention kernels: tcgen05 (bf16) and the exact fp32 CUDA-core kernels."""

from __future__ import annotations

import os
from functools import lru_cache
from ctypes import Structure, byref, c_float, c_int, c_longlong, c_void_p

import torch
from torch import Tensor

from . import _lib


def _enabled() -> bool:
    return os.environ.get("OPENTAU_B200_DENSE_ATTN", "0") != "1"


def supported(q: Tensor, k: Tensor, v: Tensor) -> bool:
    if not _enabled() or q.dtype != torch.bfloat16:
        return False
    B, Sq, H, D = q.shape
    Hkv = k.shape[2]
    g = H // Hkv
    return D % 8 == 0 and 16 <= D <= 256 and H % Hkv == 0 and g <= 128 and 128 % g == 0


def supported_bwd(q: Tensor, k: Tensor, v: Tensor) -> bool:
    if not supported(q, k, v) or os.environ.get("OPENTAU_B200_DENSE_ATTN_BWD", "0") == "1":
        return False
    g = q.shape[2] // k.shape[2]
    return g <= 32 and 32 % g == 0


def _u8(m: Tensor) -> Tensor:
    """Validity mask as bytes; a bool tensor is reinterpreted (one byte per element, 0 / 1), not converted."""
    m = m.contiguous()
    return m.view(torch.uint8) if m.dtype == torch.bool else m.to(torch.uint8)


def _prep(t: Tensor) -> Tensor:
    if t.stride(3) != 1 or any(s % 8 for s in t.stride()[:3]) or t.data_ptr() % 16:
        t = t.contiguous()
    return t


_entry = _lib.entry


def _ptr(t: Tensor | None) -> int:
    return t.data_ptr() if t is not None else 0


NUM_SMS = 148


def split_kv(B: int, Sq: int, Sk: int, H: int, Hkv: int, D: int) -> int:
    """Key splits per query tile: only when the tiles alone would leave three quarters of the SMs idle and every split
    still gets two key blocks (a 51-token suffix against a 1000-token prefix: 4 CTAs become 32)."""
    g = H // Hkv
    if D % 4 or g > 128 or 128 % g:
        return 1
    ctas = -(-Sq // (128 // g)) * Hkv * B
    nblk = -(-Sk // (64 if D > 128 else 128))
    if ctas * 4 > NUM_SMS:
        # half the chip idle and a long stream: two halves and a merge.  One pass against two halves, inside a replayed graph:
        # 16 heads of 72, 64 tiles: 21.2 / 19.0 us with 8 blocks, 35.0 / 26.6 with 15; with tiles for more than half the SMs it
        # loses.  Above a width of 128 one pass is a kernel of its own, and its blocks are half as large: 8 heads on 1 of 256, 38 - 74
        # tiles of 24 blocks 30.5 / 33.8, 47 52.4 / 53.2, 64 66.8 / 64.9, 128 126.4 / 115.5, 256 242.2 / 212.0
        return 2 if ctas * 2 <= NUM_SMS and nblk >= (64 if D > 128 else 15) else 1
    return max(1, min(8, NUM_SMS // ctas, nblk // 2))


@lru_cache(maxsize=1024)
def split_cluster(B: int, Sq: int, Sk: int, H: int, Hkv: int, D: int) -> int:
    """CTAs of the cluster that shares the keys of a 64-row query tile and merges on chip (1: not this path)."""
    g = H // Hkv
    nblk = -(-Sk // (64 if D > 128 else 128))
    if g > 64 or 64 % g or nblk < 3:
        return 1
    n = _lib.load("attention_tcgen05").otb_attn_cluster_fit(c_int(D), c_longlong(-(-Sq // (64 // g)) * Hkv * B))
    # pairs win where their streams are short: 56 tiles of 8 heads on 1 of 256 against 200, 400, 640 and 1018 keys 9.8, 13.2, 14.9 and
    # 19.8 us (best of one pass and a merge through global memory: 11.1, 14.1, 17.2, 20.5), 1500 and 3000 keys 25.1 / 22.6 and 45.1 / 33.5;
    # up to a width of 128 they lose on both ends (64 tiles of 64 against 300 9.6 / 8.0, of 128 against 2000 20.5 / 17.1)
    return 1 if n == 2 and (D <= 128 or nblk > 16) else n


def attn_fwd(q: Tensor, k: Tensor, v: Tensor, q_blk: Tensor, k_blk: Tensor, q_valid: Tensor, k_valid: Tensor,
             scale: float, nsplit: int | None = None, cluster: bool = False):
    """Returns ``(o, lse)``.  ``nsplit`` forces the CTAs that share a tile's keys, ``cluster`` that they merge on chip."""
    from . import cuda_ops
    B, Sq, H, D = q.shape
    Sk, Hkv = k.shape[1], k.shape[2]
    q, k, v = _prep(q), _prep(k), _prep(v)
    o = torch.empty(B, Sq, H * D, dtype=q.dtype, device=q.device)
    lse = torch.empty(B, H, Sq, dtype=torch.float32, device=q.device)
    qb = q_blk.to(torch.int32).contiguous()
    kb = k_blk.to(torch.int32).contiguous()
    qv = _u8(q_valid)
    kv = _u8(k_valid)
    args = (q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), qb.data_ptr(), kb.data_ptr(),
            qv.data_ptr(), kv.data_ptr(), B, Sq, Sk, H, Hkv, D, *q.stride()[:3], *k.stride()[:3], *v.stride()[:3], scale)
    kinds = 9 * "p" + 6 * "i" + 9 * "l" + "f"
    if nsplit is None:
        nsplit = split_cluster(B, Sq, Sk, H, Hkv, D)
        cluster = nsplit > 1
        if not cluster:
            nsplit = split_kv(B, Sq, Sk, H, Hkv, D)
    if nsplit > 1:
        part_o = part_ml = None
        if not cluster:
            part_o = torch.empty(nsplit, B, Sq, H, D, dtype=torch.float32, device=q.device)
            part_ml = torch.empty(nsplit, B, H, Sq, 2, dtype=torch.float32, device=q.device)
            cuda_ops.launch_count += 1
        rc = _entry("attention_tcgen05", "otb_attn_fwd_splitkv", kinds + "ipppp")(
            *args, nsplit, _ptr(part_o), _ptr(part_ml), cuda_ops.status_pointer(), cuda_ops._raw_stream())
    else:
        rc = _entry("attention_tcgen05", "otb_attn_fwd", kinds + "pp")(*args, cuda_ops.status_pointer(),
                                                                       cuda_ops._raw_stream())
    if rc != 0:
        raise RuntimeError(f"native attn_fwd failed with code {rc} (B={B} Sq={Sq} Sk={Sk} H={H} Hkv={Hkv} D={D})")
    cuda_ops.launch_count += 1
    return o, lse


@lru_cache(maxsize=1024)
def bwd_splits(B: int, Sq: int, Sk: int, H: int, Hkv: int, D: int) -> tuple[int, int, int]:
    """Parts that the streamed blocks of dQ, dK and dV are dealt to (a function of the sizes alone)."""
    n = (c_int(), c_int(), c_int())
    _lib.load("attention_bwd_tcgen05").otb_attn_bwd_splits(c_int(B), c_int(Sq), c_int(Sk), c_int(H), c_int(Hkv), c_int(D),
                                                           *(byref(x) for x in n))
    return tuple(x.value for x in n)


class _StoredBwdArgs(Structure):
    """``OtbAttnBwdStored`` of ``csrc/attention_bwd_stored_tcgen05.cu``."""

    _fields_ = [(n, c_void_p) for n in ("q", "k", "v", "o", "do", "lse", "dq", "dk", "dv", "p", "ds", "cover", "dk_parts", "dv_parts",
                                        "q_blk", "k_blk", "q_valid", "k_valid", "status")] + \
        [("strides", c_longlong * 9)] + \
        [(n, c_int) for n in ("B", "Sq", "Sk", "H", "Hkv", "D", "kv_splits")] + [("scale", c_float)]


#: bytes of P and dS together that the backward keeps at most; calls with more go a few samples at a time
BWD_STORED_LIMIT = 2 << 30


@lru_cache(maxsize=1024)
def bwd_stored_plan(B: int, Sq: int, Sk: int, H: int, Hkv: int, D: int) -> tuple[int, int, int]:
    """``(bytes of P, ints of cover, parts of dK and dV)`` of the stored backward, from the sizes alone."""
    size, cover, parts = c_longlong(), c_int(), c_int()
    _lib.load("attention_bwd_stored_tcgen05").otb_attn_bwd_stored_plan(
        c_int(B), c_int(Sq), c_int(Sk), c_int(H), c_int(Hkv), c_int(D), byref(size), byref(cover), byref(parts))
    return size.value, cover.value, parts.value


def stored_bwd_samples(B: int, Sq: int, Sk: int, H: int, Hkv: int, D: int) -> int:
    """Samples that a launch of the stored backward takes; 0, the recomputing kernels, where one alone has more P and dS than is kept
    (8 heads of more than 8192 positions) and for many short samples."""
    # A sample of up to 128 query rows and 128 keys is one tile of each recomputing kernel, with nothing to recompute, and a quarter
    # of a stored pair of 256 rows times a tile of 256 keys.  Stored / recomputing, geometric mean over 1297 such sizes of fourteen head
    # layouts by their tiles to an SM: 0.79 up to 0.3, where the chip is empty either way, 1.07 to 0.5, 1.39 to 0.7, 1.43 (0.78 - 1.85)
    # above; 2048 sequences of 6, 16 heads of 72, 5786 us and 2.2 GB of scratch against 3524 us and none.  Padding in one
    # direction or of a last tile does not turn it: with at least twice the area 0.72 (679 sizes, 0.32 - 1.22)
    if Sq * (H // Hkv) <= 128 and Sk <= 128 and B * Hkv > 0.3 * NUM_SMS:
        return 0
    return min(B, BWD_STORED_LIMIT // (2 * bwd_stored_plan(1, Sq, Sk, H, Hkv, D)[0]))


@lru_cache(maxsize=1024)
def _stored_layout(samples: int, at_once: int, B: int, Sq: int, Sk: int, H: int, Hkv: int, D: int, parts: int | None):
    """Scratch of the stored backward, ``at_once`` samples at a time: bytes of P, offset of the parts' sums and of all, bytes of a
    sample's share of a part; and the launches ``(first sample, samples, parts)``.  The parts of dK and dV, and with them the order of
    the sums, are those of ``samples`` at a time."""
    size, n_cover, _ = bwd_stored_plan(at_once, Sq, Sk, H, Hkv, D)
    sums_off, one = -(-(2 * size + 4 * n_cover) // 16) * 16, 4 * Sk * Hkv * D
    launches = []
    for g0 in range(0, B, samples):
        g1 = min(g0 + samples, B)
        m = parts or bwd_stored_plan(g1 - g0, Sq, Sk, H, Hkv, D)[2]
        launches += [(b0, min(at_once, g1 - b0), m) for b0 in range(g0, g1, at_once)]
    return size, sums_off, sums_off + max((2 * m * n * one for _, n, m in launches if m > 1), default=0), one, launches


def _attn_bwd_stored(samples: int, do, q, k, v, o, lse, qb, kb, qv, kv, dq, dk, dv, scale: float,
                     parts: int | None = None) -> bool:
    """dq, dk, dv through stored P and dS, ``samples`` at a time, or fewer where there is no room for as many; False where one
    sample finds none."""
    from . import cuda_ops
    B, Sq, H, D = q.shape
    Sk, Hkv = k.shape[1], k.shape[2]
    at_once = samples
    while True:                                  # one allocation: P, dS, cover, and the parts' fp32 dK and dV
        size, sums_off, total, one, launches = _stored_layout(samples, at_once, B, Sq, Sk, H, Hkv, D, parts)
        try:
            scratch = torch.empty(total, dtype=torch.uint8, device=q.device)
            break
        except torch.cuda.OutOfMemoryError:
            if at_once == 1:
                return False
            at_once = (at_once + 1) // 2
    s0 = scratch.data_ptr()
    fn = _entry("attention_bwd_stored_tcgen05", "otb_attn_bwd_stored", "pp")
    tensors = (q, k, v, o, do, lse, dq, dk, dv, qb, kb, qv, kv)
    at = [t.data_ptr() for t in tensors]
    strides = (c_longlong * 9)(*q.stride()[:3], *k.stride()[:3], *v.stride()[:3])
    for b0, n, m in launches:
        sums_at = (s0 + sums_off, s0 + sums_off + m * n * one) if m > 1 else (0, 0)
        args = _StoredBwdArgs(*at[:9], s0, s0 + size, s0 + 2 * size, *sums_at, *at[9:], cuda_ops.status_pointer(), strides,
                              n, Sq, Sk, H, Hkv, D, m, scale)
        rc = fn(byref(args), cuda_ops._raw_stream())
        if rc != 0:
            raise RuntimeError(f"native attn_bwd failed with code {rc} (B={B} Sq={Sq} Sk={Sk} H={H} Hkv={Hkv} D={D})")
        cuda_ops.launch_count += 3 + (m > 1)
        if b0 + n < B:
            at = [x + n * t.stride(0) * t.element_size() for x, t in zip(at, tensors)]
    return True


def attn_bwd(do: Tensor, q: Tensor, k: Tensor, v: Tensor, o: Tensor, lse: Tensor, q_blk: Tensor, k_blk: Tensor,
             q_valid: Tensor, k_valid: Tensor, scale: float, splits: tuple[int, int, int] | None = None,
             samples: int | None = None, parts: int | None = None):
    """Returns ``(dq, dk, dv)``; scratch and outputs are allocated here.  ``samples`` forces how many samples at a time go through
    stored P and dS (0: none, the recomputing kernels) and ``parts`` the parts of a tile of dK and dV there; ``splits`` forces
    the recomputing kernels and the parts that the streamed blocks of dQ, dK and dV are dealt to."""
    from . import cuda_ops
    B, Sq, H, D = q.shape
    Sk, Hkv = k.shape[1], k.shape[2]
    q, k, v = _prep(q), _prep(k), _prep(v)
    o = o.contiguous()
    do = do.contiguous()
    if do.data_ptr() % 16:                                      # a gradient may be any view; the kernels read 16 bytes at a time
        do = do.clone()
    lse = lse.contiguous()
    dq = torch.empty(B, Sq, H, D, dtype=q.dtype, device=q.device)
    dk = torch.empty(B, Sk, Hkv, D, dtype=q.dtype, device=q.device)
    dv = torch.empty(B, Sk, Hkv, D, dtype=q.dtype, device=q.device)
    qb = q_blk.to(torch.int32).contiguous()
    kb = k_blk.to(torch.int32).contiguous()
    qv = _u8(q_valid)
    kv = _u8(k_valid)
    if samples is None:
        samples = stored_bwd_samples(B, Sq, Sk, H, Hkv, D) if splits is None else 0
    if samples and _attn_bwd_stored(samples, do, q, k, v, o, lse, qb, kb, qv, kv, dq, dk, dv, scale, parts):
        return dq, dk, dv
    delta = torch.empty(B, H, Sq, dtype=torch.float32, device=q.device)
    if splits is None:
        splits = bwd_splits(B, Sq, Sk, H, Hkv, D)
    sums = [torch.empty(m, *t.shape, dtype=torch.float32, device=q.device) if m > 1 else None
            for m, t in zip(splits, (dq, dk, dv))]
    rc = _entry("attention_bwd_tcgen05", "otb_attn_bwd", 13 * "p" + 3 * "i" + 4 * "p" + 6 * "i" + 9 * "l" + "fpp")(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), do.data_ptr(), lse.data_ptr(), delta.data_ptr(),
        dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), *(_ptr(t) for t in sums), *splits, qb.data_ptr(), kb.data_ptr(),
        qv.data_ptr(), kv.data_ptr(), B, Sq, Sk, H, Hkv, D, *q.stride()[:3], *k.stride()[:3], *v.stride()[:3], scale,
        cuda_ops.status_pointer(), cuda_ops._stream())
    if rc != 0:
        raise RuntimeError(f"native attn_bwd failed with code {rc} (B={B} Sq={Sq} Sk={Sk} H={H} Hkv={Hkv} D={D})")
    cuda_ops.launch_count += 4 + sum(m > 1 for m in splits)
    return dq, dk, dv


# ------------------------------------------------------------------------------------------- exact fp32 (CUDA cores)
def supported_f32(q: Tensor, k: Tensor, v: Tensor) -> bool:
    """fp32 CUDA tensors with a head width that is a multiple of 4 up to 256 go to ``csrc/attention_f32.cu``: exact
    fp32 arithmetic without the (B, H, Sq, Sk) score tensor of the dense body."""
    if not _enabled() or q.dtype != torch.float32 or not q.is_cuda:
        return False
    D, H, Hkv = q.shape[3], q.shape[2], k.shape[2]
    return (k.dtype == v.dtype == torch.float32 and D % 4 == 0 and 4 <= D <= 256 and H % Hkv == 0
            and q.shape[0] <= 65535 and H <= 65535)                    # samples and heads are grid dimensions


#: score bytes of one 8-sample chunk up to which head widths above 128 stay on the dense evaluation
F32_DENSE_SCORE_LIMIT = 5 << 18
#: score bytes of a call above which the dense evaluation, which holds several such tensors, is not considered
F32_DENSE_MEMORY_LIMIT = 8 << 30
#: bytes of dS that the backward keeps (``F32_MAX_DS`` of ``csrc/attention_f32.cu``)
F32_DS_LIMIT = 2 << 30


@lru_cache(maxsize=1024)
def _f32_kernels_pay(B: int, Sq: int, Sk: int, H: int, Hkv: int, D: int, backward: bool) -> bool:
    """Whether the fp32 kernels are about as fast as the dense evaluation (or faster), from sizes alone and for masks that
    hide nothing (the kernels skip hidden tiles).  Microseconds, fitted to 460 sizes on a B200 (head widths 64 - 256, 1 -
    16384 samples, 1 - 4000 positions): rounds of blocks of 32 queries x 64 keys, in the backward the pairs of 32 keys x 64
    queries that are computed; for the dense evaluation its launches, its passes over pairs and operands and its batched
    products.  Padding decides: 4 queries of 4096 samples against themselves (16 heads of 72) take the kernels 2779
    forward and 6484 backward, dense 974 and 2531; 64 of 64 samples 111 and 280 against 317 and 643.  The backward
    is charged a quarter less than it takes on such masks (the kernels' forward wins that back, and what a mask hides they
    skip): by this rule no measured size takes more than 1.2 times the faster path forward, 1.25 forward and
    backward (1.35 at head width 160)."""
    tiles = lambda n, of: -(-n // of)  # noqa: E731
    pairs, elements = B * H * Sq * Sk / 1e6, B * D * (Sq * H + Sk * Hkv) / 1e6
    if not backward:
        kernels = tiles(B * H * tiles(Sq, 32), NUM_SMS) * tiles(Sk, 64) * (5 + D / 48 if D <= 128 else 7 + D / 45)
        dense = 170 + pairs * (24 + 0.06 * D) + 5 * elements + 0.01 * B * Hkv
        return kernels <= 1.15 * max(265, dense)
    kernels = B * H * tiles(Sk, 32) * 32 * tiles(Sq, 64) * 64 / 1e6 * (40 + 0.06 * D if D <= 128 else 56 + 0.133 * D)
    if B * H * Sk * tiles(Sq, 64) * 64 * 4 > F32_DS_LIMIT:
        kernels *= 1.4                                          # dS is recomputed for dQ
    dense = 290 + pairs * (20 + 0.18 * D) + 10 * elements + 0.02 * B * Hkv
    return kernels <= 1.35 * max(600, dense)


def prefer_f32_kernels(q: Tensor, k: Tensor, backward: bool = False) -> bool:
    """Which fp32 path the dispatcher takes when both can run (``OPENTAU_B200_F32_ATTN=kernel|dense`` forces one): the
    kernels, at half the dense evaluation's error against 64 bits and without its score tensors, unless they would be
    clearly slower (:func:`_f32_kernels_pay`).  Head widths above 128 with fewer score bytes than
    :data:`F32_DENSE_SCORE_LIMIT` (about 200 positions of 8 heads) stay dense, as tests hold it; that is launch-bound and
    slower (734 us against 108, forward + backward, for 100 positions of 8 heads on 1 of 256)."""
    mode = os.environ.get("OPENTAU_B200_F32_ATTN", "auto")
    if mode in ("kernel", "dense"):
        return mode == "kernel"
    B, Sq, H, D = q.shape
    Sk = k.shape[1]
    if D > 128 and min(B, 8) * H * Sq * Sk * 4 <= F32_DENSE_SCORE_LIMIT:
        return False
    return B * H * Sq * Sk * 4 > F32_DENSE_MEMORY_LIMIT or _f32_kernels_pay(B, Sq, Sk, H, k.shape[2], D,
                                                                                  backward)


def _prep_f32(t: Tensor) -> Tensor:
    if t.stride(3) != 1 or any(s % 4 for s in t.stride()[:3]) or t.data_ptr() % 16:
        t = t.contiguous()
    return t


def _f32_common(q, k, v, q_blk, k_blk, q_valid, k_valid):
    B, Sq, H, D = q.shape
    Sk, Hkv = k.shape[1], k.shape[2]
    q, k, v = _prep_f32(q), _prep_f32(k), _prep_f32(v)
    keep = (q, k, v, q_blk.to(torch.int32).contiguous(), k_blk.to(torch.int32).contiguous(), _u8(q_valid), _u8(k_valid))
    dims = [c_int(B), c_int(Sq), c_int(Sk), c_int(H), c_int(Hkv), c_int(D),
            c_longlong(q.stride(0)), c_longlong(q.stride(1)), c_longlong(q.stride(2)),
            c_longlong(k.stride(0)), c_longlong(k.stride(1)), c_longlong(k.stride(2)),
            c_longlong(v.stride(0)), c_longlong(v.stride(1)), c_longlong(v.stride(2))]
    return keep, dims


def attn_f32_fwd(q: Tensor, k: Tensor, v: Tensor, q_blk, k_blk, q_valid, k_valid, scale: float):
    from . import cuda_ops
    B, Sq, H, D = q.shape
    (q, k, v, qb, kb, qv, kv), dims = _f32_common(q, k, v, q_blk, k_blk, q_valid, k_valid)
    o = torch.empty(B, Sq, H * D, dtype=torch.float32, device=q.device)
    lse = torch.empty(B, H, Sq, dtype=torch.float32, device=q.device)
    rc = _lib.load("attention_f32").otb_attn_f32_fwd(
        c_void_p(q.data_ptr()), c_void_p(k.data_ptr()), c_void_p(v.data_ptr()), c_void_p(o.data_ptr()),
        c_void_p(lse.data_ptr()), c_void_p(qb.data_ptr()), c_void_p(kb.data_ptr()), c_void_p(qv.data_ptr()),
        c_void_p(kv.data_ptr()), *dims, c_float(scale), cuda_ops._stream())
    if rc != 0:
        raise RuntimeError(f"fp32 attn_fwd failed with code {rc} (B={B} Sq={Sq} Sk={k.shape[1]} H={H} D={D})")
    cuda_ops.launch_count += 1
    return o, lse


def attn_f32_bwd(do: Tensor, q: Tensor, k: Tensor, v: Tensor, o: Tensor, lse: Tensor, q_blk, k_blk, q_valid, k_valid,
                 scale: float, keep_ds: bool = True):
    """Returns ``(dq, dk, dv)``.  ``keep_ds=False`` recomputes dS for dQ as long sequences do, whose dS would be too big."""
    from . import cuda_ops
    B, Sq, H, D = q.shape
    Sk, Hkv = k.shape[1], k.shape[2]
    (q, k, v, qb, kb, qv, kv), dims = _f32_common(q, k, v, q_blk, k_blk, q_valid, k_valid)
    o = o.contiguous().float()
    do = do.contiguous().float()
    if do.data_ptr() % 16:
        do = do.clone()
    lse = lse.contiguous()
    lib = _lib.load("attention_f32")
    n_dq, n_dkv, n_ds = c_int(), c_int(), c_longlong()
    lib.otb_attn_f32_bwd_plan(c_int(B), c_int(Sq), c_int(Sk), c_int(H), c_int(Hkv), c_int(D), byref(n_dq), byref(n_dkv),
                              byref(n_ds))
    n_dq, n_dkv = n_dq.value, n_dkv.value
    ds = None
    if n_ds.value and keep_ds:
        try:
            ds = torch.empty(n_ds.value, dtype=torch.float32, device=q.device)
        except torch.cuda.OutOfMemoryError:                     # no room to keep it: recomputed
            pass
    # partial sums of a split backward
    dq_parts = torch.empty(n_dq, B, Sq, H, D, dtype=torch.float32, device=q.device) if n_dq > 1 else None
    dk_parts, dv_parts = torch.empty(2, n_dkv, B, Sk, Hkv, D, dtype=torch.float32, device=q.device) \
        if n_dkv > 1 else (None, None)
    dq = torch.empty(B, Sq, H, D, dtype=torch.float32, device=q.device)
    dk = torch.empty(B, Sk, Hkv, D, dtype=torch.float32, device=q.device)
    dv = torch.empty(B, Sk, Hkv, D, dtype=torch.float32, device=q.device)
    delta = torch.empty(B, H, Sq, dtype=torch.float32, device=q.device)
    rc = lib.otb_attn_f32_bwd(
        c_void_p(q.data_ptr()), c_void_p(k.data_ptr()), c_void_p(v.data_ptr()), c_void_p(o.data_ptr()),
        c_void_p(do.data_ptr()), c_void_p(lse.data_ptr()), c_void_p(delta.data_ptr()), c_void_p(dq.data_ptr()),
        c_void_p(dk.data_ptr()), c_void_p(dv.data_ptr()),
        *(c_void_p(t.data_ptr() if t is not None else 0) for t in (dq_parts, dk_parts, dv_parts, ds)), c_int(n_dq),
        c_int(n_dkv), c_void_p(qb.data_ptr()), c_void_p(kb.data_ptr()),
        c_void_p(qv.data_ptr()), c_void_p(kv.data_ptr()), *dims, c_float(scale), cuda_ops._stream())
    if rc != 0:
        raise RuntimeError(f"fp32 attn_bwd failed with code {rc} (B={B} Sq={Sq} Sk={Sk} H={H} Hkv={Hkv} D={D})")
    cuda_ops.launch_count += 3 + (n_dq > 1) + 2 * (n_dkv > 1)
    return dq, dk, dv

"""Hand-written autograd functions (ops.fused) against plain autograd of the reference bodies, fp32 CPU."""

import math

import pytest
import torch

from opentau_b200 import ops
from opentau_b200.ops import fused, prims, reference as ref


def _grads(fn, inputs):
    out = fn(*inputs)
    outs = out if isinstance(out, tuple) else (out,)
    loss = sum((o.float() * torch.linspace(0.5, 1.5, o.numel()).view_as(o)).sum() for o in outs if o is not None)
    return out, torch.autograd.grad(loss, [i for i in inputs if i.requires_grad], allow_unused=True)


def _leaf(*shape, scale=1.0):
    return (torch.randn(*shape, dtype=torch.float64) * scale).float().requires_grad_()


def test_linear_matches_reference():
    torch.manual_seed(0)
    x, w, b, r = _leaf(3, 5, 16), _leaf(24, 16), _leaf(24), _leaf(3, 5, 24)
    o1, g1 = _grads(lambda *a: fused.linear(*a), (x, w, b, r))
    o2, g2 = _grads(lambda *a: ref.linear(*a), (x, w, b, r))
    torch.testing.assert_close(o1, o2)
    for a, c in zip(g1, g2):
        torch.testing.assert_close(a, c, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("unit_offset", [True, False])
def test_rms_norm(unit_offset):
    torch.manual_seed(1)
    x, w = _leaf(4, 7, 32), _leaf(32, scale=0.1)
    o1, g1 = _grads(lambda a, b: fused.rms_norm(a, b, 1e-6, unit_offset), (x, w))
    o2, g2 = _grads(lambda a, b: ref.rms_norm(a, b, 1e-6, unit_offset), (x, w))
    torch.testing.assert_close(o1, o2)
    for a, c in zip(g1, g2):
        torch.testing.assert_close(a, c, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("per_token", [True, False])
def test_ada_rms_norm(per_token):
    torch.manual_seed(2)
    x = _leaf(3, 6, 16)
    mod = _leaf(3, 6, 48, scale=0.3) if per_token else _leaf(3, 48, scale=0.3)
    o1, g1 = _grads(lambda a, m: fused.ada_rms_norm(a, m, 1e-6), (x, mod))
    o2, g2 = _grads(lambda a, m: ref.ada_rms_norm(a, m, 1e-6), (x, mod))
    torch.testing.assert_close(o1[0], o2[0])
    torch.testing.assert_close(o1[1].expand_as(o2[1]), o2[1])
    for a, c in zip(g1, g2):
        torch.testing.assert_close(a, c, rtol=1e-4, atol=1e-5)


def test_layer_norm():
    torch.manual_seed(3)
    x, w, b = _leaf(5, 24), _leaf(24), _leaf(24)
    o1, g1 = _grads(lambda *a: fused.layer_norm(*a, 1e-6), (x, w, b))
    o2, g2 = _grads(lambda *a: ref.layer_norm(*a, 1e-6), (x, w, b))
    torch.testing.assert_close(o1, o2, rtol=1e-5, atol=1e-5)
    for a, c in zip(g1, g2):
        torch.testing.assert_close(a, c, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("act", ["gelu_tanh", "silu"])
def test_gated_mlp(act):
    torch.manual_seed(4)
    x, wg, wu, wd, r = _leaf(2, 5, 16), _leaf(64, 16, scale=0.3), _leaf(64, 16, scale=0.3), _leaf(16, 64, scale=0.3), _leaf(2, 5, 16)
    w_gu = prims.interleave_gate_up(wg.detach(), wu.detach()).requires_grad_()

    def plain(x, wg, wu, wd, r):
        h = ref.act_fn(x @ wg.t(), act) * (x @ wu.t())
        return h @ wd.t() + r

    o1, g1 = _grads(lambda x, w, d, r: fused.gated_mlp(x, w, d, act, r), (x, w_gu, wd, r))
    o2, g2 = _grads(plain, (x, wg, wu, wd, r))
    torch.testing.assert_close(o1, o2, rtol=1e-4, atol=1e-5)
    torch.testing.assert_close(g1[0], g2[0], rtol=1e-4, atol=1e-5)
    dg, du = prims.deinterleave_gate_up(g1[1])
    torch.testing.assert_close(dg, g2[1], rtol=1e-4, atol=1e-5)
    torch.testing.assert_close(du, g2[2], rtol=1e-4, atol=1e-5)
    torch.testing.assert_close(g1[2], g2[3], rtol=1e-4, atol=1e-5)
    torch.testing.assert_close(g1[3], g2[4])


def test_interleave_roundtrip():
    g, u = torch.randn(64, 8), torch.randn(64, 8)
    g2, u2 = prims.deinterleave_gate_up(prims.interleave_gate_up(g, u))
    assert torch.equal(g, g2) and torch.equal(u, u2)


def test_rope_inverse_is_backward():
    torch.manual_seed(5)
    x = _leaf(2, 6, 3, 16)
    pos = torch.arange(6)[None].expand(2, -1)
    cos, sin = ops.rope_angles(pos, 16, 10000.0)
    o1, g1 = _grads(lambda a: fused.rope(a, cos, sin), (x,))
    o2, g2 = _grads(lambda a: ref.apply_rope(a, cos, sin), (x,))
    torch.testing.assert_close(o1, o2)
    torch.testing.assert_close(g1[0], g2[0], rtol=1e-5, atol=1e-6)


def _mask_case(B, Sq, Sk, cross=0):
    att = torch.zeros(B, Sq, dtype=torch.bool)
    att[:, Sq // 2:] = True   # second half causal
    pad = torch.ones(B, Sq, dtype=torch.bool)
    pad[0, -1] = False
    q_blk, q_valid = ops.make_block_ids(pad, att)
    if cross:
        k_blk = torch.cat([torch.full((B, cross), ops.INT_MIN, dtype=torch.int32), q_blk], 1)
        k_valid = torch.cat([torch.ones(B, cross, dtype=torch.bool), q_valid], 1)
        k_valid[1, 0] = False
    else:
        k_blk, k_valid = q_blk, q_valid
    return q_blk, k_blk, q_valid, k_valid


@pytest.mark.parametrize("cross", [0, 5])
@pytest.mark.parametrize("hkv", [1, 2])
def test_block_attention(cross, hkv):
    torch.manual_seed(6)
    B, Sq, H, D = 2, 8, 4, 16
    Sk = Sq + cross
    q, k, v = _leaf(B, Sq, H, D), _leaf(B, Sk, hkv, D), _leaf(B, Sk, hkv, D)
    qb, kb, qv, kv = _mask_case(B, Sq, Sk, cross)
    scale = D ** -0.5
    o1, g1 = _grads(lambda *a: fused.block_attention(*a, qb, kb, qv, kv, scale), (q, k, v))
    o2, g2 = _grads(lambda *a: ref.block_attention(*a, qb, kb, qv, kv, scale), (q, k, v))
    valid = qv[:, :, None].expand(B, Sq, H * D)
    torch.testing.assert_close(o1[valid], o2[valid], rtol=1e-4, atol=1e-5)
    # gradients: padded query rows contribute differently (uniform softmax vs zeros) only through
    # rows that are invalid, which carry no weight in the reference either when masked out
    o1b, g1b = _grads(lambda *a: fused.block_attention(*a, qb, kb, qv, kv, scale) * valid, (q, k, v))
    o2b, g2b = _grads(lambda *a: ref.block_attention(*a, qb, kb, qv, kv, scale) * valid, (q, k, v))
    for a, c in zip(g1b, g2b):
        torch.testing.assert_close(a, c, rtol=1e-4, atol=1e-5)


def test_block_ids_reproduce_dense_mask():
    from opentau_b200.policies.pi05.modeling_pi05 import make_att_2d_masks
    pad = torch.tensor([[1, 1, 1, 1, 0, 1], [1, 1, 0, 1, 1, 1]], dtype=torch.bool)
    for att_row in ([1, 1, 1, 1, 1, 1], [0, 0, 0, 1, 1, 1], [1, 0, 1, 0, 1, 0], [0, 0, 0, 0, 0, 0]):
        att = torch.tensor([att_row, att_row])
        cs = torch.cumsum(att, 1)
        expect = (cs[:, None, :] <= cs[:, :, None]) & (pad[:, None, :] & pad[:, :, None])
        assert torch.equal(make_att_2d_masks(pad, att), expect)
    cross_pad = torch.tensor([[1, 0, 1], [1, 1, 1]], dtype=torch.bool)
    m = make_att_2d_masks(pad, att, n_cross_att_tokens=3, cross_att_pad_masks=cross_pad)
    assert m.shape == (2, 6, 9)
    assert torch.equal(m[:, :, :3], pad[:, :, None] & cross_pad[:, None, :])


def test_linear_cross_entropy():
    torch.manual_seed(7)
    h, w, b = _leaf(10, 16), _leaf(32, 16), _leaf(32)
    labels = torch.randint(0, 32, (10,))
    o1, g1 = _grads(lambda *a: fused.linear_cross_entropy(*a, labels), (h, w, b))
    o2, g2 = _grads(lambda *a: ref.linear_cross_entropy(*a, labels), (h, w, b))
    torch.testing.assert_close(o1, o2, rtol=1e-5, atol=1e-5)
    for a, c in zip(g1, g2):
        torch.testing.assert_close(a, c, rtol=1e-4, atol=1e-5)


def test_masked_mse_contract():
    u = torch.randn(2, 4, 6)
    v = torch.randn(2, 4, 6)
    pad = torch.tensor([[0, 0, 0, 1], [0, 0, 0, 0]], dtype=torch.bool)
    rad = torch.tensor([3, 6])
    loss = ops.flow_matching_masked_mse(u, v, None, pad, rad)
    mask = torch.ones(2, 4, 6, dtype=torch.bool)
    mask[0, 3] = False
    mask[0, :, 3:] = False
    expect = ((u - v) ** 2 * mask).sum() / (mask.sum() + 1e-8)
    torch.testing.assert_close(loss, expect)


def test_time_embedding_and_beta_time():
    t = torch.tensor([[0.0, 0.5, 1.0]])
    e = ops.sinusoidal_time_embedding(t, 8)
    assert e.shape == (1, 3, 8)
    frac = torch.linspace(0, 1, 4, dtype=torch.float64)
    period = 4e-3 * (4.0 / 4e-3) ** frac
    torch.testing.assert_close(e[0, 1, :4], torch.sin(2 * math.pi / period * 0.5).float())
    from opentau_b200.policies.pi05.modeling_pi05 import PI05FlowMatching
    torch.manual_seed(0)
    s = PI05FlowMatching.sample_time(20000, "cpu")
    assert 0.001 <= s.min() and s.max() <= 1.0
    assert abs(s.mean().item() - (0.6 * 0.999 + 0.001)) < 0.01   # Beta(1.5,1) has mean 0.6


def test_adamw_flat_matches_torch():
    torch.manual_seed(8)
    p = torch.randn(100)
    ref_p = p.clone().requires_grad_()
    opt = torch.optim.AdamW([ref_p], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    m, v, p32 = torch.zeros(100), torch.zeros(100), p.clone()
    for step in range(1, 4):
        g = torch.randn(100)
        ref_p.grad = g.clone()
        opt.step()
        ref.adamw_flat(p32, g, m, v, None, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=step)
        torch.testing.assert_close(p32, ref_p.detach(), rtol=1e-5, atol=1e-6)


def test_resize_with_pad_semantics():
    img = torch.rand(1, 3, 100, 200)
    out = ops.resize_with_pad(img, 224, 224, pad_value=0.0)
    assert out.shape == (1, 3, 224, 224)
    assert torch.all(out[:, :, :112, :] == 0)      # padding is on the top
    assert out[:, :, 112:, :].abs().sum() > 0


def test_forked_norms_give_the_gradients_of_norm_plus_residual():
    """``rms_norm_fork`` / ``ada_rms_norm_fork``: same values as the plain norms, and the gradient of x through
    (branch on the norm) + (residual on the second output) equals the plain two-path graph, including when only one of
    the two outputs is used."""
    import torch

    from opentau_b200 import ops
    torch.manual_seed(0)
    x = torch.randn(2, 5, 16, requires_grad=True)
    w = torch.randn(16, requires_grad=True)
    mod = torch.randn(2, 48, requires_grad=True)
    lin = torch.randn(16, 16)

    def plain():
        h = ops.rms_norm(x, w, 1e-6, True)
        y = x + h @ lin
        h2, gate = ops.ada_rms_norm(y, mod, 1e-6)
        return (y + gate * (h2 @ lin)).square().sum()

    def forked():
        h, xr = ops.rms_norm_fork(x, w, 1e-6, True)
        y = xr + h @ lin
        h2, gate, yr = ops.ada_rms_norm_fork(y, mod, 1e-6)
        return (yr + gate * (h2 @ lin)).square().sum()

    ga = torch.autograd.grad(plain(), (x, w, mod))
    gb = torch.autograd.grad(forked(), (x, w, mod))
    for a, b in zip(ga, gb):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-5)
    assert torch.allclose(plain(), forked())
    h, xr = ops.rms_norm_fork(x, w)
    torch.testing.assert_close(torch.autograd.grad(xr.sum(), x)[0], torch.ones_like(x))      # residual path alone
    h, xr = ops.rms_norm_fork(x, w)
    torch.testing.assert_close(torch.autograd.grad(h.sum(), x)[0], torch.autograd.grad(ops.rms_norm(x, w).sum(), x)[0])
    with torch.no_grad():
        h, xr = ops.rms_norm_fork(x, w)
        assert xr is x                                                                       # nothing to fork


@pytest.mark.parametrize("rows", [1, 65, 128, 129, 256])
@pytest.mark.parametrize("cols", [1024, 2056, 4096, 8192])
def test_gated_few_row_products_keep_the_gate_in_their_epilogue(rows, cols):
    """The few-row kernel alone multiplies the gate into the fp32 sum: every width that ever took it does."""
    from opentau_b200.ops import cuda_ops
    assert cuda_ops.use_skinny("nt", rows, cols, False, 0, 2048, True)
    assert cuda_ops.use_skinny("nt", rows, cols, False, 0)               # what ``gemm(gate=...)`` accepts


def test_fp32_attention_rule_follows_the_padding():
    """Sizes measured on both sides: few positions of many sequences leave the kernels' tiles empty and are clearly faster
    dense; full tiles, and calls that the dense evaluation cannot even launch in the time, are the kernels'."""
    from opentau_b200.ops.attention_native import _f32_kernels_pay as pay
    for size in ((4096, 4, 4, 16, 16, 72), (16384, 16, 16, 8, 8, 64), (64, 1, 1000, 32, 8, 128), (512, 8, 1000, 8, 1, 256),
                 (1, 1, 4000, 32, 8, 128)):
        assert not pay(*size, False), size
    for size in ((4096, 4, 4, 16, 16, 72), (64, 1, 300, 16, 16, 72), (512, 1, 300, 8, 8, 64), (512, 8, 1000, 8, 1, 256)):
        assert not pay(*size, True), size
    for size in ((2, 601, 601, 8, 1, 256), (2, 700, 700, 8, 4, 256), (1, 100, 100, 16, 16, 72), (64, 64, 64, 16, 16, 72),
                 (64, 300, 300, 8, 8, 64), (1, 50, 1000, 8, 1, 256), (8, 1, 1000, 16, 16, 72), (16, 601, 601, 16, 16, 72),
                 (4, 1227, 1227, 32, 8, 128)):
        assert pay(*size, False) and pay(*size, True), size


@pytest.mark.parametrize("which", range(8))
def test_attention_backward_refuses_misaligned_tensors_before_any_launch(which):
    """The bf16 backward reads and writes 16 bytes at a time: q, k, v, o, dO, dQ, dK and dV that start elsewhere are refused on the
    host (the addresses here are numbers that nothing may look at)."""
    from opentau_b200.ops import attention_native, build
    if not build.lib_path("attention_bwd_tcgen05").exists():
        pytest.skip("native libraries are not built")
    fn = attention_native._entry("attention_bwd_tcgen05", "otb_attn_bwd", 13 * "p" + 3 * "i" + 4 * "p" + 6 * "i" + 9 * "l" + "fpp")
    base = [1 << 20] * 10                                   # q k v o dO lse delta dQ dK dV
    base[(0, 1, 2, 3, 4, 7, 8, 9)[which]] += 8
    B, S, H, D = 1, 64, 4, 64
    strides = (S * H * D, H * D, D) * 3
    assert fn(*base, 0, 0, 0, 1, 1, 1, *[1 << 20] * 4, B, S, S, H, H, D, *strides, 0.125, 0, 0) == -6


@pytest.mark.parametrize("which", ["q", "k", "v", "o", "do", "dq", "dk", "dv", "p", "ds"])
def test_stored_attention_backward_refuses_misaligned_tensors_before_any_launch(which):
    """As above for the backward that keeps P and dS, whose blocks move in bulk copies."""
    from ctypes import byref, c_longlong

    from opentau_b200.ops import attention_native, build
    if not build.lib_path("attention_bwd_stored_tcgen05").exists():
        pytest.skip("native libraries are not built")
    fn = attention_native._entry("attention_bwd_stored_tcgen05", "otb_attn_bwd_stored", "pp")
    names = [n for n, _ in attention_native._StoredBwdArgs._fields_][:19]
    base = {n: 1 << 20 for n in names}
    base[which] += 8
    B, S, H, D = 1, 64, 4, 64
    args = attention_native._StoredBwdArgs(*base.values(), (c_longlong * 9)(*(S * H * D, H * D, D) * 3), B, S, S, H, H, D, 1, 0.125)
    assert fn(byref(args), 0) == -6


@pytest.mark.parametrize("B,S,D,room,want", [
    (4, 700, 256, None, [(0, 4, 1)]), (1, 700, 256, None, [(0, 1, 8)]),
    (1, 700, 256, "operands", None),               # room for P and dS, none for the parts' sums
    (4, 700, 256, 2, [(0, 2, 1), (2, 2, 1)]), (4, 700, 256, 1, [(i, 1, 1) for i in range(4)]), (3, 300, 64, 2, [(0, 2, 1), (2, 1, 1)]),
    (4, 700, 256, 0, None)])
def test_stored_attention_backward_takes_fewer_samples_where_memory_is_short(monkeypatch, B, S, D, room, want):
    """Room for all scratch or none is taken: every sample once, in parts that do not depend on the room; the recomputing kernels
    where not one sample finds it."""
    from opentau_b200.ops import attention_native, build, cuda_ops
    if not build.lib_path("attention_bwd_stored_tcgen05").exists():
        pytest.skip("native libraries are not built")
    H, Hkv = 8, 1
    size, cover, parts = attention_native.bwd_stored_plan(B, S, S, H, Hkv, D)
    operands = 2 * size + 4 * cover
    limit = {None: 1 << 60, "operands": operands}.get(room) if not isinstance(room, int) else operands * room // B + 64
    real, calls = torch.empty, []

    def empty(*shape, **kw):
        scratch = shape[0] if kw.get("dtype") is torch.uint8 else 0
        sums = 4 * shape[1] * shape[2] if kw.get("dtype") is torch.float32 and shape[0] == 2 else 0
        if scratch > limit or (sums and operands + sums > limit):
            raise torch.cuda.OutOfMemoryError
        return real(*shape, **kw)

    def launch(*a):
        if len(a) == 2:
            args = a[0]._obj
            b0 = (args.q - q.data_ptr()) // (2 * q.stride(0))
            calls.append((b0, args.B, args.kv_splits))
            assert args.k == k[b0].data_ptr() and args.lse == lse[b0].data_ptr()
            if args.kv_splits > 1:
                assert args.dv_parts == args.dk_parts + 4 * args.kv_splits * args.B * S * Hkv * D and args.dk_parts % 16 == 0
        else:
            calls.append("recomputed")
        return 0

    q, o, do = (real(B, S, H, D, dtype=torch.bfloat16) for _ in range(3))
    k, v = (real(B, S, Hkv, D, dtype=torch.bfloat16) for _ in range(2))
    lse = torch.zeros(B, H, S)
    blk, valid = torch.zeros(B, S, dtype=torch.int32), torch.ones(B, S, dtype=torch.bool)
    monkeypatch.setattr(attention_native, "_entry", lambda *a: launch)
    monkeypatch.setattr(cuda_ops, "_raw_stream", lambda: 0)
    monkeypatch.setattr(cuda_ops, "status_pointer", lambda: 0)
    monkeypatch.setattr(torch, "empty", empty)
    monkeypatch.setattr(attention_native, "stored_bwd_samples", lambda *a: B)
    attention_native.attn_bwd(do.view(B, S, H * D), q, k, v, o.view(B, S, H * D), lse, blk, blk, valid, valid, 0.1)
    assert calls == (want or ["recomputed"])


@pytest.mark.parametrize("kv", [1, 8, 35, 36, 37, 46, 74, 110, 184, 900])
@pytest.mark.parametrize("Sq_rows,Sk", [(2, 2), (256, 64), (300, 903), (900, 113), (5000, 5000), (256, 4000)])
def test_stored_attention_backward_deals_its_jobs_evenly(kv, Sq_rows, Sk):
    """Every dQ job goes to one CTA pair, and no pair's share is above the mean by more than the job of each kind that a share of
    whole jobs cannot avoid (and one for the rounding of equal runs)."""
    from opentau_b200.ops import _lib, build
    if not build.lib_path("attention_bwd_stored_tcgen05").exists():
        pytest.skip("native libraries are not built")
    pt, kb = -(-Sq_rows // 256), -(-Sk // 64)
    kt = -(-kb // 4)
    for splits in (1, 3):
        if splits > pt:
            continue
        n_q, n_kv = kv * pt, kv * 2 * kt * splits
        pairs = min(74, n_q + n_kv)
        more = n_kv % pairs
        more_q = _lib.load("attention_bwd_stored_tcgen05").otb_attn_bwd_stored_deal(kv, pt, kb, kt, splits, pairs)
        assert 0 <= more_q <= (n_q if more else 0)
        len_kv, len_q = 4 * -(-pt // splits) + 4, kb + 4
        run = [(more_q * (i + 1) // more - more_q * i // more) for i in range(more)]
        run += [((n_q - more_q) * (i + 1) // (pairs - more) - (n_q - more_q) * i // (pairs - more)) for i in range(pairs - more)]
        assert sum(run) == n_q
        shares = [(n_kv // pairs + (i < more)) * len_kv + r * len_q for i, r in enumerate(run)]
        assert max(shares) <= sum(shares) / pairs + len_kv + 2 * len_q, (splits, max(shares), sum(shares) / pairs)


@pytest.mark.parametrize("size,want", [
    ((2048, 6, 6, 16, 16, 72), 0), ((45, 128, 128, 8, 8, 64), 0), ((44, 128, 128, 8, 1, 64), 44), ((45, 16, 128, 8, 1, 256), 0),
    ((45, 17, 128, 8, 1, 256), 45), ((45, 16, 129, 8, 1, 256), 45), ((1, 8192, 8192, 8, 1, 256), 1), ((1, 8193, 8193, 8, 1, 256), 0),
    ((4, 4096, 4096, 8, 1, 256), 4), ((8, 4097, 4097, 8, 1, 256), 3), ((16, 1227, 1227, 8, 1, 256), 16)])
def test_attention_backward_keeps_p_and_ds_where_they_are_worth_it(size, want):
    """One tile of 128 rows and 128 keys to a sample and many samples: nothing is recomputed, and nothing is stored."""
    from opentau_b200.ops import attention_native, build
    if not build.lib_path("attention_bwd_stored_tcgen05").exists():
        pytest.skip("native libraries are not built")
    assert attention_native.stored_bwd_samples(*size) == want


@pytest.mark.parametrize("size,want", [
    ((1, 8192, 8192, 1, 1, 256), 2), ((1, 4737, 4096, 1, 1, 256), 2), ((1, 9472, 8192, 1, 1, 256), 2), ((1, 9473, 8192, 1, 1, 256), 1),
    ((1, 968, 968, 8, 1, 256), 1), ((1, 8192, 4032, 1, 1, 256), 1), ((1, 4096, 4096, 1, 1, 256), 4), ((1, 1024, 1920, 8, 8, 72), 2),
    ((1, 1024, 1792, 8, 8, 72), 1)])
def test_attention_forward_splits_long_streams_of_few_tiles(size, want):
    """Tiles for a quarter to half of the SMs: two halves from where the stream is long enough to pay for the merge."""
    from opentau_b200.ops import attention_native
    assert attention_native.split_kv(*size) == want


@pytest.mark.parametrize("M,N,K,end,want", [
    (100, 1024, 1024, "", True), (333, 2560, 1024, "", True), (400, 2560, 1024, "", True), (768, 1152, 4304, "", True),
    (512, 2048, 1152, "", False), (256, 3456, 1152, "", True), (768, 1152, 1152, "", True), (250, 3600, 1152, "", False),
    (257, 3456, 1152, "", True), (450, 2048, 2048, "", False), (550, 2048, 2048, "", True), (450, 2048, 8192, "", True),
    (400, 1024, 32, "", False), (400, 1024, 128, "", False), (384, 1024, 128, "", True), (247, 4736, 512, "", False),
    (800, 256, 1024, "", False), (64, 256, 32, "", True), (256, 4304, 1152, "act", False), (128, 4304, 1152, "act", True),
    (200, 1024, 1024, "glu", False)])
def test_line_between_the_few_row_and_the_persistent_kernel(M, N, K, end, want):
    """Products of 65 - 768 rows of an inference pass: the few-row kernel where the sum is long enough for the area."""
    from opentau_b200.ops import cuda_ops
    if not cuda_ops.SKINNY:
        pytest.skip("the few-row kernel is switched off")
    assert cuda_ops.use_skinny("nt", M, N, False, 0, K, False, end, True) is want


@pytest.mark.parametrize("cols", [8, 128, 768, 1032, 1280, 2048, 8192, 32768])
@pytest.mark.parametrize("inner", [8, 64, 256, 1088, 2048, 5120, 16384])
def test_few_row_plans_fit_the_chip(cols, inner):
    """Whatever the size, a plan covers the rows without an empty chunk and stays within shared memory; above 64 rows every CTA of
    a cluster has k-blocks and the clusters are resident at once (as a B200 holds them, two CTAs to an SM up to 64 tokens) unless
    one CTA to a sum is already too many."""
    import ctypes

    from opentau_b200.ops import _lib, build
    if not build.lib_path("gemm_skinny_tcgen05").exists():
        pytest.skip("native libraries are not built")
    fits = (ctypes.c_int * 9)(0, 148, 74, 45, 33, 26, 22, 15, 15)
    plan = (ctypes.c_int * 5)()
    for rows in (*range(1, 700), 999, 1024, 4097):
        assert _lib.load("gemm_skinny_tcgen05").otb_gemm_skinny_plan(rows, cols, inner, 148, fits, plan) == 0
        chunks, nt, splits, stages, smem = plan
        assert nt % 16 == 0 and 16 <= nt <= 256 and (chunks - 1) * nt < rows <= chunks * nt, (rows, list(plan))
        kb = -(-inner // 64)
        per = -(-kb // splits)
        assert 1 <= splits <= 8 and 1 <= stages <= min(per, 12), (rows, list(plan))
        assert smem <= (111 if nt <= 64 else 224) * 1024, (rows, list(plan))
        units = -(-cols // 128) * chunks
        if rows > 64:
            assert (splits - 1) * per < kb, (rows, list(plan))
            assert units <= fits[splits] * (2 if nt <= 64 else 1) or (splits == 1 and units > 148), (rows, list(plan))


def test_few_row_plans_share_sums_where_the_chip_is_empty():
    """100 - 400 rows of an action expert's output products: at least half the SMs work, and no CTA streams more than half the
    k-blocks of a sum that several could share."""
    import ctypes

    from opentau_b200.ops import _lib, build
    if not build.lib_path("gemm_skinny_tcgen05").exists():
        pytest.skip("native libraries are not built")
    fits = (ctypes.c_int * 9)(0, 148, 74, 45, 33, 26, 22, 15, 15)
    plan = (ctypes.c_int * 5)()
    for rows in (65, 100, 128, 150, 200, 256, 300, 400):
        for cols, inner in ((1024, 2048), (1024, 4096), (1280, 2048), (1280, 5120)):
            assert _lib.load("gemm_skinny_tcgen05").otb_gemm_skinny_plan(rows, cols, inner, 148, fits, plan) == 0
            chunks, nt, splits, _, _ = plan
            assert -(-cols // 128) * chunks * splits >= 74 and splits >= 2, (rows, cols, inner, list(plan))


@pytest.mark.parametrize("grad_mode,frozen,want", [(True, False, False), (False, False, True), (True, True, True)])
def test_products_know_whether_they_are_differentiated(monkeypatch, grad_mode, frozen, want):
    """A product that is differentiated keeps the persistent kernel's order of sums; parameters under ``no_grad`` do not count."""
    from opentau_b200.ops import cuda_ops
    seen, mm_nt = [], prims.mm_nt
    monkeypatch.setattr(prims, "mm_nt", lambda *a, no_grad=False, **kw: (seen.append(no_grad), mm_nt(*a, **kw))[1])
    w = torch.nn.Parameter(torch.randn(8, 16), requires_grad=not frozen)
    with torch.set_grad_enabled(grad_mode):
        y = fused.linear(torch.randn(3, 16), w)
    if not want:
        y.sum().backward()
        assert w.grad is not None
    assert seen == [want]
    assert cuda_ops.use_skinny("nt", 400, 1152, False, 0, 4096, False, "", want) is (want and cuda_ops.SKINNY)

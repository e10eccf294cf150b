"""tcgen05 block-causal attention against the dense fp32 reference (run on a B200)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(B, Sq, H, Hkv, D, cross, dev, seed=0, pad=True, causal_from=None):
    g = torch.Generator().manual_seed(seed)
    Sk = Sq + cross
    q = (torch.randn(B, Sq, H, D, generator=g)).to(torch.bfloat16).to(dev)
    k = (torch.randn(B, Sk, Hkv, D, generator=g)).to(torch.bfloat16).to(dev)
    v = (torch.randn(B, Sk, Hkv, D, generator=g)).to(torch.bfloat16).to(dev)
    att = torch.zeros(B, Sq, dtype=torch.bool)
    cf = Sq // 2 if causal_from is None else causal_from
    att[:, cf:] = True
    padm = torch.ones(B, Sq, dtype=torch.bool)
    if pad:
        padm[0, -3:] = False
        if Sq > 20:
            padm[-1, 5:9] = False
    from opentau_b200 import ops
    q_blk, q_valid = ops.make_block_ids(padm, att)
    if cross:
        k_blk = torch.cat([torch.full((B, cross), ops.INT_MIN, dtype=torch.int32), q_blk], 1)
        cv = torch.ones(B, cross, dtype=torch.bool)
        if pad:
            cv[0, 1::7] = False
        k_valid = torch.cat([cv, q_valid], 1)
    else:
        k_blk, k_valid = q_blk, q_valid
    return q, k, v, q_blk.to(dev), k_blk.to(dev), q_valid.to(dev), k_valid.to(dev)


@pytest.mark.parametrize("D", [64, 72, 128, 256])
@pytest.mark.parametrize("H,Hkv", [(8, 1), (8, 4), (4, 4), (16, 8)])
@pytest.mark.parametrize("Sq,cross", [(50, 0), (131, 0), (50, 203), (300, 0), (64, 64)])
def test_attn_fwd_matches_dense(D, H, Hkv, Sq, cross):
    from opentau_b200 import ops
    from opentau_b200.ops import attention_native, cuda_ops
    dev = torch.device("cuda:0")
    B = 2
    q, k, v, qb, kb, qv, kv = _case(B, Sq, H, Hkv, D, cross, dev, seed=D + Sq)
    scale = D ** -0.5
    assert attention_native.supported(q, k, v)
    o, lse = attention_native.attn_fwd(q, k, v, qb, kb, qv, kv, scale)
    cuda_ops.check_status()
    o_ref, lse_ref = ops.prims.attn_fwd(q.cpu().float(), k.cpu().float(), v.cpu().float(), qb.cpu(), kb.cpu(),
                                        qv.cpu(), kv.cpu(), scale)
    valid = qv.cpu()
    od = o.cpu().float().view(B, Sq, H, D)[valid]
    ord_ = o_ref.view(B, Sq, H, D)[valid]
    torch.testing.assert_close(od, ord_, rtol=3e-2, atol=3e-2)
    lv = lse.cpu().permute(0, 2, 1)[valid]
    lr = lse_ref.permute(0, 2, 1)[valid]
    torch.testing.assert_close(lv, lr, rtol=1e-2, atol=2e-2)
    assert torch.isfinite(o.float()).all()


def test_attn_fwd_strided_qkv_views():
    """q/k/v as column slices of one fused projection output (the layout the model produces)."""
    from opentau_b200 import ops
    from opentau_b200.ops import attention_native, cuda_ops
    dev = torch.device("cuda:0")
    B, S, H, Hkv, D = 2, 200, 8, 1, 256
    qkv = torch.randn(B, S, (H + 2 * Hkv) * D, device=dev).to(torch.bfloat16)
    q, k, v = qkv.split([H * D, Hkv * D, Hkv * D], dim=-1)
    q, k, v = q.unflatten(-1, (H, D)), k.unflatten(-1, (Hkv, D)), v.unflatten(-1, (Hkv, D))
    blk = torch.zeros(B, S, dtype=torch.int32, device=dev)
    ok = torch.ones(B, S, dtype=torch.bool, device=dev)
    o, _ = attention_native.attn_fwd(q, k, v, blk, blk, ok, ok, D ** -0.5)
    cuda_ops.check_status()
    o_ref = ops.ref.block_attention(q.float().cpu(), k.float().cpu(), v.float().cpu(), blk.cpu(), blk.cpu(),
                                    ok.cpu(), ok.cpu(), D ** -0.5)
    torch.testing.assert_close(o.cpu().float(), o_ref, rtol=3e-2, atol=3e-2)


def test_attn_large_logits_trigger_rescale():
    """Row maxima that grow late in the key sequence exercise the lazy O-rescale path."""
    from opentau_b200 import ops
    from opentau_b200.ops import attention_native, cuda_ops
    dev = torch.device("cuda:0")
    B, S, H, D = 1, 512, 4, 64
    q = torch.randn(B, S, H, D, device=dev).to(torch.bfloat16)
    k = torch.randn(B, S, H, D, device=dev).to(torch.bfloat16)
    k[:, 400:] *= 6.0
    v = torch.randn(B, S, H, D, device=dev).to(torch.bfloat16)
    blk = torch.zeros(B, S, dtype=torch.int32, device=dev)
    ok = torch.ones(B, S, dtype=torch.bool, device=dev)
    o, lse = attention_native.attn_fwd(q, k, v, blk, blk, ok, ok, 1.0)
    cuda_ops.check_status()
    o_ref, lse_ref = ops.prims.attn_fwd(q.cpu().float(), k.cpu().float(), v.cpu().float(), blk.cpu(), blk.cpu(),
                                        ok.cpu(), ok.cpu(), 1.0)
    torch.testing.assert_close(o.cpu().float(), o_ref, rtol=5e-2, atol=5e-2)
    torch.testing.assert_close(lse.cpu(), lse_ref, rtol=1e-2, atol=5e-2)


def test_attention_autograd_on_gpu_matches_cpu():
    from opentau_b200 import ops
    dev = torch.device("cuda:0")
    B, Sq, H, Hkv, D = 2, 70, 8, 1, 64
    q, k, v, qb, kb, qv, kv = _case(B, Sq, H, Hkv, D, 30, dev, seed=3)
    qc, kc, vc = (t.cpu().float().requires_grad_() for t in (q, k, v))
    q, k, v = (t.requires_grad_() for t in (q, k, v))
    o = ops.block_attention(q, k, v, qb, kb, qv, kv, D ** -0.5)
    oc = ops.block_attention(qc, kc, vc, qb.cpu(), kb.cpu(), qv.cpu(), kv.cpu(), D ** -0.5)
    w = torch.randn_like(oc) * qv.cpu()[:, :, None]
    (o.float() * w.to(dev)).sum().backward()
    (oc * w).sum().backward()
    for a, c in ((q.grad, qc.grad), (k.grad, kc.grad), (v.grad, vc.grad)):
        torch.testing.assert_close(a.cpu().float(), c, rtol=5e-2, atol=5e-2)


@pytest.mark.parametrize("D", [64, 72, 128, 256])
@pytest.mark.parametrize("H,Hkv", [(8, 1), (8, 4), (4, 4)])
@pytest.mark.parametrize("Sq,cross", [(50, 0), (131, 0), (50, 203), (300, 0)])
@pytest.mark.parametrize("samples", [2, 0])                # through stored P and dS, and recomputed
def test_attn_bwd_matches_dense(D, H, Hkv, Sq, cross, samples):
    from opentau_b200 import ops
    from opentau_b200.ops import attention_native, cuda_ops
    dev = torch.device("cuda:0")
    B = 2
    q, k, v, qb, kb, qv, kv = _case(B, Sq, H, Hkv, D, cross, dev, seed=7 * D + Sq)
    scale = D ** -0.5
    assert attention_native.supported_bwd(q, k, v)
    o, lse = attention_native.attn_fwd(q, k, v, qb, kb, qv, kv, scale)
    g = torch.Generator().manual_seed(5)
    do = (torch.randn(B, Sq, H * D, generator=g) * qv.cpu()[:, :, None]).to(torch.bfloat16).to(dev)
    dq, dk, dv = attention_native.attn_bwd(do, q, k, v, o, lse, qb, kb, qv, kv, scale, samples=samples)
    cuda_ops.check_status()
    qc, kc, vc = q.cpu().float(), k.cpu().float(), v.cpu().float()
    o_ref, lse_ref = ops.prims.attn_fwd(qc, kc, vc, qb.cpu(), kb.cpu(), qv.cpu(), kv.cpu(), scale)
    dqr, dkr, dvr = ops.prims.attn_bwd(do.cpu().float(), qc, kc, vc, o_ref, lse_ref, qb.cpu(), kb.cpu(), qv.cpu(),
                                        kv.cpu(), scale)
    valid_q = qv.cpu()
    torch.testing.assert_close(dq.cpu().float()[valid_q], dqr[valid_q], rtol=5e-2, atol=5e-2)
    valid_k = kv.cpu()
    torch.testing.assert_close(dk.cpu().float()[valid_k], dkr[valid_k], rtol=5e-2, atol=8e-2)
    torch.testing.assert_close(dv.cpu().float()[valid_k], dvr[valid_k], rtol=5e-2, atol=8e-2)
    assert torch.isfinite(dq.float()).all() and torch.isfinite(dk.float()).all() and torch.isfinite(dv.float()).all()


@pytest.mark.parametrize("B,Sq,Sk,H,Hkv,D", [(1, 51, 1019, 8, 1, 256), (2, 51, 700, 16, 8, 128), (1, 10, 300, 4, 4, 64),
                                             (1, 51, 1019, 8, 8, 72)])
@pytest.mark.parametrize("nsplit", [2, 5, 8])
def test_split_kv_matches_single_pass(B, Sq, Sk, H, Hkv, D, nsplit):
    """A suffix attending to a cached prefix plus itself: the key blocks split over several CTAs and merged give the
    single-pass result (also when some splits reach no visible key)."""
    from opentau_b200.ops import attention_native, cuda_ops
    dev = torch.device("cuda:0")
    torch.manual_seed(0)
    q = torch.randn(B, Sq, H, D, device=dev).to(torch.bfloat16)
    k = torch.randn(B, Sk, Hkv, D, device=dev).to(torch.bfloat16)
    v = torch.randn(B, Sk, Hkv, D, device=dev).to(torch.bfloat16)
    P = Sk - Sq
    k_blk = torch.cat([torch.full((B, P), -2**31, dtype=torch.int32, device=dev),
                       torch.arange(Sq, device=dev, dtype=torch.int32)[None].expand(B, -1) // 7], 1).contiguous()
    q_blk = k_blk[:, P:].contiguous()
    k_valid = torch.rand(B, Sk, device=dev) > 0.1
    q_valid = torch.ones(B, Sq, dtype=torch.bool, device=dev)
    q_valid[:, -3:] = False
    scale = D ** -0.5
    want_o, want_lse = attention_native.attn_fwd(q, k, v, q_blk, k_blk, q_valid, k_valid, scale, nsplit=1)
    got_o, got_lse = attention_native.attn_fwd(q, k, v, q_blk, k_blk, q_valid, k_valid, scale, nsplit=nsplit)
    cuda_ops.check_status()
    torch.testing.assert_close(got_o.float(), want_o.float(), atol=1e-2, rtol=1e-2)
    torch.testing.assert_close(got_lse, want_lse, atol=1e-3, rtol=1e-3)


@pytest.mark.parametrize("nsplit", [2, 3, 7, 8])
@pytest.mark.parametrize("H,Hkv,D", [(8, 1, 256), (8, 4, 256), (4, 1, 64), (16, 16, 72), (32, 8, 128), (64, 1, 40)])
@pytest.mark.parametrize("Sq,Sk", [(1, 77), (1, 1019), (50, 322), (51, 1018), (9, 130)])
def test_cluster_merge_matches_single_pass(H, Hkv, D, Sq, Sk, nsplit):
    """Keys of a 64-row tile shared by a cluster: tiles with one row and partly filled ones, ranks that own no row, splits
    without a key, rows that see nothing.  Differs from one pass by fp32 rounding of the merge before bf16 (2^-8)."""
    from opentau_b200.ops import attention_native, cuda_ops
    B = 2
    g = torch.Generator(device="cuda").manual_seed(Sk)
    q, k, v = (torch.randn(B, S, h, D, device="cuda", generator=g).to(torch.bfloat16)
               for S, h in ((Sq, H), (Sk, Hkv), (Sk, Hkv)))
    kb = torch.cat([torch.full((B, Sk - Sq), -2**31, device="cuda"), torch.arange(Sq, device="cuda").expand(B, -1) // 7], 1).int()
    qb, kv = kb[:, Sk - Sq:].contiguous(), torch.rand(B, Sk, device="cuda", generator=g) > 0.2
    kv[1, :] = False                                       # nothing to see for this sample
    qv = torch.ones(B, Sq, dtype=torch.bool, device="cuda")
    qv[:, Sq // 2 + 1:Sq // 2 + 3] = False
    args = (q, k, v, qb, kb, qv, kv, D ** -0.5)
    want_o, want_lse = attention_native.attn_fwd(*args, nsplit=1)
    o, lse = attention_native.attn_fwd(*args, nsplit=nsplit, cluster=True)
    cuda_ops.check_status()
    assert _rel(o, want_o.double()) < 2 ** -8
    torch.testing.assert_close(lse, want_lse, atol=1e-4, rtol=1e-5)
    assert float(o[1].abs().max()) == 0.0


@pytest.mark.parametrize("nsplit", [3, 8])
@pytest.mark.parametrize("H,Hkv,D", [(8, 1, 256), (4, 1, 64), (16, 16, 72)])
def test_cluster_merge_keeps_nan(H, Hkv, D, nsplit):
    """A NaN in a query row or in a key's value reaches the same outputs as in one pass: a partial whose weight is zero
    because its row sum is NaN is not one that saw nothing."""
    from opentau_b200.ops import attention_native, cuda_ops
    B, Sq, Sk = 2, 50, 700
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v = (torch.randn(B, S, h, D, device="cuda", generator=g).to(torch.bfloat16)
               for S, h in ((Sq, H), (Sk, Hkv), (Sk, Hkv)))
    q[0, 7, H // 2, 1] = q[1, 20] = v[1, 500, 0, 3] = float("nan")
    zero, ok = (lambda S: torch.zeros(B, S, dtype=torch.int32, device="cuda"),
                lambda S: torch.ones(B, S, dtype=torch.bool, device="cuda"))
    args = (q, k, v, zero(Sq), zero(Sk), ok(Sq), ok(Sk), D ** -0.5)
    want = attention_native.attn_fwd(*args, nsplit=1)[0]
    got = attention_native.attn_fwd(*args, nsplit=nsplit, cluster=True)[0]
    cuda_ops.check_status()
    assert torch.equal(got.isnan(), want.isnan())
    assert want.view(B, Sq, H, D)[0, 7, H // 2].isnan().all() and want.view(B, Sq, H, D)[1, 20].isnan().all()
    assert want.view(B, Sq, H, D)[1, 30, 0, 3].isnan() and not want[0, 8].isnan().any()


@pytest.mark.parametrize("D", [32, 72, 128, 160, 256])
@pytest.mark.parametrize("H,Hkv", [(8, 1), (6, 3), (4, 4)])
@pytest.mark.parametrize("Sq,cross", [(50, 0), (131, 0), (50, 203), (33, 64)])
def test_fp32_attention_kernels_match_the_dense_fp32_reference(D, H, Hkv, Sq, cross, monkeypatch):
    """The exact fp32 kernels (forward, dQ, dK / dV over the whole GQA group) against the CPU fp32 dense evaluation,
    at fp32 tolerances: block-causal mask, pads, a cross-attention prefix with block id INT_MIN, strided inputs."""
    from opentau_b200 import ops
    from opentau_b200.ops import attention_native
    dev = torch.device("cuda:0")
    B = 2
    qh, kh, vh, qb, kb, qv, kv = _case(B, Sq, H, Hkv, D, cross, dev, seed=3 * D + Sq)
    g = torch.Generator().manual_seed(11)
    Sk = Sq + cross
    # q as a strided view of a fused (B, Sq, H + 2 Hkv, D) projection, as the models produce it
    fused = torch.randn(B, Sq, H + 2 * Hkv, D, generator=g).to(dev)
    q = fused[:, :, :H]
    k = torch.randn(B, Sk, Hkv, D, generator=g).to(dev)
    v = torch.randn(B, Sk, Hkv, D, generator=g).to(dev)
    scale = D ** -0.5
    assert attention_native.supported_f32(q, k, v) and not attention_native.supported(q, k, v)
    from opentau_b200.ops import attention as dispatch
    monkeypatch.setenv("OPENTAU_B200_F32_ATTN", "kernel")               # at small sizes "auto" may take the dense body
    o, lse = dispatch.attn_fwd(q, k, v, qb, kb, qv, kv, scale)
    assert attention_native.prefer_f32_kernels(q, k)
    monkeypatch.setenv("OPENTAU_B200_F32_ATTN", "auto")
    assert attention_native.prefer_f32_kernels(q, k) == (D <= 128)      # these score tensors are far below the limit
    qc, kc, vc = q.cpu().contiguous(), k.cpu(), v.cpu()
    o_ref, lse_ref = ops.prims.attn_fwd(qc, kc, vc, qb.cpu(), kb.cpu(), qv.cpu(), kv.cpu(), scale)
    vq, vk = qv.cpu(), kv.cpu()
    torch.testing.assert_close(o.cpu().view(B, Sq, H, D)[vq], o_ref.view(B, Sq, H, D)[vq], rtol=2e-4, atol=2e-5)
    torch.testing.assert_close(lse.cpu().permute(0, 2, 1)[vq], lse_ref.permute(0, 2, 1)[vq], rtol=1e-5, atol=2e-5)
    do = (torch.randn(B, Sq, H * D, generator=g) * vq[:, :, None]).to(dev)
    dq, dk, dv = attention_native.attn_f32_bwd(do, q, k, v, o, lse, qb, kb, qv, kv, scale)
    dqr, dkr, dvr = ops.prims.attn_bwd(do.cpu(), qc, kc, vc, o_ref, lse_ref, qb.cpu(), kb.cpu(), vq, vk, scale)
    torch.testing.assert_close(dq.cpu()[vq], dqr[vq], rtol=5e-4, atol=5e-5)
    torch.testing.assert_close(dk.cpu()[vk], dkr[vk], rtol=5e-4, atol=1e-4)
    torch.testing.assert_close(dv.cpu()[vk], dvr[vk], rtol=5e-4, atol=1e-4)
    hidden = ~vq                                               # rows that see nothing: zero output, zero gradient
    if hidden.any():
        assert float(o.cpu().view(B, Sq, H, D)[hidden].abs().max()) == 0.0
        assert float(dq.cpu()[hidden].abs().max()) == 0.0


def test_fp32_attention_through_autograd_on_gpu(monkeypatch):
    """fp32 CUDA tensors through ``ops.block_attention`` (the autograd function the models call) take the fp32 kernels
    and give the CPU gradients."""
    from opentau_b200 import ops
    monkeypatch.setenv("OPENTAU_B200_F32_ATTN", "kernel")
    dev = torch.device("cuda:0")
    B, Sq, H, Hkv, D = 2, 70, 8, 2, 64
    _, _, _, qb, kb, qv, kv = _case(B, Sq, H, Hkv, D, 0, dev, seed=9)
    g = torch.Generator().manual_seed(3)
    q = torch.randn(B, Sq, H, D, generator=g)
    k = torch.randn(B, Sq, Hkv, D, generator=g)
    v = torch.randn(B, Sq, Hkv, D, generator=g)
    w = torch.randn(B, Sq, H * D, generator=g) * qv.cpu()[:, :, None]
    outs = []
    for device in ("cpu", dev):
        a, b_, c = (t.clone().to(device).requires_grad_(True) for t in (q, k, v))
        o = ops.block_attention(a, b_, c, qb.to(device), kb.to(device), qv.to(device), kv.to(device), D ** -0.5)
        (o * w.to(device)).sum().backward()
        outs.append((o.detach().cpu(), a.grad.cpu(), b_.grad.cpu(), c.grad.cpu()))
    (o_c, dq_c, dk_c, dv_c), (o_g, dq_g, dk_g, dv_g) = outs
    vq = qv.cpu()
    torch.testing.assert_close(o_g[vq], o_c[vq], rtol=5e-4, atol=5e-5)
    torch.testing.assert_close(dq_g[vq], dq_c[vq], rtol=5e-4, atol=1e-4)
    torch.testing.assert_close(dk_g[vq], dk_c[vq], rtol=5e-4, atol=1e-4)
    torch.testing.assert_close(dv_g[vq], dv_c[vq], rtol=5e-4, atol=1e-4)


@pytest.mark.parametrize("B,S,H,Hkv,D,kernels", [(2, 250, 8, 1, 256, True), (1, 90, 8, 1, 256, False), (2, 40, 4, 4, 72, True)])
def test_fp32_attention_reaches_its_kernels(B, S, H, Hkv, D, kernels):
    """``ops.block_attention`` on fp32 CUDA tensors launches them (forward and backward) where the rule says so, and
    gives the dense statement's answer where masks broadcast."""
    from opentau_b200 import ops
    from opentau_b200.ops import cuda_ops
    q, k, v = (torch.randn(B, S, h, D, device="cuda").requires_grad_() for h in (H, Hkv, Hkv))
    blk = torch.arange(S, device="cuda").int().expand(B, -1)
    ok = torch.ones(B, S, dtype=torch.bool, device="cuda")
    before = cuda_ops.launch_count
    o = ops.block_attention(q, k, v, blk, blk, ok, ok, D ** -0.5)
    o.sum().backward()
    assert (cuda_ops.launch_count > before) == kernels
    wide = ops.block_attention(q, k, v, blk[:1], blk[:1], ok[:1], ok[:1], D ** -0.5)
    assert _rel(wide.detach(), o.detach().double()) < 256 * 2 ** -24


def _fp64(q, k, v, do, qb, kb, qv, kv, scale):
    """``(o, dq, dk, dv)`` of the masked attention in 64 bits."""
    B, Sq, H, D = q.shape
    K = k.shape[2]
    a = [q.double(), k.double().repeat_interleave(H // K, 2), v.double().repeat_interleave(H // K, 2)]
    a = [t.requires_grad_() for t in a]
    m = (qv[:, :, None] & kv[:, None, :] & (kb[:, None, :] <= qb[:, :, None]))[:, None]
    s = (torch.einsum("bqhd,bkhd->bhqk", a[0], a[1]) * scale).masked_fill(~m, -1e300)
    p = torch.where(m, torch.softmax(s, -1), 0.0)
    o = torch.einsum("bhqk,bkhd->bqhd", p, a[2]).reshape(B, Sq, H * D)
    dq, dk, dv = torch.autograd.grad(o, a, do.double())
    return o.detach(), dq, dk.view(B, -1, K, H // K, D).sum(3), dv.view(B, -1, K, H // K, D).sum(3)


def _rel(got, want):
    return ((got.double() - want).norm() / want.norm().clamp_min(1e-30)).item()


@pytest.mark.parametrize("D", [4, 28, 72, 132, 256])
@pytest.mark.parametrize("Sq,cross", [(1, 0), (31, 1), (32, 32), (33, 63), (64, 0), (65, 0), (129, 70), (400, 0)])
@pytest.mark.parametrize("H,Hkv", [(8, 1), (4, 4)])
def test_fp32_attention_kernels_at_the_edges_of_their_tiles(D, Sq, cross, H, Hkv):
    """32 owner rows, 64 streamed rows, widths that pad to 16, split sums (400 positions under one kv head), against 64
    bits.  Bound: an inner product of n terms rounds to within n 2^-24 of the sum of its magnitudes (n = 256 at most here,
    the sums over rows average out).  A hidden key may hold anything, NaN included."""
    from opentau_b200.ops import attention_native
    B, Sk = 2, Sq + cross
    g = torch.Generator(device="cuda").manual_seed(D + Sq)
    q, k, v, do = (torch.randn(*shape, device="cuda", generator=g)
                   for shape in ((B, Sq, H, D), (B, Sk, Hkv, D), (B, Sk, Hkv, D), (B, Sq, H * D)))
    kb = torch.cat([torch.full((B, cross), -2**31, device="cuda"), torch.arange(Sq, device="cuda").expand(B, -1) // 5], 1).int()
    qb, kv = kb[:, cross:].contiguous(), torch.rand(B, Sk, device="cuda", generator=g) > 0.1
    qv = torch.rand(B, Sq, device="cuda", generator=g) > 0.1
    kv[:, 0] = qv[:, -1] = True
    do = do * qv[:, :, None]
    want = _fp64(q, k, v, do, qb, kb, qv, kv, D ** -0.5)
    k[~kv], v[~kv] = float("nan"), float("nan")
    o, lse = attention_native.attn_f32_fwd(q, k, v, qb, kb, qv, kv, D ** -0.5)
    got = (o, *attention_native.attn_f32_bwd(do, q, k, v, o, lse, qb, kb, qv, kv, D ** -0.5))
    again = attention_native.attn_f32_bwd(do, q, k, v, o, lse, qb, kb, qv, kv, D ** -0.5, keep_ds=False)
    for name, x, w in zip(("o", "dq", "dk", "dv", "dq recomputed"), (*got, again[0]), (*want, want[1])):      # inputs of unit scale: their count bounds cancellation
        assert (x.double() - w).norm() < 256 * 2 ** -24 * (w.norm() + w.numel() ** 0.5), name


@pytest.mark.parametrize("B,S,H,Hkv,D", [(4, 333, 16, 16, 72), (2, 1300, 8, 1, 128), (3, 200, 32, 32, 64), (5, 129, 16, 16, 24),
                                         (2, 641, 16, 16, 96), (160, 65, 1, 1, 128)])
def test_forward_with_two_tiles_per_sm(B, S, H, Hkv, D):
    """More tiles than SMs up to width 128: probabilities in tensor memory, last blocks and tiles of one row, rows that see
    nothing, against 64 bits.  Probabilities and results are rounded to bf16, 2^-9 each."""
    from opentau_b200.ops import attention_native, cuda_ops
    g = torch.Generator(device="cuda").manual_seed(D + S)
    q, k, v = (torch.randn(B, S, h, D, device="cuda", generator=g).to(torch.bfloat16) for h in (H, Hkv, Hkv))
    blk = (torch.arange(S, device="cuda") - S // 2).clamp_min(0).expand(B, -1).int().contiguous()
    valid = torch.ones(B, S, dtype=torch.bool, device="cuda")
    valid[1, S - 7:] = False
    o, lse = attention_native.attn_fwd(q, k, v, blk, blk, valid, valid, D ** -0.5)
    cuda_ops.check_status()
    see = valid[:, None, :, None] & valid[:, None, None, :] & (blk[:, None, None, :] <= blk[:, None, :, None])
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double().repeat_interleave(H // Hkv, 2)) * D ** -0.5
    s = s.masked_fill(~see, float("-inf"))
    want = torch.einsum("bhqk,bkhd->bqhd", s.softmax(-1).nan_to_num(0.0), v.double().repeat_interleave(H // Hkv, 2))
    assert _rel(o.view_as(q), want) < 2 ** -8
    ref = torch.logsumexp(s, -1)
    ref = torch.where(ref.isinf(), torch.zeros_like(ref), ref)
    assert (lse.double() - ref).abs().max() < 1e-3


@pytest.mark.parametrize("B,Sq,Sk,H,Hkv,D", [(1, 50, 1018, 8, 1, 256), (1, 60, 1018, 8, 1, 256), (1, 1, 700, 8, 1, 256),
                                             (1, 50, 1074, 8, 4, 256), (2, 17, 400, 4, 2, 128), (1, 33, 322, 32, 1, 64),
                                             (1, 3, 515, 64, 1, 64)])
def test_cluster_tiles_of_32_and_64_rows(B, Sq, Sk, H, Hkv, D):
    """Tiles whose keys a cluster shares, on both sides of the line between 32 and 64 rows, against 64 bits."""
    from opentau_b200.ops import attention_native, cuda_ops
    g = torch.Generator(device="cuda").manual_seed(Sq + Sk)
    q, k, v = (torch.randn(B, n, h, D, device="cuda", generator=g).to(torch.bfloat16) for n, h in ((Sq, H), (Sk, Hkv), (Sk, Hkv)))
    k_ok = torch.rand(B, Sk, device="cuda", generator=g) > 0.2
    q_ok = torch.ones(B, Sq, dtype=torch.bool, device="cuda")
    q_ok[-1, -1] = Sq == 1
    zq, zk = (torch.zeros(B, n, dtype=torch.int32, device="cuda") for n in (Sq, Sk))
    assert attention_native.split_cluster(B, Sq, Sk, H, Hkv, D) > 1
    o, lse = attention_native.attn_fwd(q, k, v, zq, zk, q_ok, k_ok, D ** -0.5)
    cuda_ops.check_status()
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double().repeat_interleave(H // Hkv, 2)) * D ** -0.5
    s = s.masked_fill(~(q_ok[:, None, :, None] & k_ok[:, None, None]), float("-inf"))
    want = torch.einsum("bhqk,bkhd->bqhd", s.softmax(-1).nan_to_num(0.0), v.double().repeat_interleave(H // Hkv, 2))
    assert _rel(o.view_as(q), want) < 2 ** -8
    ref = torch.logsumexp(s, -1)
    assert (lse.double() - torch.where(ref.isinf(), torch.zeros_like(ref), ref)).abs().max() < 1e-3


@pytest.mark.parametrize("D,H,Hkv", [(256, 8, 1), (256, 8, 4), (200, 2, 2), (136, 64, 1)])
@pytest.mark.parametrize("Sq,Sk", [(1, 1), (15, 64), (17, 65), (33, 128), (130, 129), (65, 300), (200, 513)])
@pytest.mark.parametrize("big", [1.0, 12.0])
def test_unsplit_forward_above_width_128(D, H, Hkv, Sq, Sk, big):
    """Blocks that two groups of warps take in turn: one block, two, an odd and an even number; tiles with a row more or less; block ids
    in no order, rows that see nothing, rows whose first visible key comes late; scores that make either group rescale.  Against
    64 bits: P and the result are rounded to bf16 (2^-9 each)."""
    from opentau_b200.ops import attention_native, cuda_ops
    B = 2
    g = torch.Generator(device="cuda").manual_seed(D + 7 * Sq + Sk)
    q, k, v = (torch.randn(*shape, device="cuda", generator=g) for shape in ((B, Sq, H, D), (B, Sk, Hkv, D), (B, Sk, Hkv, D)))
    k *= torch.linspace(0.1, big, Sk, device="cuda")[None, :, None, None]     # the maximum keeps growing
    q, k, v = (t.to(torch.bfloat16) for t in (q, k, v))
    qb = torch.randint(0, 6, (B, Sq), device="cuda", generator=g, dtype=torch.int32)
    kb = torch.randint(0, 8, (B, Sk), device="cuda", generator=g, dtype=torch.int32)
    kb[1, :Sk // 2] = 9
    qv = torch.rand(B, Sq, device="cuda", generator=g) > 0.1
    kv = torch.rand(B, Sk, device="cuda", generator=g) > 0.1
    qb[0, :Sq // 3] = -1                                               # sees nothing
    o, lse = attention_native.attn_fwd(q, k, v, qb, kb, qv, kv, D ** -0.5, nsplit=1)
    cuda_ops.check_status()
    see = qv[:, None, :, None] & kv[:, None, None, :] & (kb[:, None, None, :] <= qb[:, None, :, None])
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double().repeat_interleave(H // Hkv, 2)) * D ** -0.5
    s = s.masked_fill(~see, -torch.inf)
    want_lse = s.logsumexp(-1).nan_to_num(neginf=0.0)
    p = (s - want_lse[..., None]).exp().masked_fill(~see, 0.0)
    want = torch.einsum("bhqk,bkhd->bqhd", p, v.double().repeat_interleave(H // Hkv, 2)).reshape(B, Sq, H * D)
    assert _rel(o, want) < 2 ** -8
    assert float((lse.double() - want_lse).abs().max()) < 1e-4 * big ** 2 + 1e-5      # fp32 sums of scores up to about 5 big


@pytest.mark.parametrize("D,H,Hkv", [(256, 8, 1), (256, 2, 2), (160, 4, 4), (136, 64, 1)])
@pytest.mark.parametrize("Sk", [1, 20, 64, 65, 128, 192, 193, 256, 300])
def test_forward_of_one_query_tile_gives_the_bits_of_several(D, H, Hkv, Sk):
    """A tile to a kv head and a few blocks of keys take another kernel than several tiles, where both sum in one order."""
    from opentau_b200.ops import attention_native, cuda_ops
    B, one = 3, 128 * Hkv // H
    gen = torch.Generator(device="cuda").manual_seed(D + Sk)
    q, k, v = (torch.randn(*s, device="cuda", generator=gen).to(torch.bfloat16)
               for s in ((B, 2 * one + 1, H, D), (B, Sk, Hkv, D), (B, Sk, Hkv, D)))
    qb = torch.randint(0, 6, q.shape[:2], device="cuda", generator=gen, dtype=torch.int32)
    kb = torch.randint(0, 7, (B, Sk), device="cuda", generator=gen, dtype=torch.int32)
    qv, kv = torch.rand(q.shape[:2], device="cuda", generator=gen) > 0.1, torch.rand(B, Sk, device="cuda", generator=gen) > 0.1
    all_o, all_lse = attention_native.attn_fwd(q, k, v, qb, kb, qv, kv, D ** -0.5, nsplit=1)
    for n in (1, one):
        o, lse = attention_native.attn_fwd(q[:, :n].contiguous(), k, v, qb[:, :n], kb, qv[:, :n], kv, D ** -0.5, nsplit=1)
        assert torch.equal(o, all_o[:, :n]) and torch.equal(lse, all_lse[:, :, :n])
    cuda_ops.check_status()


@pytest.mark.parametrize("D,H,Hkv,S", [(256, 8, 1, 513), (256, 2, 2, 1000), (200, 4, 4, 449), (136, 8, 4, 65), (128, 4, 2, 1025),
                                       (96, 2, 2, 129), (64, 8, 1, 900), (24, 4, 4, 1000), (16, 32, 1, 130)])
@pytest.mark.parametrize("samples", [2, 0])
def test_backward_with_fixed_tiles_in_tensor_memory(D, H, Hkv, S, samples):
    """Rings that wrap twice, last blocks and tiles of one column or row, head widths off the 64-column pieces, against 64 bits.
    P, dS and the results are rounded to bf16 (2^-9 each): the sums' relative error stays below two of them."""
    from opentau_b200.ops import attention_native, cuda_ops
    B = 2
    g = torch.Generator(device="cuda").manual_seed(D + S)
    q, k, v, do = (torch.randn(*shape, device="cuda", generator=g).to(torch.bfloat16)
                   for shape in ((B, S, H, D), (B, S, Hkv, D), (B, S, Hkv, D), (B, S, H, D)))
    blk = (torch.arange(S, device="cuda") - S // 2).clamp_min(0).expand(B, -1).int().contiguous()
    valid = torch.ones(B, S, dtype=torch.bool, device="cuda")
    valid[1, S - 7:] = False
    o, lse = attention_native.attn_fwd(q, k, v, blk, blk, valid, valid, D ** -0.5)
    do[~valid] = 0
    got = attention_native.attn_bwd(do.view(B, S, -1), q, k, v, o, lse, blk, blk, valid, valid, D ** -0.5, samples=samples)
    cuda_ops.check_status()
    qd, kd, vd = (t.double().requires_grad_() for t in (q, k, v))
    see = valid[:, None, :, None] & valid[:, None, None, :] & (blk[:, None, None, :] <= blk[:, None, :, None])
    s = torch.einsum("bqhd,bkhd->bhqk", qd, kd.repeat_interleave(H // Hkv, 2)) * D ** -0.5
    p = s.masked_fill(~see, -1e30).softmax(-1).masked_fill(~see, 0.0)
    out = torch.einsum("bhqk,bkhd->bqhd", p, vd.repeat_interleave(H // Hkv, 2))
    want = torch.autograd.grad(out, (qd, kd, vd), do.double())
    for name, x, w in zip(("dq", "dk", "dv"), got, want):
        assert _rel(x, w) < 2 ** -8, (name, _rel(x, w))


@pytest.mark.parametrize("D,H,Hkv,S", [(64, 4, 1, 900), (72, 16, 16, 260), (128, 8, 2, 641), (200, 4, 4, 449), (256, 8, 1, 1027)])
@pytest.mark.parametrize("samples", [2, 1, 0])
def test_backward_of_strided_views_and_repeats(D, H, Hkv, S, samples):
    """q, k and v as views of one q/k/v buffer (the fixed tiles are addressed by hand), a second sample and a gradient that starts
    off a 16-byte boundary: the same bits as contiguous tensors give, and the same bits again every time (a block's scores go
    over the columns that the block before has just read, rings wrap many times)."""
    from opentau_b200.ops import attention_native, cuda_ops
    B = 2
    g = torch.Generator(device="cuda").manual_seed(D + S)
    qkv = torch.randn(B, S, (H + 2 * Hkv) * D, device="cuda", generator=g).to(torch.bfloat16)
    q = qkv[..., :H * D].unflatten(-1, (H, D))
    k, v = (t.unflatten(-1, (Hkv, D)) for t in qkv[..., H * D:].chunk(2, -1))
    blk = (torch.arange(S, device="cuda") - S // 2).clamp_min(0).expand(B, -1).int().contiguous()
    valid = torch.ones(B, S, dtype=torch.bool, device="cuda")
    valid[1, S - 7:] = False
    raw = torch.randn(B * S * H * D + 1, device="cuda", generator=g).to(torch.bfloat16)
    do = raw[1:].view(B, S, H * D)
    assert not q.is_contiguous() and not v.is_contiguous() and do.data_ptr() % 16
    o, lse = attention_native.attn_fwd(q, k, v, blk, blk, valid, valid, D ** -0.5)
    args = (o, lse, blk, blk, valid, valid, D ** -0.5)
    want = attention_native.attn_bwd(do.clone(), q.contiguous(), k.contiguous(), v.contiguous(), *args, samples=samples)
    for _ in range(4):
        got = attention_native.attn_bwd(do, q, k, v, *args, samples=samples)
        assert all(torch.equal(x, y) for x, y in zip(got, want))
    cuda_ops.check_status()


@pytest.mark.parametrize("D,H,Hkv", [(256, 8, 1), (256, 8, 4), (200, 2, 2), (128, 32, 1), (72, 4, 4), (64, 8, 2)])
@pytest.mark.parametrize("Sq,Sk", [(1, 1), (17, 63), (16, 64), (33, 65), (130, 257), (257, 130), (300, 513)])
@pytest.mark.parametrize("samples,parts", [(1, None), (3, None), (2, 3)])
def test_stored_backward_matches_the_recomputing_one(D, H, Hkv, Sq, Sk, samples, parts):
    """Query tiles, stored blocks of 64 and key tiles of 256 with one row more or less; block ids in no order, a tile that sees
    nothing, keys that nobody sees, queries without a key; several launches for a batch; parts of dK and dV, empty ones among them.
    Both paths round P and dS to bf16 and sum in fp32: what differs is delta's order of summation and the result's rounding (2^-8).
    A query that sees one key has dS = 0 but for what dP and delta, fp32 sums of D products of unit normals, lose where they
    cancel: D 2^-24 of sum |o dO| = 0.64 D, times the scale D^-1/2, below 2^-12 at D = 256, whatever the size of the result."""
    from opentau_b200.ops import attention_native, cuda_ops
    B = 3
    g = torch.Generator(device="cuda").manual_seed(D + 7 * Sq + Sk)
    q, k, v, do = (torch.randn(*shape, device="cuda", generator=g).to(torch.bfloat16)
                   for shape in ((B, Sq, H, D), (B, Sk, Hkv, D), (B, Sk, Hkv, D), (B, Sq, H * D)))
    qb = torch.randint(0, 6, (B, Sq), device="cuda", generator=g, dtype=torch.int32)
    kb = torch.randint(0, 8, (B, Sk), device="cuda", generator=g, dtype=torch.int32)
    kb[1, Sk // 2:] = 9                                                # hidden from every query
    kb[2] = -2147483648                                                # cached keys
    qv = torch.rand(B, Sq, device="cuda", generator=g) > 0.1
    kv = torch.rand(B, Sk, device="cuda", generator=g) > 0.1
    qv[0, Sq // 2:] = False
    qb[1, :Sq // 3] = -1                                               # sees nothing
    o, lse = attention_native.attn_fwd(q, k, v, qb, kb, qv, kv, D ** -0.5)
    args = (do, q, k, v, o, lse, qb, kb, qv, kv, D ** -0.5)
    want = attention_native.attn_bwd(*args, samples=0)
    got = attention_native.attn_bwd(*args, samples=samples, parts=parts)
    again = attention_native.attn_bwd(*args, samples=samples, parts=parts)
    cuda_ops.check_status()
    for name, x, y, w in zip(("dq", "dk", "dv"), got, again, want):
        assert torch.equal(x, y), name
        diff = (x.double() - w.double()).norm().item()
        assert bool(torch.isfinite(x).all()) and diff <= 2 ** -8 * w.double().norm().item() + 2 ** -12 * x.numel() ** 0.5, (name, diff)
    assert float(got[1][1, Sk // 2:].abs().sum()) == 0.0 and float(got[0][0, Sq // 2:].abs().sum()) == 0.0


@pytest.mark.parametrize("D,H,Hkv", [(256, 8, 1), (256, 8, 4), (200, 2, 2), (128, 32, 1), (72, 4, 4), (64, 8, 2)])
@pytest.mark.parametrize("seen,asked", [(300, 333), (64, 700), (257, 130), (1, 1), (449, 513)])
@pytest.mark.parametrize("samples", [1, 2, 0])
def test_backward_reads_no_key_or_query_behind_the_last_visible_block(D, H, Hkv, seen, asked, samples):
    """NaN in the keys behind the block that holds the last visible one (64 keys, 128 up to head width 128), and in the query rows behind
    the last valid one's, leaves every gradient as if zeros stood there, bit for bit."""
    from opentau_b200.ops import attention_native, cuda_ops
    B, S, g = 2, 700, H // Hkv
    gen = torch.Generator(device="cuda").manual_seed(D + seen)
    q, k, v, do = (torch.randn(*shape, device="cuda", generator=gen).to(torch.bfloat16)
                   for shape in ((B, S, H, D), (B, S, Hkv, D), (B, S, Hkv, D), (B, S, H, D)))
    block = 64 if D > 128 else 128
    keys, rows = -(-seen // block) * block, -(-asked * g // block) * block // g
    blk = torch.zeros(B, S, dtype=torch.int32, device="cuda")
    qv, kv = (torch.arange(S, device="cuda").expand(B, -1) < n for n in (asked, seen))
    out = []
    for fill in (float("nan"), 0.0):
        k[:, keys:], v[:, keys:], q[:, rows:], do[:, rows:] = fill, fill, fill, fill
        o, lse = attention_native.attn_fwd(q, k, v, blk, blk, qv, kv, D ** -0.5, nsplit=1)
        grads = attention_native.attn_bwd(do.reshape(B, S, H * D), q, k, v, o, lse, blk, blk, qv, kv, D ** -0.5, samples=samples)
        out.append((o.view(B, S, H, D)[:, :asked], *grads))
    cuda_ops.check_status()
    for name, x, want in zip(("o", "dq", "dk", "dv"), *out):
        assert torch.equal(x, want), name


def test_backward_recomputes_where_there_is_no_room_for_p_and_ds(monkeypatch):
    """A call whose P and dS are more than is kept goes a sample at a time, then without them; so does one that finds no memory."""
    from opentau_b200.ops import attention_native, cuda_ops
    B, S, H, Hkv, D = 2, 200, 8, 1, 64
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v, do = (torch.randn(*shape, device="cuda", generator=g).to(torch.bfloat16)
                   for shape in ((B, S, H, D), (B, S, Hkv, D), (B, S, Hkv, D), (B, S, H * D)))
    blk, valid = torch.zeros(B, S, dtype=torch.int32, device="cuda"), torch.ones(B, S, dtype=torch.bool, device="cuda")
    o, lse = attention_native.attn_fwd(q, k, v, blk, blk, valid, valid, D ** -0.5)
    args = (do, q, k, v, o, lse, blk, blk, valid, valid, D ** -0.5)
    want = {n: attention_native.attn_bwd(*args, samples=n) for n in (2, 1, 0)}
    assert all(_rel(x, w.double()) < 2 ** -8 for n in (2, 1) for x, w in zip(want[n], want[0]))
    both = attention_native.bwd_stored_plan(1, S, S, H, Hkv, D)[0] * 2
    entry, taken = attention_native._entry, []
    monkeypatch.setattr(attention_native, "_entry", lambda lib, *a: (taken.append(lib), entry(lib, *a))[1])
    for limit, samples in ((2 * both, 2), (both, 1), (both - 1, 0)):
        monkeypatch.setattr(attention_native, "BWD_STORED_LIMIT", limit)
        assert attention_native.stored_bwd_samples(B, S, S, H, Hkv, D) == samples
        taken.clear()
        got = attention_native.attn_bwd(*args)
        cuda_ops.check_status()
        assert taken == ["attention_bwd_stored_tcgen05" if samples else "attention_bwd_tcgen05"]
        assert all(torch.equal(x, w) for x, w in zip(got, want[samples]))
    monkeypatch.undo()
    real = torch.empty

    def empty(*a, **kw):
        if kw.get("dtype") is torch.uint8:
            raise torch.cuda.OutOfMemoryError
        return real(*a, **kw)

    monkeypatch.setattr(torch, "empty", empty)
    got = attention_native.attn_bwd(*args)
    monkeypatch.undo()
    assert all(torch.equal(x, w) for x, w in zip(got, want[0]))


@pytest.mark.parametrize("B,Sq,Sk,H,Hkv,D", [(36, 2, 2, 32, 1, 256), (9, 113, 113, 8, 4, 256), (23, 34, 903, 2, 2, 256), (3, 106, 106, 12, 12, 64),
                                             (110, 244, 7, 1, 1, 128), (37, 300, 70, 1, 1, 72), (74, 20, 300, 1, 1, 64)])
def test_stored_backward_of_many_kv_heads(B, Sq, Sk, H, Hkv, D):
    """(sample, kv head)s whose jobs are no multiple of the CTA pairs, dealt in every way; against the recomputing kernels as above."""
    from opentau_b200.ops import attention_native, cuda_ops
    g = torch.Generator(device="cuda").manual_seed(B + Sq)
    q, k, v, do = (torch.randn(*shape, device="cuda", generator=g).to(torch.bfloat16)
                   for shape in ((B, Sq, H, D), (B, Sk, Hkv, D), (B, Sk, Hkv, D), (B, Sq, H * D)))
    qb, kb = (torch.randint(0, n, (B, s), device="cuda", generator=g, dtype=torch.int32) for n, s in ((6, Sq), (8, Sk)))
    qv, kv = (torch.rand(B, s, device="cuda", generator=g) > 0.1 for s in (Sq, Sk))
    o, lse = attention_native.attn_fwd(q, k, v, qb, kb, qv, kv, D ** -0.5)
    args = (do, q, k, v, o, lse, qb, kb, qv, kv, D ** -0.5)
    got, want = attention_native.attn_bwd(*args, samples=B), attention_native.attn_bwd(*args, samples=0)
    cuda_ops.check_status()
    for name, x, w in zip(("dq", "dk", "dv"), got, want):
        diff = (x.double() - w.double()).norm().item()
        assert bool(torch.isfinite(x).all()) and diff <= 2 ** -8 * w.double().norm().item() + 2 ** -12 * x.numel() ** 0.5, (name, diff)


@pytest.mark.parametrize("D,H,Hkv", [(256, 8, 1), (128, 8, 2), (64, 4, 4), (72, 16, 16)])
@pytest.mark.parametrize("splits", [(2, 3, 2), (4, 16, 7)])
def test_split_backward_matches_the_unsplit_one(D, H, Hkv, splits):
    """Parts of every size, empty ones among them (a causal tail leaves late key tiles with few query blocks).  Split sums
    differ from the running one by rounding in fp32 and agree after the one rounding to bf16 but for ties (2^-8)."""
    from opentau_b200.ops import attention_native, cuda_ops
    B, S = 2, 333
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v, do = (torch.randn(*shape, device="cuda", generator=g).to(torch.bfloat16)
                   for shape in ((B, S, H, D), (B, S, Hkv, D), (B, S, Hkv, D), (B, S, H * D)))
    blk = (torch.arange(S, device="cuda") - 40).clamp_min(0).expand(B, -1).int().contiguous()
    valid = torch.ones(B, S, dtype=torch.bool, device="cuda")
    valid[1, 300:] = False
    args = (q, k, v, blk, blk, valid, valid, D ** -0.5)
    o, lse = attention_native.attn_fwd(*args)
    args = (do, q, k, v, o, lse, blk, blk, valid, valid, D ** -0.5)
    one = attention_native.attn_bwd(*args, splits=(1, 1, 1))
    got = attention_native.attn_bwd(*args, splits=splits)
    cuda_ops.check_status()
    for name, x, w in zip(("dq", "dk", "dv"), got, one):
        x, w = x[valid], w[valid]
        assert _rel(x, w.double()) < 2 ** -8, name
    for x in got[1:]:
        assert float(x[1, 300:].abs().max()) == 0.0


@pytest.mark.parametrize("bad_keys", [False, True])
@pytest.mark.parametrize("H,Hkv,D", [(4, 1, 64), (8, 1, 256)])
def test_fp32_attention_keeps_nan_and_infinite_scores(H, Hkv, D, bad_keys):
    """A NaN or infinite row or key of the inputs shows in ``block_attention``'s output where the dense evaluation shows
    it: a row of nothing but NaN or -inf scores is not one that sees no key."""
    from opentau_b200 import ops
    from opentau_b200.ops import prims
    B, S = 1, 260
    g = torch.Generator().manual_seed(D)
    q, k, v, do = (torch.randn(B, S, h, D, generator=g) for h in (H, Hkv, Hkv, H))
    k[..., 0] = 2.0
    q[0, 5, 0], q[0, 70, H - 1, 3] = float("nan"), float("nan")      # all scores of a row NaN
    q[0, 33, 1, 0], q[0, 200, 0, 0] = 3e38, -3e38                    # all +inf, all -inf
    if bad_keys:
        k[0, 250] = float("nan")                                     # for the rows that see it
    blk = (torch.arange(S) // 20).int()[None]
    ok = torch.ones(B, S, dtype=torch.bool)
    ok[0, 100:110] = False                                           # rows that see nothing stay zero
    args = (blk, blk, ok, ok, D ** -0.5)
    dev_args = (*(t.cuda() for t in args[:4]), args[4])
    o_w, lse_w = prims.attn_fwd(q, k, v, *args)
    a = [t.cuda().requires_grad_() for t in (q, k, v)]
    lse = prims.attn_fwd(*(t.detach() for t in a), *dev_args)[1]
    o = ops.block_attention(*a, *dev_args)
    pairs = [("o", o.detach(), o_w), ("lse", lse, lse_w)]
    if not bad_keys:                # (the dense backward also spreads NaN between rows and keys that do not meet)
        dq_w, _, dv_w = prims.attn_bwd(do.reshape(B, S, -1), q, k, v, o_w, lse_w, *args)
        dq, _, dv = torch.autograd.grad(o, a, do.reshape(B, S, -1).cuda())
        pairs += [("dq", dq, dq_w), ("dv", dv, dv_w)]
    for name, x, w in pairs:
        x = x.cpu()
        assert torch.equal(x.isnan(), w.isnan()) and torch.equal(x.isposinf(), w.isposinf()), name
        assert torch.equal(x.isneginf(), w.isneginf()), name
        torch.testing.assert_close(x[w.isfinite()], w[w.isfinite()], rtol=1e-4, atol=1e-4)
    assert not o_w[0, 105].any() and not lse_w[0, :, 105].any()


def test_fp32_attention_takes_more_sequences_than_a_grid_has_rows():
    """65 536 sequences of a few positions (temporal attention of a batch of clips) take the dense evaluation."""
    from opentau_b200 import ops
    B, S, H, D = 65536, 3, 1, 8
    q, k, v = (torch.randn(B, S, H, D, device="cuda").requires_grad_() for _ in range(3))
    blk = torch.arange(S, device="cuda").int().expand(B, -1)
    ok = torch.ones(B, S, dtype=torch.bool, device="cuda")
    o = ops.block_attention(q, k, v, blk, blk, ok, ok, D ** -0.5)
    grads = torch.autograd.grad(o.square().sum(), (q, k, v))
    a = [t.detach()[-40:].requires_grad_() for t in (q, k, v)]
    w = ops.block_attention(*a, blk[:40], blk[:40], ok[:40], ok[:40], D ** -0.5)
    for x, y in zip((o, *grads), (w, *torch.autograd.grad(w.square().sum(), a))):
        torch.testing.assert_close(x[-40:], y, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("H,Hkv,D", [(8, 1, 256), (8, 4, 256), (16, 16, 72), (32, 1, 128)])
@pytest.mark.parametrize("B,S", [(1, 400), (1, 4096), (8, 1300), (1, 131072), (8, 65536)])
def test_split_backward_scratch_is_bounded(H, Hkv, D, B, S):
    """The parts of one output never pass 256 MB, in bf16's backward as in fp32's (sizes only: nothing is allocated)."""
    from ctypes import byref, c_int, c_longlong
    from opentau_b200.ops import _lib, attention_native
    outs = [4 * B * S * H * D] + [4 * B * S * Hkv * D] * 2
    parts = [attention_native.bwd_splits(B, S, S, H, Hkv, D)]
    dq, dkv, ds = c_int(), c_int(), c_longlong()
    _lib.load("attention_f32").otb_attn_f32_bwd_plan(B, S, S, H, Hkv, D, byref(dq), byref(dkv), byref(ds))
    parts.append((dq.value, dkv.value, dkv.value))
    for m in parts:
        assert all(n >= 1 and (n == 1 or n * out <= 1 << 28) for n, out in zip(m, outs)), m
    assert 4 * ds.value <= attention_native.F32_DS_LIMIT
    if (B, S, H, Hkv) == (1, 4096, 8, 1):
        assert min(parts[0][1:]) > 4                        # where they pay they are kept


@pytest.mark.parametrize("forward", [True, False])
@pytest.mark.parametrize("backward", [True, False])
def test_fp32_attention_may_take_either_path_in_each_direction(forward, backward, monkeypatch):
    """Kernels and dense evaluation hand each other O and LSE: every combination gives the 64-bit gradients to fp32
    rounding (256 * 2^-24 of the norm: inner products of at most 256 terms)."""
    from opentau_b200 import ops
    from opentau_b200.ops import attention_native, cuda_ops
    monkeypatch.setattr(attention_native, "_f32_kernels_pay", lambda *a: backward if a[-1] else forward)
    B, S, H, Hkv, D = 2, 75, 6, 2, 72
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v, do = (torch.randn(B, S, h, D, device="cuda", generator=g) for h in (H, Hkv, Hkv, H))
    blk = (torch.arange(S, device="cuda") // 9).int().expand(B, -1).contiguous()
    ok = torch.rand(B, S, device="cuda", generator=g) > 0.15
    ok[:, 0] = True
    do = (do * ok[:, :, None, None]).reshape(B, S, -1)
    want = _fp64(q, k, v, do, blk, blk, ok, ok, D ** -0.5)
    a = [t.requires_grad_() for t in (q, k, v)]
    before = cuda_ops.launch_count
    o = ops.block_attention(*a, blk, blk, ok, ok, D ** -0.5)
    assert (cuda_ops.launch_count > before) == forward
    before = cuda_ops.launch_count
    grads = torch.autograd.grad(o, a, do)
    assert (cuda_ops.launch_count > before) == backward
    for x, w in zip((o.detach(), *grads), want):
        assert _rel(x, w) < 256 * 2 ** -24


def test_fp32_backward_recomputes_ds_where_there_is_no_room_for_it(monkeypatch):
    from opentau_b200.ops import attention_native
    B, S, H, D = 1, 70, 2, 64
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v, do = (torch.randn(B, S, H, D, device="cuda", generator=g) for _ in range(4))
    blk = torch.arange(S, device="cuda").int()[None]
    args = (blk, blk, torch.ones(B, S, dtype=torch.bool, device="cuda"), torch.ones(B, S, dtype=torch.bool, device="cuda"), D ** -0.5)
    o, lse = attention_native.attn_f32_fwd(q, k, v, *args)
    want = attention_native.attn_f32_bwd(do.reshape(B, S, -1), q, k, v, o, lse, *args, keep_ds=False)
    empty = torch.empty

    def full(*size, **kw):
        if len(size) == 1:                                  # the scratch of dS alone has one dimension
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*size, **kw)

    monkeypatch.setattr(torch, "empty", full)
    got = attention_native.attn_f32_bwd(do.reshape(B, S, -1), q, k, v, o, lse, *args)
    for x, y in zip(got, want):
        assert torch.equal(x, y)

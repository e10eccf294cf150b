"""Tiny pi0.5 on the GPU through the native kernels: parity with the CPU oracle, training step, sampler
replayed from a CUDA graph."""

import pytest
import torch

from helpers import tiny_batch, tiny_pi05, tiny_pi05_config
from opentau_b200.datasets.synthetic import identity_stats

pytestmark = pytest.mark.gpu


def _pair(seed=0):
    cpu = tiny_pi05(seed=seed)
    gpu = tiny_pi05(seed=seed)
    gpu.load_state_dict(cpu.state_dict())
    return cpu, gpu.to("cuda").to(torch.bfloat16)


def test_loss_parity_with_cpu_fp32_oracle():
    from opentau_b200.ops import cuda_ops
    cpu, gpu = _pair()
    for n, p in cpu.named_parameters():        # open the adaptive-norm gates so the expert path matters
        if ".dense." in n:
            torch.nn.init.normal_(p, std=0.05)
    gpu.load_state_dict(cpu.state_dict())
    gpu = gpu.to("cuda").to(torch.bfloat16)
    b = tiny_batch()
    noise, time = torch.randn(4, 10, 32), torch.full((4,), 0.4)
    ref = cpu(b, noise=noise, time=time)
    bg = {k: v.cuda() for k, v in b.items()}
    out = gpu(bg, noise=noise.cuda(), time=time.cuda())
    cuda_ops.check_status()
    assert abs(out["MSE"].item() - ref["MSE"].item()) / ref["MSE"].item() < 3e-2
    assert abs(out["CE"].item() - ref["CE"].item()) / ref["CE"].item() < 3e-2
    (out["MSE"] + out["CE"]).backward()
    (ref["MSE"] + ref["CE"]).backward()
    cuda_ops.check_status()
    checked = 0
    for (n, pc), (_, pg) in zip(cpu.named_parameters(), gpu.named_parameters()):
        if pc.grad is None or pc.grad.abs().max() < 1e-6 or pc.numel() < 512:
            continue
        a, c = pg.grad.float().cpu().flatten(), pc.grad.flatten()
        cos = torch.nn.functional.cosine_similarity(a, c, dim=0).item()
        assert cos > 0.98, f"{n}: cosine {cos}"
        checked += 1
    assert checked > 10


def test_training_reduces_loss_on_gpu():
    from opentau_b200.ops import cuda_ops
    from opentau_b200.parallel.engine import OptimHyper, TrainEngine
    pol = tiny_pi05(seed=1).to(torch.bfloat16).train()
    eng = TrainEngine(pol, OptimHyper(lr=2e-3, grad_clip_norm=1.0), device="cuda")
    b = tiny_batch(device="cuda")
    noise, time = torch.randn(4, 10, 32, device="cuda"), torch.full((4,), 0.5, device="cuda")
    first = last = None
    for _ in range(12):
        out = pol(b, noise=noise, time=time)
        loss = out["MSE"] + out["CE"]
        loss.backward()
        eng.optimizer_step()
        first = loss.item() if first is None else first
        last = loss.item()
    cuda_ops.check_status()
    assert last < 0.8 * first


def test_cuda_graph_sampler_matches_eager():
    from opentau_b200.ops import cuda_ops
    pol = tiny_pi05(seed=2).to("cuda").to(torch.bfloat16).eval()
    b = tiny_batch(device="cuda")
    noise = torch.randn(4, 10, 32, device="cuda")
    eager = pol.sample_actions(b, noise=noise)
    pol.enable_cuda_graphs(True)
    g1 = pol.sample_actions(b, noise=noise)
    g2 = pol.sample_actions(b, noise=noise)           # replay
    other = pol.sample_actions(b, noise=noise * 0.5)  # replay with new inputs
    cuda_ops.check_status()
    torch.testing.assert_close(g1, eager, rtol=1e-3, atol=1e-3)
    assert torch.equal(g1, g2)
    assert not torch.allclose(other, g1)
    assert pol._graph_runner.num_graphs == 1


def test_replayed_requests_refuse_infinite_statistics_of_their_own_rows():
    """Two datasets, the second without usable statistics: requests of the first are served, requests of the second are
    refused, also when the graph is already captured and the buffer was written through ``.data``."""
    from opentau_b200.policies.pi05.modeling_pi05 import PI05Policy
    torch.manual_seed(2)
    pol = PI05Policy(tiny_pi05_config("cuda"), per_dataset_stats=[identity_stats(), identity_stats()],
                     dataset_names=["a", "b"]).to("cuda").to(torch.bfloat16).eval()
    for stat in (*pol.normalize_inputs.parameters(), *pol.unnormalize_outputs.parameters()):
        stat.data[1] = float("inf")
    b = tiny_batch(device="cuda")
    B = b["state"].shape[0]
    noise = torch.randn(B, 10, 32, device="cuda")
    first = dict(b, dataset_index=torch.zeros(B, dtype=torch.long, device="cuda"))
    second = dict(b, dataset_index=torch.ones(B, dtype=torch.long, device="cuda"))
    eager = pol.sample_actions(first, noise=noise)
    pol.enable_cuda_graphs(True)
    torch.testing.assert_close(pol.sample_actions(first, noise=noise), eager, rtol=1e-3, atol=1e-3)
    with pytest.raises(AssertionError, match="infinity"):
        pol.sample_actions(second, noise=noise)
    pol.normalize_inputs.buffer_state["max"].data[0] = float("inf")
    with pytest.raises(AssertionError, match="infinity"):
        pol.sample_actions(first, noise=noise)


def test_replayed_requests_of_several_kinds_keep_their_captures():
    """Serving one and several candidates in turn captures each kind once."""
    from opentau_b200.policies.candidates import MEDOID, configure_candidates
    pol = tiny_pi05(seed=2).to("cuda").to(torch.bfloat16).eval()
    b = tiny_batch(device="cuda")
    B = b["state"].shape[0]
    configure_candidates(pol, 3, MEDOID, device=torch.device("cuda"))
    pol.enable_cuda_graphs(True)
    runners = {}
    for n in (1, 3, 1, 3):
        pol.sample_actions(b, noise=torch.randn(B * n, 10, 32, device="cuda"), n_candidates=n)
        assert runners.setdefault(n, pol._graph_runner) is pol._graph_runner and pol._graph_runner.num_graphs == 1
    assert runners[1] is not runners[3]


def _open_policy(**over):
    """A tiny policy whose adaptive norms are open, as a trained checkpoint's are (zero at the start of training)."""
    from opentau_b200.models.layers import AdaRMSNorm
    pol = tiny_pi05(seed=2, **over).to("cuda").to(torch.bfloat16).eval()
    with torch.no_grad():
        for m in pol.modules():
            if isinstance(m, AdaRMSNorm):
                m.dense.weight.normal_(std=0.05)
                m.dense.bias.normal_(std=0.3)
        pol.model.time_mlp_in.weight.normal_(std=0.15)
        pol.model.time_mlp_out.weight.normal_(std=0.15)
    return pol


def test_replayed_samplers_follow_candidates_and_steps():
    """Text prompts replay the sampler alone: other candidate counts and step counts are other captures, each with the
    eager call's actions."""
    from opentau_b200.policies.candidates import MEDOID, configure_candidates
    pol = _open_policy()
    b = {k: v for k, v in tiny_batch(device="cuda").items() if not k.startswith("lang_")}
    B = b["state"].shape[0]
    b["prompt"] = ["pick up the cup"] * B
    configure_candidates(pol, 3, MEDOID, device=torch.device("cuda"))
    for n, steps in ((1, 10), (3, 10), (1, 5), (1, 10)):
        pol.config.num_steps = steps
        noise = torch.randn(B * n, 10, 32, device="cuda")
        pol._use_graphs = False
        eager = pol.sample_actions(b, noise=noise, n_candidates=n)
        if not hasattr(pol, "_request_runners"):
            pol.enable_cuda_graphs(True)
        pol._use_graphs = True
        torch.testing.assert_close(pol.sample_actions(b, noise=noise, n_candidates=n), eager, rtol=1e-3, atol=1e-3)
    assert len(pol._request_runners) == 3


@pytest.mark.parametrize("text", [False, True])
@pytest.mark.parametrize("delay", [3, "per sample"])
def test_frozen_rows_without_a_prefix_stay_free_when_replayed(text, delay):
    """A delay without committed actions only sets the frozen rows' diffusion time; with a prefix they are held at it."""
    pol = _open_policy()
    b = tiny_batch(device="cuda")
    B = b["state"].shape[0]
    if text:
        b = {k: v for k, v in b.items() if not k.startswith("lang_")} | {"prompt": ["pick up the cup"] * B}
    if delay != 3:
        delay = torch.arange(B, device="cuda") % 4
    noise, prefix = torch.randn(B, 10, 32, device="cuda"), torch.randn(B, 10, 32, device="cuda")
    calls = (dict(delay=delay), dict(delay=delay, action_prefix=prefix), dict())
    eager = [pol.sample_actions(b, noise=noise, **kw) for kw in calls]
    pol.enable_cuda_graphs(True)
    for kw, want in zip(calls, eager):
        torch.testing.assert_close(pol.sample_actions(b, noise=noise, **kw), want, rtol=1e-3, atol=1e-3)


def test_replayed_requests_refuse_infinite_statistics_of_every_feature_that_comes():
    """An input that the sampler does not read is normalised, and refused, all the same."""
    from opentau_b200.configs.types import FeatureType, NormalizationMode, PolicyFeature
    from opentau_b200.policies.pi05.modeling_pi05 import PI05Policy
    cfg = tiny_pi05_config("cuda")
    cfg.input_features["environment"] = PolicyFeature(FeatureType.ENV, (4,))
    cfg.normalization_mapping = dict(cfg.normalization_mapping, ENV=NormalizationMode.MIN_MAX)
    stats = dict(identity_stats(), environment={"min": torch.zeros(4), "max": torch.full((4,), float("inf"))})
    pol = PI05Policy(cfg, per_dataset_stats=[stats]).to("cuda").to(torch.bfloat16).eval()
    b = tiny_batch(device="cuda")
    for graphs in (False, True):
        pol.enable_cuda_graphs(graphs)
        pol.sample_actions(b)
        with pytest.raises(AssertionError, match="infinity"):
            pol.sample_actions(dict(b, environment=torch.zeros(b["state"].shape[0], 4, device="cuda")))


def test_replayed_responses_match_the_eager_ones():
    """The first request of a kind with a response runs eagerly, the second captures, later ones replay: the same tokens and
    actions each time, and those of a policy without graphs."""
    pol = _open_policy(predict_response=True, response_max_length=6)
    b = tiny_batch(device="cuda")
    noise = torch.randn(b["state"].shape[0], 10, 32, device="cuda")
    want = pol.sample_actions(b, noise=noise)
    tokens, masks = pol.model.last_response_tokens, pol.model.last_response_masks
    pol.enable_cuda_graphs(True)
    for graphs in (0, 1, 1):
        got = pol.sample_actions(b, noise=noise)
        assert pol._graph_runner.num_graphs == graphs
        assert torch.equal(pol.model.last_response_tokens, tokens) and torch.equal(pol.model.last_response_masks, masks)
        torch.testing.assert_close(got, want, rtol=1e-3, atol=1e-3)


@pytest.mark.parametrize("B", [4, 12, 30])                 # 40, 120 and 300 rows: each way the row products take
@pytest.mark.parametrize("delay", [0, 3, "per sample"])
@pytest.mark.parametrize("prefix", [False, True])
def test_planned_loop_matches_the_step_by_step_one(B, delay, prefix, monkeypatch):
    """Conditions of all steps computed at once and picked per token (frozen ones at time 0) give the velocities of the
    loop that computes them step by step.  Both round to bf16 (2^-8 at most, in their own order) what a step adds to the sample;
    other frozen rows move the result by a third."""
    pol = _open_policy()
    b = tiny_batch(device="cuda", batch_size=B)
    if delay == "per sample":
        delay = torch.arange(B, device="cuda") % 6
    kw = dict(noise=torch.randn(B, 10, 32, device="cuda"), delay=delay)
    if prefix:
        kw["action_prefix"] = torch.randn(B, 10, 32, device="cuda")
    got = pol.sample_actions(b, **kw)
    calls = []
    monkeypatch.setattr(pol.model, "_can_plan_loop", lambda *a: calls.append(a))
    want = pol.sample_actions(b, **kw)
    assert calls
    move = want - kw["noise"]
    assert (got - want).norm() < 2 ** -8 * move.norm()
    other = pol.sample_actions(b, **dict(kw, delay=6))
    assert (other - want).norm() > 2 ** -3 * move.norm()        # frozen rows are seen by the others


def test_replayed_candidates_are_the_eager_ones():
    from opentau_b200.policies.candidates import MEDOID, configure_candidates
    pol = _open_policy()
    b = tiny_batch(device="cuda")
    B = b["state"].shape[0]
    configure_candidates(pol, 3, MEDOID, device=torch.device("cuda"))
    for n in (3, 7):
        noise = torch.randn(B * n, 10, 32, device="cuda")
        pol.enable_cuda_graphs(False)
        want = pol.sample_actions(b, noise=noise, n_candidates=n)
        pol.enable_cuda_graphs(True)
        torch.testing.assert_close(pol.sample_actions(b, noise=noise, n_candidates=n), want, rtol=1e-3, atol=1e-3)


def test_replayed_requests_leave_every_module_in_eval_mode():
    """A vision tower left in training mode is out of it after the call, also when the request is replayed, and a capture is
    made in eval mode."""
    pol = _open_policy(dropout=0.1)
    b = tiny_batch(device="cuda")
    noise = torch.randn(b["state"].shape[0], 10, 32, device="cuda")
    want = pol.sample_actions(b, noise=noise)
    pol.enable_cuda_graphs(True)
    for part in (pol, pol.model.wrapper.paligemma.vision_tower, pol.model.wrapper.decoder):
        part.train()
        torch.testing.assert_close(pol.sample_actions(b, noise=noise), want, rtol=1e-3, atol=1e-3)
        assert not any(m.training for m in pol.modules())

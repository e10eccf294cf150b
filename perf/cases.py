"""What a user of this framework has it do, as measurable cases.

Three kinds of work, each through the entry point a user's program calls:

* ``sample``: one action chunk from a served policy (``policy.sample_actions`` with graph replay armed, as the gRPC and
  websocket servers arm it);
* ``train``: one optimizer step of ``TrainEngine.train_step``;
* ``attention``: forward and backward of ``ops.block_attention``, the op that custom models call directly.

``listed()`` names the cases, ``draw()`` gives more of the same ranges.  Weights are random with the scales of a trained
network where the scale decides what runs or how errors grow (open adaptive-norm gates, depth-scaled residual writes).
"""

from __future__ import annotations

import gc
import math

import torch

from opentau_b200 import ops
from opentau_b200.configs.types import FeatureType, PolicyFeature
from opentau_b200.datasets.synthetic import SyntheticSpec, identity_stats, make_synthetic_batch
from opentau_b200.models.layers import AdaRMSNorm, DecoderLayer
from opentau_b200.parallel.engine import OptimHyper, TrainEngine
from opentau_b200.policies.candidates import MEDOID, configure_candidates
from opentau_b200.policies.pi05.configuration_pi05 import PI05Config
from opentau_b200.policies.pi05.modeling_pi05 import PI05Policy
from opentau_b200.policies.pi06.configuration_pi06 import PI06Config
from opentau_b200.policies.pi06.modeling_pi06 import PI06Policy

CHUNK, ACTION_DIM = 50, 32

# The small pi0.5 of the tests and of ``bench.py --tiny``: two layers everywhere.
TINY = dict(
    vlm=dict(hidden_size=256, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=1, head_dim=64,
             intermediate_size=1024, vocab_size=1024),
    expert=dict(hidden_size=128, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=1, head_dim=64,
                intermediate_size=512, vocab_size=1024),
    vision=dict(hidden_size=128, intermediate_size=256, num_hidden_layers=2, num_attention_heads=4))

# (width, layers, q heads, kv heads, head dim, MLP width) of backbone and expert; (width, layers, MLP width, patches,
# tokens) of the vision tower for one camera; vocabulary
GEOMETRY = {
    "tiny": ((256, 2, 4, 1, 64, 1024), (128, 2, 4, 1, 64, 512), (128, 2, 256, 256, 256), 1024),
    "pi05": ((2048, 18, 8, 1, 256, 16384), (1024, 18, 8, 1, 256, 4096), (1152, 27, 4304, 256, 256), 257152),
    "pi06": ((2560, 34, 8, 4, 256, 10240), (1280, 34, 8, 4, 256, 5120), (1152, 27, 4304, 1024, 256), 262208),
}


def _sample(name, model="pi05", batch=1, cams=3, prompt=200, steps=10, candidates=1, delay=0, response=0, ragged=False):
    return dict(name=name, kind="sample", model=model, batch=batch, cams=cams, prompt=prompt, steps=steps,
                candidates=candidates, delay=delay, response=response, ragged=ragged)


def _train(name, model="pi05", batch=8, cams=3, prompt=200, fast=256, expert_only=False, dropout=0.1):
    return dict(name=name, kind="train", model=model, batch=batch, cams=cams, prompt=prompt, fast=fast,
                expert_only=expert_only, dropout=dropout)


def _attention(name, batch, seq, heads, kv_heads, dim, tail, dtype="bf16"):
    return dict(name=name, kind="attention", batch=batch, seq=seq, heads=heads, kv_heads=kv_heads, dim=dim, tail=tail,
                dtype=dtype)


def listed():
    return [
        # a test-sized policy served to one robot: nothing but launches and host work
        _sample("sample tiny", model="tiny", cams=1, prompt=16),
        # the standard request: one observation of three cameras, ten Euler steps
        _sample("sample pi05"),
        # four simulator environments evaluated together: two cameras, prompts of different lengths padded to 77 tokens,
        # a camera missing in one of them, five actions of the last chunk still to be executed
        _sample("sample pi05 batch 4", batch=4, cams=2, prompt=77, delay=5, ragged=True),
        # best of eight candidates over one prefix
        _sample("sample pi05 best of 8", candidates=8),
        # the backbone writes a subtask before the expert acts: 52 tokens, one at a time
        _sample("sample pi05 response", response=52),
        # the larger policy: 448-pixel cameras, five steps
        _sample("sample pi06", model="pi06", prompt=256, steps=5),
        # a training step of the test-sized policy, as in continuous integration and debugging
        _train("train tiny", model="tiny", batch=4, cams=1, prompt=16, fast=8),
        # fine-tuning the action expert (and the action-token head) behind a frozen backbone
        _train("train pi05 expert", batch=16, expert_only=True),
        # full fine-tuning with knowledge insulation and co-trained action tokens
        _train("train pi05 full", batch=8),
        # an attention layer of a long multi-frame context: bidirectional prefix, causal text behind it
        _attention("attention bf16 long", batch=1, seq=4096, heads=8, kv_heads=1, dim=256, tail=1024),
        # the exact fp32 path: evaluation against a float32 checkpoint, odd length
        _attention("attention fp32", batch=2, seq=601, heads=8, kv_heads=1, dim=256, tail=100, dtype="fp32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sample", "sample", "sample", "train", "train", "attention"])
    if kind == "sample":
        what = rng.choice(["tiny", "one", "batch", "candidates", "response", "pi06"])
        cams = rng.randint(1, 3)
        if what == "tiny":
            case = _sample("", model="tiny", batch=_log(rng, 1, 16), cams=cams, prompt=_log(rng, 8, 64),
                           steps=rng.randint(5, 10))
        elif what == "response":
            case = _sample("", cams=cams, prompt=_log(rng, 16, 200), response=rng.randint(8, 52), steps=rng.randint(5, 10))
        else:
            case = _sample("", model="pi06" if what == "pi06" else "pi05", cams=cams, prompt=_log(rng, 16, 256),
                           batch=rng.randint(2, 6) if what == "batch" else 1,
                           candidates=rng.randint(3, 12) if what == "candidates" else 1,
                           steps=rng.randint(4, 6) if what == "pi06" else rng.randint(5, 10),
                           delay=rng.choice([0, 0, rng.randint(1, 12)]), ragged=rng.random() < 0.5)
    elif kind == "train":
        what = rng.choice(["tiny", "expert", "full"])
        cams, dropout = rng.randint(1, 3), rng.choice([0.1, 0.1, 0.0])
        if what == "tiny":
            case = _train("", model="tiny", batch=_log(rng, 1, 32), cams=cams, prompt=_log(rng, 8, 64),
                          fast=_log(rng, 4, 32), dropout=dropout)
        else:
            case = _train("", batch=_log(rng, 1, 16 if what == "expert" else 8), cams=cams, prompt=_log(rng, 32, 200),
                          fast=_log(rng, 16, 256), expert_only=what == "expert", dropout=dropout)
    else:
        heads, kv_heads, dim = rng.choice([(8, 1, 256), (8, 4, 256), (16, 16, 72), (32, 8, 128)])
        dtype = rng.choice(["bf16", "bf16", "fp32"])
        seq = _log(rng, 200, 4096) if dtype == "bf16" else _log(rng, 100, 700)
        case = _attention("", rng.randint(1, 2), seq, heads, kv_heads, dim, int(seq * rng.random() * 0.5), dtype)
    del case["name"]
    return case


# ------------------------------------------------------------------------------------------------ policies
def _policy(case, seed, *, train):
    tiny, pi06 = case["model"] == "tiny", case["model"] == "pi06"
    side = 448 if pi06 else 224
    feats = {f"camera{i}": PolicyFeature(FeatureType.VISUAL, (3, side, side)) for i in range(case["cams"])}
    feats["state"] = PolicyFeature(FeatureType.STATE, (32,))
    kw = dict(chunk_size=CHUNK, n_action_steps=CHUNK, prompt_max_length=case["prompt"], device="cuda",
              input_features=feats, output_features={"actions": PolicyFeature(FeatureType.ACTION, (ACTION_DIM,))})
    if tiny:
        kw.update(TINY, discrete_action_vocab_size=256)
    if train:
        kw.update(dropout=case["dropout"], discrete_action_max_length=case["fast"],
                  train_expert_only=case["expert_only"])
    else:
        kw.update(dropout=0.0, num_steps=case["steps"])
        if case["response"]:
            kw.update(predict_response=True, response_max_length=case["response"])
    torch.manual_seed(seed)
    before = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        with torch.device("cuda"):
            policy = (PI06Policy(PI06Config(**kw), per_dataset_stats=[identity_stats()]) if pi06 else
                      PI05Policy(PI05Config(**kw), per_dataset_stats=[identity_stats()]))
    finally:
        torch.set_default_dtype(before)
    policy.to(device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        for m in policy.modules():
            if isinstance(m, AdaRMSNorm):             # zero at the start of pretraining; open in a trained checkpoint
                m.dense.weight.normal_(std=0.02)
                m.dense.bias.normal_(std=0.3)
            elif isinstance(m, DecoderLayer):
                depth = (2 * m.cfg.num_hidden_layers) ** -0.5
                m.self_attn.o_proj.weight.mul_(depth)
                m.mlp.down_proj.weight.mul_(depth)
    return policy.train(train)


def _batch(case, seed, fast=8):
    side = 448 if case["model"] == "pi06" else 224
    vocab = GEOMETRY[case["model"]][3]
    spec = SyntheticSpec(batch_size=case["batch"], num_cams=case["cams"], resolution=(side, side),
                         prompt_len=case["prompt"], vocab_size=vocab, state_dim=32, action_dim=ACTION_DIM,
                         chunk_size=CHUNK, discrete_action_len=fast,
                         discrete_action_vocab=256 if case["model"] == "tiny" else 2048, image_dtype=torch.bfloat16)
    return make_synthetic_batch(spec, device="cuda", seed=seed)


def _prepare_sample(case, seed):
    policy = _policy(case, seed, train=False)
    batch = _batch(case, seed + 1)
    B, n = case["batch"], case["candidates"]
    if case["ragged"]:
        lengths = torch.tensor([max(4, case["prompt"] * (8 - i % 5) // 8) for i in range(B)], device="cuda")
        batch["lang_masks"] = torch.arange(case["prompt"], device="cuda")[None, :] < lengths[:, None]
        if case["cams"] > 1:
            batch["img_is_pad"][0, -1] = True
    policy.enable_cuda_graphs(True)
    if n > 1:
        configure_candidates(policy, n, MEDOID, device=torch.device("cuda"))
    gen = torch.Generator(device="cuda").manual_seed(seed + 2)
    kw = dict(noise=torch.randn(B * n, CHUNK, ACTION_DIM, device="cuda", generator=gen))
    if case["delay"]:
        kw.update(delay=case["delay"],
                  action_prefix=torch.randn(B, case["delay"], ACTION_DIM, device="cuda", generator=gen))
    if n > 1:
        kw["n_candidates"] = n
    return dict(kind="sample", policy=policy, batch=batch, kw=kw)


def _prepare_train(case, seed):
    policy = _policy(case, seed, train=True)
    engine = TrainEngine(policy, OptimHyper(), device="cuda")
    return dict(kind="train", engine=engine, batch=_batch(case, seed + 1, case["fast"]), seed=seed)


def _prepare_attention(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = torch.float32 if case["dtype"] == "fp32" else torch.bfloat16
    B, S, H, K, D = case["batch"], case["seq"], case["heads"], case["kv_heads"], case["dim"]

    def t(*shape):
        return torch.randn(*shape, device="cuda", generator=gen).to(dt)

    att = torch.zeros(B, S, dtype=torch.bool, device="cuda")
    att[:, S - case["tail"]:] = True                                   # every token of the tail opens a block
    valid = torch.ones(B, S, dtype=torch.bool, device="cuda")
    valid[-1, S - max(1, S // 16):] = False                            # the last sample is padded
    blk, valid = ops.make_block_ids(valid, att)
    q, k, v = (x.requires_grad_() for x in (t(B, S, H, D), t(B, S, K, D), t(B, S, K, D)))
    return dict(kind="attention", q=q, k=k, v=v, do=t(B, S, H * D), blk=blk, valid=valid, scale=D ** -0.5)


def prepare(case, seed):
    gc.collect()            # a policy and its graph refer to each other: the last one's memory comes back first
    return {"sample": _prepare_sample, "train": _prepare_train, "attention": _prepare_attention}[case["kind"]](case, seed)


def run(state):
    if state["kind"] == "sample":
        return state["policy"].sample_actions(state["batch"], **state["kw"])
    if state["kind"] == "train":
        torch.manual_seed(state["seed"])                               # noise, times and dropout of this step
        engine = state["engine"]
        out = engine.train_step(state["batch"])
        opt = engine.state_dict()
        return {"loss": out["loss"], "mse": out["MSE"], "ce": out["CE"], "grad_norm": out["grad_norm"],
                "params": [g.data for g in engine.store.groups],
                "moments": [opt[f"group{i}.{k}"] for i in range(len(engine.store.groups)) for k in ("m", "v")]}
    q, k, v = state["q"], state["k"], state["v"]
    o = ops.block_attention(q, k, v, state["blk"], state["blk"], state["valid"], state["valid"], state["scale"])
    return (o.detach(), *torch.autograd.grad(o, (q, k, v), state["do"]))


# ------------------------------------------------------------------------------------------------ work
def _layer_params(g):
    width, layers, heads, kv, dim, mlp = g
    return layers * (width * (heads + 2 * kv) * dim + heads * dim * width + 3 * width * mlp)


def _tower_flops(g, rows):
    return 2.0 * rows * _layer_params(g)


def _attn_flops(g, q_rows, keys):
    return 4.0 * g[1] * q_rows * keys * g[2] * g[4]


def _vision(v, images):
    """(parameters, flops) of the vision tower over ``images`` cameras."""
    width, layers, mlp, patches, _ = v
    params = layers * (4 * width * width + 2 * width * mlp)
    return params, 2.0 * images * patches * params + 4.0 * layers * images * patches * patches * width


def work(case):
    if case["kind"] == "attention":
        B, S, H, K, D = case["batch"], case["seq"], case["heads"], case["kv_heads"], case["dim"]
        size = 4 if case["dtype"] == "fp32" else 2
        T = case["tail"]
        P = S - T
        pairs = B * (P * P + T * P + T * (T + 1) / 2)                  # query / key pairs that see each other
        return {"flops": 14.0 * pairs * H * D, "bytes": float(size * B * S * D * (4 * H + 4 * K))}
    vlm, exp, vis, vocab = GEOMETRY[case["model"]]
    B, n_img = case["batch"], case["cams"] * vis[4]
    vis_params, vis_flops = _vision(vis, B * case["cams"])
    ada = (2 * exp[1] + 1) * exp[0] * 3 * exp[0]
    vlm_p, exp_p = _layer_params(vlm), _layer_params(exp) + ada
    if case["kind"] == "sample":
        S = n_img + case["prompt"]
        rows, steps, room = B * case["candidates"], case["steps"], S + case["response"] + CHUNK
        flops = vis_flops + _tower_flops(vlm, B * S) + _attn_flops(vlm, B * S, S)
        flops += steps * (_tower_flops(exp, rows * CHUNK) + _attn_flops(exp, rows * CHUNK, room) + 2.0 * rows * ada)
        size = 2.0 * (vis_params + vlm_p + steps * exp_p)
        if case["response"]:
            flops += case["response"] * B * 2.0 * (vlm_p + vocab * vlm[0])
            size += 2.0 * case["response"] * (vlm_p + vocab * vlm[0])
        return {"flops": flops, "bytes": size}
    S = n_img + case["prompt"] + 3 + case["fast"]
    # a frozen backbone still passes gradients down to the action-token embedding, which trains: no weight gradients
    flops = vis_flops + (2.0 if case["expert_only"] else 3.0) * _tower_flops(vlm, B * S) + 3.5 * _attn_flops(vlm, B * S, S)
    flops += 3.0 * _tower_flops(exp, B * CHUNK) + 3.5 * _attn_flops(exp, B * CHUNK, S + CHUNK)
    trained = exp_p + (0 if case["expert_only"] else vlm_p + vocab * vlm[0])
    # weights once forward and once backward, gradients written and read, fp32 master and two moments read and written
    size = 2.0 * (vis_params + 2 * vlm_p + 2 * exp_p) + trained * (2 + 2 + 24 + 2)
    return {"flops": flops, "bytes": size}


def tolerance(case):
    if case["kind"] == "attention":
        return {"rel": 1e-5, "max": 1e-3} if case["dtype"] == "fp32" else {"rel": 1e-2, "max": 0.2}
    # bf16 activations through the whole network; the second moment doubles a gradient's relative error
    return {"rel": 1e-2} if case["kind"] == "sample" else {"rel": 2e-2, "max": 0.99}

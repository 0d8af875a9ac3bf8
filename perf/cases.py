"""What the speed of this framework is measured on.

The cases are what its users have it do at the WALL-OSS size (``wallx_b200.config.wall_oss_config``: 36 decoder layers of
width 2048 with two experts per feed-forward, 32 vision blocks of width 1280), bf16 throughout:

* ``chunk``     one action chunk from the serving engine (``FlowEngine``): vision tower, prefix pass, ten Euler evaluations;
* ``predict``   the same through ``model(mode="predict")``, for callers whose observation layout changes from call to call;
* ``generate``  greedy text decoding (question answering, FAST action ids), prefill and one token at a time;
* ``score``     a forward pass that returns the logits of every position (validation);
* ``train``     forward, backward and optimizer step of one micro-batch through ``TrainEngine``, flow or FAST loss. A quarter
                of the blocks (9 decoder layers, 8 vision blocks, one of them with full attention), so that a state with its
                fp32 optimizer copies leaves room for others; every block of the full model does the same work;
* ``ffn``       the token-routed expert feed-forward of one layer, forward and backward (the kernel sweep's path).

Weights and observations are random: uniform pixels and prompt ids, N(0, 1) proprioception and noise, actions in [-1, 1].
"""
from __future__ import annotations

import math

import torch

from wallx_b200.config import wall_oss_config
from wallx_b200.data.collator import add_pack_info, to_device
from wallx_b200.data.synthetic import images_to_patches, make_batch, make_processor, smart_resize
from wallx_b200.models import Qwen2_5_VLMoEForAction
from wallx_b200.models.inference import FlowEngine
from wallx_b200.models.layers import RMSNorm
from wallx_b200.models.llm import SparseMoeBlock
from wallx_b200.ops import functional as F_
from wallx_b200.parallel.engine import TrainEngine

DEV = "cuda"
ACTION_VOCAB = 2048
FAST_TOKENS = 48
EULER = 10
LR = 9e-5


def listed():
    def obs(kind, name, batch, views, height, width, prompt, ragged=0, **kw):
        return dict(name=name, kind=kind, batch=batch, views=views, height=height, width=width, prompt=prompt, ragged=ragged, **kw)

    return [
        # one robot at its control rate: latency is what counts
        obs("chunk", "chunk_b1", 1, 3, 256, 256, 64, horizon=32),
        # a few robots sharing a GPU, two cameras that are not square, prompts of different lengths, an odd horizon
        obs("chunk", "chunk_b5_odd", 5, 2, 240, 320, 77, ragged=30, horizon=31),
        # a fleet, or simulated evaluation: throughput
        obs("chunk", "chunk_b32", 32, 3, 256, 256, 64, horizon=32),
        # an evaluation script: every call brings another layout, nothing can be captured ahead
        obs("predict", "predict_b1", 1, 2, 224, 280, 41, horizon=32),
        # a question about one picture, answered token by token
        obs("generate", "generate_b1", 1, 1, 448, 448, 100, new=32),
        # several prompts of different lengths decoded together, as many ids as a FAST action chunk has
        obs("generate", "generate_b6_ragged", 6, 2, 256, 256, 90, ragged=40, new=FAST_TOKENS),
        # validation of FAST targets with the logits of all positions
        obs("score", "score_b3", 3, 3, 256, 256, 64, ragged=17),
        # the smallest fine-tuning micro-batch: launches and host time count
        obs("train", "train_flow_b2", 2, 3, 256, 256, 64, horizon=32, loss="flow"),
        # the example configuration's batch per GPU, prompts of different lengths
        obs("train", "train_flow_b8_ragged", 8, 3, 256, 256, 80, ragged=37, horizon=32, loss="flow"),
        # the benchmark's micro-batch
        obs("train", "train_flow_b32", 32, 3, 256, 256, 64, horizon=32, loss="flow"),
        # FAST fine-tuning: language-model head and cross entropy over the action ids
        obs("train", "train_fast_b8", 8, 3, 256, 256, 64, horizon=32, loss="fast"),
        # the kernel sweep's smallest size, a quarter of the tokens are action tokens
        dict(name="ffn_2k", kind="ffn", tokens=2048, action=0.25),
    ]


def draw(rng):
    """A case of the ranges above: 1 to 32 samples, 1 to 3 cameras of 112 to 448 pixels a side, prompts of 16 to 160 tokens,
    horizons of 8 to 64 actions, 4 to 48 generated ids, feed-forwards of 256 to 32768 tokens."""
    def log(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    most = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(["chunk", "chunk", "predict", "generate", "score", "train", "train", "ffn"])
        if kind == "ffn":
            c = dict(kind=kind, tokens=log(256, 32768), action=round(rng.uniform(0.02, 0.6), 3))
        else:
            prompt = rng.randint(16, 160)
            c = dict(kind=kind, batch=log(1, {"generate": 8, "score": 8}.get(kind, 32)), views=rng.randint(1, 3),
                     height=rng.randint(112, 448), width=rng.randint(112, 448), prompt=prompt,
                     ragged=rng.choice([0, rng.randint(0, prompt - 8)]))
            if kind == "generate":
                c["new"] = log(4, 48)
            elif kind != "score":
                c["horizon"] = log(8, 64)
            if kind == "train":
                c["loss"] = rng.choice(["flow", "flow", "fast"])
        if work(c)["flops"] <= most * {"train": 0.5, "predict": 0.5}.get(kind, 1.0):
            return c


# ------------------------------------------------------------------------------------------------ sizes of a case
def _prompts(case):
    """Prompt length of every sample: from ``prompt`` down to ``prompt - ragged``."""
    b = case["batch"]
    return [case["prompt"] - (case["ragged"] * i) // max(1, b - 1) for i in range(b)]


def _grid(case):
    h, w = smart_resize(case["height"], case["width"])
    return h // 14, w // 14


def _tail(case):
    """Tokens after the proprioception token."""
    if case["kind"] == "generate":
        return 2
    return FAST_TOKENS + 3 if case["kind"] == "score" or case.get("loss") == "fast" else case["horizon"]


def _blocks(case):
    """(decoder layers, vision blocks)."""
    return (9, 8) if case["kind"] == "train" else (36, 32)


H, QKV, VLM, ACT, V_H, V_I = 2048, 2560, 11008, 2048, 1280, 3420
VOCAB = 151936 + 2 + ACTION_VOCAB
ATTN_W = H * QKV + H * H            # parameters of a decoder layer's attention
VIT_W = 4 * V_H * V_H + 3 * V_H * V_I
VIT_ENDS = 1176 * V_H + (4 * V_H) ** 2 + 4 * V_H * H
HEAD_W = 4 * 20 * H + 3 * H * H + H * 20


def work(case):
    if case["kind"] == "ffn":
        t, a = case["tokens"], int(round(case["tokens"] * case["action"]))
        w = 3 * H * (VLM + ACT)
        # forward reads x and the weights and writes y; backward reads x, dy and the weights and writes dx and dW
        return {"bytes": 2.0 * (3 * w + 6 * t * H), "flops": 3 * 2.0 * 3 * H * ((t - a) * VLM + a * ACT)}
    layers, vblocks = _blocks(case)
    gh, gw = _grid(case)
    n_img = case["batch"] * case["views"]
    patches = n_img * gh * gw
    full = [i for i in (7, 15, 23, 31) if i < vblocks]
    # a window holds at most 8 x 8 patches
    vit = 2.0 * patches * (VIT_W * vblocks + VIT_ENDS / 4 + 1176 * V_H * 0.75)
    vit += 4.0 * V_H * (len(full) * n_img * (gh * gw) ** 2 + (vblocks - len(full)) * patches * min(64, gh * gw))
    pre = [p + case["views"] * (gh * gw // 4 + 2) + 1 for p in _prompts(case)]
    tail = _tail(case)
    n_pre = sum(pre)
    vlm = ATTN_W + 3 * H * VLM
    act = ATTN_W + 3 * H * ACT
    w_vit = VIT_W * vblocks + VIT_ENDS
    pairs = sum(p * p / 2 for p in pre)
    pixels = 2.0 * patches * 1176
    kind = case["kind"]
    if kind in ("chunk", "predict"):
        rows = case["batch"] * case["horizon"]
        step = 2.0 * rows * act * layers + 4.0 * H * layers * case["horizon"] * sum(p + case["horizon"] for p in pre) + 2.0 * rows * HEAD_W
        flops = vit + 2.0 * n_pre * vlm * layers + 4.0 * H * layers * pairs + EULER * step
        kv = 2.0 * layers * 2 * 256 * n_pre
        # an evaluation needs the one before it, and the action weights are larger than any on-chip memory: read each time
        byts = 2.0 * (w_vit + layers * vlm + EULER * layers * act) + pixels + kv * (1 + EULER) + 4.0 * rows * 20
    elif kind == "generate":
        b, new = case["batch"], case["new"]
        n_pre += tail * b
        flops = vit + 2.0 * n_pre * vlm * layers + 4.0 * H * layers * pairs
        flops += (new - 1) * 2.0 * b * vlm * layers + new * 2.0 * b * VOCAB * H + new * 4.0 * H * layers * n_pre
        byts = 2.0 * (w_vit + layers * vlm * new + VOCAB * H * new) + pixels + 2.0 * layers * 2 * 256 * n_pre * new
    else:
        fast = kind == "score" or case.get("loss") == "fast"
        n_all = n_pre + tail * case["batch"]
        flops = vit + 4.0 * H * layers * sum((p + tail) ** 2 / 2 for p in pre)
        flops += 2.0 * layers * (n_all * vlm if fast else n_pre * vlm + tail * case["batch"] * act)
        params = w_vit + layers * (ATTN_W + 3 * H * (VLM + (0 if fast else ACT))) + VOCAB * H * (2 if fast else 1)
        if kind == "score":
            flops += 2.0 * n_all * VOCAB * H + 2.0 * case["batch"] * (FAST_TOKENS + 1) * VOCAB * H
            byts = 2.0 * params + pixels + 2.0 * n_all * VOCAB
        else:
            flops += 2.0 * case["batch"] * ((FAST_TOKENS + 1) * VOCAB * H if fast else tail * HEAD_W)
            flops *= 3
            # weights and fp32 master, moments read; the same written
            byts = params * (2.0 + 2.0 + 12.0 + 12.0) + pixels
    return {"bytes": byts, "flops": flops}


def tolerance(case):
    """bf16 activations and weights, fp32 sums. Measured against the same model in fp32 on the CPU (2-norm, then the largest
    difference over the rms): action chunks 0.006 to 0.011 and 0.03; first moments after a flow step 0.007 to 0.011 and after
    a FAST step 0.02, where the differences of single entries reach the rms; updated weights 0.002."""
    kind = case["kind"]
    if kind == "generate":
        return {"differ": 0.01}
    if kind in ("chunk", "predict"):
        return {"rel": 0.03, "max": 0.12}
    return {"rel": 0.015 if kind == "ffn" else 0.03}


# ------------------------------------------------------------------------------------------------ states
def _config(case):
    layers, vblocks = _blocks(case)
    cfg = wall_oss_config(action_expert_intermediate=ACT, action_vocab=ACTION_VOCAB, num_hidden_layers=layers)
    cfg.vision_config.depth = vblocks
    cfg.vision_config.fullatt_block_indexes = [i for i in cfg.vision_config.fullatt_block_indexes if i < vblocks]
    return cfg


def _model(cfg, proc, fast):
    old = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        with torch.device(DEV):
            return Qwen2_5_VLMoEForAction(cfg, processor=proc, use_fast_tokenizer=fast)
    finally:
        torch.set_default_dtype(old)


def _batch(case, cfg, proc, seed, pack):
    """Left-padded batch of ``case`` on the GPU, as the collator and the image processor leave it."""
    mode = "fast" if case["kind"] in ("generate", "score") or case.get("loss") == "fast" else "flow"
    gen = torch.Generator().manual_seed(seed)
    rows, width = [], None
    for prompt in _prompts(case):
        rows.append(make_batch(cfg, proc, 1, views=case["views"], image_hw=(case["height"], case["width"]), prompt_len=prompt,
                               horizon=case.get("horizon", 32), mode=mode, fast_tokens=FAST_TOKENS, generator=gen, raw_images=True,
                               pad_to=width))
        width = rows[0]["input_ids"].shape[1]
    b = {k: torch.cat([r[k] for r in rows]) if torch.is_tensor(rows[0][k]) else sum((r[k] for r in rows), []) for k in rows[0]}
    if case["kind"] == "generate":  # the prompt ends where the assistant's turn begins
        cut = width - FAST_TOKENS - 1
        b.pop("labels")
        for k in ("input_ids", "attention_mask", "moe_token_types"):
            b[k] = b[k][:, :cut].contiguous()
    if pack:
        b = add_pack_info(b, cfg)
    vc = cfg.vision_config
    b = to_device(b, DEV, torch.bfloat16)
    b["pixel_values"], _ = images_to_patches(b.pop("images_uint8"), vc.patch_size, vc.temporal_patch_size, vc.spatial_merge_size,
                                             torch.bfloat16)
    b.pop("frame_index")
    return b


def _randn(shape, seed):
    return torch.randn(shape, device=DEV, generator=torch.Generator(DEV).manual_seed(seed)).to(torch.bfloat16)


class _Training(dict):
    """A training state. The engine's parameter hooks refer back to it from C++, where no collector sees the cycle: it is
    closed with the state, as a program does that trains several models in turn."""

    def __del__(self):
        self["engine"].close()


def prepare(case, seed):
    kind = case["kind"]
    torch.manual_seed(seed)
    if kind == "ffn":
        t, a = case["tokens"], int(round(case["tokens"] * case["action"]))
        cfg = wall_oss_config(action_expert_intermediate=ACT)
        with torch.device(DEV):
            norm, block = RMSNorm(H, eps=cfg.rms_norm_eps).to(torch.bfloat16), SparseMoeBlock(cfg, 2).to(torch.bfloat16)
        params = list(norm.parameters()) + list(block.parameters())
        for p in params[1:]:
            torch.nn.init.normal_(p, std=cfg.initializer_range)
        types = torch.zeros(t, dtype=torch.int32, device=DEV)
        types[torch.randperm(t, device=DEV)[:a]] = 1
        return {"kind": kind, "norm": norm, "block": block, "params": params, "types": types,
                "x": _randn((t, H), seed).requires_grad_(True), "dy": _randn((t, H), seed + 1) * 0.1}
    cfg = _config(case)
    proc = make_processor(cfg, ACTION_VOCAB)
    model = _model(cfg, proc, kind == "score" or case.get("loss") == "fast")
    s = {"kind": kind, "model": model}
    if kind == "train":
        model.train()
        s = _Training(s, engine=TrainEngine(model, lr=LR, weight_decay=0.1, max_grad_norm=1.0))
        s["batch"] = _batch(case, cfg, proc, seed, pack=True)
        if case["loss"] == "flow":  # what the noise schedule would draw, from the seed
            chunk = s["batch"]["action_chunk"]
            s["batch"]["flow_noise"] = _randn(chunk.shape, seed)
            s["batch"]["flow_time"] = torch.rand(chunk.shape[0], device=DEV).pow(1 / 1.5).to(torch.bfloat16)
        return s
    model.eval()
    b = _batch(case, cfg, proc, seed, pack=kind == "score")
    if kind == "generate":
        # A trained model is sure of most of its tokens, random weights of none. Embeddings of unit size and a head that
        # looks for the next id give the greedy choice a margin of several standard deviations of the other logits.
        model.model.embed_tokens.weight.data.normal_()
        model.lm_head.weight.data.copy_(model.model.embed_tokens.weight.data.roll(1, 0))
        s["new"] = case["new"]
        b.pop("moe_token_types")
    elif kind != "score":
        b.pop("action_chunk")
        s["noise"] = _randn((case["batch"], case["horizon"], 20), seed)
        if kind == "chunk":
            s["engine"] = FlowEngine(model, b, num_inference_timesteps=EULER)
    s["batch"] = b
    return s


def run(s):
    kind = s["kind"]
    if kind == "chunk":
        return s["engine"](s["batch"], noise=s["noise"])["predict_action"]
    if kind == "predict":
        return s["model"](mode="predict", predict_mode="diffusion", noise=s["noise"], num_inference_timesteps=EULER,
                          **s["batch"])["predict_action"]
    if kind == "generate":
        return s["model"].generate(max_new_tokens=s["new"], **s["batch"])
    if kind == "score":
        out = s["model"](mode="validate", **s["batch"])
        return {"logits": out.logits, "loss": out.loss}
    if kind == "train":
        e = s["engine"]
        out = s["model"](mode="train", **s["batch"])
        e.backward(out.loss)
        norm_sq = e.optimizer_step(LR)
        # after a first step the first moment is the clipped gradient times (1 - beta1)
        return {"loss": out.loss.detach(), "norm_sq": norm_sq.clone(), "params": [b.param for b in e.buffers],
                "moments": [b.exp_avg for b in e.buffers]}
    x, params = s["x"], s["params"]
    x.grad = None
    for p in params:
        p.grad = None
    plan = F_.make_route_plan(s["types"], 2)
    y = s["block"](s["norm"](x, dest=plan.dest, out_rows=plan.rows), x, plan)
    y.backward(s["dy"])
    return {"y": y.detach(), "dx": x.grad, "dw": [p.grad for p in params]}

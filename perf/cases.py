"""Performance cases: the work that training a Qwen2.5-VL model on one GPU consists of.

Every case goes through the package's public classes, the way ``trainers/`` composes them: ``VisionEncoder`` and
``TextDecoder`` with ``ZeroAdamW`` over their parameters, and ``Qwen2_5_VLModel`` for evaluation.

kind            one pass
``encode``      vision encoder without gradients (evaluation, computing embeddings): images -> merged tokens
``vision``      vision half of a training step: forward and backward from the gradient the text half returns
``text``        text half of a training step: embedding, splice of the vision rows, decoder, loss, backward
``evaluate``    whole model without gradients: images and ids -> logits of every token
``train``       one optimisation step of the whole model: both halves forward and backward, and the updates
``optimizer``   global gradient norm, clipping and AdamW over one flat buffer

A case is a dict of plain values.  ``images`` lists the pixel extents (height x width, multiples of 28) of the images
of a batch, ``texts`` the text tokens of its samples; in ``text`` cases the k-th image belongs to the k-th sample.
``layers`` and ``depth`` keep that many of the decoder's and of the encoder's layers, each of the full width and in
the models' proportion of window and full attention: three sets of weights, gradients and optimizer state then fit
on one GPU, and the bf16 rounding of a random-init model, which grows with its depth, stays within the tolerance.
"""
from __future__ import annotations

import dataclasses
import math
from types import SimpleNamespace

import torch
import torch.utils.checkpoint

from multimodal_training_b200.config.model_configs import get_model_config
from multimodal_training_b200.data.synthetic import Sample
from multimodal_training_b200.models.text import TextDecoder, mrope_cos_sin
from multimodal_training_b200.models.vision import VisionEncoder, prepare_plan
from multimodal_training_b200.models.vlm import Qwen2_5_VLModel
from multimodal_training_b200.ops.attention import SeqInfo
from multimodal_training_b200.parallel.handoff import pack_text_batch, splice_rows
from multimodal_training_b200.parallel.sp import build_vision_plan
from multimodal_training_b200.parallel.zero import ZeroAdamW

DEV = "cuda"
BF16 = torch.bfloat16


def listed() -> list[dict]:
    return [
        # the encoder of the 7B model on one small image: every kernel is short, latency and launches count
        dict(name="encode_7b_224", kind="encode", model="qwen2_5_vl_7b", images="224x224"),
        # the benchmark's image, one per GPU and step: the vision half of the headline training step
        dict(name="vision_7b_896", kind="vision", model="qwen2_5_vl_7b", images="896x896", recompute=False),
        # a batch of a real data set: photos of different extents, windows cut at the edges, activations recomputed
        # (the default of the sample configuration)
        dict(name="vision_7b_photos", kind="vision", model="qwen2_5_vl_7b",
             images="616x812+476x644+1036x392+252x364+700x924", recompute=True),
        # the 32B configuration's image (its encoder: 32 layers, MLP 3456, merger to 5120)
        dict(name="vision_32b_1792", kind="vision", model="qwen2_5_vl_32b", images="1792x1792", recompute=False),
        # the long-sequence sweep: 36864 patches in one image, four layers attend over all of them
        dict(name="vision_7b_2688", kind="vision", model="qwen2_5_vl_7b", images="2688x2688", recompute=True),
        # the headline step's text half: 1024 text tokens around 1024 vision tokens
        dict(name="text_7b_2048", kind="text", model="qwen2_5_vl_7b", layers=4, images="896x896", texts="1024",
             recompute=False),
        # packed samples of odd lengths, two of them without an image
        dict(name="text_7b_packed", kind="text", model="qwen2_5_vl_7b", layers=4, images="616x812+476x644+252x364",
             texts="391+87+1203+2044+33", recompute=True),
        # one sample of the 32B configuration: 2048 text tokens and an 1792x1792 image
        dict(name="text_32b_6144", kind="text", model="qwen2_5_vl_32b", layers=2, images="1792x1792", texts="2048",
             recompute=False),
        # evaluating a prompt with the 3B model
        dict(name="evaluate_3b", kind="evaluate", model="qwen2_5_vl_3b", layers=12, images="448x448", texts="187"),
        # the small model of the smoke runs and tests, full precision of the optimizer: many short kernels
        dict(name="train_smoke", kind="train", model="smoke", images="448x448+448x448", texts="256+256",
             recompute=True, master=True, lr=1e-3),
        # the 3B model (tied embedding) on the benchmark's sample, forward to update
        dict(name="train_3b_896", kind="train", model="qwen2_5_vl_3b", depth=8, layers=4, images="896x896",
             texts="1024", recompute=False, master=True, lr=1e-5),
        # clipping and AdamW over the parameters of the 7B vision encoder (32 layers, 676 million elements)
        dict(name="optimizer_676m", kind="optimizer", numel=676550656, master=True),
    ]


def _log_uniform(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_image(rng, lo_patches: float, hi_patches: float) -> str:
    patches = _log_uniform(rng, lo_patches, hi_patches)
    aspect = _log_uniform(rng, 0.5, 2.0)
    h = max(2, round(math.sqrt(patches * aspect) / 2))
    w = max(2, round(math.sqrt(patches / aspect) / 2))
    return f"{28 * h}x{28 * w}"


def draw(rng) -> dict:
    kind = rng.choice(["encode", "vision", "vision", "text", "text", "evaluate", "train", "optimizer"])
    big = ["qwen2_5_vl_3b", "qwen2_5_vl_7b", "qwen2_5_vl_32b"]
    if kind == "encode":
        return dict(kind=kind, model=rng.choice(big), images=_draw_image(rng, 200, 9000))
    if kind == "vision":
        images = [_draw_image(rng, 200, 5000) for _ in range(rng.randint(1, 5))] if rng.random() < 0.7 \
            else [_draw_image(rng, 5000, 28000)]
        return dict(kind=kind, model=rng.choice(big), images="+".join(images), recompute=rng.random() < 0.5)
    if kind == "text":
        n = rng.randint(1, 5)
        return dict(kind=kind, model=rng.choice(big), layers=2,
                    images="+".join(_draw_image(rng, 200, 3000) for _ in range(rng.randint(1, n))),
                    texts="+".join(str(int(_log_uniform(rng, 30, 1500))) for _ in range(n)),
                    recompute=rng.random() < 0.5)
    if kind == "evaluate":
        return dict(kind=kind, model="qwen2_5_vl_3b", layers=12, images=_draw_image(rng, 200, 5000),
                    texts=str(int(_log_uniform(rng, 16, 1200))))
    if kind == "train":
        n = rng.randint(1, 4)
        return dict(kind=kind, model="smoke", images="+".join(_draw_image(rng, 100, 4000) for _ in range(n)),
                    texts="+".join(str(int(_log_uniform(rng, 30, 1000))) for _ in range(n)),
                    recompute=rng.random() < 0.5, master=rng.random() < 0.5, lr=1e-3)
    return dict(kind=kind, numel=128 * int(_log_uniform(rng, 2e4, 6e6)), master=rng.random() < 0.5)


# --------------------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------------------
def _grids(case, cfg) -> list[tuple[int, int, int]]:
    p = cfg.vision.patch_size
    return [(1, int(h) // p, int(w) // p) for h, w in (s.split("x") for s in case["images"].split("+"))]


def _config(case):
    cfg = get_model_config(case["model"])
    if "layers" in case:
        cfg = dataclasses.replace(cfg, text=dataclasses.replace(cfg.text, num_hidden_layers=case["layers"]))
    if "depth" in case:
        full = [i for i in cfg.vision.fullatt_block_indexes if i < case["depth"]]
        cfg = dataclasses.replace(cfg, vision=dataclasses.replace(cfg.vision, depth=case["depth"],
                                                                  fullatt_block_indexes=full))
    return cfg


def _trained(model, gen):
    """Biases and norm weights of a model that has been trained for a while (they are initialised to 0 and 1)."""
    with torch.no_grad():
        for n, p in model.named_parameters():
            if p.dim() == 1:
                p.add_(torch.randn(p.shape, generator=gen, device=DEV).to(p.dtype), alpha=0.02)
    return model


def _vision_plan(grids, cfg):
    v = cfg.vision
    plan = build_vision_plan(grids, sp=1, rank=0, spatial_merge_size=v.spatial_merge_size, window_size=v.window_size,
                             patch_size=v.patch_size, head_dim=v.head_dim)
    return prepare_plan(plan, torch.device(DEV))


def _samples(case, cfg, grids, seed) -> list[Sample]:
    """Samples with uniform-random ids, the image's placeholders in the middle, labels ignored at those places."""
    g = torch.Generator().manual_seed(seed)
    top = min(cfg.vision_start_token_id, cfg.vision_end_token_id, cfg.image_token_id, cfg.text.vocab_size)
    out = []
    for i, n in enumerate(int(t) for t in case["texts"].split("+")):
        mine = grids[i:i + 1]
        merged = sum(t * h * w for t, h, w in mine) // cfg.vision.merge_unit
        ids = torch.randint(1, top, (n,), generator=g)
        ids = torch.cat([ids[:n // 2], torch.full((merged,), cfg.image_token_id, dtype=torch.long), ids[n // 2:]])
        labels = ids.clone()
        labels[n // 2:n // 2 + merged] = -100
        out.append(Sample(ids, labels, None, mine, i))
    return out


def _pixels(grids, cfg, gen):
    n = sum(t * h * w for t, h, w in grids)
    return torch.randn(n, cfg.vision.patch_dim, generator=gen, device=DEV).to(BF16)


def _prepare_vision(s, case, cfg, grids, gen, seed, grad: bool):
    s.plan = _vision_plan(grids, cfg)
    s.pixels = _pixels(grids, cfg, gen).index_select(0, s.plan.local_patch_index.to(DEV))
    s.vision = _trained(VisionEncoder(cfg.vision, dtype=BF16, device=DEV, seed=seed,
                                      activation_checkpointing=bool(case.get("recompute", False))), gen)
    if grad:
        s.vision_opt = ZeroAdamW(s.vision.named_parameters(), lr=case.get("lr", 1e-5), weight_decay=0.01,
                                 master_weights=bool(case.get("master", False)))


def _prepare_text(s, case, cfg, grids, gen, seed):
    t = cfg.text
    tb = pack_text_batch(_samples(case, cfg, grids, seed), image_token_id=cfg.image_token_id,
                         vision_start_token_id=cfg.vision_start_token_id,
                         spatial_merge_size=cfg.vision.spatial_merge_size, pad_token_id=cfg.pad_token_id)
    s.ids, s.labels = tb.input_ids.to(DEV), tb.shifted_labels.to(DEV)
    s.seq = SeqInfo.from_list(tb.cu_seqlens, DEV)
    s.cos, s.sin = mrope_cos_sin(tb.position_ids, t.head_dim, t.rope_theta, t.mrope_section, device=DEV)
    rows = torch.cat([torch.from_numpy(r) for r in tb.image_rows])
    s.rows = rows.to(DEV)
    s.text = _trained(TextDecoder(t, dtype=BF16, device=DEV, seed=seed + 1,
                                  activation_checkpointing=bool(case["recompute"])), gen)
    s.text_opt = ZeroAdamW(s.text.named_parameters(), lr=case.get("lr", 1e-5), weight_decay=0.01,
                           master_weights=bool(case.get("master", False)))


def prepare(case: dict, seed: int):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    kind = case["kind"]
    s = SimpleNamespace(kind=kind)
    if kind == "optimizer":
        n = case["numel"]
        p = torch.nn.Parameter((torch.randn(n, generator=gen, device=DEV) * 0.02).to(BF16))
        s.opt = ZeroAdamW([("w", p)], lr=1e-4, weight_decay=0.01, master_weights=case["master"])
        for lo in range(0, n, 1 << 26):          # in pieces: the fp32 noise of the whole buffer is not needed at once
            hi = min(n, lo + (1 << 26))
            noise = torch.randn(hi - lo, generator=gen, device=DEV)
            s.opt.flat_grad[lo:hi].copy_(noise * 1e-3)
            s.opt.exp_avg[lo:hi].copy_(noise.roll(1) * 3e-4)
            s.opt.exp_avg_sq[lo:hi].copy_(noise.roll(2).square() * 1e-6 + 1e-8)
        s.opt.step_count = 100
        p.grad_written = True
        return s
    cfg = _config(case)
    grids = _grids(case, cfg)
    if kind == "evaluate":
        s.model = _trained(Qwen2_5_VLModel(cfg, dtype=BF16, device=DEV, seed=seed), gen)
        s.ids = _samples(case, cfg, grids, seed)[0].input_ids.unsqueeze(0).to(DEV)
        s.pixels, s.grids = _pixels(grids, cfg, gen), grids
        return s
    if kind in ("encode", "vision", "train"):
        _prepare_vision(s, case, cfg, grids, gen, seed, grad=kind != "encode")
    if kind in ("text", "train"):
        _prepare_text(s, case, cfg, grids, gen, seed)
    if kind == "vision":     # the gradient of a mean loss over a few thousand tokens
        s.grad = (torch.randn(s.pixels.shape[0] // cfg.vision.merge_unit, cfg.vision.out_hidden_size, generator=gen,
                              device=DEV) * 1e-4).to(BF16)
    if kind == "text":       # what the merger of a random-init encoder emits
        s.merged = torch.randn(s.rows.numel(), cfg.text.hidden_size, generator=gen, device=DEV).to(BF16)
    return s


# --------------------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------------------
def _text_step(s, merged):
    x = s.text.embed(s.ids)
    leaf = merged.detach().requires_grad_(True)
    x = splice_rows(x, leaf, s.rows)
    loss = s.text.loss(s.text(x, s.cos, s.sin, s.seq), s.labels)
    loss.backward()
    return loss.detach(), leaf.grad


def run(s):
    if s.kind == "encode":
        with torch.no_grad():
            return {"merged": s.vision(s.pixels, s.plan)}
    if s.kind == "evaluate":
        with torch.no_grad():
            return {"logits": s.model(s.ids, s.pixels, s.grids)}
    if s.kind == "vision":
        s.vision_opt.zero_grad()
        merged = s.vision(s.pixels, s.plan)
        merged.backward(s.grad)
        return {"merged": merged.detach(), "grad": s.vision_opt.flat_grad}
    if s.kind == "text":
        s.text_opt.zero_grad()
        loss, grad = _text_step(s, s.merged)
        return {"loss": loss, "vision_grad": grad, "grad": s.text_opt.flat_grad}
    if s.kind == "train":
        s.vision_opt.zero_grad()
        s.text_opt.zero_grad()
        merged = s.vision(s.pixels, s.plan)
        loss, grad = _text_step(s, merged)
        merged.backward(grad)
        s.text_opt.step()
        s.vision_opt.step()
        return {"loss": loss, "vision_grad": s.vision_opt.flat_grad, "text_grad": s.text_opt.flat_grad,
                "vision": s.vision_opt.flat_param, "text": s.text_opt.flat_param}
    o = s.opt
    shard = o.reduce_gradients()
    own, replicated = o.grad_norm_sq_local(shard)
    norm = (own + replicated).sqrt()
    o.step(grad_scale=torch.clamp(1.0 / (norm + 1e-6), max=1.0), shard=shard)
    out = {"norm": norm, "param": o.flat_param, "exp_avg": o.exp_avg, "exp_avg_sq": o.exp_avg_sq}
    if o.master is not None:
        out["master"] = o.master
    return out


# --------------------------------------------------------------------------------------
# The same pass in 64 bits: plain PyTorch on the weights, tables and inputs that prepare() makes
# --------------------------------------------------------------------------------------
F64 = torch.float64


def _checkpointed(fn, *args):
    return torch.utils.checkpoint.checkpoint(fn, *args, use_reentrant=False) if torch.is_grad_enabled() else fn(*args)


def _norm64(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rotate64(x, cos, sin):
    """x [T, heads, dim]"""
    a, b = x.chunk(2, dim=-1)
    return x * cos[:, None] + torch.cat((-b, a), -1) * sin[:, None]


def _softmax64(q, k, v, causal):
    s = q @ k.transpose(-1, -2) / math.sqrt(q.shape[-1])
    if causal:
        s = s.masked_fill(torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).triu(1), -math.inf)
    return s.softmax(-1) @ v


def _attention64(q, k, v, cu, causal):
    """q [T, heads, dim], k and v [T, kv heads, dim]; sequences of one length together, long ones head by head."""
    rep, heads = q.shape[1] // k.shape[1], q.shape[1]
    out = torch.zeros_like(q)
    lengths: dict[int, list[int]] = {}
    for a, b in zip(cu[:-1], cu[1:]):
        if b > a:
            lengths.setdefault(b - a, []).append(a)
    for n, starts in lengths.items():
        rows = torch.tensor(starts, device=q.device)[:, None] + torch.arange(n, device=q.device)
        if n > 1024:
            for r in rows:
                out = out.index_copy(0, r, torch.stack([
                    _checkpointed(_softmax64, q[r, h], k[r, h // rep], v[r, h // rep], causal)
                    for h in range(heads)], 1))
            continue
        flat = rows.flatten()
        qs, ks, vs = (t[flat].view(len(starts), n, t.shape[1], -1).transpose(1, 2) for t in (q, k, v))
        ks, vs = (t.repeat_interleave(rep, 1) for t in (ks, vs))
        out = out.index_copy(0, flat, _softmax64(qs, ks, vs, causal).transpose(1, 2).reshape(flat.numel(), heads, -1))
    return out


def _block64(x, w, cos, sin, cu, causal, heads, kv, eps):
    T, d = x.shape[0], cos.shape[1]
    bias = lambda y, b: y if b is None else y + b  # noqa: E731
    qkv = bias(_norm64(x, w["n1"], eps) @ w["qkv"].T, w["qkv_b"]).view(T, -1, d)
    rot = _rotate64(qkv[:, :heads + kv], cos, sin)
    a = _attention64(rot[:, :heads], rot[:, heads:], qkv[:, heads + kv:], cu, causal)
    x = x + bias(a.reshape(T, -1) @ w["o"].T, w["o_b"])
    g, u = bias(_norm64(x, w["n2"], eps) @ w["gu"].T, w["gu_b"]).chunk(2, dim=-1)
    return x + bias((torch.nn.functional.silu(g) * u) @ w["down"].T, w["down_b"])


def _weights64(model, grad: bool) -> dict:
    return {n: p.detach().to(F64).requires_grad_(grad) for n, p in model.named_parameters()}


def _vision64(W, v, pixels, plan):
    cos, sin = plan.cos_dev.to(F64), plan.sin_dev.to(F64)
    x = pixels.to(F64) @ W["patch_embed_w"].T
    for i in range(v.depth):
        w = {a: W.get(f"blocks.{i}.{b}") for a, b in (
            ("n1", "norm1_w"), ("qkv", "qkv_w"), ("qkv_b", "qkv_b"), ("o", "proj_w"), ("o_b", "proj_b"), ("n2", "norm2_w"),
            ("gu", "gate_up_w"), ("gu_b", "gate_up_b"), ("down", "down_w"), ("down_b", "down_b"))}
        cu = plan.full_cu if i in v.fullatt_block_indexes else plan.win_cu
        x = _checkpointed(lambda t, w=w, cu=cu: _block64(t, w, cos, sin, cu, False, v.num_heads, v.num_heads,
                                                         v.rms_norm_eps), x)
    x = _norm64(x, W["ln_q_w"], v.rms_norm_eps).reshape(-1, v.hidden_size * v.merge_unit)
    x = torch.nn.functional.gelu(x @ W["merger_fc1_w"].T + W["merger_fc1_b"])
    return x @ W["merger_fc2_w"].T + W["merger_fc2_b"]


def _text64(W, t, x, cos, sin, cu):
    for i in range(t.num_hidden_layers):
        w = {a: W.get(f"layers.{i}.{b}") for a, b in (
            ("n1", "ln1_w"), ("qkv", "qkv_w"), ("qkv_b", "qkv_b"), ("o", "o_w"), ("o_b", ""), ("n2", "ln2_w"),
            ("gu", "gate_up_w"), ("gu_b", ""), ("down", "down_w"), ("down_b", ""))}
        x = _checkpointed(lambda y, w=w: _block64(y, w, cos, sin, cu, True, t.num_attention_heads,
                                                  t.num_key_value_heads, t.rms_norm_eps), x)
    return _norm64(x, W["norm_w"], t.rms_norm_eps), W.get("lm_head", W["embed_tokens"])


def _text_loss64(W, t, s, merged):
    x = W["embed_tokens"][s.ids].index_copy(0, s.rows, merged)
    h, head = _text64(W, t, x, s.cos.to(F64), s.sin.to(F64), s.seq.host)
    rows = (s.labels >= 0).nonzero().flatten()
    return _checkpointed(lambda a, b: torch.nn.functional.cross_entropy(a @ b.T, s.labels[rows]), h[rows], head)


def _flat64(opt, pieces: dict):
    """The tensors of `pieces` (by parameter name) where the optimizer's flat buffers hold them, zeros between."""
    out = torch.zeros(opt.total, dtype=F64, device=DEV)
    for n, o in zip(opt.names, opt.offsets):
        out[o:o + pieces[n].numel()] = pieces[n].detach().flatten()
    return out


def _adamw64(opt, p, g, m, v, step):
    """Weights and moments after one update in 64 bits; the decayed parameters lie in front."""
    b1, b2 = opt.betas
    m, v = b1 * m + (1 - b1) * g, b2 * v + (1 - b2) * g * g
    update = (m / (1 - b1 ** step)) / ((v / (1 - b2 ** step)).sqrt() + opt.eps)
    update[:opt.n_decay] += opt.weight_decay * p[:opt.n_decay]
    return p - opt.lr * update, m, v


def exact(case: dict, seed: int):
    if case["kind"] == "optimizer":
        s = prepare(case, seed)
        o = s.opt
        norm = torch.sqrt(sum(c.to(F64).square().sum() for c in o.flat_grad.split(1 << 26)))
        g = o.flat_grad.to(F64) * torch.clamp(1.0 / (norm + 1e-6), max=1.0)
        p, m, v = _adamw64(o, (o.flat_param if o.master is None else o.master).to(F64), g, o.exp_avg.to(F64),
                           o.exp_avg_sq.to(F64), o.step_count + 1)
        out = {"norm": norm.reshape(1), "param": p, "exp_avg": m, "exp_avg_sq": v}
        return out if o.master is None else {**out, "master": p}
    if work(case)["flops"] > 1.5e14:       # over 20 seconds in 64 bits
        return None
    s, cfg = prepare(case, seed), _config(case)
    v, t = cfg.vision, cfg.text
    if s.kind in ("encode", "evaluate"):
        with torch.no_grad():
            if s.kind == "encode":
                return {"merged": _vision64(_weights64(s.vision, False), v, s.pixels, s.plan)}
            plan = _vision_plan(s.grids, cfg)
            merged = _vision64(_weights64(s.model.visual, False), v,
                               s.pixels.index_select(0, plan.local_patch_index.to(DEV)), plan)
            merged = torch.empty_like(merged).index_copy(0, plan.local_merged_ids.to(DEV), merged)
            W, ids = _weights64(s.model.language_model, False), s.ids[0]
            x = W["embed_tokens"][ids].index_copy(0, (ids == cfg.image_token_id).nonzero().flatten(), merged)
            pos, _ = s.model.get_rope_index(s.ids, s.grids)
            cos, sin = mrope_cos_sin(pos[:, 0], t.head_dim, t.rope_theta, t.mrope_section)
            h, head = _text64(W, t, x, cos.to(DEV, F64), sin.to(DEV, F64), [0, ids.numel()])
            return {"logits": h @ head.T}
    out = {}
    if s.kind in ("vision", "train"):
        Wv = _weights64(s.vision, True)
        merged = _vision64(Wv, v, s.pixels, s.plan)
    if s.kind in ("text", "train"):
        Wt = _weights64(s.text, True)
        leaf = (s.merged.to(F64) if s.kind == "text" else merged.detach()).requires_grad_(True)
        loss = _text_loss64(Wt, t, s, leaf)
        loss.backward()
        text_grad = _flat64(s.text_opt, {n: w.grad for n, w in Wt.items()})
    if s.kind == "text":
        return {"loss": loss.detach(), "vision_grad": leaf.grad, "grad": text_grad}
    merged.backward(s.grad.to(F64) if s.kind == "vision" else leaf.grad)
    vision_grad = _flat64(s.vision_opt, {n: w.grad for n, w in Wv.items()})
    if s.kind == "vision":
        return {"merged": merged.detach(), "grad": vision_grad}
    out = {"loss": loss.detach(), "vision_grad": vision_grad, "text_grad": text_grad}
    for name, opt, grad in (("vision", s.vision_opt, vision_grad), ("text", s.text_opt, text_grad)):
        p = opt.flat_param.to(F64)
        out[name] = _adamw64(opt, p, grad, torch.zeros_like(p), torch.zeros_like(p), 1)[0]
    return out


# --------------------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------------------
def _vision_counts(grids, v) -> tuple[int, int, float]:
    """(parameters, patches, forward flops)"""
    C, I, M = v.hidden_size, v.intermediate_size, v.hidden_size * v.merge_unit
    layer = 4 * C * C + 3 * C * I
    merger = M * M + M * v.out_hidden_size
    T = sum(t * h * w for t, h, w in grids)
    edge = v.window_size // v.patch_size
    pairs_full = sum(t * (h * w) ** 2 for t, h, w in grids)
    pairs_win = sum(t * sum(min(edge, h - i) ** 2 for i in range(0, h, edge))
                    * sum(min(edge, w - j) ** 2 for j in range(0, w, edge)) for t, h, w in grids)
    full = len(v.fullatt_block_indexes)
    attention = 4.0 * C * (full * pairs_full + (v.depth - full) * pairs_win)
    params = v.depth * (layer + 6 * C + 2 * I) + merger + C * v.patch_dim + C + M + v.out_hidden_size
    matmul = 2.0 * T * (v.depth * layer + C * v.patch_dim) + 2.0 * T / v.merge_unit * merger
    return params, T, matmul + attention, attention


def _text_counts(lens, t, logit_rows) -> tuple[int, int, float]:
    H, I, d = t.hidden_size, t.intermediate_size, t.head_dim
    q, kv = t.num_attention_heads * d, t.num_key_value_heads * d
    layer = H * (q + 2 * kv) + q * H + 3 * H * I
    T, L = sum(lens), t.num_hidden_layers
    attention = L * sum(4.0 * q * n * (n + 1) / 2 for n in lens)
    params = L * (layer + q + 2 * kv + 2 * H) + t.vocab_size * H * (1 if t.tie_word_embeddings else 2) + H
    return params, T, 2.0 * T * L * layer + 2.0 * logit_rows * H * t.vocab_size + attention, attention


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "optimizer":
        # gradient, weight and state read, weight and state written; the norm has to see every gradient first
        n = case["numel"]
        return {"bytes": n * (30 if case["master"] else 16), "flops": 16.0 * n}
    cfg = _config(case)
    grids = _grids(case, cfg)
    v = cfg.vision
    bytes_ = flops = 0.0
    if kind in ("encode", "vision", "evaluate", "train"):
        params, T, forward, attention = _vision_counts(grids, v)
        once = 2.0 * T * v.patch_dim + 2.0 * T / v.merge_unit * v.out_hidden_size
        if kind in ("encode", "evaluate"):
            bytes_, flops = bytes_ + 2.0 * params + once, flops + forward
        else:      # the pixels need no gradient; attention's backward has five products to the forward's two
            flops += 3.0 * forward - 0.5 * attention - 2.0 * T * v.hidden_size * v.patch_dim
            bytes_ += 4.0 * params + once
    if kind in ("text", "evaluate", "train"):
        t = cfg.text
        merged = [a * b * c // v.merge_unit for a, b, c in grids]
        texts = [int(x) for x in case["texts"].split("+")]
        lens = [n + (merged[i] if i < len(merged) else 0) for i, n in enumerate(texts)]
        # rows whose next token is an image placeholder (and a sample's last one) have no label
        rows = sum(lens) if kind == "evaluate" else sum(texts) - len(texts)
        params, T, forward, attention = _text_counts(lens, t, rows)
        if kind == "evaluate":
            bytes_, flops = bytes_ + 2.0 * params + 2.0 * T * t.vocab_size, flops + forward
        else:
            flops += 3.0 * forward - 0.5 * attention
            bytes_ += 4.0 * params + 4.0 * T * t.hidden_size
    if kind == "train":
        both = _vision_counts(grids, v)[0] + params
        bytes_ += both * (28 if case["master"] else 14)
    return {"bytes": bytes_, "flops": flops}


def tolerance(case: dict) -> dict:
    if case["kind"] == "optimizer":
        # fp32 arithmetic; the bf16 weights (and bf16 moments) differ by one unit in the last place, 2^-7 of the value,
        # where a sum falls on the other side of a rounding boundary
        return {"rel": 1e-4, "max": 0.01}
    # Against the same network in 64 bits (plain PyTorch, same weights): merged tokens 0.021, logits 0.04, gradients
    # 0.023 to 0.035 for the large models and 0.008 for the small one; single values of the gradients, where a row's
    # terms cancel, are off by more than the gradient's root mean square.
    return {"rel": 0.03, "max": 0.9}

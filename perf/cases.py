"""Performance cases: what users of the framework run, from the smallest calls to the largest.

Kinds (all through the public entry points):
  train      one optimizer step of ``Trainer.train_step`` (forward, backward, gradient clip, AdamW) on Wan2.1 or
             HunyuanVideo models, micro-batches of latents, text states and noise that are already on the GPU;
  denoise    one sampling step of the Wan pipeline: the DiT on the prompt and on the negative prompt, classifier-free
             guidance, one Euler step;
  hunyuan    ``HunyuanVideoPipeline`` for two sampling steps (embedded guidance: one DiT call per step);
  encode     ``WanVideoVAE.encode`` of a clip (what encoder ranks do for every training sample);
  decode     ``WanVideoVAE.decode`` of latents, in the pipeline's 30 x 52 tiles or whole;
  text       ``encode_prompt`` with the full-size umT5 encoder.

Sizes are the repository's own: Wan2.1-1.3B / 14B and HunyuanVideo-13B widths, 256P / 480P / 720P clips of 1 to 81
frames, 512 umT5 text states, 257 CLIP tokens.  ``layers`` is the depth that is run: the layers of these models are
all alike, so the large cases run a few of them (the optimizer's share shrinks with them), the small ones all thirty,
because there the number of calls is what counts.
"""
from __future__ import annotations

import itertools
import math

import torch

from teletron_b200.infer.hunyuan_pipeline import HunyuanVideoPipeline
from teletron_b200.models import FlowMatchScheduler, HunyuanVideoModel, WanModel, hunyuan_config, wan_config
from teletron_b200.models.encoders.umt5 import UMT5Encoder, encode_prompt
from teletron_b200.models.encoders.wan_vae import WanVideoVAE
from teletron_b200.train import Trainer, make_forward_step, make_hunyuan_forward_step, parse_args

DEVICE = "cuda"
BF16 = torch.bfloat16
TEXT_TOKENS, TEXT_DIM, CLIP_TOKENS, CLIP_DIM = 512, 4096, 257, 1280
HUNYUAN_TEXT_TOKENS, HUNYUAN_POOLED = 256, 768
GUIDANCE = 5.0

T2V_1B, I2V_14B, HUNYUAN = "wan2.1-1.3b-t2v", "wan2.1-14b-i2v", "hunyuanvideo-13b-t2v"


def listed():
    return [
        # the smallest sampling call: a 256P still (256 tokens); 30 layers of short kernels, so launches and latency count
        dict(name="denoise_1b_256p_1f", kind="denoise", model=T2V_1B, layers=30, frames=1, height=256, width=256),
        # a sampling step of the framework's headline clip, 480P x 81 frames (32,760 tokens)
        dict(name="denoise_1b_480p_81f", kind="denoise", model=T2V_1B, layers=30, frames=81, height=480, width=832),
        # image-to-video sampling on the 14B width, a short clip with an odd grid (5 x 29 x 53 = 7,685 tokens)
        dict(name="denoise_14b_i2v_17f", kind="denoise", model=I2V_14B, layers=8, frames=17, height=464, width=848),
        # HunyuanVideo sampling with padded text (9 x 34 x 45 = 13,770 + 256 tokens)
        dict(name="hunyuan_544p_33f", kind="hunyuan", model=HUNYUAN, layers=2, singles=4, frames=33, height=544, width=720),
        # low-resolution pre-training: two 256P x 17-frame clips in a micro-batch, two micro-batches per step
        dict(name="train_1b_256p_17f", kind="train", model=T2V_1B, layers=30, frames=17, height=256, width=256, batch=2,
             micro_batches=2, recompute=False),
        # the headline training clip
        dict(name="train_1b_480p_81f", kind="train", model=T2V_1B, layers=8, frames=81, height=480, width=832, batch=1,
             micro_batches=1, recompute=False),
        # 14B image-to-video training with full activation recompute
        dict(name="train_14b_i2v_480p_81f", kind="train", model=I2V_14B, layers=2, frames=81, height=480, width=832,
             batch=1, micro_batches=1, recompute=True),
        # HunyuanVideo training, ragged token count and padded text (9 x 25 x 45 = 10,125 + 256 tokens)
        dict(name="train_hunyuan_400p_33f", kind="train", model=HUNYUAN, layers=2, singles=4, frames=33, height=400,
             width=720, batch=1, micro_batches=1, recompute=False),
        # encoding one training clip, long enough to go through the VAE in temporal chunks
        dict(name="encode_480p_49f", kind="encode", frames=49, height=480, width=832),
        # encoding one still image for image training
        dict(name="encode_256p_1f", kind="encode", frames=1, height=256, width=256),
        # decoding a short sampled clip the way the pipeline does, in overlapping tiles (the decoder runs in fp32)
        dict(name="decode_480p_9f_tiled", kind="decode", frames=9, height=480, width=832, tiled=True),
        # text states of one prompt and its negative prompt
        dict(name="text_2x512", kind="text", batch=2, tokens=512),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: another size of one of the kinds, never more work than the largest listed case of its kind and
    model."""
    while True:
        like = dict(rng.choice(listed()))
        like.pop("name")
        if like["kind"] == "text":
            like["batch"], like["tokens"] = rng.choice([1, 2, 3, 4]), 8 * _log_int(rng, 8, 64)
        else:
            like["frames"] = 4 * rng.choice([0, 1, 2, 3, 4, 6, 8, 12, 16, 20]) + 1
            side = 16 * _log_int(rng, 12, 45)
            like["height"] = side
            like["width"] = 16 * max(12, int(round(side / 16 * rng.uniform(0.75, 1.8))))
            if like["kind"] == "decode":
                like["tiled"] = rng.choice([True, False])
            if like["kind"] == "train":
                like["batch"] = rng.choice([1, 1, 2, 3])
                like["micro_batches"] = rng.choice([1, 2])
                if like["model"] == T2V_1B:
                    like["recompute"] = rng.choice([True, False])
                    like["layers"] = 30 if _tokens(like) * like["batch"] <= 4096 else 8
            if like["kind"] == "denoise" and like["model"] == T2V_1B:
                like["layers"] = 30
        cap = max(_cost(c) for c in listed() if c["kind"] == like["kind"] and c.get("model") == like.get("model"))
        plain = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
        if _cost(like) <= cap and like not in plain:
            return like


# ------------------------------------------------------------------------------------------------ sizes and work
def _grid(case):
    return (case["frames"] - 1) // 4 + 1, case["height"] // 8, case["width"] // 8


def _tokens(case):
    f, h, w = _grid(case)
    return f * (h // 2) * (w // 2)


def _wan_forward(case):
    """(flops, parameters) of one forward pass of one sample."""
    cfg = wan_config(case["model"], num_layers=case["layers"])
    n, c = _tokens(case), cfg.dim
    i2v = cfg.has_image_input
    ctx = TEXT_TOKENS + (CLIP_TOKENS if i2v else 0)
    per_token = 6 * c * c + 2 * c * cfg.ffn_dim                       # qkv, o, cross q, cross o, ffn
    per_ctx = 2 * c * c
    layer = 2 * n * per_token + 2 * ctx * per_ctx + 4 * n * n * c + 4 * n * ctx * c
    embed = 2 * n * c * (4 * cfg.in_dim + 4 * cfg.out_dim) + 2 * TEXT_TOKENS * (TEXT_DIM * c + c * c)
    embed += 2 * CLIP_TOKENS * (CLIP_DIM * CLIP_DIM + CLIP_DIM * c) if i2v else 0
    params = case["layers"] * (8 * c * c + 2 * c * cfg.ffn_dim + (2 * c * c if i2v else 0)) + 8 * c * c + TEXT_DIM * c
    return case["layers"] * layer + embed, params


def _hunyuan_forward(case):
    cfg = hunyuan_config(case["model"])
    n, t, c = _tokens(case), HUNYUAN_TEXT_TOKENS, cfg.hidden_size
    m = int(c * cfg.mlp_ratio)
    s = n + t
    mats = 4 * c * c + 2 * c * m
    attn = 4 * s * s * c
    blocks = case["layers"] + case["singles"]
    refiner = cfg.num_refiner_layers * mats
    flops = blocks * (2 * s * mats + attn) + 2 * t * (refiner + TEXT_DIM * c) + 2 * n * c * 128
    params = case["layers"] * (2 * mats + 12 * c * c) + case["singles"] * (mats + 3 * c * c) + refiner + 2 * 2 * c * c
    params += TEXT_DIM * c + 4 * c * c
    return flops, params


def _vae_flops(frames, h, w, decoder):
    """Multiply-adds x 2 of the convolutions (dims 96 / 192 / 384 / 384, two or three residual blocks per stage) at
    pixel size h x w."""
    dims, total = [96, 192, 384, 384], 0

    def conv(vox, a, b, taps=27):
        return 2 * vox * a * b * taps

    f = [frames, frames, (frames - 1) // 2 + 1, (frames - 1) // 4 + 1]     # frames at each resolution
    vox = [f[i] * (h >> i) * (w >> i) for i in range(4)]
    if not decoder:
        total += conv(vox[0], 3, 96)
        for i, d in enumerate(dims):
            a = dims[max(i - 1, 0)]
            total += conv(vox[i], a, d) + 3 * conv(vox[i], d, d) + (conv(vox[i], a, d, 1) if a != d else 0)
            if i < 3:
                total += conv(vox[i] // 4, d, d, 9) + (conv(vox[i + 1], d, d, 3) if i else 0)
        total += 4 * conv(vox[3], 384, 384) + conv(vox[3], 384, 32)
    else:
        total += conv(vox[3], 16, 384) + 4 * conv(vox[3], 384, 384) + conv(vox[0], 96, 3)
        ins = [96, 192, 192, 384]
        for i in (3, 2, 1, 0):
            d = dims[i]
            total += conv(vox[i], ins[i], d) + 5 * conv(vox[i], d, d) + (conv(vox[i], ins[i], d, 1) if ins[i] != d else 0)
            if i:
                total += (conv(vox[i], d, 2 * d, 3) if i > 1 else 0) + conv(f[i - 1] * (h >> (i - 1)) * (w >> (i - 1)), d, d // 2, 9)
    n = (h >> 3) * (w >> 3)
    return total + f[3] * (4 * n * n * 384 + 2 * n * 384 * 384 * 4)


def _tiles(case):
    """Latent tiles that the blended decode visits."""
    _, h, w = _grid(case)

    def starts(n, tile, stride):
        s = list(range(0, max(n - tile, 0) + 1, stride)) or [0]
        return s + [n - tile] if s[-1] + tile < n else s

    return len(starts(h, 30, 15)) * len(starts(w, 52, 26)), min(h, 30), min(w, 52)


def work(case):
    kind = case["kind"]
    if kind == "text":
        n, d, ff, layers = case["batch"] * case["tokens"], 4096, 10240, 24
        mats = layers * (4 * d * d + 3 * d * ff)
        return dict(flops=2.0 * n * mats + layers * 4.0 * case["batch"] * case["tokens"] ** 2 * d,
                    bytes=2.0 * (mats + 2 * n * d))
    if kind in ("encode", "decode"):
        f, h, w = _grid(case)
        flops = _vae_flops(case["frames"], 8 * h, 8 * w, kind == "decode")
        if case.get("tiled"):
            n, th, tw = _tiles(case)
            flops = n * _vae_flops(case["frames"], 8 * th, 8 * tw, True)
        return dict(flops=float(flops), bytes=2.0 * (3 * case["frames"] * 64 * h * w + 16 * f * h * w + 60e6))
    f, h, w = _grid(case)
    latent = 16 * f * h * w
    if kind == "denoise":
        flops, params = _wan_forward(case)
        return dict(flops=2.0 * flops, bytes=2.0 * (params + 2 * latent + 2 * TEXT_TOKENS * TEXT_DIM))
    if kind == "hunyuan":
        flops, params = _hunyuan_forward(case)
        return dict(flops=2.0 * flops, bytes=2.0 * (2 * params + 4 * latent))
    flops, params = (_hunyuan_forward if case["model"] == HUNYUAN else _wan_forward)(case)
    samples = case["batch"] * case["micro_batches"]
    # backward is twice the forward; recompute adds one forward; AdamW reads and writes master / m / v, reads the fp32
    # gradient and writes the bf16 weight
    return dict(flops=samples * flops * (4.0 if case["recompute"] else 3.0),
                bytes=params * (2.0 * 2 + 2 * 4 + 6 * 4 + 2) + 4.0 * samples * latent)


def _cost(case):
    w = work(case)
    return max(w["flops"] / 1e15, w["bytes"] / 6e12)


def tolerance(case):
    """Largest differences between two correct implementations.  Seen against the same computation in fp32: denoise
    0.015 (max 0.06) after 30 layers, train 0.009 for the gradients, encode 0.006 (max 0.036), text 0.022 (max 0.13),
    decode (TF32 convolutions) 0.0013 (max 0.008).  Single gradient elements whose sum over the tokens cancels are off
    by a whole root mean square: ``max`` says nothing more about them."""
    if case["kind"] == "decode":
        return dict(rel=0.005, max=0.035)
    return dict(rel=0.03, max=dict(denoise=0.3, hunyuan=0.3, encode=0.15, text=0.6, train=0.99)[case["kind"]])


# ------------------------------------------------------------------------------------------------------- inputs
def _randn(*shape, dtype=BF16):
    return torch.randn(*shape, device=DEVICE, dtype=dtype)


def _text(batch, tokens, dim, lens):
    """Text states, zero past each prompt's length."""
    keep = torch.arange(tokens, device=DEVICE)[None, :, None] < torch.tensor(lens, device=DEVICE)[:, None, None]
    return torch.where(keep, _randn(batch, tokens, dim), 0.0).to(BF16)


def _image_condition(f, h, w, batch):
    mask = torch.zeros(batch, 4, f, h, w, device=DEVICE, dtype=BF16)
    mask[:, :, 0] = 1
    return torch.cat([mask, _randn(batch, 16, f, h, w)], dim=1)


def _lens(n, lo, hi):
    return torch.randint(lo, hi + 1, (n,)).tolist()


def _prepare_train(case, seed):
    hunyuan = case["model"] == HUNYUAN
    argv = ["--model", "ParallelHunyuanVideoModel" if hunyuan else "ParallelWanModel", "--model-preset", case["model"],
            "--num-layers", str(case["layers"]), "--bf16", "--micro-batch-size", str(case["batch"]),
            "--global-batch-size", str(case["batch"] * case["micro_batches"]), "--train-iters", "1000000",
            "--lr", "1e-5", "--weight-decay", "1e-2", "--clip-grad", "1.0", "--num-frames", str(case["frames"]),
            "--video-resolution", str(case["height"]), str(case["width"]), "--synthetic-latents", "--log-interval",
            "1000000", "--seed", str(seed), "--init-on-device"]
    if case["model"] == I2V_14B:
        argv += ["--task-type", "i2v"]
    if case["recompute"]:
        argv += ["--recompute-granularity", "full", "--recompute-method", "block", "--recompute-num-layers", "1000"]
    args = parse_args(argv=argv)
    if hunyuan:
        args.num_single_layers = case["singles"]
    trainer = Trainer(args, build_data=False)
    torch.manual_seed(seed)
    f, h, w = _grid(case)
    b, batches = case["batch"], []
    for _ in range(case["micro_batches"]):
        item = dict(latents=_randn(b, 16, f, h, w), noise=_randn(b, 16, f, h, w))
        if hunyuan:
            lens = _lens(b, HUNYUAN_TEXT_TOKENS // 4, HUNYUAN_TEXT_TOKENS)
            mask = torch.arange(HUNYUAN_TEXT_TOKENS)[None, :] < torch.tensor(lens)[:, None]
            item.update(prompt_embeds=_randn(b, HUNYUAN_TEXT_TOKENS, TEXT_DIM), prompt_mask=mask.long().to(DEVICE),
                        clip_text_embed=_randn(b, HUNYUAN_POOLED))
        else:
            item["context"] = _text(b, TEXT_TOKENS, TEXT_DIM, _lens(b, 20, 300))
            if case["model"] == I2V_14B:
                item.update(clip_feature=_randn(b, CLIP_TOKENS, CLIP_DIM), image_emb_y=_image_condition(f, h, w, b))
        batches.append(item)
    make = make_hunyuan_forward_step if hunyuan else make_forward_step
    step = make(timestep_generator=torch.Generator().manual_seed(seed))
    return dict(trainer=trainer, step=step, data=itertools.cycle(batches))


def _prepare_denoise(case, seed):
    torch.manual_seed(seed)
    with torch.device(DEVICE):
        dit = WanModel(wan_config(case["model"], num_layers=case["layers"])).to(BF16).eval().requires_grad_(False)
    sched = FlowMatchScheduler(shift=5, sigma_min=0.0, extra_one_step=True)
    sched.set_timesteps(50)
    f, h, w = _grid(case)
    state = dict(dit=dit, sched=sched, t=sched.timesteps[int(torch.randint(5, 45, (1,)))], latents=_randn(1, 16, f, h, w),
                 pos=_text(1, TEXT_TOKENS, TEXT_DIM, _lens(1, 20, 300)), neg=_text(1, TEXT_TOKENS, TEXT_DIM, _lens(1, 20, 300)),
                 clip=None, y=None)
    if case["model"] == I2V_14B:
        state.update(clip=_randn(1, CLIP_TOKENS, CLIP_DIM), y=_image_condition(f, h, w, 1))
    return state


def _prepare_hunyuan(case, seed):
    torch.manual_seed(seed)
    cfg = hunyuan_config(case["model"], num_layers=case["layers"], num_single_layers=case["singles"])
    with torch.device(DEVICE):
        dit = HunyuanVideoModel(cfg).to(BF16).eval().requires_grad_(False)
    mask = (torch.arange(HUNYUAN_TEXT_TOKENS) < _lens(1, HUNYUAN_TEXT_TOKENS // 4, HUNYUAN_TEXT_TOKENS)[0]).long()
    return dict(pipe=HunyuanVideoPipeline(dit, device=DEVICE), seed=seed, height=case["height"], width=case["width"],
                frames=case["frames"], text=_randn(1, HUNYUAN_TEXT_TOKENS, TEXT_DIM), mask=mask[None].to(DEVICE),
                pooled=_randn(1, HUNYUAN_POOLED))


def _prepare_vae(case, seed):
    torch.manual_seed(seed)
    with torch.device(DEVICE):
        vae = WanVideoVAE()
        for m in (vae.model.encoder.middle[1], vae.model.decoder.middle[1]):
            torch.nn.init.normal_(m.proj.weight, std=0.02)      # zero when new, never in a checkpoint
        vae = vae.to(BF16 if case["kind"] == "encode" else torch.float32).eval().requires_grad_(False)
    vae.reset_constants(torch.device(DEVICE))
    f, h, w = _grid(case)
    if case["kind"] == "encode":
        return dict(vae=vae, videos=[(torch.rand(3, case["frames"], 8 * h, 8 * w, device=DEVICE) * 2 - 1).to(BF16)])
    return dict(vae=vae, latents=_randn(1, 16, f, h, w, dtype=torch.float32), tiled=case["tiled"])


def _prepare_text(case, seed):
    torch.manual_seed(seed)
    with torch.device("meta"):
        enc = UMT5Encoder().to(BF16)
    enc = enc.to_empty(device=DEVICE).eval().requires_grad_(False)
    for name, p in enc.named_parameters():
        if "norm" in name:
            p.fill_(1.0)
        elif "embedding" in name:
            p.normal_(std=1.0 if name.startswith("token") else 4096 ** -0.5)
        else:                                                    # q so that logits have unit variance, as T5 starts
            p.normal_(std=(p.shape[1] * (64 if ".q." in name else 1)) ** -0.5)
    b, n = case["batch"], case["tokens"]
    mask = torch.zeros(b, n, dtype=torch.long)
    for i, k in enumerate(_lens(b, min(16, n), max(16, n * 3 // 4))):
        mask[i, :k] = 1
    ids = torch.randint(1, 256384, (b, n)) * mask
    return dict(enc=enc, ids=ids.to(DEVICE), mask=mask.to(DEVICE))


def prepare(case, seed):
    make = dict(train=_prepare_train, denoise=_prepare_denoise, hunyuan=_prepare_hunyuan, encode=_prepare_vae,
                decode=_prepare_vae, text=_prepare_text)[case["kind"]]
    return dict(make(case, seed), kind=case["kind"])


# --------------------------------------------------------------------------------------------------------- runs
def _train(s):
    losses, _, norm, _ = s["trainer"].train_step(s["step"], s["data"])
    buf = s["trainer"].buffer
    out = dict(loss=losses["loss"], grad_norm=norm, params=buf.params)
    for r in buf.regions():                                      # matrices; biases, norms and modulation
        out["matrix_grads" if r.wd else "vector_grads"] = buf.grads[r.start:r.end]
    return out


@torch.no_grad()
def _denoise(s):
    ts = s["t"].reshape(1).to(DEVICE, torch.float32)
    v_pos = s["dit"](s["latents"], ts, s["pos"], s["clip"], s["y"])
    v_neg = s["dit"](s["latents"], ts, s["neg"], s["clip"], s["y"])
    v = v_neg + GUIDANCE * (v_pos - v_neg)
    return s["sched"].step(v.float(), s["t"], s["latents"].float()).to(BF16), v_pos, v_neg


def _hunyuan(s):
    return s["pipe"](s["text"], s["mask"], s["pooled"], height=s["height"], width=s["width"], num_frames=s["frames"],
                     num_inference_steps=2, seed=s["seed"])


def _encode(s):
    return s["vae"].encode(s["videos"])


def _decode(s):
    return s["vae"].decode(s["latents"], tiled=s["tiled"], tile_size=(30, 52), tile_stride=(15, 26))


@torch.no_grad()
def _text_states(s):
    return encode_prompt(s["enc"], s["ids"], s["mask"])


def run(state):
    return dict(train=_train, denoise=_denoise, hunyuan=_hunyuan, encode=_encode, decode=_decode,
                text=_text_states)[state["kind"]](state)

"""Workloads whose speed is tracked: calls a user of this package makes, at the sizes they are made at.

A case is a dict of plain values. `listed()` names twelve, `draw(rng)` gives more of the same ranges, `prepare` builds
what a program holds before the call (weights, handles, inputs on the GPU), `run` is one pass through the public entry
points and returns its outputs whole. `work` counts the bytes and operations a pass cannot do without and `tolerance`
says how far another correct implementation of the same precision may be from this one.

Kinds:
  step    one evaluation of the transformer (step.H3Runtime.step): embedding, fused blocks, output projection
  attn    the attention override of RapidH3Int8Attention on [1, H, S, 128] (head-major q, k, v of a host framework)
  linear  one quantized linear as the node pack patches it in (nodes._QuantLinear): row quantizer + W8A8 GEMM + bias
  te      one text-encoder linear (te_quant._TELinear, fp32 in and out, second pass on the outlier rows)
  vae     the causal conv3d decoder, latent to RGB (vae.VAEDecoder.decode)
  ff      the feed-forward block of the fp16 transformer decoder (vae_fast._ff_forward)
"""
import math

import torch

from rapid_h3_b200 import kernels, model, nodes, step, te_quant, vae, vae_fast

DEV = "cuda"


def listed():
    return [
        # the smallest configuration of the tests and the smoke run: every launch is tiny, so latency is what counts
        dict(name="step_tiny", kind="step", d=256, mlp=512, blocks=2, text_dim=256, grid_t=2, grid_h=6, grid_w=9,
             audio=7, batch=1, text=33, mode="int8_rowwise", rotate=False),
        # one picture (a single latent frame) at the full resolution and model width, CFG batch 2
        dict(name="step_still", kind="step", d=4096, mlp=16384, blocks=2, text_dim=4096, grid_t=1, grid_h=24, grid_w=42,
             audio=0, batch=2, text=512, mode="int8_rowwise", rotate=False),
        # a short clip in the production recipe: H256-rotated linears, token-scaled attention
        dict(name="step_clip_rot", kind="step", d=4096, mlp=16384, blocks=1, text_dim=4096, grid_t=6, grid_h=24,
             grid_w=42, audio=148, batch=2, text=512, mode="int8_rot", rotate=True),
        # the draft pass at 0.7 x the spatial size (odd grid, ragged last tiles), one block of it
        dict(name="step_draft", kind="step", d=4096, mlp=16384, blocks=1, text_dim=4096, grid_t=36, grid_h=17, grid_w=29,
             audio=148, batch=2, text=512, mode="int8_rowwise", rotate=False),
        # the full-resolution pass, 768 x 1344 x 141 frames, one of its 48 blocks
        dict(name="step_full", kind="step", d=4096, mlp=16384, blocks=1, text_dim=4096, grid_t=36, grid_h=24, grid_w=42,
             audio=148, batch=2, text=512, mode="int8_rowwise", rotate=False),
        # attention alone as a host framework calls it, production numerics, the sequence of a 3-second clip
        dict(name="attn_tok_22k", kind="attn", heads=32, s=22332, rotate=True),
        # a linear on a handful of rows (conditioning tokens): bound by reading the weight once
        dict(name="linear_few_rows", kind="linear", m=37, n=4096, k=4096, mode="int8_rowwise"),
        # the e4m3 recipe on a ragged number of tokens, qkv-shaped
        dict(name="linear_fp8_qkv", kind="linear", m=5003, n=12288, k=4096, mode="fp8_rowwise"),
        # text-encoder projection of one prompt; one row in seven is an outlier row
        dict(name="te_prompt", kind="te", m=512, n=4096, k=4096, mode="int8_rot"),
        # a preview decode of a few latent frames at a quarter of the resolution
        dict(name="vae_preview", kind="vae", t=3, h=12, w=21),
        # the full decode, latent 16 x 36 x 24 x 42 to 3 x 141 x 768 x 1344
        dict(name="vae_full", kind="vae", t=36, h=24, w=42),
        # feed-forward block of the fp16 transformer decoder, two tiles of 1797 tokens
        dict(name="ff_two_tiles", kind="ff", batch=2, s=1797, k=2048, f=8192),
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], spread over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "attn", "linear", "linear", "te", "vae", "ff"])
    if kind == "step":
        if rng.random() < 0.2:  # the test-sized model
            return dict(kind=kind, d=256 * rng.randint(1, 3), mlp=512 * rng.randint(1, 3), blocks=rng.randint(1, 3),
                        text_dim=256, grid_t=rng.randint(1, 4), grid_h=rng.randint(3, 12), grid_w=rng.randint(3, 17),
                        audio=rng.randint(0, 40), batch=rng.randint(1, 2), text=rng.randint(8, 90),
                        mode=rng.choice(["int8_rowwise", "int8_rot"]), rotate=rng.random() < 0.4)
        t = _log(rng, 1, 36)
        size = rng.uniform(0.6, 1.0)
        rotate = rng.random() < 0.4
        if rotate:
            t = min(t, 18)  # the token-scaled kernel at the full sequence costs more than the largest listed case
        return dict(kind=kind, d=4096, mlp=16384, blocks=1, text_dim=4096, grid_t=t, grid_h=max(1, round(24 * size)),
                    grid_w=max(1, round(42 * size)), audio=rng.choice([0, 4 * t, 148]), batch=rng.randint(1, 2),
                    text=rng.randint(64, 512), mode=rng.choice(["int8_rowwise", "int8_rot"]), rotate=rotate)
    if kind == "attn":
        return dict(kind=kind, heads=rng.choice([8, 16, 24, 32]), s=_log(rng, 1024, 24000), rotate=rng.random() < 0.5)
    if kind == "linear":
        return dict(kind=kind, m=_log(rng, 1, 36436), n=rng.choice([1024, 4096, 5376, 12288]),
                    k=rng.choice([1024, 2048, 4096, 16384]), mode=rng.choice(["int8_rowwise", "int8_rot", "fp8_rowwise"]))
    if kind == "te":
        return dict(kind=kind, m=_log(rng, 16, 2048), n=rng.choice([1024, 4096, 8192]), k=rng.choice([2048, 4096]),
                    mode=rng.choice(["int8_rot", "int8_rot_plain"]))
    if kind == "vae":
        return dict(kind=kind, t=_log(rng, 1, 30), h=rng.randint(6, 24), w=rng.randint(8, 42))
    return dict(kind=kind, batch=rng.randint(1, 4), s=_log(rng, 64, 4000), k=2048, f=rng.choice([6144, 8192]))


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(*shape, device=DEV, generator=g)


def _hadamard256_row(i):
    """Row i of the +-1 matrix H4 x H4 x H4 x H4 (H4 = ones with -1 on the anti-diagonal)."""
    h4 = torch.ones(4, 4, device=DEV)
    h4[torch.arange(4), 3 - torch.arange(4)] = -1.0
    h = h4
    for _ in range(3):
        h = torch.kron(h, h4)
    return h[i]


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    bf16, f16 = torch.bfloat16, torch.float16
    if kind == "step":
        cfg = model.H3Config(d_model=case["d"], heads=case["d"] // 128, mlp_hidden=case["mlp"], n_blocks=case["blocks"],
                             text_dim=case["text_dim"])
        rt = step.H3Runtime.random(cfg, seed=seed, device=DEV, mode=case["mode"])
        t, h, w, b = case["grid_t"], case["grid_h"], case["grid_w"], case["batch"]
        return dict(kind=kind, rt=rt, numerics="reference" if case["rotate"] else "fast",
                    args=(_randn(g, b, cfg.latent_ch, t, h, w).to(bf16), _randn(g, b, case["audio"], cfg.latent_ch).to(bf16),
                          _randn(g, b, 2, cfg.d_model).to(bf16), step.rope_table_for_grid(t, h, w, case["audio"]).to(DEV),
                          _randn(g, b, case["text"], cfg.text_dim).to(bf16)))
    if kind == "attn":
        s, h = case["s"], case["heads"]
        q, v = _randn(g, 1, h, s, 128).to(bf16), _randn(g, 1, h, s, 128).to(bf16)
        k = (_randn(g, 1, h, s, 128) + 2 * _randn(g, 1, h, 1, 128)).to(bf16)  # per-channel offset: what smoothing removes
        _, override = nodes.RapidH3Int8Attention().patch(None, numerics="reference" if case["rotate"] else "fast")
        return dict(kind=kind, fn=override, q=q, k=k, v=v, heads=h)
    if kind == "linear":
        x = _randn(g, case["m"], case["k"])
        x[:, torch.randperm(case["k"], device=DEV, generator=g)[:max(1, case["k"] // 100)]] *= 20.0  # outlier channels
        mod = torch.nn.Linear(case["k"], case["n"], device=DEV, dtype=bf16)
        mod.requires_grad_(False)
        mod.weight.copy_(0.02 * _randn(g, case["n"], case["k"]))
        mod.bias.copy_(0.01 * _randn(g, case["n"]))
        lin = nodes._QuantLinear(mod, "blocks.0.attn.qkv_proj", case["mode"])
        lin.qweight_for()
        return dict(kind=kind, fn=lin, x=x.to(bf16))
    if kind == "te":
        x = _randn(g, case["m"], case["k"])
        x[::7, 256:512] += 6.0 * _hadamard256_row(5)  # rows that the rotation concentrates into one channel
        w = (_randn(g, case["n"], case["k"]) / case["k"] ** 0.5).to(bf16)
        lin = te_quant._TELinear(kernels.quantize_weight(w, "int8_rot"), 0.1 * _randn(g, case["n"]), case["mode"])
        return dict(kind=kind, fn=lin, x=x)
    if kind == "vae":
        dec = vae.VAEDecoder(seed=seed, device=DEV)
        return dict(kind=kind, dec=dec, z=_randn(g, 1, 16, case["t"], case["h"], case["w"]).to(bf16))
    k, f = case["k"], case["f"]

    def rotated(n, kk):  # codes and scales of a rotated weight, as a checkpoint stores them
        ws = (0.8 + 0.4 * torch.rand(n, device=DEV, generator=g)) * 4.0 / (127.0 * math.sqrt(kk))
        wq = (_randn(g, n, kk) * (127.0 / 4.0)).round().clamp(-127, 127).to(torch.int8)
        return vae_fast.Int8Linear(wq, ws, (0.05 * _randn(g, n)).to(f16))

    w1, w2 = rotated(2 * f, k), rotated(k, f)
    shape = (case["batch"], case["s"], k)
    return dict(kind=kind, w1=w1, w2=w2, x=_randn(g, *shape).to(f16), nw=(1 + 0.1 * _randn(g, k)).to(f16),
                resid=_randn(g, *shape).to(f16), rs=(1 + 0.1 * _randn(g, k)).to(f16))


def run(state):
    kind = state["kind"]
    if kind == "step":
        nodes.RapidH3Int8Attention().patch(None, numerics=state["numerics"])
        return state["rt"].step(*state["args"])
    if kind == "attn":
        return state["fn"](None, state["q"], state["k"], state["v"], heads=state["heads"], skip_reshape=True)
    if kind in ("linear", "te"):
        return state["fn"](state["x"])
    if kind == "vae":
        return state["dec"].decode(state["z"])
    return vae_fast._ff_forward(state["w1"], state["w2"], state["x"], state["nw"], 1e-6, state["resid"], state["rs"])


def work(case):
    kind = case["kind"]
    if kind == "step":
        d, f, td, text, b = case["d"], case["mlp"], case["text_dim"], case["text"], case["batch"]
        sites = case["grid_t"] * case["grid_h"] * case["grid_w"]
        s = sites + case["audio"]
        weights = 3 * d * d + d * d + 2 * d * d + 3 * f * d       # int8: qkv, out, cross q and out, fc1, fc2
        block_flops = 2 * s * weights + 2 * text * td * 2 * d + 4 * s * s * d + 4 * s * text * d + 2 * 2 * d * 6 * d
        block_bytes = weights + td * 2 * d + 2 * 6 * d * d        # + kv projection (int8) and the modulation (bf16)
        ends = 2 * 2 * s * 16 * d * b                             # embedding and output projection
        io = b * (2 * 2 * s * 16 + 2 * text * td + 2 * 2 * d) + s * 48 * 4 * 2
        return {"bytes": case["blocks"] * block_bytes + io, "flops": case["blocks"] * b * block_flops + ends}
    if kind == "attn":
        e = case["heads"] * case["s"] * 128
        return {"bytes": 4 * 2 * e, "flops": 4 * e * case["s"]}
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * m * k + n * k + 4 * n + 2 * n + 2 * m * n, "flops": 2 * m * n * k}
    if kind == "te":
        m, n, k = case["m"], case["n"], case["k"]
        rows = m + (-(-m // 7) if case["mode"] == "int8_rot" else 0)
        return {"bytes": 4 * m * k + n * k + 8 * n + 4 * m * n, "flops": 2 * rows * n * k}
    if kind == "vae":
        widths, t, h, w = (512, 256, 128), case["t"], case["h"], case["w"]
        sites = t * h * w
        flops, weights, io = 2 * sites * 16 * widths[0] * 27, 27 * 16 * widths[0], 2 * 16 * sites
        for i, c in enumerate(widths):
            flops += 2 * sites * c * c * 27 * 4
            weights += 27 * c * c * 4
            if i + 1 < len(widths):
                t, h, w = 2 * t - 1, 2 * h, 2 * w
                sites = t * h * w
                flops += 2 * sites * c * widths[i + 1] * 27
                weights += 27 * c * widths[i + 1]
        flops += 2 * sites * widths[-1] * 192 * 27
        weights += 27 * widths[-1] * 192
        return {"bytes": 2 * weights + io + 2 * sites * 192, "flops": flops}
    m, k, f = case["batch"] * case["s"], case["k"], case["f"]
    return {"bytes": 3 * 2 * m * k + 3 * f * k + 4 * (2 * f + k), "flops": 2 * m * 3 * f * k}


# Largest relative 2-norm error per kind, about four times what was measured on a B200:
#   attn    the same call with the keys in another order of whole 128-key tiles: 2.0e-3 (e4m3 P and V) and 0.9e-3
#           (token-scaled); what moves is the fp32 sums and, through the means of K and V, a few codes
#   linear  against the product, scales and bias in 64 bits with one rounding: 2.3e-3 (the bias is added in bf16)
#   te      against both passes in 64 bits: 1.7e-3 (the first pass is a bf16 product)
#   ff      against the route that rounds w1's output to fp16 before the SwiGLU: 1.4e-3
#   vae     against fp32 convolutions with a bf16 rounding per layer: 6.9e-3 over the whole chain
#   step    the keys of the self-attention in another order: 4.4e-2. Every row quantizer turns a difference far below
#           its step into flipped int8 codes (a step is 3 % of a row's deviation), so that a change of one bf16 rounding
#           early in a block ends at the quantizers' own step; stated at twice the measurement, not four times
TOLERANCE = {"attn": 8e-3, "linear": 1e-2, "te": 6e-3, "ff": 6e-3, "vae": 2.5e-2, "step": 9e-2}


def tolerance(case):
    return {"rel": 4e-3 if case["kind"] == "attn" and case["rotate"] else TOLERANCE[case["kind"]]}

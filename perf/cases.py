"""What the performance of this package is measured on.

Each case is one call that a user's program makes, through the public entry points: the policy
engine on host frames (``chunk``), the policy model without a captured graph (``policy``), the DiT
denoiser (``denoise``) and its runner contract (``runner``), the callables that are hooked into a
host framework's modules (``mlp``, ``ffn_tail``), and the W8A16 linear and the attention on their own
(``linear``, ``attention``).
Sizes are those of ``tybok_b200/shapes.py``, of the tests and of ``bench.py``, and ragged ones between them.
"""

from __future__ import annotations

import math

import torch

from tybok_b200 import hooks, ops
from tybok_b200.dit import DiTBlock, DiTDenoiser, rotary_parts
from tybok_b200.engine import PI05B200Engine
from tybok_b200.pi05 import PI05Model
from tybok_b200.shapes import DIT_FULL, PI05_FULL, W8_SWEEP_NK
from tybok_b200.weights import quantize_dit_block, quantize_w8, random_dit_block_params, random_pi05_params

DEVICE = "cuda"
#: Widths of the feed-forward pairs (model width, intermediate width) that the ``mlp`` cases run:
#: the action expert's and the prefix decoder's.
MLP_WIDTHS = ((1024, 4096), (2048, 16384))


def listed() -> list[dict]:
    return [
        # One robot asks for its next action chunk: the serving latency. Frames arrive on the host at the
        # model's resolution, the chunk goes back to the host.
        {"name": "chunk_b1", "kind": "chunk", "batch": 1, "steps": 10, "prompt": 32, "height": 224, "width": 224},
        # A small fleet in one batch, camera frames at the camera's own resolution, prompts shorter than their slot.
        {"name": "chunk_b8_camera", "kind": "chunk", "batch": 8, "steps": 10, "prompt": 19, "height": 240, "width": 320},
        # Batched serving at its throughput end.
        {"name": "chunk_b32", "kind": "chunk", "batch": 32, "steps": 10, "prompt": 27, "height": 224, "width": 224},
        # A policy with three cameras and the long prompt slot of a checkpoint's default tokenizer length, run
        # without a captured graph, as a program does whose shapes change from call to call.
        {"name": "policy_3cam_eager", "kind": "policy", "batch": 1, "cams": 3, "lang": 200, "prompt": 131, "steps": 10},
        # The denoiser on a short sequence: 30 blocks, four flow steps, fewer tokens than weights to stream.
        {"name": "denoise_106", "kind": "denoise", "tokens": 106, "blocks": 30, "steps": 4, "context": 77},
        # The fused runner of a host framework: 50 action tokens attend to the video's keys and values.
        {"name": "runner_50", "kind": "runner", "tokens": 50, "video": 4096, "blocks": 30, "context": 129},
        # One token through one projection: the smallest call, launches and host work count.
        {"name": "linear_1", "kind": "linear", "tokens": 1, "n": 2560, "k": 2048, "epilogue": "none"},
        # A batch of tokens through the wide projection, with bias and GELU.
        {"name": "linear_800", "kind": "linear", "tokens": 800, "n": 16384, "k": 2048, "epilogue": "gelu"},
        # The action expert's feed-forward hook at its decode size.
        {"name": "mlp_50", "kind": "mlp", "tokens": 50, "width": 1024, "inner": 4096},
        # The prefix decoder's feed-forward hook on a prompt of odd length.
        {"name": "mlp_333", "kind": "mlp", "tokens": 333, "width": 2048, "inner": 16384},
        # The DiT block's feed-forward tail hook at the video + action sequence length.
        {"name": "ffn_tail_4146", "kind": "ffn_tail", "batch": 1, "tokens": 4146},
        # The DiT block's self-attention at that length.
        {"name": "attention_4146", "kind": "attention", "batch": 1, "tokens": 4146, "keys": 4146, "heads": 24, "kv_heads": 24,
         "head_dim": 128, "masked": False},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(("chunk", "chunk", "policy", "denoise", "runner", "linear", "linear", "mlp", "mlp", "ffn_tail", "ffn_tail",
                       "attention", "attention"))
    if kind == "chunk":
        height, width = rng.choice(((224, 224), (224, 224), (240, 320), (256, 256)))
        return {"kind": kind, "batch": _log_int(rng, 1, 32), "steps": rng.randint(4, 10), "prompt": rng.randint(4, 32),
                "height": height, "width": width}
    if kind == "policy":
        lang = rng.randint(16, 200)
        return {"kind": kind, "batch": rng.randint(1, 3), "cams": rng.randint(1, 3), "lang": lang,
                "prompt": rng.randint(4, lang), "steps": rng.randint(4, 10)}
    if kind == "denoise":
        return {"kind": kind, "tokens": _log_int(rng, 16, 128), "blocks": rng.randint(4, 30), "steps": rng.randint(1, 4),
                "context": rng.randint(16, 160)}
    if kind == "runner":
        return {"kind": kind, "tokens": _log_int(rng, 16, 128), "video": _log_int(rng, 256, 4096),
                "blocks": rng.randint(4, 30), "context": rng.randint(16, 160)}
    if kind == "linear":
        n, k = rng.choice(W8_SWEEP_NK)
        return {"kind": kind, "tokens": _log_int(rng, 1, 1600), "n": n, "k": k, "epilogue": rng.choice(("none", "gelu", "residual"))}
    if kind == "mlp":
        width, inner = rng.choice(MLP_WIDTHS)
        return {"kind": kind, "tokens": _log_int(rng, 1, 1600), "width": width, "inner": inner}
    if kind == "ffn_tail":
        return {"kind": kind, "batch": rng.randint(1, 2), "tokens": _log_int(rng, 64, 2073)}
    form = rng.choice(("self", "cross", "prefix", "suffix"))
    if form == "self":
        n = _log_int(rng, 106, 4146)
        return {"kind": kind, "batch": 1, "tokens": n, "keys": n, "heads": 24, "kv_heads": 24, "head_dim": 128, "masked": False}
    if form == "cross":
        return {"kind": kind, "batch": 1, "tokens": _log_int(rng, 106, 4146), "keys": rng.randint(16, 160), "heads": 24,
                "kv_heads": 24, "head_dim": 128, "masked": True}
    n = rng.randint(260, 968)
    return {"kind": kind, "batch": _log_int(rng, 1, 8), "tokens": n if form == "prefix" else 50,
            "keys": n if form == "prefix" else n + 50, "heads": 8, "kv_heads": 1, "head_dim": 256, "masked": True}


# ------------------------------------------------------------------------------------ inputs and handles
def _gen(seed: int, device: str = DEVICE) -> torch.Generator:
    return torch.Generator(device=device).manual_seed(seed)


def _normal(gen, *shape, std: float = 1.0, dtype=torch.float32) -> torch.Tensor:
    return torch.empty(*shape, device=gen.device).normal_(0.0, std, generator=gen).to(dtype)


def _frames(case: dict, seed: int) -> list[dict]:
    """Client frames on the host: pinned camera images in [0, 1], prompt ids with their mask, a state."""
    g = _gen(seed, "cpu")
    frames = []
    for _ in range(case["batch"]):
        frame = {f"observation.images.camera{c + 1}": torch.rand(3, case["height"], case["width"], generator=g).pin_memory()
                 for c in range(PI05_FULL.n_cams)}
        frame["observation.state"] = torch.randn(8, generator=g)
        frame["task"] = "pick up the red block"
        frame["observation.language.tokens"] = torch.randint(0, PI05_FULL.vocab, (case["prompt"],), generator=g)
        frame["observation.language.attention_mask"] = torch.ones(case["prompt"], dtype=torch.bool)
        frames.append(frame)
    return frames


def _denoiser(blocks: int, seed: int) -> DiTDenoiser:
    den = DiTDenoiser([], DIT_FULL, device=DEVICE)
    for i in range(blocks):
        den.blocks.append(DiTBlock(quantize_dit_block(random_dit_block_params(DIT_FULL, seed=1000 * seed + i, device=DEVICE)),
                                   DIT_FULL, device=DEVICE))
    return den


def _rotary(tokens: int) -> torch.Tensor:
    d = DIT_FULL.head_dim
    ang = torch.outer(torch.arange(tokens, dtype=torch.float64),
                      1.0 / torch.pow(10000, torch.arange(0, d, 2, dtype=torch.float64) / d))
    return torch.polar(torch.ones_like(ang), ang)[:, None, :]


class _Linear:
    """The attributes of a host framework's fp8 linear module."""

    def __init__(self, gen, n: int, k: int, bias: bool):
        self.weight, self.weight_scale = quantize_w8(_normal(gen, n, k, std=0.02, dtype=torch.bfloat16))
        self.bias = _normal(gen, n, std=0.02, dtype=torch.bfloat16) if bias else None


class _Module:
    pass


def _context_mask(n: int) -> torch.Tensor:
    mask = torch.ones(n, dtype=torch.bool)
    mask[-5:-1] = False  # a text shorter than its slot, before the proprioception token
    return mask


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    bf16 = torch.bfloat16
    g = _gen(seed)
    if kind == "chunk":
        engine = PI05B200Engine(f"synthetic:pi05_full@{seed}", device=DEVICE, batch_size=case["batch"], num_steps=case["steps"])
        noise = torch.randn(case["batch"], PI05_FULL.chunk, PI05_FULL.max_action_dim, generator=_gen(seed, "cpu"))
        return {"case": case, "engine": engine, "frames": _frames(case, seed), "noise": noise}
    if kind == "policy":
        shape = PI05_FULL.with_(n_cams=case["cams"], lang_len=case["lang"], steps=case["steps"])
        model = PI05Model(random_pi05_params(shape, seed=seed, device=DEVICE), shape, device=DEVICE, vision_dtype=torch.float16)
        b, res = case["batch"], shape.vision.image
        tokens = torch.randint(0, shape.vocab, (b, case["lang"]), generator=g, device=DEVICE)
        masks = (torch.arange(case["lang"], device=DEVICE) < case["prompt"])[None].expand(b, -1).contiguous()
        return {"case": case, "model": model,
                "args": ([torch.empty(b, 3, res, res, device=DEVICE).uniform_(-1, 1, generator=g) for _ in range(case["cams"])],
                         [torch.ones(b, dtype=torch.bool, device=DEVICE) for _ in range(case["cams"])], tokens, masks,
                         _normal(g, b, shape.chunk, shape.max_action_dim))}
    h = DIT_FULL.hidden
    if kind == "denoise":
        den = _denoiser(case["blocks"], seed)
        den.prepare_context(_normal(g, case["context"], h, dtype=bf16), _context_mask(case["context"]))
        cos, sin = rotary_parts(_rotary(case["tokens"]), DEVICE)
        t_mods = _normal(g, case["steps"], 6, h, std=0.5, dtype=bf16)
        return {"case": case, "den": den, "x": _normal(g, case["tokens"], h, dtype=bf16), "t_mods": t_mods, "cos": cos,
                "sin": sin, "deltas": [-1.0 / case["steps"]] * case["steps"]}
    if kind == "runner":
        den = _denoiser(case["blocks"], seed)
        kv = lambda n: _normal(g, 1, n, h, dtype=bf16)  # noqa: E731
        return {"case": case, "den": den, "tokens": kv(case["tokens"]), "t_mod": _normal(g, 1, 6, h, std=0.5, dtype=bf16),
                "freqs": _rotary(case["tokens"]).to(DEVICE),
                "video": [{"k": kv(case["video"]), "v": kv(case["video"])} for _ in range(case["blocks"])],
                "cross": [(kv(case["context"]), kv(case["context"])) for _ in range(case["blocks"])],
                "mask": _context_mask(case["context"]).to(DEVICE)}
    if kind == "linear":
        lin = _Linear(g, case["n"], case["k"], bias=True)
        state = {"case": case, "w8": lin.weight, "scale": lin.weight_scale, "bias": lin.bias,
                 "x": _normal(g, case["tokens"], case["k"], dtype=bf16), "residual": None}
        if case["epilogue"] == "residual":
            state["residual"] = _normal(g, case["tokens"], case["n"], dtype=bf16)
        return state
    if kind == "mlp":
        mlp = _Module()
        mlp.gate_proj, mlp.up_proj = (_Linear(g, case["inner"], case["width"], bias=False) for _ in range(2))
        mlp.down_proj = _Linear(g, case["width"], case["inner"], bias=False)
        return {"case": case, "fn": hooks.make_mlp_forward(mlp), "x": _normal(g, 1, case["tokens"], case["width"], dtype=bf16)}
    if kind == "ffn_tail":
        blk = _Module()
        blk.ffn = [_Linear(g, DIT_FULL.ffn, h, bias=True), None, _Linear(g, h, DIT_FULL.ffn, bias=True)]
        mods = _normal(g, case["batch"], 6, h, std=0.5, dtype=bf16)  # the modulation table; its rows are strided views
        return {"case": case, "fn": hooks.make_fused_ffn_tail(blk), "x": _normal(g, case["batch"], case["tokens"], h, dtype=bf16),
                "mods": tuple(mods[:, i : i + 1] for i in (3, 4, 5))}
    if kind == "attention":
        b, n, d = case["batch"], case["keys"], case["head_dim"]
        valid = None
        if case["masked"]:  # keys past the end of the prompt or text do not count; the last ones (the query's own) do
            valid = torch.ones(b, n, dtype=torch.uint8, device=DEVICE)
            valid[:, n - n // 8 : n - n // 16] = 0
        return {"case": case, "q": _normal(g, b * case["tokens"], case["heads"] * d, dtype=bf16),
                "k": _normal(g, b, case["kv_heads"], n, d, dtype=bf16), "v": _normal(g, b, case["kv_heads"], n, d, dtype=bf16),
                "valid": valid}
    raise ValueError(f"unknown kind {kind!r}")


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "chunk":
        if case["batch"] == 1:
            return state["engine"].predict_action_chunk(state["frames"][0], noise=state["noise"][0])
        return state["engine"].predict_action_chunks(state["frames"], noise=state["noise"])
    if kind == "policy":
        return state["model"].sample_actions(*state["args"])
    if kind == "denoise":
        return state["den"].denoise(state["x"], state["t_mods"], state["cos"], state["sin"], state["deltas"])
    if kind == "runner":
        return state["den"].run_action_layers(state["tokens"], state["t_mod"], state["freqs"], state["video"], state["cross"],
                                              state["mask"])
    if kind == "linear":
        epilogue = {"none": ops.EPI_NONE, "gelu": ops.EPI_GELU, "residual": ops.EPI_RESIDUAL}[case["epilogue"]]
        return ops.w8a16_linear(state["x"], state["w8"], state["scale"], state["bias"], epilogue=epilogue,
                                residual=state["residual"])
    if kind == "mlp":
        return state["fn"](state["x"])
    if kind == "ffn_tail":
        return state["fn"](state["x"], *state["mods"])
    return ops.attention(state["q"], state["k"], state["v"], state["valid"], tokens=case["tokens"], keys=case["keys"],
                         scale=case["head_dim"] ** -0.5)[0]


# ------------------------------------------------------------------------------------ what a pass cannot do without
def _policy_work(batch: int, cams: int, lang: int, steps: int) -> tuple[float, float]:
    """(bytes, flops) of one chunk: tower, projector and both decoders; weights once, frames in, actions out."""
    s = PI05_FULL
    v = s.vision
    vis = v.layers * (4 * v.hidden * v.hidden + 2 * v.hidden * v.mlp_dim) + 3 * v.patch * v.patch * v.hidden + v.hidden * s.vlm.width
    vt = batch * cams * v.tokens
    flops = 2.0 * vis * vt + 4.0 * v.layers * vt * v.tokens * v.hidden
    lp = cams * v.tokens + lang

    def decoder(spec):
        a, kv = spec.num_heads * spec.head_dim, spec.num_kv_heads * spec.head_dim
        return spec.depth * (spec.width * (2 * a + 2 * kv) + 3 * spec.width * spec.mlp_dim), spec.depth * 4.0 * a

    wp, ap = decoder(s.vlm)
    we, ae = decoder(s.expert)
    flops += batch * lp * (2.0 * wp + ap * lp) + steps * batch * s.chunk * (2.0 * we + ae * (lp + s.chunk))
    byts = 2.0 * vis + wp + we + batch * (cams * 3 * v.image * v.image * 4 + lang * (8 + 2 * s.vlm.width)
                                          + 2 * s.chunk * s.max_action_dim * 4)
    return byts, flops


def work(case: dict) -> dict:
    kind = case["kind"]
    h, f = DIT_FULL.hidden, DIT_FULL.ffn
    if kind == "chunk":
        byts, flops = _policy_work(case["batch"], PI05_FULL.n_cams, PI05_FULL.lang_len, case["steps"])
    elif kind == "policy":
        byts, flops = _policy_work(case["batch"], case["cams"], case["lang"], case["steps"])
    elif kind == "denoise":
        t, c = case["tokens"], case["context"]
        byts = case["blocks"] * (6 * h * h + 2 * h * f + 4 * c * h) + 4 * t * h
        flops = case["steps"] * case["blocks"] * (2.0 * t * (6 * h * h + 2 * h * f) + 4.0 * t * (t + c) * h)
    elif kind == "runner":
        t, c, v = case["tokens"], case["context"], case["video"]
        byts = case["blocks"] * (6 * h * h + 2 * h * f + 4 * (c + v) * h) + 4 * t * h
        flops = case["blocks"] * (2.0 * t * (6 * h * h + 2 * h * f) + 4.0 * t * (t + v + c) * h)
    elif kind == "linear":
        m, n, k = case["tokens"], case["n"], case["k"]
        byts = n * k + 6 * n + 2 * m * k + 2 * m * n * (2 if case["epilogue"] == "residual" else 1)
        flops = 2.0 * m * n * k
    elif kind == "mlp":
        m, w, i = case["tokens"], case["width"], case["inner"]
        byts = 3 * w * i + 4 * m * w
        flops = 6.0 * m * w * i
    elif kind == "attention":
        b, t, n, d = case["batch"], case["tokens"], case["keys"], case["head_dim"]
        byts = 4 * b * d * (t * case["heads"] + n * case["kv_heads"])
        flops = 4.0 * b * case["heads"] * t * n * d
    else:
        m = case["batch"] * case["tokens"]
        byts = 2 * h * f + 4 * m * h
        flops = 4.0 * m * h * f
    return {"bytes": byts, "flops": flops}


def tolerance(case: dict) -> dict:
    # bf16 activations between the layers; deep stacks carry each layer's rounding on, so another correct
    # summation order shows more there than in one linear or one feed-forward block.
    if case["kind"] in ("linear", "mlp", "ffn_tail", "attention"):
        return {"rel": 5e-3}
    return {"rel": 1.5e-2}

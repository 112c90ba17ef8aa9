"""What a program that uses this library has it do, as cases that can be timed and compared.

Every case goes through a public entry point: the patched ``F.linear`` (conditioning vectors, text rows, token rows),
the two attention functions that replace the engine's dispatch points, the AdaLN and QK-norm row kernels, and one
block of each model through its step engine.  Widths, head counts and sequence lengths are those of the two
architectures the library runs (3072 wide with 24 heads, 5120 wide with 40) and of their shards on 2, 4 and 8 GPUs."""
import math

import torch
import torch.nn as nn
import torch.nn.functional as F

from diffsynth_engine_b200 import attention, flux, ops, quant, wan

DEV = "cuda"
# (in, out) features of the token Linears of the two architectures
LINEARS = ((3072, 3072), (3072, 9216), (3072, 12288), (12288, 3072), (3072, 21504), (15360, 3072),
           (5120, 5120), (5120, 13824), (13824, 5120), (4096, 5120))
FORMATS = ("fp8_tensor", "fp8_channel", "int8_channel", "bf16")
AFTER_LN = {"bf16": ops.FMT_BF16, "e4m3": ops.FMT_E4M3, "int8": ops.FMT_INT8}


def listed():
    return [
        # AdaLN modulation of one block: the conditioning vector of a step, one row, bound by the weight's bytes
        {"name": "linear_vector", "kind": "linear", "fmt": "fp8_tensor", "rows": 1, "k": 3072, "n": 18432},
        # feed-forward of the 512 text tokens: a weight-sized Linear on few rows
        {"name": "linear_text", "kind": "linear", "fmt": "fp8_channel", "rows": 512, "k": 3072, "n": 12288},
        # an odd token count (6889 image and 256 text tokens) with INT8 weights
        {"name": "linear_int8_odd", "kind": "linear", "fmt": "int8_channel", "rows": 7145, "k": 3072, "n": 9216},
        # unquantised weights at a 1024 x 1024 image's 4096 + 512 tokens
        {"name": "linear_bf16", "kind": "linear", "fmt": "bf16", "rows": 4608, "k": 3072, "n": 3072},
        # LayerNorm + modulation + row quantisation over an 81-frame 480p video's tokens
        {"name": "adaln_rows", "kind": "adaln", "out": "e4m3", "rows": 32760, "d": 5120},
        # full-width query / key RMSNorm + RoPE over the same tokens
        {"name": "qk_norm_rows", "kind": "qk_norm", "rows": 32760, "d": 5120},
        # joint attention of a 1024 x 1024 image with its text
        {"name": "attn_joint", "kind": "attn_joint", "heads": 24, "sq": 4608, "batch": 1},
        # a small image: odd token count, one wave of tiles, two samples
        {"name": "attn_joint_odd", "kind": "attn_joint", "heads": 24, "sq": 1061, "batch": 2},
        # cross-attention of a video's tokens with 512 text tokens
        {"name": "attn_cross", "kind": "attn_video", "heads": 40, "sq": 32760, "sk": 512},
        # one double-stream and one single-stream block at 1024 x 1024, as a captured step
        {"name": "flux_double_block", "kind": "flux", "fmt": "fp8_tensor", "double": 1, "single": 0, "h": 128, "w": 128,
         "text": 512},
        {"name": "flux_single_block", "kind": "flux", "fmt": "fp8_tensor", "double": 0, "single": 1, "h": 128, "w": 128,
         "text": 512},
        # one block of the video model over the whole 480p video
        {"name": "wan_block", "kind": "wan", "fmt": "fp8_channel", "frames": 21, "h": 60, "w": 104, "text": 512},
    ]


def _spread(rng, lo, hi):
    """A whole number in [lo, hi], even over its logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(("linear", "linear", "linear", "adaln", "qk_norm", "attn_joint", "attn_joint", "attn_video",
                       "attn_video", "flux", "wan"))
    if kind == "linear":
        k, n = rng.choice(LINEARS)
        return {"kind": kind, "fmt": rng.choice(FORMATS), "rows": _spread(rng, 1, 32760), "k": k, "n": n}
    if kind == "adaln":
        return {"kind": kind, "out": rng.choice(sorted(AFTER_LN)), "rows": _spread(rng, 200, 32760),
                "d": rng.choice((3072, 5120))}
    if kind == "qk_norm":
        return {"kind": kind, "rows": _spread(rng, 200, 32760), "d": rng.choice((3072, 5120))}
    if kind == "attn_joint":
        return {"kind": kind, "heads": rng.choice((12, 24, 24, 40)), "sq": _spread(rng, 200, 8192),
                "batch": rng.choice((1, 1, 2))}
    if kind == "attn_video":
        sq = _spread(rng, 500, 16380)
        return {"kind": kind, "heads": rng.choice((5, 10, 20, 40)), "sq": sq,
                "sk": rng.choice((sq, sq, 512, 257, _spread(rng, 20, 512)))}
    if kind == "flux":
        double = rng.randint(0, 1)
        return {"kind": kind, "fmt": rng.choice(FORMATS), "double": double, "single": 1 - double,
                "h": 2 * _spread(rng, 12, 64), "w": 2 * _spread(rng, 12, 64), "text": rng.choice((512, 256, rng.randint(20, 500)))}
    return {"kind": kind, "fmt": rng.choice(FORMATS), "frames": rng.randint(1, 13), "h": 2 * rng.randint(15, 30),
            "w": 2 * rng.randint(15, 52), "text": rng.choice((512, rng.randint(20, 512)))}


# ------------------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(gen, *shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(shape, generator=gen, device=DEV) * std).to(dtype)


def _tokens(gen, rows, d):
    """Hidden-state rows: unit noise with a few channels that are far larger than the rest, as a DiT's are."""
    x = torch.randn((rows, d), generator=gen, device=DEV)
    x *= 1.0 + 4.0 * (torch.rand(d, generator=gen, device=DEV) < 0.01)
    return x.bfloat16()


def _rope(gen, rows):
    ang = torch.rand((rows, 64), generator=gen, device=DEV) * 6.0
    return torch.stack([ang.cos(), ang.sin()], dim=-1).contiguous()


def _linear_inputs(case, seed):
    gen = _gen(seed)
    w = _randn(gen, case["n"], case["k"], std=0.02)
    return _tokens(gen, case["rows"], case["k"]), w, _randn(gen, case["n"], std=0.1)


def _adaln_inputs(case, seed):
    gen = _gen(seed)
    d = case["d"]
    return (_tokens(gen, case["rows"], d), _randn(gen, d, std=0.3, dtype=torch.float32),
            _randn(gen, d, std=0.3, dtype=torch.float32))


def _qk_norm_inputs(case, seed):
    gen = _gen(seed)
    return (_tokens(gen, case["rows"], case["d"]), 1.0 + _randn(gen, case["d"], std=0.05, dtype=torch.float32),
            _rope(gen, case["rows"]))


def _attn_inputs(case, seed):
    """q and k with the spread that a per-head norm gives them; [B, H, S, D] for the joint attention, whose q, k and v
    are views of one projection, [B, S, H*D] for the video model's."""
    gen = _gen(seed)
    h, sq = case["heads"], case["sq"]
    if case["kind"] == "attn_joint":
        qkv = _randn(gen, case["batch"], sq, 3, h, 128)
        return tuple(qkv[:, :, i].transpose(1, 2) for i in range(3))
    q = _randn(gen, 1, sq, h * 128, std=1.2)
    return q, _randn(gen, 1, case["sk"], h * 128, std=1.2), _randn(gen, 1, case["sk"], h * 128)


def _weights(shapes, seed):
    gen = _gen(seed)
    out = {}
    for name, shape in shapes.items():
        t = torch.randn(shape, generator=gen, device=DEV) * (shape[-1] ** -0.5 if name.endswith("modulation") else 0.02)
        out[name] = ((t + 1.0) if ("norm" in name and len(shape) == 1 and name.endswith("weight")) else t).bfloat16()
    return out


def _with(shapes, name, n_out, n_in):
    shapes[name + ".weight"], shapes[name + ".bias"] = (n_out, n_in), (n_out,)


def _flux_inputs(case, seed):
    d, s = 3072, {}
    for e in ("time_embedder.timestep_embedder", "guidance_embedder.timestep_embedder"):
        _with(s, e + ".0", d, 256), _with(s, e + ".2", d, d)
    _with(s, "pooled_text_embedder.0", d, 768), _with(s, "pooled_text_embedder.2", d, d)
    _with(s, "context_embedder", d, 4096), _with(s, "x_embedder", d, 64)
    if case["double"]:
        for a in "ab":
            _with(s, f"blocks.0.norm1_{a}.linear", 6 * d, d)
            _with(s, f"blocks.0.attn.{a}_to_qkv", 3 * d, d), _with(s, f"blocks.0.attn.{a}_to_out", d, d)
            s[f"blocks.0.attn.norm_q_{a}.weight"] = s[f"blocks.0.attn.norm_k_{a}.weight"] = (128,)
            _with(s, f"blocks.0.ff_{a}.0", 4 * d, d), _with(s, f"blocks.0.ff_{a}.2", d, 4 * d)
    if case["single"]:
        _with(s, "single_blocks.0.norm.linear", 3 * d, d), _with(s, "single_blocks.0.to_qkv_mlp", 7 * d, d)
        s["single_blocks.0.norm_q_a.weight"] = s["single_blocks.0.norm_k_a.weight"] = (128,)
        _with(s, "single_blocks.0.proj_out", d, 5 * d)
    _with(s, "final_norm_out.linear", 2 * d, d), _with(s, "final_proj_out", 64, d)
    gen = _gen(seed + 1)
    return _weights(s, seed), {
        "latents": _randn(gen, 1, 16, case["h"], case["w"]), "timestep": torch.full((1,), 500.0, device=DEV),
        "prompt": _randn(gen, 1, case["text"], 4096), "pooled": _randn(gen, 1, 768, dtype=torch.float32),
        "guidance": torch.full((1,), 3.5, device=DEV)}


def _wan_inputs(case, seed):
    d, ffn, s = 5120, 13824, {"patch_embedding.weight": (5120, 16, 1, 2, 2), "patch_embedding.bias": (5120,)}
    _with(s, "text_embedding.0", d, 4096), _with(s, "text_embedding.2", d, d)
    _with(s, "time_embedding.0", d, 256), _with(s, "time_embedding.2", d, d), _with(s, "time_projection.1", 6 * d, d)
    for a in ("self_attn", "cross_attn"):
        for n in "qkvo":
            _with(s, f"blocks.0.{a}.{n}", d, d)
        s[f"blocks.0.{a}.norm_q.weight"] = s[f"blocks.0.{a}.norm_k.weight"] = (d,)
    s["blocks.0.norm3.weight"] = s["blocks.0.norm3.bias"] = (d,)
    _with(s, "blocks.0.ffn.0", ffn, d), _with(s, "blocks.0.ffn.2", d, ffn)
    s["blocks.0.modulation"] = (1, 6, d)
    _with(s, "head.head", 64, d)
    s["head.modulation"] = (1, 2, d)
    gen = _gen(seed + 1)
    return _weights(s, seed), {
        "latents": _randn(gen, 1, 16, case["frames"], case["h"], case["w"]),
        "timestep": torch.full((1,), 417.0, device=DEV), "context": _randn(gen, 1, case["text"], 4096)}


# -------------------------------------------------------------------------------------------------- the timed program
def prepare(case, seed):
    kind = case["kind"]
    if kind == "linear":
        x, w, b = _linear_inputs(case, seed)
        layer = nn.Linear(case["k"], case["n"], device="meta")
        layer.weight, layer.bias = nn.Parameter(w, requires_grad=False), nn.Parameter(b, requires_grad=False)
        quant.enable_b200_linear(layer, case["fmt"])
        return {"kind": kind, "x": x, "layer": layer}
    if kind == "adaln":
        x, shift, scale = _adaln_inputs(case, seed)
        return {"kind": kind, "x": x, "shift": shift, "scale": scale, "fmt": AFTER_LN[case["out"]]}
    if kind == "qk_norm":
        x, w, rope = _qk_norm_inputs(case, seed)
        return {"kind": kind, "x": x, "w": w, "rope": rope, "out": torch.empty_like(x)}
    if kind in ("attn_joint", "attn_video"):
        return {"kind": kind, "qkv": _attn_inputs(case, seed), "heads": case["heads"]}
    if kind == "flux":
        w, inputs = _flux_inputs(case, seed)
        eng = flux.FluxDiTEngine(w, fmt=case["fmt"], device="cuda:0", n_double=case["double"], n_single=case["single"],
                                 num_heads=24, release_source=True)
        eng.prepare(case["text"], case["h"], case["w"])
        eng.set_inputs(inputs["latents"], inputs["timestep"], inputs["prompt"], inputs["pooled"], inputs["guidance"])
        return {"kind": kind, "engine": eng.capture(), "inputs": inputs}
    w, inputs = _wan_inputs(case, seed)
    eng = wan.WanDiTEngine(w, fmt=case["fmt"], device="cuda:0", num_layers=1, num_heads=40, release_source=True)
    eng.prepare(case["frames"], case["h"], case["w"], case["text"])
    return {"kind": kind, "engine": eng, "inputs": inputs}


def run(state):
    kind = state["kind"]
    if kind == "linear":
        with quant.b200_inference():
            return state["layer"](state["x"])
    if kind == "adaln":
        return ops.ln_modulate(state["x"], state["shift"], state["scale"], 1e-6, state["fmt"])
    if kind == "qk_norm":
        return ops.rmsnorm_full(state["x"], state["w"], state["rope"], out=state["out"])
    if kind == "attn_joint":
        return attention.b200_attn(*state["qkv"])
    if kind == "attn_video":
        return attention.b200_wan_attention(*state["qkv"], state["heads"])
    eng, i = state["engine"], state["inputs"]
    if kind == "flux":
        eng.set_inputs(i["latents"], i["timestep"], i["prompt"], i["pooled"], i["guidance"])
    else:
        eng.set_inputs(i["latents"], i["context"], i["timestep"])
    return eng.step()


# ------------------------------------------------------------------------------------------------ work and tolerances
def _wbytes(fmt):
    return 2 if fmt == "bf16" else 1


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": 2 * m * k + _wbytes(case["fmt"]) * k * n + 2 * m * n, "flops": 2 * m * k * n}
    if kind == "adaln":
        return {"bytes": case["rows"] * case["d"] * (4 if case["out"] == "bf16" else 3), "flops": 0}
    if kind == "qk_norm":
        return {"bytes": case["rows"] * (4 * case["d"] + 512), "flops": 0}
    if kind in ("attn_joint", "attn_video"):
        h, sq, sk, b = case["heads"], case["sq"], case.get("sk", case["sq"]), case.get("batch", 1)
        return {"bytes": b * h * 128 * 2 * (2 * sq + 2 * sk), "flops": 4 * b * h * sq * sk * 128}
    if kind == "flux":
        d, img, txt = 3072, case["h"] * case["w"] // 4, case["text"]
        s = img + txt
        block = (24 * d * d + 4 * s * d) * s        # 12 d^2 weights per token and stream, q k^T and p v
        vectors = 2 * (2 * 256 * d + 2 * d * d) // 2 + 768 * d + d * d + (12 if case["double"] else 3) * d * d + 2 * d * d
        weights = (24 if case["double"] else 12) * d * d + vectors + 4096 * d + 128 * d
        return {"bytes": weights * _wbytes(case["fmt"]) + 2 * (128 * img + 4096 * txt),
                "flops": block + 2 * vectors + 2 * d * (64 * 2 * img + 4096 * txt)}
    d, ffn, s, txt = 5120, 13824, case["frames"] * case["h"] * case["w"] // 4, case["text"]
    flops = 2 * s * (6 * d * d + 2 * d * ffn) + 4 * s * s * d + 4 * s * txt * d + 4 * s * 64 * d
    weights = 6 * d * d + 2 * d * ffn + 256 * d + 7 * d * d + 128 * d
    # the prompt's own projections (text embedding, cross-attention keys and values) are made once per prompt
    return {"bytes": weights * _wbytes(case["fmt"]) + 2 * 128 * s + 4 * txt * d, "flops": flops + 2 * (256 * d + 7 * d * d)}


def tolerance(case):
    kind = case["kind"]
    if kind == "linear":
        return {"rel": 2e-3}                       # one bf16 rounding of sums that may be taken in another order
    if kind == "adaln":
        # a value next to a rounding boundary may fall on either side: 2^-8 of it in bf16, 2^-3 in e4m3
        return {"rel": 2e-3} if case["out"] == "bf16" else {"rel": 5e-3, "max": 0.15, "differ": 2e-3}
    if kind == "qk_norm":
        return {"rel": 2e-3}
    if kind in ("attn_joint", "attn_video"):
        return {"rel": 4e-3}                       # probabilities are rounded to bf16 in front of the second product
    # A block: a changed rounding in one tensor moves codes of the next quantised one; two evaluations of the same
    # formula in another summation order differ by up to 2e-2 (8-bit operands) and 4e-3 (bf16).
    return {"rel": 1e-2} if case["fmt"] == "bf16" else {"rel": 3e-2}


# ------------------------------------------------------------------------------------------- the same in 64 bits
def _rounded(w, fmt):
    """The values that a weight of this format holds, in 64 bits."""
    if fmt == "bf16":
        return w.double()
    w, top = w.float(), 127.0 if fmt == "int8_channel" else 448.0
    amax = w.abs().amax() if fmt == "fp8_tensor" else w.abs().amax(dim=1, keepdim=True)
    s = torch.where(amax > 0, amax / top, torch.ones_like(amax))
    q = (w / s).clamp(-top, top)
    q = q.round() if fmt == "int8_channel" else q.to(torch.float8_e4m3fn)
    return q.double() * s.double()


def _attend(q, k, v):
    """[H, S, D] each, one head and a slice of the queries at a time."""
    out = torch.empty_like(q)
    for h in range(q.shape[0]):
        kt = k[h].t() * q.shape[-1] ** -0.5
        for r in range(0, q.shape[1], 8192):
            out[h, r:r + 8192] = torch.softmax(q[h, r:r + 8192] @ kt, dim=-1) @ v[h]
    return out


def _norm(x, eps=1e-6):
    return F.layer_norm(x, (x.shape[-1],), eps=eps)


def _rms(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * w.double()


def _rotate(x, cos, sin):
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([cos * a - sin * b, sin * a + cos * b], dim=-1).flatten(-2)


def _split(x, heads):
    return x.unflatten(-1, (heads, 128)).transpose(0, 1)


def _join(x):
    return x.transpose(0, 1).flatten(1)


def _gelu(x):
    return F.gelu(x, approximate="tanh")


def _angles(pos, dim):
    return pos.double()[:, None] * 10000.0 ** (-torch.arange(0, dim, 2, device=DEV).double() / dim)


def _sinusoid(t, dim):
    ang = _angles(t, dim)
    return torch.cat([ang.cos(), ang.sin()], dim=-1).bfloat16().double()   # the sinusoid is bf16 in front of its MLP


def _exact_flux(case, seed):
    w, i = _flux_inputs(case, seed)
    heads, txt = 24, case["text"]

    def lin(x, name):
        return x @ _rounded(w[name + ".weight"], case["fmt"]).t() + w[name + ".bias"].double()

    def mlp(x, name):
        return lin(F.silu(lin(x, name + ".0")), name + ".2")

    cond = (mlp(_sinusoid(i["timestep"], 256), "time_embedder.timestep_embedder")
            + mlp(_sinusoid(i["guidance"] * 1000.0, 256), "guidance_embedder.timestep_embedder")
            + mlp(i["pooled"].double(), "pooled_text_embedder"))
    act = F.silu(cond)
    gh, gw = case["h"] // 2, case["w"] // 2
    rows = torch.arange(gh * gw, device=DEV)
    zero = torch.zeros(txt, device=DEV)
    ang = torch.cat([_angles(torch.cat([zero, rows * 0]), 16), _angles(torch.cat([zero, rows // gw]), 56),
                     _angles(torch.cat([zero, rows % gw]), 56)], dim=1)
    cos, sin = ang.cos(), ang.sin()
    patches = i["latents"].double()[0].reshape(16, gh, 2, gw, 2).permute(1, 3, 0, 2, 4).reshape(gh * gw, 64)
    xi, xt = lin(patches, "x_embedder"), lin(i["prompt"][0].double(), "context_embedder")

    def qk(q, name):
        return _rms(_split(q, heads), w[name])

    if case["double"]:
        pre = "blocks.0."
        mod = {a: lin(act, pre + f"norm1_{a}.linear")[0].chunk(6) for a in "ab"}
        parts = {a: lin(_norm(x) * (1 + mod[a][1]) + mod[a][0], pre + f"attn.{a}_to_qkv").chunk(3, dim=-1)
                 for a, x in (("b", xt), ("a", xi))}
        q, k = (_rotate(torch.cat([qk(parts[a][n], pre + f"attn.norm_{c}_{a}.weight") for a in "ba"], dim=1), cos, sin)
                for n, c in ((0, "q"), (1, "k")))
        att = _join(_attend(q, k, torch.cat([_split(parts[a][2], heads) for a in "ba"], dim=1)))
        new = {}
        for a, x, o in (("a", xi, att[txt:]), ("b", xt, att[:txt])):
            x = x + mod[a][2] * lin(o, pre + f"attn.{a}_to_out")
            hid = _gelu(lin(_norm(x) * (1 + mod[a][4]) + mod[a][3], pre + f"ff_{a}.0"))
            new[a] = x + mod[a][5] * lin(hid, pre + f"ff_{a}.2")
        xi, xt = new["a"], new["b"]
    x = torch.cat([xt, xi])
    if case["single"]:
        pre = "single_blocks.0."
        shift, scale, gate = lin(act, pre + "norm.linear")[0].chunk(3)
        hid = lin(_norm(x) * (1 + scale) + shift, pre + "to_qkv_mlp")
        q, k, v = hid[:, :9216].chunk(3, dim=-1)
        att = _attend(_rotate(qk(q, pre + "norm_q_a.weight"), cos, sin), _rotate(qk(k, pre + "norm_k_a.weight"), cos, sin),
                      _split(v, heads))
        x = x + gate * lin(torch.cat([_join(att), _gelu(hid[:, 9216:])], dim=1), pre + "proj_out")
    scale, shift = lin(act, "final_norm_out.linear")[0].chunk(2)
    out = lin(_norm(x[txt:]) * (1 + scale) + shift, "final_proj_out")
    return out.reshape(gh, gw, 16, 2, 2).permute(2, 0, 3, 1, 4).reshape(1, 16, case["h"], case["w"])


def _exact_wan(case, seed):
    w, i = _wan_inputs(case, seed)
    heads, d = 40, 5120

    def lin(x, name):
        return x @ _rounded(w[name + ".weight"].flatten(1), case["fmt"]).t() + w[name + ".bias"].double()

    t = lin(F.silu(lin(_sinusoid(i["timestep"], 256), "time_embedding.0")), "time_embedding.2")
    mod = w["blocks.0.modulation"].double()[0] + lin(F.silu(t), "time_projection.1").reshape(6, d)
    ctx = lin(_gelu(lin(i["context"][0].double(), "text_embedding.0")), "text_embedding.2")
    fr, gh, gw = case["frames"], case["h"] // 2, case["w"] // 2
    r = torch.arange(fr * gh * gw, device=DEV)
    ang = torch.cat([_angles(r // (gh * gw), 44), _angles(r // gw % gh, 42), _angles(r % gw, 42)], dim=1)
    cos, sin = ang.cos(), ang.sin()
    x = lin(i["latents"].double()[0].reshape(16, fr, gh, 2, gw, 2).permute(1, 2, 4, 0, 3, 5).reshape(-1, 64),
            "patch_embedding")

    def qkv(xq, xkv, a):
        q = _rms(lin(xq, a + ".q"), w[a + ".norm_q.weight"])
        return _split(q, heads), _split(_rms(lin(xkv, a + ".k"), w[a + ".norm_k.weight"]), heads), _split(lin(xkv, a + ".v"), heads)

    n = _norm(x) * (1 + mod[1]) + mod[0]
    q, k, v = qkv(n, n, "blocks.0.self_attn")
    x = x + mod[2] * lin(_join(_attend(_rotate(q, cos, sin), _rotate(k, cos, sin), v)), "blocks.0.self_attn.o")
    n = _norm(x) * w["blocks.0.norm3.weight"].double() + w["blocks.0.norm3.bias"].double()
    x = x + lin(_join(_attend(*qkv(n, ctx, "blocks.0.cross_attn"))), "blocks.0.cross_attn.o")
    hid = _gelu(lin(_norm(x) * (1 + mod[4]) + mod[3], "blocks.0.ffn.0"))
    x = x + mod[5] * lin(hid, "blocks.0.ffn.2")
    shift, scale = w["head.modulation"].double()[0] + t
    out = lin(_norm(x) * (1 + scale) + shift, "head.head")
    return out.reshape(fr, gh, gw, 2, 2, 16).permute(5, 0, 1, 3, 2, 4).reshape(1, 16, fr, case["h"], case["w"])


def exact(case, seed):
    kind = case["kind"]
    if kind == "linear":
        x, w, b = _linear_inputs(case, seed)
        return x.double() @ _rounded(w, case["fmt"]).t() + b.double()
    if kind == "adaln":
        x, shift, scale = (t.double() for t in _adaln_inputs(case, seed))
        y = _norm(x) * (1 + scale) + shift
        if case["out"] == "bf16":
            return y, None
        s = y.abs().amax(dim=1) / (448.0 if case["out"] == "e4m3" else 127.0)
        return (y / s[:, None] if case["out"] == "e4m3" else None), s
    if kind == "qk_norm":
        x, w, rope = _qk_norm_inputs(case, seed)
        y = _rms(x.double(), w).unflatten(1, (-1, 128))
        return _rotate(y, rope[:, None, :, 0].double(), rope[:, None, :, 1].double()).flatten(1)
    if kind == "attn_joint":
        return torch.stack([_attend(*(t[b].double() for t in _attn_inputs(case, seed))) for b in range(case["batch"])])
    if kind == "attn_video":
        return _join(_attend(*(_split(t[0].double(), case["heads"]) for t in _attn_inputs(case, seed))))[None]
    return _exact_flux(case, seed) if kind == "flux" else _exact_wan(case, seed)

"""Performance cases: what a user of this package has it do, through its public entry points.

``listed()`` names fixed cases over the range of real use, ``draw()`` gives further ones of the same
ranges, ``prepare()`` builds what a program has in hand before the call, ``run()`` is one pass, ``work()``
the bytes and operations a pass cannot do without and ``tolerance()`` what correct implementations of the
same precision may differ by.  The package is inference only: there is no backward pass.

Kinds of case
  op    ``dot_product_attention_cpp`` on CUDA tensors: q, k, v [B1, B2, S, D], a bias [B2, S, S] shared by
        the B1 batch rows and a key mask.  ``qk`` is bf16, f32 (an fp32 caller) or fp8 (e4m3 with
        per-head scales)
  grid  the grid (triangle) self-attention module on a pair representation [N, N, C]
  self  ``self_attention_cpp``: single / diffusion attention with pair bias on tokens [N, C]
  host  ``dot_product_attention_cpp`` on pinned host tensors, result in host memory
"""
import math

import torch

import af3_kernels_b200 as A


def listed():
    return [
        # a short chain: one call of a few microseconds, host time and launches are everything
        dict(name="op_single_77", kind="op", B1=1, B2=16, S=77, D=24, qk="bf16", bias="f32", mask="tail", pad=9),
        # single attention with pair bias over 512 tokens, fp32 bias as a CPU caller of the reference holds it
        dict(name="op_single_512", kind="op", B1=1, B2=16, S=512, D=32, qk="bf16", bias="f32", mask="tail", pad=64),
        # single attention of a large complex, head width 24, wide bias
        dict(name="op_single_1536", kind="op", B1=1, B2=16, S=1536, D=24, qk="bf16", bias="bf16", mask="tail", pad=128),
        # diffusion-transformer token attention: five samples share one pair bias
        dict(name="op_diffusion_5x1536", kind="op", B1=5, B2=16, S=1536, D=48, qk="bf16", bias="bf16", mask="tail", pad=96),
        # triangle attention over all rows of a 768-token pair representation: the ordinary large call
        dict(name="op_rows_768", kind="op", B1=768, B2=4, S=768, D=32, qk="bf16", bias="f32", mask="random", pad=0),
        # the largest call: 2048 rows of 2048 keys, q and k quantised to e4m3
        dict(name="op_rows_fp8_2048", kind="op", B1=2048, B2=4, S=2048, D=32, qk="fp8", bias="bf16", mask="random", pad=0),
        # the whole module on a small pair: a dozen short launches
        dict(name="grid_64", kind="grid", N=64, C=128, H=4, dtype="bf16", transpose=False),
        # ragged size, fp32 pair and weights, ending-node (transposed) orientation
        dict(name="grid_389_f32_t", kind="grid", N=389, C=128, H=4, dtype="f32", transpose=True),
        # the ordinary large module call
        dict(name="grid_768", kind="grid", N=768, C=128, H=4, dtype="bf16", transpose=False),
        # a narrow pair stack: 64 channels
        dict(name="grid_c64_256", kind="grid", N=256, C=64, H=4, dtype="bf16", transpose=False),
        # single attention block: projections, query bias, attention, gate
        dict(name="self_1536", kind="self", N=1536, C=384, H=16, dtype="bf16"),
        # what a caller of the CPU reference holds: host tensors in, host tensor out
        dict(name="host_rows_256", kind="host", B1=256, B2=4, S=256, D=32, qk="bf16", bias="f32", mask="random", pad=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "single", "diffusion", "rows", "rows", "fp8", "grid", "grid", "grid", "self", "self", "host"])
    if kind in ("single", "diffusion"):
        S = _log(rng, 16, 2048)
        return dict(kind="op", B1=1 if kind == "single" else rng.randint(2, 8), B2=16, S=S, D=rng.choice([24, 32, 48]),
                    qk="f32" if kind == "single" and rng.random() < 0.2 else "bf16", bias=rng.choice(["bf16", "f32"]),
                    mask="tail", pad=rng.randint(0, S // 6))
    if kind == "rows":
        S = _log(rng, 32, 1024)
        return dict(kind="op", B1=S, B2=4, S=S, D=32, qk="bf16", bias=rng.choice(["bf16", "f32"]), mask="random", pad=0)
    if kind == "fp8":
        S = _log(rng, 128, 1536)
        return dict(kind="op", B1=S, B2=4, S=S, D=32, qk="fp8", bias="bf16", mask="random", pad=0)
    if kind == "grid":
        return dict(kind="grid", N=_log(rng, 24, 1024), C=rng.choice([128, 128, 128, 64]), H=4,
                    dtype=rng.choice(["bf16", "bf16", "f32"]), transpose=rng.random() < 0.5)
    if kind == "self":
        return dict(kind="self", N=_log(rng, 24, 2048), C=rng.choice([384, 768]), H=16, dtype=rng.choice(["bf16", "bf16", "f32"]))
    S = _log(rng, 48, 448)
    return dict(kind="host", B1=S, B2=4, S=S, D=32, qk="bf16", bias=rng.choice(["bf16", "f32"]), mask="random", pad=0)


_modules = []        # a program keeps the modules it has loaded for as long as it runs

_DTYPE = {"bf16": torch.bfloat16, "f32": torch.float32}


def _key_mask(c, rows, S, g):
    if c["mask"] == "tail":                        # padding tokens behind the sequence
        mask = torch.ones(rows, S, dtype=torch.bool, device="cuda")
        mask[:, S - c["pad"]:] = False
        return mask
    return torch.rand(rows, S, generator=g, device="cuda") >= 0.05


def _quantised(x):
    scale = (x.abs().amax(dim=(0, 2, 3)).clamp_min(1e-12) / 448.0).float()
    return (x / scale.view(1, -1, 1, 1)).to(torch.float8_e4m3fn), scale


def prepare(case, seed):
    c = case
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, std=1.0):
        return torch.randn(*shape, generator=g, device="cuda") * std

    if c["kind"] in ("op", "host"):
        shape = (c["B1"], c["B2"], c["S"], c["D"])
        st = {"kind": c["kind"], "q_scale": None, "k_scale": None}
        if c["qk"] == "fp8":
            st["q"], st["q_scale"] = _quantised(normal(*shape))
            st["k"], st["k_scale"] = _quantised(normal(*shape))
            st["v"] = normal(*shape).to(torch.bfloat16)
        else:
            for name in "qkv":
                st[name] = normal(*shape).to(_DTYPE[c["qk"]])
        st["bias"] = normal(c["B2"], c["S"], c["S"]).to(_DTYPE[c["bias"]])
        st["mask"] = _key_mask(c, c["B1"], c["S"], g)
        if c["kind"] == "host":
            for name in ("q", "k", "v", "bias", "mask"):
                st[name] = st[name].cpu().pin_memory()
        return st

    dtype, C, H, N = _DTYPE[c["dtype"]], c["C"], c["H"], c["N"]
    if c["kind"] == "grid":
        with torch.device("cuda"):
            module = A.GridSelfAttentionCpp(C, H, c["transpose"])
        with torch.no_grad():
            for name, p in module.named_parameters():
                p.copy_(normal(*p.shape, std=C ** -0.5 if p.dim() == 2 else 0.1))
            module.act_norm.weight.add_(1.0)
        module = module.to(dtype).eval()
        _modules.append(module)
        pair = (normal(N, N, C) * 2.0 + 0.25).to(dtype)
        return {"kind": "grid", "module": module, "pair": pair, "mask": torch.rand(N, N, generator=g, device="cuda") >= 0.05}

    weights = [normal(C, C, std=C ** -0.5).to(dtype) for _ in range(4)]      # [in, out]
    mask = torch.ones(N, dtype=torch.bool, device="cuda")
    mask[N - N // 12:] = False
    return {"kind": "self", "x": normal(N, C).to(dtype), "mask": mask, "bias": normal(H, N, N).to(dtype), "weights": weights,
            "q_bias": normal(C, std=0.1).to(dtype), "H": H}


def run(state):
    s = state
    with torch.no_grad():
        if s["kind"] in ("op", "host"):
            return A.dot_product_attention_cpp(s["q"], s["k"], s["v"], s["mask"], s["bias"], q_scale=s["q_scale"], k_scale=s["k_scale"])
        if s["kind"] == "grid":
            return s["module"](s["pair"], s["mask"])
        w_q, w_k, w_v, w_g = s["weights"]
        return A.self_attention_cpp(s["x"], s["mask"], s["bias"], w_q, s["q_bias"], w_k, w_v, w_g, s["H"])


_BYTES = {"bf16": 2, "f32": 4, "fp8": 1}


def work(case):
    c = case
    if c["kind"] in ("op", "host"):
        B1, B2, S, D = c["B1"], c["B2"], c["S"], c["D"]
        qk, v = _BYTES[c["qk"]], 4 if c["qk"] == "f32" else 2
        return {"bytes": B1 * B2 * S * D * (2 * qk + 2 * v) + B2 * S * S * _BYTES[c["bias"]] + B1 * S,
                "flops": 4 * B1 * B2 * S * S * D}
    N, C, H, es = c["N"], c["C"], c["H"], _BYTES[c["dtype"]]
    if c["kind"] == "grid":                          # five C x C projections and the bias projection around the attention
        return {"bytes": 2 * N * N * C * es + N * N + (5 * C * C + H * C + 2 * C) * es,
                "flops": 4 * N * N * N * C + 2 * N * N * C * (5 * C + H)}
    return {"bytes": 2 * N * C * es + H * N * N * es + 4 * C * C * es + N,
            "flops": 4 * N * N * C + 2 * N * C * 4 * C}


def tolerance(case):
    # operands, softmax weights and results are rounded to bf16 (relative 2^-9 each) whatever the
    # caller's type; sums are fp32
    return {"rel": 1e-2}

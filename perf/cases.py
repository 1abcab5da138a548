"""Performance cases: the layers and operators that a prediction, a scoring run or a generation spends its time in.

Every case goes through the modules a program builds (``models.*``) with the kernel implementation switched on, in
bf16, the type all of them run in on a GPU.  Sizes are those of the repository's configurations and benchmarks: pair
stacks of 48 to 1536 tokens, alignments of up to 1024 sequences, samplers of 1 to 5 samples over up to 12768 atoms,
hidden width 4096 for the genomic decoder, 960 to 1152 for the protein encoder.  The one workload with a backward pass
(design by inversion) runs plain PyTorch statements and is left out: no kernel of this package is on its path.

``exact`` restates each path in float64 with torch alone.
"""
import math

import torch
import torch.nn.functional as F

from uplifting_biomolecular_modeling_b200.models import diffusion, evo2, msa, pairformer, plm

BF = torch.bfloat16


# ---------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one Pairformer block on a short chain with a few padding tokens: ~40 launches on little work each
        {"name": "pairformer_block_137", "kind": "pairformer_block", "n": 137, "mask": True},
        # the three operators of the pair track on their own, up to the benchmark's 1536 tokens
        {"name": "trimul_incoming_1021", "kind": "trimul", "n": 1021, "outgoing": False, "mask": True},
        {"name": "triatt_starting_1536", "kind": "triatt", "n": 1536, "starting": True, "mask": False},
        {"name": "transition_1536", "kind": "transition", "n": 1536},
        # the two operators of the MSA track with a full-depth alignment
        {"name": "pair_averaging_1024x768", "kind": "pwa", "s": 1024, "n": 768},
        {"name": "outer_product_1024x768", "kind": "opm", "s": 1024, "n": 768, "full": True},
        # the sampler: two layers of the token transformer and the atom transformer, 5 samples
        {"name": "token_layers_5x1536", "kind": "token_layers", "b": 5, "n": 1536},
        {"name": "atom_layers_5x12768", "kind": "atom_layers", "b": 5, "a": 12768},
        # prefill of the long and the medium convolution operator of the genomic decoder
        {"name": "hyena_long_8192", "kind": "hyena", "op": "hcl", "b": 1, "l": 8192, "d": 4096},
        {"name": "hyena_medium_8192", "kind": "hyena", "op": "hcm", "b": 1, "l": 8192, "d": 4096},
        # one decoding step of a decoder with one block of each operator: the smallest call, host and launches count
        {"name": "decode_step_4096", "kind": "decode", "b": 1, "l": 4096},
        # protein encoder layer on a scoring batch of ragged length
        {"name": "encoder_layer_8x2047", "kind": "encoder", "config": "esmc_300m", "b": 8, "l": 2047},
    ]


def _log(rng, lo, hi, m=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / m)) * m))


def draw(rng):
    kind = rng.choice(["pairformer_block", "trimul", "triatt", "transition", "pwa", "opm", "token_layers",
                       "atom_layers", "hyena", "hyena", "decode", "encoder"])
    flip = lambda: rng.random() < 0.5  # noqa: E731
    if kind == "pairformer_block":
        return {"kind": kind, "n": _log(rng, 48, 400), "mask": flip()}
    if kind == "trimul":
        return {"kind": kind, "n": _log(rng, 128, 1536), "outgoing": flip(), "mask": flip()}
    if kind == "triatt":
        return {"kind": kind, "n": _log(rng, 128, 1400), "starting": flip(), "mask": flip()}
    if kind == "transition":
        return {"kind": kind, "n": _log(rng, 48, 1536)}
    if kind in ("pwa", "opm"):
        c = {"kind": kind, "s": _log(rng, 16, 1024), "n": _log(rng, 64, 768)}
        return {**c, "full": flip()} if kind == "opm" else c
    if kind == "token_layers":
        return {"kind": kind, "b": rng.randint(1, 5), "n": _log(rng, 64, 1536)}
    if kind == "atom_layers":
        return {"kind": kind, "b": rng.randint(1, 5), "a": _log(rng, 512, 12768, 32)}
    if kind == "hyena":
        b = rng.randint(1, 2)
        return {"kind": kind, "op": rng.choice(["hcs", "hcm", "hcl"]), "b": b,
                "l": _log(rng, 200, 16384 // b), "d": rng.choice([1920, 4096])}
    if kind == "decode":
        return {"kind": kind, "b": rng.randint(1, 8), "l": _log(rng, 128, 16384)}
    return {"kind": kind, "config": rng.choice(["esmc_300m", "esmc_600m"]), "b": rng.randint(1, 8),
            "l": _log(rng, 64, 2048)}


# ---------------------------------------------------------------------------------------------- inputs
def _weights(module, gen):
    """Weights of a trained network's scale: matrices keep the variance of their input, norms lie near one."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            r = torch.randn(p.shape, device=p.device, generator=gen)
            if p.dim() >= 2 and "fir" not in name and not name.endswith(("h", "log_poles", "residues", "clade_bias")):
                p.copy_(r / math.sqrt(p.shape[-1]))
            elif name.endswith("log_poles"):
                # decays from a few positions to a few thousand
                u = torch.rand(p.shape, device=p.device, generator=gen) * 3.2 + 0.3
                p.copy_(torch.log1p(-torch.pow(10.0, -u)))
            elif name.endswith(("h", "fir", "residues")):
                p.copy_(r / math.sqrt(p.shape[-1]))
            elif p.dim() == 1 and name.endswith(("weight", "scale", ".D")) or name == "D":
                p.copy_(1.0 + 0.1 * r)
            else:
                p.copy_(0.1 * r)
    module.eval().requires_grad_(False)
    return module


def _make(seed, build, dtype=BF):
    gen = torch.Generator("cuda").manual_seed(seed)
    with torch.device("cuda"):
        m = build()
    return _weights(m.to(dtype), gen), gen


def _randn(gen, *shape, dtype=BF):
    return torch.randn(shape, device="cuda", generator=gen).to(dtype)


def _tokens(n, padded):
    """Keep-mask [1, n] of the tokens: a twentieth of them padding at the end."""
    keep = torch.ones(1, n, device="cuda", dtype=BF)
    if padded:
        keep[:, n - max(1, n // 20):] = 0
    return keep


def _decoder():
    return evo2.StripedHyena2(evo2.replace(evo2.CONFIGS["evo2_7b"], n_layers=4, attn_layers=(3,)))


def _inputs(case, seed):
    """Module with plain weights, generator-made inputs."""
    k = case["kind"]
    if k == "pairformer_block":
        m, g = _make(seed, pairformer.PairformerLayer)
        keep = _tokens(case["n"], case["mask"])
        mask = keep if case["mask"] else None
        return {"m": m, "s": _randn(g, 1, case["n"], 384), "z": _randn(g, 1, case["n"], case["n"], 128), "mask": mask,
                "pair_mask": None if mask is None else keep[:, :, None] * keep[:, None, :]}
    if k in ("trimul", "triatt"):
        build = (lambda: pairformer.TriangleMultiplication(128, case["outgoing"])) if k == "trimul" else \
            (lambda: pairformer.TriangleAttention(starting=case["starting"]))
        m, g = _make(seed, build)
        keep = _tokens(case["n"], case["mask"])
        return {"m": m, "z": _randn(g, 1, case["n"], case["n"], 128),
                "mask": keep[:, :, None] * keep[:, None, :] if case["mask"] else None}
    if k == "transition":
        m, g = _make(seed, lambda: pairformer.Transition(128, 512))
        return {"m": m, "z": _randn(g, 1, case["n"], case["n"], 128)}
    if k == "pwa":
        m, g = _make(seed, msa.PairWeightedAveraging)
        return {"m": m, "x": _randn(g, 1, case["s"], case["n"], 64), "z": _randn(g, 1, case["n"], case["n"], 128),
                "mask": torch.ones(1, case["n"], case["n"], device="cuda", dtype=BF)}
    if k == "opm":
        m, g = _make(seed, msa.OuterProductMean)
        mask = torch.ones(1, case["s"], case["n"], device="cuda", dtype=BF)
        if not case["full"]:        # sequences that cover a part of the target
            mask = (torch.rand(mask.shape, device="cuda", generator=g) < 0.9).to(BF)
        m.full_mask = case["full"]
        return {"m": m, "x": _randn(g, 1, case["s"], case["n"], 64), "mask": mask}
    if k == "token_layers":
        m, g = _make(seed, lambda: diffusion.DiffusionTransformer(2, 768, 768, 16))
        n = case["n"]
        return {"m": m, "a": _randn(g, case["b"], n, 768), "s": _randn(g, 1, n, 768),
                "bias": [_randn(g, 16, n, (n + 7) // 8 * 8) for _ in range(2)]}
    if k == "atom_layers":
        m, g = _make(seed, lambda: diffusion.DiffusionTransformer(3, 128, 128, 4))
        n = case["a"]
        return {"m": m, "a": _randn(g, case["b"], n, 128), "c": _randn(g, 1, n, 128),
                "bias": [_randn(g, 1, 4, n // 32, 32, 128) for _ in range(3)]}
    if k == "hyena":
        cfg = evo2.CONFIGS["evo2_7b" if case["d"] == 4096 else "evo2_1b"]
        m, g = _make(seed, lambda: evo2.HyenaOperator(cfg, case["op"]))
        return {"m": m, "x": _randn(g, case["b"], case["l"], case["d"])}
    if k == "decode":
        m, g = _make(seed, _decoder)
        b, c = case["b"], m.cfg
        states = []
        for i in range(4):
            kind = c.layer_kind(i)
            if kind == "attn":
                st = {n: _randn(g, b, case["l"], c.n_heads, 128) for n in ("k", "v")}
            else:
                st = {"fir_tail": _randn(g, b, c.fir_len - 1, 3 * c.d_model)}
                if kind == "hcl":
                    st["poles"] = _randn(g, b, c.d_model, c.state_dim, dtype=torch.float32)
                else:
                    st["inner_tail"] = _randn(g, b, (c.short_len if kind == "hcs" else c.medium_len) - 1, c.d_model)
            states.append(st)
        return {"m": m, "token": torch.randint(0, c.vocab, (b, 1), device="cuda", generator=g), "states": states}
    cfg = plm.CONFIGS[case["config"]]
    m, g = _make(seed, lambda: plm.EncoderBlock(cfg, 0))
    pos = torch.arange(case["l"], device="cuda", dtype=torch.int32).repeat(case["b"])
    return {"m": m, "cfg": cfg, "x": _randn(g, case["b"], case["l"], cfg.d_model), "pos": pos}


def prepare(case, seed):
    st = _inputs(case, seed)
    st["kind"], m = case["kind"], st["m"]
    if st["kind"] in ("hyena", "encoder"):
        m.impl = "fused"
    elif st["kind"] == "decode":
        m.set_impl("fused")
        m.make_static_states(st["states"], case["l"] + 64)
        st["keep"] = [{n: t.clone() for n, t in s.items() if n in ("fir_tail", "inner_tail", "poles")}
                      for s in st["states"]]
    else:
        pairformer.set_impl(m, "fused")
    if st["kind"] == "token_layers":        # pair biases of a prediction's 200 steps, made once by DiffusionModule
        st["planes"] = [pairformer.BiasPlanes((b.float() * 1.4426950408889634).to(BF)[:, :, :case["n"]])
                        for b in st["bias"]]
    if st["kind"] == "atom_layers":
        st["planes"] = [diffusion.WindowBias(b) for b in st["bias"]]
        st["hoisted"] = [layer.hoist(st["c"]) for layer in m.layers]
    return st


@torch.no_grad()
def run(st):
    k, m = st["kind"], st["m"]
    if k == "pairformer_block":
        return m(st["s"], st["z"], st["mask"], st["pair_mask"])
    if k in ("trimul", "triatt"):
        return m(st["z"], st["mask"], residual=True)
    if k == "transition":
        return m(st["z"], residual=True)
    if k == "pwa":
        return m(st["x"], st["z"], st["mask"])
    if k == "opm":
        return m(st["x"], st["mask"])
    if k == "token_layers":                 # the conditioning changes with the noise level: projected every step
        return m(st["a"], st["s"], st["planes"], None, multiplicity=st["a"].shape[0], hoisted=m.hoist_all(st["s"]))
    if k == "atom_layers":
        return m(st["a"], st["c"], st["planes"], hoisted=st["hoisted"], window=(32, 128))
    if k == "hyena":
        state = {}
        return m(st["x"], state, evo2.fused_linear), state
    if k == "decode":                       # the same step from the same state every time
        for s, keep in zip(st["states"], st["keep"]):
            for n, t in keep.items():
                s[n].copy_(t)
        logits = m.step(st["token"], st["states"])
        return logits, [{n: s[n] for n in keep} for s, keep in zip(st["states"], st["keep"])]
    return m(st["x"], st["pos"])


# ---------------------------------------------------------------------------------------------- cost and tolerance
def work(case):
    """Operands read once, results written once; multiply-adds of the contractions as two operations each."""
    k = case["kind"]
    if k in ("pairformer_block", "trimul", "triatt", "transition"):
        n = case["n"]
        p = n * n
        z = 2 * p * 128 * 2
        mul = 2 * p * 128 * (512 + 256) + 2 * 128 * n ** 3
        att = 2 * p * 128 * (512 + 4 + 128) + 4 * n ** 3 * 128
        tra = 2 * p * 128 * 512 * 3
        if k != "pairformer_block":
            return {"bytes": z, "flops": {"trimul": mul, "triatt": att, "transition": tra}[k]}
        single = 2 * n * 384 * (5 * 384 + 3 * 1536) + 4 * n * n * 384 + 2 * p * 128 * 16
        return {"bytes": z + 2 * n * 384 * 2 + 2 * (128 * 128 * 30 + 384 * 384 * 17), "flops": 2 * mul + 2 * att + tra + single}
    if k == "pwa":
        s, n = case["s"], case["n"]
        return {"bytes": 2 * s * n * 64 * 2 + n * n * 130 * 2,
                "flops": 2 * s * n * 64 * 768 + 2 * n * n * 128 * 8 + 2 * s * n * n * 256}
    if k == "opm":
        s, n = case["s"], case["n"]
        return {"bytes": s * n * 65 * 2 + n * n * 128 * 2,
                "flops": 2 * s * n * 64 * 64 + 2 * s * (n * 32) ** 2 + 2 * n * n * 1024 * 128}
    if k == "token_layers":
        b, n, c = case["b"], case["n"], 768
        flops = 2 * (2 * n * c * 6 * c + 2 * b * n * c * c * (5 + 8) + 4 * b * n * n * c)
        return {"bytes": 2 * b * n * c * 2 + n * c * 2 + 2 * 16 * n * n * 2 + 2 * 2 * c * c * 19, "flops": flops}
    if k == "atom_layers":
        b, n, c = case["b"], case["a"], 128
        flops = 3 * (2 * b * n * c * c * (5 + 8) + 4 * b * n * 128 * c)
        return {"bytes": 2 * b * n * c * 2 + 3 * (6 * n * c * 2 + 4 * n * 128 * 2 + 2 * c * c * 13), "flops": flops}
    if k == "hyena":
        t, d = case["b"] * case["l"], case["d"]
        taps = {"hcs": 7, "hcm": 128, "hcl": 32}[case["op"]]
        return {"bytes": 2 * t * d * 2 + 4 * d * d * 2, "flops": 2 * t * d * 4 * d + 2 * t * d * (taps + 9)}
    if k == "decode":
        b, l = case["b"], case["l"]
        w = 4 * (4 * 4096 * 4096 + 3 * 4096 * 11008) + 512 * 4096
        return {"bytes": 2 * w + 2 * b * l * 4096 * 2 + b * 4096 * (16 * 8 + 2 * 2 * 6 * 3 + 2 * 2 * 133),
                "flops": 2 * b * w + 4 * b * l * 4096}
    cfg = plm.CONFIGS[case["config"]]
    t, d = case["b"] * case["l"], cfg.d_model
    w = 4 * d * d + 3 * d * cfg.ffn
    return {"bytes": 2 * t * d * 2 + 2 * w, "flops": 2 * t * w + 4 * t * case["l"] * d}


# About four times the measured distance to float64 (bf16 operands of every product, bf16 intermediates): 0.0025 for the
# triangle multiplication, 0.0017 triangle attention, 0.0022 transition, 0.0036 pair averaging, 0.0021 outer product,
# 0.005 the sampler's layers and the convolution operators, 0.0095 the logits of a decoding step, 0.0032 the encoder
# layer.  The block's rows of padding tokens attend to nothing and have no defined value; the bound is that of the others.
REL = {"pairformer_block": 0.015, "trimul": 0.01, "triatt": 0.007, "transition": 0.009, "pwa": 0.015, "opm": 0.009,
       "token_layers": 0.02, "atom_layers": 0.02, "hyena": 0.02, "decode": 0.04, "encoder": 0.013}


def tolerance(case):
    return {"rel": REL[case["kind"]]}


# ---------------------------------------------------------------------------------------------- float64 statements
def _d(t):
    return None if t is None else t.double()


def _lin(x, layer):
    return F.linear(x, _d(layer.weight), _d(layer.bias))


def _ln(x, layer):
    return F.layer_norm(x, (x.shape[-1],), _d(layer.weight), _d(layer.bias), layer.eps)


def _rows(f, x, *more, block=1 << 18):
    """f over blocks of rows, the results in one tensor."""
    flat = x.reshape(-1, x.shape[-1])
    return torch.cat([f(flat[i:i + block], *(t[i:i + block] for t in more)) for i in range(0, flat.shape[0], block)])


def _x_transition(m, x):
    f = lambda r: _lin(F.silu(_lin(_ln(r, m.norm), m.fc1)) * _lin(_ln(r, m.norm), m.fc2), m.fc3)  # noqa: E731
    return _rows(f, x).view_as(x)


def _x_trimul(m, z, mask):
    n = z.shape[0]
    zn = _ln(z, m.norm_in)
    planes = []
    for h in range(2):
        w = slice(128 * h, 128 * h + 128)
        p = F.linear(zn, _d(m.p_in.weight)[w]) * torch.sigmoid(F.linear(zn, _d(m.g_in.weight)[w]))
        planes.append((p if mask is None else p * mask[..., None]).permute(2, 0, 1))
    a, b = planes
    x = torch.empty(n, n, 128, dtype=torch.float64, device=z.device)
    for c in range(128):
        x[..., c] = a[c] @ b[c].T if m.outgoing else a[c].T @ b[c]
    del planes, a, b
    return z + _lin(_ln(x, m.norm_out), m.p_out) * torch.sigmoid(_lin(zn, m.g_out))


def _x_attend(q, k, v, bias):
    """[..., H, n, D] with bias broadcast to [..., H, n, n]."""
    return torch.softmax(q @ k.transpose(-1, -2) / math.sqrt(q.shape[-1]) + bias, -1) @ v


def _x_triatt(m, z, mask):
    n, a = z.shape[0], m.mha
    x = z if m.starting else z.transpose(0, 1)
    keep = None if mask is None else (mask if m.starting else mask.T)
    xn = _ln(x, m.layer_norm)
    bias = F.linear(xn, _d(m.linear.weight)).permute(2, 0, 1)
    upd = torch.empty(n, n, 128, dtype=torch.float64, device=z.device)
    for i in range(0, n, 8):
        r = xn[i:i + 8]
        q, k, v = (_lin(r, w).view(-1, n, 4, 32).transpose(1, 2) for w in (a.linear_q, a.linear_k, a.linear_v))
        b = bias if keep is None else bias + ((keep[i:i + 8] - 1) * 1e30)[:, None, None, :]
        o = _x_attend(q, k, v, b).transpose(1, 2).reshape(-1, n, 128)
        upd[i:i + 8] = _lin(o * torch.sigmoid(_lin(r, a.linear_g)), a.linear_o)
    return z + (upd if m.starting else upd.transpose(0, 1))


def _x_apb(m, s, bias):
    """s: [B, n, c]; bias: [H, n, n] (mask included)."""
    b, n, c = s.shape
    q, k, v = (_lin(s, w).view(b, n, m.heads, -1).transpose(1, 2) for w in (m.proj_q, m.proj_k, m.proj_v))
    o = torch.stack([_x_attend(q[i], k[i], v[i], bias) for i in range(b)])
    return _lin(o.transpose(1, 2).reshape(b, n, c) * torch.sigmoid(_lin(s, m.proj_g)), m.proj_o)


def _x_adaln(m, a, s):
    sn = _ln(s, m.s_norm)
    return torch.sigmoid(_lin(sn, m.s_scale)) * F.layer_norm(a, (a.shape[-1],)) + _lin(sn, m.s_bias)


def _x_dit_layer(m, a, s, attend):
    a = a + torch.sigmoid(_lin(s, m.output_projection_linear)) * attend(m.pair_bias_attn, _x_adaln(m.adaln, a, s))
    t = m.transition
    x = _x_adaln(t.adaln, a, s)
    val, gate = _lin(x, t.swish_gate[0]).chunk(2, -1)
    u = F.silu(gate) * val * _lin(x, t.a_to_b)
    return a + torch.sigmoid(_lin(s, t.output_projection[0])) * _lin(u, t.b_to_a)


def _x_windows(m, x, bias):
    """Windows of 32 queries over the 128 keys around them.  x: [B, A, 128]; bias: [H, A / 32, 32, 128]."""
    b, n, _ = x.shape
    at = torch.arange(n // 32, device=x.device)[:, None] * 32 + torch.arange(128, device=x.device) - 48
    out_of = ((at < 0) | (at >= n))[:, None, :]
    out = torch.empty_like(x)
    for i in range(b):
        q, k, v = (_lin(x[i], w).view(n, 4, 32).transpose(0, 1) for w in (m.proj_q, m.proj_k, m.proj_v))
        k, v = (t[:, at.clamp(0, n - 1)] for t in (k, v))
        o = _x_attend(q.view(4, -1, 32, 32), k, v, bias.masked_fill(out_of, -math.inf))
        out[i] = _lin(o.view(4, n, 32).transpose(0, 1).reshape(n, 128) * torch.sigmoid(_lin(x[i], m.proj_g)), m.proj_o)
    return out


def _x_fir(x, h):
    """Causal depthwise convolution over dimension 1 by shifted sums.  x: [B, L, C]; h: [C, K]."""
    y = x * h[:, 0]
    for j in range(1, min(h.shape[1], x.shape[1])):
        y[:, j:] += x[:, :-j] * h[:, j]
    return y


def _x_hyena(m, x):
    z = _lin(x, m.in_proj)
    x1, x2, v = _x_fir(z, _d(m.fir)).chunk(3, -1)
    u = x1 * v
    state = {"fir_tail": z[:, -(m.fir.shape[1] - 1):].clone()}
    L = x.shape[1]
    if m.kind == "hcl":
        y = torch.empty_like(u)
        poles = u.new_empty(*u.shape[::2], m.log_poles.shape[1])
        t = torch.arange(L, device=x.device, dtype=torch.float64)
        for c in range(0, m.d, 64):
            lam = torch.exp(_d(m.log_poles[c:c + 64]))[..., None] ** t
            h = torch.einsum("cs,cst->ct", _d(m.residues[c:c + 64]), lam)
            f = torch.fft.rfft(u[:, :, c:c + 64].transpose(1, 2), n=2 * L) * torch.fft.rfft(h, n=2 * L)
            y[:, :, c:c + 64] = torch.fft.irfft(f, n=2 * L)[..., :L].transpose(1, 2)
            poles[:, c:c + 64] = torch.einsum("blc,csl->bcs", u[:, :, c:c + 64], lam.flip(-1))
        state["poles"] = poles
    else:
        y = _x_fir(u, _d(m.h))
        k = m.h.shape[1] - 1
        state["inner_tail"] = F.pad(u, (0, 0, max(0, k - L), 0))[:, -k:].clone()
    return _lin(x2 * (y + u * _d(m.D)), m.out_proj), state


def _x_rms(x, m):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + m.eps) * _d(m.scale)


def _x_rotary(x, pos, rot, base=10000.0):
    """x: [..., L, H, D]; rotates interleaved pairs of the first rot dimensions."""
    inv = base ** (-torch.arange(0, rot, 2, device=x.device, dtype=torch.float64) / rot)
    ang = pos.double()[:, None, None] * inv
    a, b = x[..., 0:rot:2], x[..., 1:rot:2]
    r = torch.stack([a * ang.cos() - b * ang.sin(), a * ang.sin() + b * ang.cos()], -1).flatten(-2)
    return torch.cat([r, x[..., rot:]], -1)


def _x_decode(m, token, states, pos):
    x = _d(m.embedding.weight)[token]                                    # [B, 1, d]
    out = []
    for blk, st in zip(m.blocks, states):
        n, mix = _x_rms(x, blk.pre_norm), blk.mixer
        new = {}
        if blk.kind == "attn":
            q, k, v = _lin(n, mix.qkv).view(n.shape[0], 1, 3, -1, 128).unbind(2)
            at = torch.tensor([pos], device=x.device)
            k = torch.cat([_d(st["k"][:, :pos]), _x_rotary(k, at, 128)], 1).transpose(1, 2)
            v = torch.cat([_d(st["v"][:, :pos]), v], 1).transpose(1, 2)
            o = _x_attend(_x_rotary(q, at, 128).transpose(1, 2), k, v, 0.0).transpose(1, 2).flatten(-2)
        else:
            z = torch.cat([_d(st["fir_tail"]), _lin(n, mix.in_proj)], 1)
            x1, x2, v = _x_fir(z, _d(mix.fir))[:, -1:].chunk(3, -1)
            u = x1 * v
            new["fir_tail"] = z[:, 1:]
            if blk.kind == "hcl":
                p = _d(st["poles"]) * torch.exp(_d(mix.log_poles)) + u[:, 0, :, None]
                y = (p * _d(mix.residues)).sum(-1)[:, None]
                new["poles"] = p
            else:
                t = torch.cat([_d(st["inner_tail"]), u], 1)
                y = _x_fir(t, _d(mix.h))[:, -1:]
                new["inner_tail"] = t[:, 1:]
            o = x2 * (y + u * _d(mix.D))
        x = x + _lin(o, mix.out_proj)
        n = _x_rms(x, blk.post_norm)
        x = x + _lin(F.silu(_lin(n, blk.mlp.l1)) * _lin(n, blk.mlp.l2), blk.mlp.l3)
        out.append({k: new[k] for k in ("fir_tail", "inner_tail", "poles") if k in new})
    return F.linear(_x_rms(x, m.norm), _d(m.embedding.weight)), out


def _x_encoder(m, cfg, x, pos):
    b, l, d = x.shape
    q, k, v = _lin(_ln(x, m.ln1), m.wqkv).chunk(3, -1)
    p = pos[:l]
    q, k = (_x_rotary(_ln(t, ln).view(b, l, cfg.heads, -1), p, cfg.rot).transpose(1, 2)
            for t, ln in ((q, m.q_ln), (k, m.k_ln)))
    v = v.view(b, l, cfg.heads, -1).transpose(1, 2)
    o = torch.stack([_x_attend(q[i], k[i], v[i], 0.0) for i in range(b)]).transpose(1, 2).reshape(b, l, d)
    x = x + _lin(o, m.wo) / m.scale
    f = lambda r: _lin(F.silu(_lin(r, m.w1).chunk(2, -1)[0]) * _lin(r, m.w1).chunk(2, -1)[1], m.w2)  # noqa: E731
    return x + _rows(f, _ln(x, m.ln2), block=4096).view_as(x) / m.scale


@torch.no_grad()
def exact(case, seed):
    st = _inputs(case, seed)
    k, m = st["kind"] if "kind" in st else case["kind"], st["m"]
    if k == "transition":
        z = st["z"].double()
        return z + _x_transition(m, z)
    if k in ("trimul", "triatt"):
        f = _x_trimul if k == "trimul" else _x_triatt
        return f(m, _d(st["z"])[0], None if st["mask"] is None else _d(st["mask"])[0])[None]
    if k == "pairformer_block":
        z, s = _d(st["z"])[0], _d(st["s"])
        pm = None if st["pair_mask"] is None else _d(st["pair_mask"])[0]
        z = _x_trimul(m.tri_mul_in, _x_trimul(m.tri_mul_out, z, pm), pm)
        z = _x_triatt(m.tri_att_end, _x_triatt(m.tri_att_start, z, pm), pm)
        z = z + _x_transition(m.transition_z, z)
        at = m.attention
        bias = _lin(_ln(z, at.proj_z[0]), at.proj_z[1]).permute(2, 0, 1)
        if st["mask"] is not None:
            bias = bias + (_d(st["mask"])[0] - 1) * 1e30
        s = s + _x_apb(at, _ln(s, m.pre_norm_s), bias)
        return s + _x_transition(m.transition_s, s), z[None]
    if k == "pwa":
        x, z = _d(st["x"])[0], _d(st["z"])[0]
        w = torch.softmax(_lin(_ln(z, m.norm_z), m.proj_z).permute(2, 0, 1), -1)          # [H, i, j]
        out = torch.empty_like(x)
        for i in range(0, x.shape[0], 64):
            n = _ln(x[i:i + 64], m.norm_m)
            v = _lin(n, m.proj_m).view(*n.shape[:2], m.heads, -1)
            o = torch.einsum("hij,sjhc->sihc", w, v).flatten(-2)
            out[i:i + 64] = _lin(torch.sigmoid(_lin(n, m.proj_g)) * o, m.proj_o)
        return out[None]
    if k == "opm":
        x, mask = _d(st["x"])[0], _d(st["mask"])[0]
        n = _ln(x, m.norm)
        a, b = (_lin(n, w) * mask[..., None] for w in (m.proj_a, m.proj_b))
        N = x.shape[1]
        out = torch.empty(N, N, 128, dtype=torch.float64, device=x.device)
        cnt = (mask.T @ mask).clamp(min=1.0)
        for i in range(0, N, 32):
            t = torch.einsum("sic,sjd->ijcd", a[:, i:i + 32], b).flatten(-2) / cnt[i:i + 32, :, None]
            out[i:i + 32] = _lin(t, m.proj_o)
        return out[None]
    if k in ("token_layers", "atom_layers"):
        a = _d(st["a"])
        for layer, b in zip(m.layers, st["bias"]):
            if k == "token_layers":
                a = _x_dit_layer(layer, a, _d(st["s"]), lambda at, x: _x_apb(at, x, _d(b)[:, :, :case["n"]]))
            else:
                a = _x_dit_layer(layer, a, _d(st["c"]), lambda at, x: _x_windows(at, x, _d(b)[0]))
        return a
    if k == "hyena":
        return _x_hyena(m, _d(st["x"]))
    if k == "decode":
        return _x_decode(m, st["token"], st["states"], case["l"])
    return _x_encoder(m, st["cfg"], _d(st["x"]), st["pos"])

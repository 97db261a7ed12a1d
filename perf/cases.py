"""The work that users of this framework have it do, as cases that can be timed and compared.

Two kinds of program use it: one that runs prompts to logits (scoring, the first step of a generation),
and one that decodes, token by token, behind a prompt. Both exist for the three decoders (Complexity with
token-routed experts and mu guidance; Pimezen; Rugedra) and the token-routed layer is used by itself too.

  prompt     model(ids).logits for a batch of prompts, ids from pinned host memory; "graph": the same through
             PrefillGraph, as a server does that always sees the same shape
  portions   a prompt in portions behind one another on a state from the model's pool (chunked prefill)
  decode     DecodeGraph: `steps` given tokens (replay, scoring of a continuation) behind `cached` ones, the
             logits of every step kept; the cached tokens are those of a prompt run in advance
  layer      TokenRoutedMLP.forward on the activations of a batch

Weights are random, at the scales of the models' own initialisation or of unit-variance activations.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

VOCAB = 32000
GRID = {"bf16": torch.bfloat16, "f32": torch.float32}

# ------------------------------------------------------------------------------------------- sizes
# (hidden, intermediate, layers, query heads, key heads, experts): the presets of ComplexityConfig and the 18-layer
# model of the README's parity figures
COMPLEXITY = {"tiny": (256, 704, 6, 4, 2, 4), "small": (512, 1408, 8, 8, 4, 4), "150m": (768, 2048, 12, 12, 4, 4),
              "readme": (768, 2048, 18, 12, 4, 4), "1b": (2048, 5632, 24, 16, 8, 8)}
# the two widths that bench.py has, and one whose sizes no power of two divides
PIMEZEN = {"w600": dict(width=600, layers=4, heads=6, kv=2, dim=40, vdim=56, window=300, keep=5, rheads=3, rdim=36,
                        rvdim=52, ff=1000),
           "w1024": dict(width=1024, layers=8, heads=8, kv=4, dim=128, vdim=128, window=512, keep=4, rheads=4, rdim=128,
                         rvdim=128, ff=2816),
           "w2048": dict(width=2048, layers=8, heads=16, kv=8, dim=128, vdim=128, window=1024, keep=4, rheads=8, rdim=128,
                         rvdim=128, ff=5632)}
RUGEDRA = {"w600": dict(width=600, layers=4, heads=6, dim=40, rot=24, vdim=56, rank=104, dheads=6, dkv=3, ddim=36, dvdim=52,
                        conv=3, inner=20, experts=12, groups=4, keep=2, top=3, ff=1000, mff=200),
           "w1024": dict(width=1024, layers=8, heads=8, dim=128, rot=64, vdim=128, rank=512, dheads=8, dkv=8, ddim=128,
                         dvdim=128, conv=4, inner=128, experts=32, groups=8, keep=4, top=4, ff=2816, mff=704),
           "w2048": dict(width=2048, layers=8, heads=16, dim=128, rot=64, vdim=128, rank=512, dheads=16, dkv=16, ddim=128,
                         dvdim=128, conv=4, inner=128, experts=64, groups=8, keep=4, top=8, ff=5632, mff=704)}
TAU, LIMIT, EPS, BRANCH, MULT, ROT_BASE, POSITIONS = 16.0, 7.0, 1e-6, 0.7, 0.5, 1e4, 8192
LATENT_EVERY = 4            # every fourth Rugedra layer, the first included, is latent attention; layer 0 is dense


def _case(name, kind, family, size, batch, seq, dtype="bf16", cached=0, steps=0, portion=0, graph=False):
    return {"name": name, "kind": kind, "family": family, "size": size, "dtype": dtype, "batch": batch, "seq": seq,
            "cached": cached, "steps": steps, "portion": portion, "graph": graph}


def listed():
    return [
        # one short question to a small model, called as it comes: launches and latency
        _case("complexity_150m_prompt_1x37", "prompt", "complexity", "150m", 1, 37),
        # a server's fixed shape on the README's model
        _case("complexity_readme_prompt_4x512", "prompt", "complexity", "readme", 4, 512, graph=True),
        # the headline: the 1B-class model on 65 536 tokens
        _case("complexity_1b_prompt_32x2048", "prompt", "complexity", "1b", 32, 2048),
        # one user's answer from a small model: a step is as short as steps get
        _case("complexity_150m_decode_1", "decode", "complexity", "150m", 1, 1, cached=301, steps=16),
        # a server's decode batch on the 1B-class model
        _case("complexity_1b_decode_32", "decode", "complexity", "1b", 32, 1, cached=2048, steps=16),
        # the token-routed layer by itself, at the size of its isolated benchmark
        _case("routed_layer_16384", "layer", "layer", "e8_h2048_i5632", 8, 2048),
        # prompts of the window / linear attention decoder
        _case("pimezen_w2048_prompt_8x2048", "prompt", "pimezen", "w2048", 8, 2048),
        # its decode batch, with the window full
        _case("pimezen_w1024_decode_32", "decode", "pimezen", "w1024", 32, 1, cached=1100, steps=16),
        # 32-bit storage (evaluation runs): a ragged prompt
        _case("pimezen_w1024_f32_prompt_2x509", "prompt", "pimezen", "w1024", 2, 509, dtype="f32"),
        # prompts of the latent attention / delta rule decoder
        _case("rugedra_w2048_prompt_8x2048", "prompt", "rugedra", "w2048", 8, 2048),
        # the same decoder fed in portions, as a server does that mixes prompts with decoding; ragged
        _case("rugedra_w1024_portions_4x1000", "portions", "rugedra", "w1024", 4, 1000, portion=150),
        # its decode batch
        _case("rugedra_w2048_decode_64", "decode", "rugedra", "w2048", 64, 1, cached=1500, steps=16),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """Prompts of 16 to 65 536 tokens in all, decode batches of 1 to 64, every model and storage type above."""
    kind = rng.choice(["prompt", "prompt", "prompt", "portions", "decode", "decode", "layer"])
    if kind == "layer":
        seq = _log(rng, 16, 2048)
        c = _case("", kind, "layer", rng.choice(["e8_h2048_i5632", "e8_h2048_i704", "e4_h768_i512"]), _log(rng, 1, 8), seq)
    else:
        family = rng.choice(["complexity", "pimezen", "rugedra"] if kind != "portions" else ["pimezen", "rugedra"])
        size = rng.choice(sorted({"complexity": COMPLEXITY, "pimezen": PIMEZEN, "rugedra": RUGEDRA}[family]))
        dtype = "f32" if family != "complexity" and size != "w2048" and rng.random() < 0.25 else "bf16"
        if kind == "decode":
            c = _case("", kind, family, size, _log(rng, 1, 64 if dtype == "bf16" else 8), 1, dtype, cached=_log(rng, 32, 2048),
                      steps=rng.randint(4, 16))
        else:
            most = 65536 if family == "complexity" else 16384 if dtype == "bf16" else 2048
            seq = _log(rng, 16, 2048)
            batch = _log(rng, 1, max(1, min(32, most // seq)))
            c = _case("", kind, family, size, batch, seq, dtype, portion=_log(rng, 16, 512) if kind == "portions" else 0,
                      graph=kind == "prompt" and rng.random() < 0.4)
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------- weights
def _layer_sizes(case):
    e, h, i = (int(x[1:]) for x in case["size"].split("_"))
    return e, h, i


def _latent(i):
    return i % LATENT_EVERY == 0


class _Draws:
    """Random tensors on the GPU in the case's storage type, in a fixed order."""

    def __init__(self, case, seed):
        self.g = torch.Generator(device="cuda").manual_seed(7919 * int(seed) + 11)
        self.dtype = GRID[case["dtype"]]

    def normal(self, *shape, std=1.0):
        return torch.empty(shape, device="cuda").normal_(0.0, std, generator=self.g).to(self.dtype)

    def lean(self, rows, cols):
        """Projections of queries and keys that lean the same way, as in a trained recurrent head: a token's own part of
        the result is then not noise around zero, which the head norm behind it would blow up at the first tokens."""
        q = torch.empty(rows, cols, device="cuda").normal_(0.0, cols ** -0.5, generator=self.g)
        k = torch.empty(rows, cols, device="cuda").normal_(0.0, cols ** -0.5, generator=self.g)
        return q.to(self.dtype), (0.6 * q + 0.8 * k).to(self.dtype)

    def uniform(self, lo, hi, *shape):
        return torch.empty(shape, device="cuda").uniform_(lo, hi, generator=self.g).to(self.dtype)

    def lin(self, rows, cols, gain=1.0):
        return self.normal(rows, cols, std=gain * cols ** -0.5)

    def near(self, at, *shape):
        return (at + 0.1 * torch.empty(shape, device="cuda").normal_(generator=self.g)).to(self.dtype)


def _zipf(vocab):
    p = torch.arange(1, vocab + 1, dtype=torch.float64).pow(-1.1)
    return (p / p.sum()).float()


def _ids(case, seed, tokens):
    g = torch.Generator(device="cuda").manual_seed(104729 * int(seed) + 3)
    u = torch.rand(case["batch"], tokens, device="cuda", dtype=torch.float64, generator=g)
    return torch.searchsorted(_zipf(VOCAB).double().cumsum(0).cuda(), u).clamp(max=VOCAB - 1)


_TABLES = {}


def _table(experts):
    """The routing table for the frequencies of the ids: tokens in order of frequency, each to the lightest expert."""
    if experts not in _TABLES:
        freq, load, table = _zipf(VOCAB).tolist(), [0.0] * experts, [0] * VOCAB
        for t in range(VOCAB):                       # the frequencies fall with the token id
            e = min(range(experts), key=load.__getitem__)
            table[t] = e
            load[e] += freq[t]
        _TABLES[experts] = torch.tensor(table)
    return _TABLES[experts]


def _routed_weights(d, p, hidden, inner, experts, out_std):
    return {p + "gate_proj_w": d.normal(experts, hidden, inner, std=0.02), p + "up_proj_w": d.normal(experts, hidden, inner, std=0.02),
            p + "down_proj_w": d.normal(experts, inner, hidden, std=out_std), p + "shared_gate.weight": d.normal(inner, hidden, std=0.02),
            p + "shared_up.weight": d.normal(inner, hidden, std=0.02), p + "shared_down.weight": d.normal(hidden, inner, std=out_std)}


def _complexity_weights(case, seed):
    d = _Draws(case, seed)
    H, I, L, hq, hkv, E = COMPLEXITY[case["size"]]
    D, res = H // hq, 0.02 / (2 * L) ** 0.5
    w = {"embed_tokens.weight": d.normal(VOCAB, H, std=0.02), "norm.weight": d.near(1, H), "mu_init": d.normal(1, 1, H, std=0.1)}
    for i in range(L):
        p = f"layers.{i}."
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = d.near(1, H), d.near(1, H)
        for n, rows in (("q_proj", hq), ("k_proj", hkv), ("v_proj", hkv), ("mu_to_q", hq), ("mu_to_k", hkv), ("mu_to_v", hkv)):
            w[f"{p}self_attn.{n}.weight"] = d.normal(rows * D, H, std=0.02)
        w[p + "self_attn.o_proj.weight"] = d.normal(H, hq * D, std=res)
        w[p + "self_attn.q_norm.weight"], w[p + "self_attn.k_norm.weight"] = d.near(1, D), d.near(1, D)
        w.update(_routed_weights(d, p + "mlp.", H, I // E, E, res))
        w[p + "mu_guidance.mu"], w[p + "mu_guidance.mu_proj.weight"] = d.near(1, H), d.normal(H, H, std=0.02)
    return w


def _pimezen_weights(case, seed):
    d, z = _Draws(case, seed), PIMEZEN[case["size"]]
    W, H, G, R = z["width"], z["heads"], z["kv"], z["rheads"]
    w = {"embed_tokens.weight": d.normal(VOCAB, W, std=0.5), "norm.weight": d.near(0, W)}
    for i in range(z["layers"]):
        p = f"layers.{i}."
        a, b = p + "mixers.branches.left.", p + "mixers.branches.right."
        w[p + "norm1.weight"], w[p + "norm2.weight"] = d.near(0, W), d.near(0, W)
        w[p + "ls1"], w[p + "ls2"] = d.near(0.5, W), d.near(0.5, W)
        w[a + "q_proj.weight"], w[a + "k_proj.weight"] = d.lin(H * z["dim"], W), d.lin(G * z["dim"], W)
        w[a + "v_proj.weight"], w[a + "o_proj.weight"] = d.lin(G * z["vdim"], W), d.lin(W, H * z["vdim"])
        w[a + "q_norm"], w[a + "k_norm"] = d.near(1, z["dim"]), d.near(1, z["dim"])
        w[a + "r1"], w[a + "r2"] = d.uniform(0.1, 1.0, H), d.uniform(0.1, 1.0, H)
        w[a + "talk"] = (torch.eye(H, device="cuda") + d.normal(H, H, std=0.2)).to(d.dtype)
        w[b + "q_proj.weight"], w[b + "k_proj.weight"] = d.lean(R * z["rdim"], W)
        w[b + "v_proj.weight"], w[b + "g_proj.weight"] = d.lin(R * z["rvdim"], W), d.lin(R * z["rvdim"], W)
        w[b + "o_proj.weight"], w[b + "norm"] = d.lin(W, R * z["rvdim"]), d.near(1, z["rvdim"])
        w[b + "a1_proj.weight"], w[b + "a2_proj.weight"] = d.lin(16, W), d.lin(R * z["rdim"], 16)
        w[b + "a2_proj.bias"] = d.uniform(-1.0, 4.0, R * z["rdim"])
        for n in ("gate", "up"):
            w[f"{p}mlp.{n}_proj.weight"] = d.lin(z["ff"], W)
        w[p + "mlp.down_proj.weight"] = d.lin(W, z["ff"])
    return w


def _rugedra_weights(case, seed):
    d, z = _Draws(case, seed), RUGEDRA[case["size"]]
    W, H, R, D, G = z["width"], z["heads"], z["rank"], z["dheads"], z["dkv"]
    w = {"embed_tokens.weight": d.normal(VOCAB, W), "embed_positions.weight": d.normal(POSITIONS, W, std=0.3),
         "norm.weight": d.near(1, W), "lm_head.weight": d.lin(VOCAB, W)}
    for i in range(z["layers"]):
        p = f"layers.{i}."
        m = p + "mixers.branches.mix."
        w[p + "norm1.weight"], w[p + "norm2.weight"] = d.near(1, W), d.near(1, W)
        if _latent(i):
            w[m + "q_proj.weight"], w[m + "kv_proj.weight"] = d.lin(H * (z["dim"] + z["rot"]), W), d.lin(R + z["rot"], W)
            w[m + "kv_norm"], w[m + "g_proj.weight"] = d.near(1, R), d.lin(H, W)
            w[m + "uk_proj.weight"], w[m + "uv_proj.weight"] = d.lin(H * z["dim"], R), d.lin(H * z["vdim"], R)
            w[m + "o_proj.weight"] = d.lin(W, H * z["vdim"])
        else:
            w[m + "q_proj.weight"], w[m + "k_proj.weight"] = d.lean(G * z["ddim"], W)
            w[m + "v_proj.weight"] = d.lin(D * z["dvdim"], W)
            w[m + "q_conv"] = d.normal(G * z["ddim"], z["conv"], std=0.5)
            w[m + "k_conv"] = (w[m + "q_conv"] + d.normal(G * z["ddim"], z["conv"], std=0.2)).to(d.dtype)
            w[m + "v_conv"] = d.normal(D * z["dvdim"], z["conv"], std=0.5)
            w[m + "b_proj.weight"], w[m + "norm"] = d.lin(D, W), d.near(1, z["dvdim"])
            w[m + "A_log"], w[m + "dt_bias"] = d.uniform(-2.0, 1.0, D), d.uniform(-5.0, 0.0, D * z["ddim"])
            w[m + "a1_proj.weight"], w[m + "a2_proj.weight"] = d.lin(z["inner"], W), d.lin(D * z["ddim"], z["inner"], 0.5)
            w[m + "g1_proj.weight"], w[m + "g2_proj.weight"] = d.lin(z["inner"], W), d.lin(D * z["dvdim"], z["inner"])
            w[m + "o_proj.weight"] = d.lin(W, D * z["dvdim"])
        if i == 0:
            w[p + "mlp.up_proj.weight"], w[p + "mlp.down_proj.weight"] = d.lin(z["ff"], W), d.lin(W, z["ff"], 0.5)
        else:
            w[p + "mlp.router.weight"] = d.lin(z["experts"], W, 3.0)
            w[p + "mlp.gate_proj"] = d.normal(z["experts"], z["mff"], W, std=W ** -0.5)
            w[p + "mlp.up_proj"] = d.normal(z["experts"], z["mff"], W, std=W ** -0.5)
            w[p + "mlp.down_proj"] = d.normal(z["experts"], W, z["mff"], std=0.5 * z["mff"] ** -0.5)
    return w


def _weights(case, seed):
    if case["family"] == "layer":
        e, h, i = _layer_sizes(case)
        return _routed_weights(_Draws(case, seed), "", h, i, e, 0.02)
    return {"complexity": _complexity_weights, "pimezen": _pimezen_weights, "rugedra": _rugedra_weights}[case["family"]](case, seed)


# ------------------------------------------------------------------------------------------- models
def _pimezen_config(z):
    layer = {"type": "parallel",
             "mixer": {"left": {"heads": z["heads"], "kv_heads": z["kv"], "dim": z["dim"], "vdim": z["vdim"],
                                "scale": z["dim"] ** -0.5, "mask": {"size": z["window"], "keep_first": z["keep"]}},
                       "right": {"heads": z["rheads"], "dim": z["rdim"], "vdim": z["rvdim"], "tau": TAU},
                       "left_scale": BRANCH, "right_scale": BRANCH},
             "mlp": {"kind": "dense", "ff": z["ff"], "limit": LIMIT}}
    return {"vocab": VOCAB, "width": z["width"], "norm": {"eps": EPS}, "layers": [layer] * z["layers"]}


def _rugedra_config(z):
    latent = {"heads": z["heads"], "dim": z["dim"], "rot_dim": z["rot"], "vdim": z["vdim"], "kv_rank": z["rank"],
              "scale": (z["dim"] + z["rot"]) ** -0.5, "rot": {"base": ROT_BASE, "dims": z["rot"]}}
    delta = {"heads": z["dheads"], "kv_heads": z["dkv"], "dim": z["ddim"], "vdim": z["dvdim"], "conv": z["conv"]}
    moe = {"kind": "moe", "expert": {"ff": z["mff"], "limit": LIMIT},
           "router": {"experts": z["experts"], "top": z["top"], "groups": {"count": z["groups"], "keep": z["keep"]}}}
    layers = [{"type": "latent_attention" if _latent(i) else "channel_delta", "mixer": latent if _latent(i) else delta,
               "mlp": {"kind": "dense", "ff": z["ff"]} if i == 0 else moe} for i in range(z["layers"])]
    return {"vocab": VOCAB, "width": z["width"], "max_positions": POSITIONS, "norm": {"eps": EPS}, "residual_mult": MULT,
            "logit_scale": 1.0, "layers": layers}


@torch.no_grad()
def _model(case, weights):
    import complexity_deep_b200 as cd
    from complexity_deep_b200.models import PimezenConfig, PimezenModel, RugedraConfig, RugedraModel
    with torch.device("cuda"):
        if case["family"] == "layer":
            e, h, i = _layer_sizes(case)
            model = cd.TokenRoutedMLP(h, e * i, e, VOCAB, True, None)
        elif case["family"] == "complexity":
            H, I, L, hq, hkv, E = COMPLEXITY[case["size"]]
            model = cd.ComplexityModel(cd.ComplexityConfig(
                vocab_size=VOCAB, hidden_size=H, intermediate_size=I, num_hidden_layers=L, num_attention_heads=hq,
                num_key_value_heads=hkv, num_experts=E))
        elif case["family"] == "pimezen":
            model = PimezenModel(PimezenConfig.from_dict(_pimezen_config(PIMEZEN[case["size"]])))
        else:
            cfg = RugedraConfig.from_dict(_rugedra_config(RUGEDRA[case["size"]]))
            for layer in cfg.layers:
                if layer.mixer.kind == "channel_delta":
                    layer.mixer.rank = layer.mixer.gate_rank = RUGEDRA[case["size"]]["inner"]
            model = RugedraModel(cfg)
    model = model.to(GRID[case["dtype"]]).requires_grad_(False).eval()
    params = dict(model.named_parameters())
    params.pop("lm_head.weight", None) if case["family"] == "complexity" else None     # tied to the embedding
    if set(params) != set(weights):
        raise ValueError(f"weights for {sorted(set(weights) ^ set(params))}")
    for name, p in params.items():
        p.copy_(weights[name])
    for name, b in model.named_buffers():
        if name.endswith("token_to_expert"):
            b.copy_(_table(len(model.layers[0].mlp.gate_proj_w) if case["family"] == "complexity" else model.num_experts))
    return model


# ------------------------------------------------------------------------------------------- prepare and run
def _tokens(case):
    return case["cached"] + case["steps"] if case["kind"] == "decode" else case["seq"]


def _activations(case, seed):
    g = torch.Generator(device="cuda").manual_seed(15485863 * int(seed) + 5)
    h = _layer_sizes(case)[1]
    return torch.empty(case["batch"], case["seq"], h, device="cuda").normal_(generator=g).to(GRID[case["dtype"]])


@torch.no_grad()
def prepare(case, seed):
    from complexity_deep_b200.models import DecodeGraph, PrefillGraph
    model = _model(case, _weights(case, seed))
    ids = _ids(case, seed, _tokens(case))
    state = {"kind": case["kind"], "model": model}
    if case["kind"] == "decode":
        B, n = case["batch"], case["cached"]
        prompt, state["ids"] = ids[:, :n], ids[:, n:].t().contiguous().view(-1, B, 1)
        state["decode"] = dec = DecodeGraph(model, batch=B, capacity=n + case["steps"])
        if case["family"] == "complexity":
            past = [model(prompt[b:b + 8].contiguous(), use_cache=True).past_key_values for b in range(0, B, 8)]
            dec.cache.load([tuple(torch.cat([p[i][j] for p in past]) for j in (0, 1)) for i in range(len(past[0]))])
        else:
            none = torch.empty(0, dtype=torch.int64, device="cuda")
            prefix = model.new_state(B)
            for a in range(0, n, 512):
                model(prompt[:, a:a + 512].contiguous(), past_key_values=prefix, use_cache=True, logit_rows=none)
            state["prefix"] = prefix
        state["cached"] = n
    else:
        state["ids"] = ids.cpu().pin_memory()
    if case["kind"] == "prompt" and case["graph"]:
        state["graph"] = PrefillGraph(model, case["batch"], case["seq"])
    if case["kind"] == "portions":
        state["pool"], state["portion"] = model.state_pool(case["batch"]), case["portion"]
    if case["kind"] == "layer":
        state["x"] = _activations(case, seed)
    return state


@torch.no_grad()
def run(state):
    kind, model, ids = state["kind"], state["model"], state["ids"]
    if kind == "decode":
        dec = state["decode"]
        if "prefix" in state:
            dec.cache.load(state["prefix"])
        else:
            dec.cache.set_length(state["cached"])
        return torch.stack([dec.step(x).clone() for x in ids])
    ids = ids.to("cuda", non_blocking=True)
    if kind == "layer":
        return model(state["x"], ids)
    if kind == "portions":
        request = state["pool"].get("request")
        logits = [model(ids[:, a:a + state["portion"]].contiguous(), past_key_values=request, use_cache=True).logits
                  for a in range(0, ids.shape[1], state["portion"])]
        state["pool"].release("request")
        return logits
    return state["graph"](ids) if "graph" in state else model(ids).logits


# ------------------------------------------------------------------------------------------- work
def _per_layer(case):
    """[(matrix products as (inputs, outputs, applied, held), score columns per key, state bytes per sequence)] for
    every layer: `applied` of the `held` matrices multiply a token; a cached token costs `score` multiply-adds and
    `row` bytes, as far as `reach` tokens back."""
    if case["family"] == "layer":
        e, h, i = _layer_sizes(case)
        return [dict(mats=[(h, 3 * i, 1, e), (h, 3 * i, 1, 1)], score=0, row=0, reach=0, state=0, step=0)]
    if case["family"] == "complexity":
        H, I, L, hq, hkv, E = COMPLEXITY[case["size"]]
        D = H // hq
        one = dict(mats=[(2 * H, (hq + 2 * hkv) * D, 1, 1), (hq * D, H, 1, 1), (H, 3 * (I // E), 1, E), (H, 3 * (I // E), 1, 1), (H, H, 1, 1)],
                   score=2 * hq * D, row=2 * hkv * D, reach=1 << 30, state=0, step=0)
        return [one] * L
    if case["family"] == "pimezen":
        z = PIMEZEN[case["size"]]
        W, H, G, R = z["width"], z["heads"], z["kv"], z["rheads"]
        one = dict(mats=[(W, H * z["dim"] + G * (z["dim"] + z["vdim"]) + R * 2 * (z["rdim"] + z["rvdim"]) + 16, 1, 1), (16, R * z["rdim"], 1, 1),
                         (H * z["vdim"] + R * z["rvdim"], W, 1, 1), (W, 3 * z["ff"], 1, 1)],
                   score=H * (z["dim"] + z["vdim"] + H), row=G * (z["dim"] + z["vdim"]), reach=z["window"] + z["keep"],
                   state=4 * R * z["rdim"] * z["rvdim"], step=2 * R * z["rdim"] * z["rvdim"])
        return [one] * z["layers"]
    z, out = RUGEDRA[case["size"]], []
    W, H, D, G = z["width"], z["heads"], z["dheads"], z["dkv"]
    for i in range(z["layers"]):
        if _latent(i):
            one = dict(mats=[(W, H * (z["dim"] + z["rot"]) + z["rank"] + z["rot"] + H, 1, 1), (z["rank"], H * (z["dim"] + z["vdim"]), 1, 1),
                             (H * z["vdim"], W, 1, 1)],
                       score=H * (z["dim"] + z["rot"] + z["vdim"]), row=z["rank"] + z["rot"], reach=1 << 30, state=0, step=0)
        else:
            one = dict(mats=[(W, 2 * G * z["ddim"] + D * z["dvdim"] + D + 2 * z["inner"], 1, 1), (z["inner"], D * (z["ddim"] + z["dvdim"]), 1, 1),
                             (D * z["dvdim"], W, 1, 1)],
                       score=0, row=0, reach=0, state=4 * D * z["ddim"] * z["dvdim"], step=3 * D * z["ddim"] * z["dvdim"])
        one["mats"] += [(W, 2 * z["ff"], 1, 1)] if i == 0 else [(W, z["experts"], 1, 1), (W, 3 * z["mff"], z["top"], z["experts"])]
        out.append(one)
    return out


def work(case):
    """Every weight that is used read once per call of the model, ids in and logits out, cached tokens and states read
    (and states written) once per call; two operations per weight and token, per state element and per visible key."""
    item, logit = (4 if case["dtype"] == "f32" else 2), (2 if case["family"] == "complexity" else 4)
    B, head = case["batch"], 0 if case["family"] == "layer" else VOCAB
    if case["kind"] == "decode":
        calls = [(case["cached"] + i, 1) for i in range(case["steps"])]
    else:
        step = case["portion"] or case["seq"]
        calls = [(a, min(step, case["seq"] - a)) for a in range(0, case["seq"], step)]
    layers = _per_layer(case)
    width = layers[0]["mats"][-1][0]
    flops = byts = 0.0
    for seen, new in calls:
        T = B * new
        flops += 2.0 * T * width * head
        byts += item * width * head + T * (8 + logit * head) + (2 * item * T * width if not head else 0)
        for layer in layers:
            for k, n, applied, held in layer["mats"]:
                flops += 2.0 * T * k * n * applied
                byts += item * k * n * min(held, T * applied)
            keys = sum(min(seen + t + 1, layer["reach"]) for t in range(new))
            flops += 2.0 * B * keys * layer["score"] + 2.0 * T * layer["step"]
            old = min(seen, layer["reach"])
            byts += item * B * layer["row"] * (old + new) + 2.0 * B * layer["state"]
    return {"bytes": byts, "flops": flops}


def tolerance(case):
    """About four times the distance from 64 bits that is measured over these ranges: 2.3e-6 (f32), 2.4e-3 (layer),
    3.5e-3 (Complexity), 6.1e-3 (Pimezen). In Rugedra a router's choice between two experts that are a rounding apart
    moves a whole row: 6e-3 to 9e-3 in all, 3.5e-3 in the median row, 7e-2 in the worst."""
    if case["dtype"] == "f32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"layer": {"rel": 0.01, "max": 0.1}, "complexity": {"rel": 0.014, "max": 0.1}, "pimezen": {"rel": 0.025, "max": 0.25},
            "rugedra": {"rel": 0.03, "max": 0.95}}[case["family"]]


# ------------------------------------------------------------------------------------------- in 64 bits
def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _routed(x, w, p, ids, table):
    """x [n, hidden], one id each."""
    out = (F.silu(x @ w[p + "shared_gate.weight"].t()) * (x @ w[p + "shared_up.weight"].t())) @ w[p + "shared_down.weight"].t()
    chosen = table[ids]
    for e in range(w[p + "gate_proj_w"].shape[0]):
        at = (chosen == e).nonzero()[:, 0]
        y = (F.silu(x[at] @ w[p + "gate_proj_w"][e]) * (x[at] @ w[p + "up_proj_w"][e])) @ w[p + "down_proj_w"][e]
        out.index_add_(0, at, y)
    return out


def _softmax_attention(q, k, v, scale, hidden, bias=None, mix=None):
    """q [S, H, d], k [S, G, d], v [S, G, e] -> [S, H, e]; hidden [S, S]: keys that a row does not see."""
    rep = q.shape[1] // k.shape[1]
    s = torch.einsum("ihd,jhd->hij", q * scale, k.repeat_interleave(rep, 1))
    if bias is not None:
        s -= bias
    s = s.masked_fill_(hidden, -math.inf).softmax(-1)
    if mix is not None:
        s = torch.einsum("hg,gij->hij", mix, s)
    return torch.einsum("hij,jhe->ihe", s, v.repeat_interleave(rep, 1))


def _complexity_exact(case, w, ids):
    H, _, L, hq, hkv, E = COMPLEXITY[case["size"]]
    B, S = ids.shape
    D, table = H // hq, _table(E).cuda()
    freq = 1.0 / (10000.0 ** (torch.arange(0, D, 2, dtype=torch.float64, device="cuda") / D))
    angle = torch.outer(torch.arange(S, dtype=torch.float64, device="cuda"), freq)
    cos, sin = (torch.cat([f(angle)] * 2, -1)[:, None] for f in (torch.cos, torch.sin))
    hidden = torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1)
    turn = lambda t: t * cos + torch.cat([-t[..., D // 2:], t[..., : D // 2]], -1) * sin   # noqa: E731
    out = []
    for b in range(B):
        x = w["embed_tokens.weight"][ids[b]]
        mu = w["mu_init"].view(1, -1).expand(S, -1)
        for i in range(L):
            p = f"layers.{i}."
            a = p + "self_attn."
            h = _rms(x, 1e-6) * w[p + "input_layernorm.weight"]
            q, k, v = ((h @ w[f"{a}{n}_proj.weight"].t() + mu @ w[f"{a}mu_to_{n}.weight"].t()).view(S, -1, D) for n in "qkv")
            q, k = turn(_rms(q, 1e-6) * w[a + "q_norm.weight"]), turn(_rms(k, 1e-6) * w[a + "k_norm.weight"])
            x = x + _softmax_attention(q, k, v, D ** -0.5, hidden).reshape(S, -1) @ w[a + "o_proj.weight"].t()
            h = _rms(x, 1e-6) * w[p + "post_attention_layernorm.weight"]
            x = x + _routed(h, w, p + "mlp.", ids[b], table)
            mu = w[p + "mu_guidance.mu"].clamp(0.0, 2.0) + x @ w[p + "mu_guidance.mu_proj.weight"].t()
            mu = mu.clamp(-2.0, 2.0)
        out.append((_rms(x, 1e-6) * w["norm.weight"]) @ w["embed_tokens.weight"].t())
    return torch.stack(out)


def _glu(h, gate, up, down):
    g, u = (h @ gate.t()).clamp(max=LIMIT), (h @ up.t()).clamp(-LIMIT, LIMIT)
    return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ down.t()


def _pimezen_exact(case, w, ids):
    z = PIMEZEN[case["size"]]
    B, S = ids.shape
    at = torch.arange(S, device="cuda")
    gap = at[:, None] - at[None]
    hidden = (gap < 0) | ((gap >= z["window"]) & (at[None] >= z["keep"]))
    x = w["embed_tokens.weight"][ids]
    for i in range(z["layers"]):
        p = f"layers.{i}."
        a, r = p + "mixers.branches.left.", p + "mixers.branches.right."
        h = _rms(x, EPS) * (1.0 + w[p + "norm1.weight"])
        q, k = ((h @ w[f"{a}{n}_proj.weight"].t()).view(B, S, -1, z["dim"]) for n in "qk")
        q, k = _rms(q, EPS) * w[a + "q_norm"], _rms(k, EPS) * w[a + "k_norm"]
        v = (h @ w[a + "v_proj.weight"].t()).view(B, S, -1, z["vdim"])
        bias = w[a + "r1"].view(-1, 1, 1) * torch.log1p(w[a + "r2"].view(-1, 1, 1) * gap.clamp(min=0))
        left = torch.stack([_softmax_attention(q[b], k[b], v[b], z["dim"] ** -0.5, hidden, bias, w[a + "talk"]) for b in range(B)])
        q, k = ((h @ w[f"{r}{n}_proj.weight"].t()).view(B, S, -1, z["rdim"]) for n in "qk")
        v = (h @ w[r + "v_proj.weight"].t()).view(B, S, -1, z["rvdim"])
        g = F.logsigmoid((h @ w[r + "a1_proj.weight"].t()) @ w[r + "a2_proj.weight"].t() + w[r + "a2_proj.bias"])
        g = (g / TAU).exp().view_as(q)
        s, o = torch.zeros(B, z["rheads"], z["rdim"], z["rvdim"], dtype=x.dtype, device="cuda"), torch.empty_like(v)
        for t in range(S):
            s.mul_(g[:, t, ..., None]).add_(k[:, t, ..., None] * v[:, t, :, None])
            o[:, t] = (q[:, t, :, None] @ s)[:, :, 0]
        o = (_rms(o * z["rdim"] ** -0.5, EPS) * w[r + "norm"]).flatten(2) * F.silu(h @ w[r + "g_proj.weight"].t())
        y = left.flatten(2) @ w[a + "o_proj.weight"].t() + o @ w[r + "o_proj.weight"].t()
        x = x + BRANCH * y * w[p + "ls1"]
        h = _rms(x, EPS) * (1.0 + w[p + "norm2.weight"])
        x = x + w[p + "ls2"] * _glu(h, *(w[f"{p}mlp.{n}_proj.weight"] for n in ("gate", "up", "down")))
    return (_rms(x, EPS) * (1.0 + w["norm.weight"])) @ w["embed_tokens.weight"].t()


def _experts_exact(h, w, p, z):
    s = (h @ w[p + "router.weight"].t()).softmax(-1)
    size = z["experts"] // z["groups"]
    best = s.view(-1, z["groups"], size).amax(-1).topk(z["keep"], -1).indices
    kept = torch.zeros(len(s), z["groups"], dtype=torch.bool, device="cuda").scatter_(1, best, True).repeat_interleave(size, 1)
    weight, chosen = s.masked_fill(~kept, -1.0).topk(z["top"], -1)
    weight = weight / (weight.sum(-1, keepdim=True) + 1e-20)
    out = torch.zeros_like(h)
    for e in range(z["experts"]):
        row, col = (chosen == e).nonzero(as_tuple=True)
        y = _glu(h[row], w[p + "gate_proj"][e], w[p + "up_proj"][e], w[p + "down_proj"][e])
        out.index_add_(0, row, y * weight[row, col, None])
    return out


def _rugedra_exact(case, w, ids):
    z = RUGEDRA[case["size"]]
    B, S = ids.shape
    norm = lambda t, n: _rms(t - t.mean(-1, keepdim=True), EPS) * w[n]                       # noqa: E731
    freq = ROT_BASE ** (-torch.arange(0, z["rot"], 2, dtype=torch.float64, device="cuda") / z["rot"])
    angle = torch.outer(torch.arange(S, dtype=torch.float64, device="cuda"), freq)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def turn(t):                                                                            # [..., S, heads, rot]
        u, v = t[..., 0::2], t[..., 1::2]
        return torch.stack([u * cos - v * sin, v * cos + u * sin], -1).flatten(-2)

    def conv(t, taps):
        K = taps.shape[1]
        return F.silu(sum(F.pad(t, (0, 0, K - 1 - j, 0))[:, :S] * taps[:, j] for j in range(K)))

    unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)                # noqa: E731
    hidden = torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1)
    x = w["embed_tokens.weight"][ids] + w["embed_positions.weight"][:S]
    for i in range(z["layers"]):
        p = f"layers.{i}."
        m = p + "mixers.branches.mix."
        h = norm(x, p + "norm1.weight")
        if _latent(i):
            both = h @ w[m + "kv_proj.weight"].t()
            lat = _rms(both[..., : z["rank"]], EPS) * w[m + "kv_norm"]
            key = turn(both[..., None, z["rank"]:])
            q = (h @ w[m + "q_proj.weight"].t()).view(B, S, z["heads"], -1)
            q = torch.cat([q[..., : z["dim"]], turn(q[..., z["dim"]:])], -1)
            k = (lat @ w[m + "uk_proj.weight"].t()).view(B, S, z["heads"], -1)
            k = torch.cat([k, key.expand(-1, -1, z["heads"], -1)], -1)
            v = (lat @ w[m + "uv_proj.weight"].t()).view(B, S, z["heads"], -1)
            scale = (z["dim"] + z["rot"]) ** -0.5
            o = torch.stack([_softmax_attention(q[b], k[b], v[b], scale, hidden) for b in range(B)])
            o = o * torch.sigmoid(h @ w[m + "g_proj.weight"].t())[..., None]
        else:
            D, rep = z["dheads"], z["dheads"] // z["dkv"]
            q, k, v = (conv(h @ w[f"{m}{n}_proj.weight"].t(), w[f"{m}{n}_conv"]) for n in "qkv")
            q, k = (unit(t.view(B, S, z["dkv"], -1)).repeat_interleave(rep, 2) for t in (q, k))
            v = v.view(B, S, D, -1)
            g = F.softplus((h @ w[m + "a1_proj.weight"].t()) @ w[m + "a2_proj.weight"].t() + w[m + "dt_bias"]).view(B, S, D, -1)
            g = torch.exp(-w[m + "A_log"].exp().view(-1, 1) * g)
            beta = torch.sigmoid(h @ w[m + "b_proj.weight"].t())
            s, o = torch.zeros(B, D, z["ddim"], z["dvdim"], dtype=x.dtype, device="cuda"), torch.empty_like(v)
            for t in range(S):
                s.mul_(g[:, t, ..., None])
                u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None] @ s)[:, :, 0])
                s.add_(k[:, t, ..., None] * u[:, :, None])
                o[:, t] = (q[:, t, :, None] @ s)[:, :, 0]
            gate = torch.sigmoid((h @ w[m + "g1_proj.weight"].t()) @ w[m + "g2_proj.weight"].t())
            o = _rms(o * z["ddim"] ** -0.5, EPS) * w[m + "norm"] * gate.view_as(o)
        x = x + MULT * (o.flatten(2) @ w[m + "o_proj.weight"].t())
        h = norm(x, p + "norm2.weight")
        if i == 0:
            y = (h @ w[p + "mlp.up_proj.weight"].t()).relu().square() @ w[p + "mlp.down_proj.weight"].t()
        else:
            y = _experts_exact(h.flatten(0, 1), w, p + "mlp.", z).view_as(h)
        x = x + MULT * y
    return norm(x, "norm.weight") @ w["lm_head.weight"].t()


@torch.no_grad()
def exact(case, seed):
    """The outputs in 64 bits from the same weights and ids; the whole sequence at once, whatever the case's portions."""
    cost = dict(case, kind="prompt", seq=_tokens(case), portion=0)
    if work(cost)["flops"] > 1.2e14:
        return None
    w = {k: v.double() for k, v in _weights(case, seed).items()}
    ids = _ids(case, seed, _tokens(case))
    if case["kind"] == "layer":
        x = _activations(case, seed).double()
        e = _layer_sizes(case)[0]
        return _routed(x.flatten(0, 1), w, "", ids.flatten(), _table(e).cuda()).view_as(x)
    logits = {"complexity": _complexity_exact, "pimezen": _pimezen_exact, "rugedra": _rugedra_exact}[case["family"]](case, w, ids)
    if case["kind"] == "decode":
        return logits[:, case["cached"]:].transpose(0, 1).unsqueeze(2)
    if case["kind"] == "portions":
        return list(logits.split(case["portion"], 1))
    return logits

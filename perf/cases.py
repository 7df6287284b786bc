"""Workloads of the framework's hot paths, one dictionary of plain numbers each, with their inputs, one pass through the public entry
points, the bytes and operations a pass cannot do without, and a float64 statement of the result in plain torch.

The kinds and what they stand for in use:

* ``sample``       choosing the next tokens of a batch from fp32 logits over a whole vocabulary (temperature, top-k, top-p)
* ``linear``       one projection of the LLaMA stack, with the norm before it, the gated activation or the residual sum behind it, from a
                   decode batch to a prompt
* ``attn_prompt``  causal attention of a prompt's queries over the cache just written (left-padded rows, grouped heads)
* ``attn_decode``  rotation, cache append and attention of one new token per row over a long cache
* ``llama``        a whole request to a LLaMA engine: prompt, then tokens fed one at a time, logits read back
* ``folirax``      the same for an engine of the hybrid family (gated linear attention and softmax attention)
* ``mixer``        one sequence mixer of the hybrid family over prompts, its cache or state starting empty
* ``ff``           one feed-forward of the hybrid family: dense or experts, in bfloat16 or in true float32
"""
from __future__ import annotations

import math

import torch

from jax_llama_b200.config import (AttentionMixerSpec, DeltaMixerSpec, DenseMlpSpec, FoliraxConfig, GlaMixerSpec, LatentAttentionMixerSpec,
                                   LLaMAConfig, MoeMlpSpec, RetentionMixerSpec, RotarySpec, StateSpaceMixerSpec)
from jax_llama_b200.models.engine import B200Engine
from jax_llama_b200.models.feedforward import DenseFeedForward, MoeFeedForward
from jax_llama_b200.models.hybrid_engine import HybridCache, HybridEngine
from jax_llama_b200.models.mixers import MIXERS, rotary_table
from jax_llama_b200.ops import kernels as K

F64 = torch.float64
EPS = 1e-5


def listed():
    return [
        # a sampling step of a serving batch over a 128k vocabulary (temperature 0.8, nucleus 0.95)
        dict(name="sample_nucleus_b4", kind="sample", B=4, V=128256, temperature=0.8, top_k=0, top_p=0.95),
        # gate and up projection of an 8B-sized layer for a decode batch of 16, norm and SwiGLU included
        dict(name="linear_swiglu_b16", kind="linear", M=16, N=28672, K=4096, mode="swiglu"),
        # its down projection for a prompt of 2048 tokens, added to the residual stream
        dict(name="linear_down_prompt", kind="linear", M=2048, N=4096, K=14336, mode="residual"),
        # attention of a 3000-token prompt, 32 query heads over 8 key / value heads
        dict(name="attn_prompt_3000", kind="attn_prompt", B=1, S=3000, nh=32, nkv=8, hd=128, pad=0),
        # one token for each of 24 rows with about 4000 cached tokens
        dict(name="attn_decode_b24", kind="attn_decode", B=24, T=4096, length=4000, nh=32, nkv=8, hd=128, pad=500),
        # one interactive request: short prompt, tokens streamed (layers of the 8B size, four of them)
        dict(name="llama_request", kind="llama", B=1, P=100, steps=24, width=4096, heads=32, kv=8, ff=14336, layers=4, vocab=32000),
        # two left-padded requests to a hybrid model (the size the framework's own comparison uses)
        dict(name="folirax_request", kind="folirax", B=2, P=60, steps=24, width=2048, heads=16, kv=4, ff=8192, layers=8, vocab=32000),
        # recurrent layers over a prompt: one decay per key channel, and the delta rule
        dict(name="gla_prompt", kind="mixer", mixer="gla", dtype="bf16", B=1, S=2048, width=2048, H=16, D=64, Dv=128, window=0),
        dict(name="delta_prompt", kind="mixer", mixer="delta", dtype="bf16", B=2, S=1000, width=2048, H=16, D=64, Dv=128, window=0),
        # latent attention over a prompt, 128 + 64 wide heads, sliding window
        dict(name="latent_prompt", kind="mixer", mixer="latent", dtype="bf16", B=1, S=2048, width=2048, H=16, D=128, Dv=128, window=1024),
        # experts with a shared one over a prompt's tokens
        dict(name="experts_prompt", kind="ff", ff_kind="moe", dtype="bf16", M=2048, width=2048, ff=1024, experts=32, top=4, shared=1360),
        # the exact float32 path, a gated layer over a short prompt
        dict(name="dense_f32", kind="ff", ff_kind="dense", dtype="f32", M=200, width=2048, ff=5464, experts=0, top=0, shared=0),
    ]


def _log_int(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, int(round(v / multiple)) * multiple)


def draw(rng):
    """One more case of the ranges above; sizes are logarithmically spread and seldom round."""
    kind = rng.choice(["sample", "linear", "attn_prompt", "attn_decode", "llama", "folirax", "mixer", "mixer", "ff"])
    if kind == "sample":
        return dict(kind=kind, B=_log_int(rng, 1, 64), V=_log_int(rng, 8000, 128256), temperature=round(rng.uniform(0.5, 1.2), 2),
                    top_k=rng.choice([0, 0, 50, 400]), top_p=rng.choice([1.0, 0.9, 0.95]))
    if kind == "linear":
        mode = rng.choice(["swiglu", "residual", "plain"])
        return dict(kind=kind, M=_log_int(rng, 1, 2048), N=_log_int(rng, 1024, 28672, 256), K=_log_int(rng, 1024, 4096, 256), mode=mode)
    if kind == "attn_prompt":
        B = rng.randint(1, 4)
        S = _log_int(rng, 32, 3000 // B)
        nkv = rng.choice([4, 8])
        return dict(kind=kind, B=B, S=S, nh=nkv * rng.choice([1, 2, 4]), nkv=nkv, hd=rng.choice([128, 128, 64]), pad=rng.choice([0, S // 5]))
    if kind == "attn_decode":
        T = _log_int(rng, 64, 4096, 8)
        length = rng.randint(T // 2, T - 1)
        nkv = rng.choice([4, 8])
        return dict(kind=kind, B=_log_int(rng, 1, 24), T=T, length=length, nh=nkv * rng.choice([1, 2, 4]), nkv=nkv, hd=rng.choice([128, 128, 64]),
                    pad=rng.choice([0, length // 4]))
    if kind == "llama":
        width = rng.choice([1024, 2048, 4096])
        B = _log_int(rng, 1, 24)
        return dict(kind=kind, B=B, P=_log_int(rng, 20, max(40, 900 // B)), steps=rng.randint(8, 16), width=width, heads=width // 128,
                    kv=width // 512, ff=_log_int(rng, width * 2, width * 7 // 2, 256), layers=rng.randint(2, 4), vocab=32000)
    if kind == "folirax":
        width = rng.choice([1024, 2048])
        return dict(kind=kind, B=_log_int(rng, 1, 8), P=_log_int(rng, 20, 200), steps=rng.randint(8, 24), width=width, heads=width // 128,
                    kv=width // 512, ff=_log_int(rng, width * 2, width * 4, 8), layers=rng.choice([4, 8]), vocab=32000)
    if kind == "mixer":
        mixer = rng.choice(["gla", "retention", "state_space", "delta", "latent"])
        B = rng.randint(1, 4)
        S = _log_int(rng, 24, 2048 // B)
        H = rng.choice([4, 8, 16])
        if mixer == "latent":
            D, Dv, window = 128, 128, rng.choice([0, 512, 1024])
        elif mixer == "state_space":
            D, Dv, window = rng.choice([64, 128]), 64, 0
        else:
            D, Dv, window = rng.choice([32, 64, 128]), rng.choice([64, 128]), 0
        dtype = rng.choice(["bf16", "bf16", "bf16", "f32"])
        return dict(kind=kind, mixer=mixer, dtype=dtype, B=B, S=S, width=rng.choice([1024, 2048]), H=H, D=D, Dv=Dv, window=window)
    width = rng.choice([1024, 2048])
    if rng.random() < 0.5:
        return dict(kind=kind, ff_kind="moe", dtype="bf16", M=_log_int(rng, 1, 2048), width=width, ff=_log_int(rng, 256, 1024, 8), experts=32,
                    top=rng.choice([2, 4]), shared=rng.choice([0, 1360]))
    f32 = rng.random() < 0.5
    return dict(kind=kind, ff_kind="dense", dtype="f32" if f32 else "bf16", M=_log_int(rng, 1, 400 if f32 else 2048), width=width,
                ff=_log_int(rng, 1024, 5464, 8), experts=0, top=0, shared=0)


# ------------------------------------------------------------------------------------------ inputs
class _Draws:
    """Random tensors on the GPU from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def normal(self, *shape, scale=1.0, dtype=torch.float32):
        return (torch.randn(shape, generator=self.g, device="cuda") * scale).to(dtype)

    def matrix(self, n, k, dtype=torch.bfloat16):
        return self.normal(n, k, scale=k ** -0.5, dtype=dtype)

    def gain(self, n, dtype=torch.bfloat16, around=1.0):
        return (around + 0.1 * torch.randn(n, generator=self.g, device="cuda")).to(dtype)

    def ints(self, hi, *shape):
        return torch.randint(0, hi, shape, generator=self.g, device="cuda")


def _dtype(case):
    return torch.float32 if case.get("dtype") == "f32" else torch.bfloat16


def _pads(case, B):
    """Left padding per row: from none to `pad`, spread over the rows."""
    return [case["pad"] * b // max(B - 1, 1) for b in range(B)]


def _request_pads(case):
    return [(case["P"] // 4) * b // max(case["B"] - 1, 1) for b in range(case["B"])]


def _llama_tree(case, d):
    W, H, G, F, V = case["width"], case["heads"], case["kv"], case["ff"], case["vocab"]

    def kernel(i, o):
        return {"kernel": d.normal(i, o, scale=i ** -0.5, dtype=torch.bfloat16)}

    layers = {}
    for i in range(case["layers"]):
        layers[str(i)] = {"attention": {"wq": kernel(W, H * 128), "wk": kernel(W, G * 128), "wv": kernel(W, G * 128), "wo": kernel(H * 128, W)},
                          "feed_forward": {"w1": kernel(W, F), "w3": kernel(W, F), "w2": kernel(F, W)},
                          "attention_norm": {"kernel": d.gain(W)}, "ffn_norm": {"kernel": d.gain(W)}}
    return {"transformer": {"wte": {"embedding": d.normal(V, W, dtype=torch.bfloat16)}, "ln_f": {"kernel": d.gain(W)}, "h": layers},
            "lm_head": kernel(W, V)}


def _folirax_layers(case):
    H, G = case["heads"], case["kv"]
    att = {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "rot": {"dims": 64, "base": 10000.0}}
    gla = {"heads": H, "dim": 64, "vdim": 128, "tau": 16.0}
    mlp = {"kind": "dense", "ff": case["ff"]}
    out = []
    for i in range(case["layers"]):
        out.append([{"type": "gla", "mixer": gla, "mlp": None}, {"type": "attention", "mixer": att, "mlp": mlp},
                    {"type": "attention", "mixer": dict(att, kv_from=i - 1), "mlp": mlp}, {"type": "gla", "mixer": gla, "mlp": mlp}][i % 4])
    return out


def _folirax_tensors(case, d):
    W, H, G, V = case["width"], case["heads"], case["kv"], case["vocab"]
    t = {"embed": d.normal(V, W, dtype=torch.bfloat16), "final.norm": d.gain(W, around=0.0), "head": d.matrix(V, W)}
    for i, l in enumerate(_folirax_layers(case)):
        p = f"l{i}."
        t[p + "norm1"], t[p + "norm1b"] = d.gain(W, around=0.0), d.gain(W, around=0.0)
        if l["type"] == "gla":
            t.update({p + "mix." + k: v for k, v in _gla_weights(d, W, H, 64, 128, torch.bfloat16).items()})
        else:
            t[p + "mix.q"], t[p + "mix.g"], t[p + "mix.o"] = d.matrix(H * 128, W), d.matrix(H, W), d.matrix(W, H * 128)
            if l["mixer"].get("kv_from") is None:
                t[p + "mix.k"], t[p + "mix.v"] = d.matrix(G * 128, W), d.matrix(G * 128, W)
        if l["mlp"] is not None:
            t[p + "norm2"], t[p + "norm2b"] = d.gain(W, around=0.0), d.gain(W, around=0.0)
            t[p + "mlp.up"], t[p + "mlp.down"] = d.matrix(case["ff"], W), d.matrix(W, case["ff"])
    return t


def _gla_weights(d, W, H, D, Dv, dt):
    return {"q": d.matrix(H * D, W, dt), "k": d.matrix(H * D, W, dt), "v": d.matrix(H * Dv, W, dt), "g": d.matrix(H * Dv, W, dt),
            "a1": d.matrix(16, W, dt), "a2": d.matrix(H * D, 16, dt), "a2.b": (2.0 + 2.0 * d.normal(H * D)).to(dt), "norm": d.gain(Dv, dt),
            "o": d.matrix(W, H * Dv, dt)}


def _latent_ranks(case):
    return 3 * case["width"] // 8, 512, 64            # query rank, key / value rank, rotated channels


def _decays(H):
    return [1.0 - 0.05 * 0.1 ** (h / max(H - 1, 1)) for h in range(H)]


def _mixer_weights(case, d):
    W, H, D, Dv, dt = case["width"], case["H"], case["D"], case["Dv"], _dtype(case)
    m = case["mixer"]
    if m == "gla":
        return _gla_weights(d, W, H, D, Dv, dt)
    if m == "retention":
        return {"q": d.matrix(H * D, W, dt), "k": d.matrix(H * D, W, dt), "v": d.matrix(H * Dv, W, dt), "g": d.matrix(H * Dv, W, dt),
                "o": d.matrix(W, H * Dv, dt)}
    if m == "state_space":
        inner = H * Dv
        return {"in": d.matrix(2 * inner + 2 * D + H, W, dt), "conv": d.normal(inner + 2 * D, 4, scale=0.5, dtype=dt),
                "conv.b": d.normal(inner + 2 * D, scale=0.1, dtype=dt), "dt_bias": (d.normal(H) - 2.0).to(dt), "A_log": d.normal(H, scale=0.5, dtype=dt),
                "D": d.normal(H, scale=0.5, dtype=dt), "norm": d.gain(inner, dt), "o": d.matrix(W, inner, dt)}
    if m == "delta":
        w = {"q": d.matrix(H * D, W, dt), "k": d.matrix(H * D, W, dt), "v": d.matrix(H * Dv, W, dt), "g": d.matrix(H * Dv, W, dt),
             "b": d.matrix(H, W, dt), "a": d.matrix(H, W, dt), "dt_bias": (d.normal(H) - 3.0).to(dt), "A_log": d.normal(H, scale=0.5, dtype=dt),
             "norm": d.gain(Dv, dt), "o": d.matrix(W, H * Dv, dt)}
        for n, c in (("q", H * D), ("k", H * D), ("v", H * Dv)):
            w[n + ".conv"] = d.normal(c, 4, scale=0.5, dtype=dt)
        return w
    qr, kr, rd = _latent_ranks(case)
    return {"dq": d.matrix(qr, W, dt), "dq.norm": d.gain(qr, dt), "uq": d.matrix(H * (D + rd), qr, dt), "dkv": d.matrix(kr + rd, W, dt),
            "dkv.norm": d.gain(kr, dt), "uk": d.matrix(H * D, kr, dt), "uv": d.matrix(H * Dv, kr, dt), "o": d.matrix(W, H * Dv, dt)}


def _mixer_spec(case):
    H, D, Dv, m = case["H"], case["D"], case["Dv"], case["mixer"]
    if m == "gla":
        return GlaMixerSpec(heads=H, dim=D, vdim=Dv, tau=16.0)
    if m == "retention":
        return RetentionMixerSpec(heads=H, dim=D, vdim=Dv, decay=_decays(H), rot=RotarySpec(D, 10000.0, "half"))
    if m == "state_space":
        return StateSpaceMixerSpec(heads=H, vdim=Dv, state=D, groups=1, conv=4, norm_groups=1)
    if m == "delta":
        return DeltaMixerSpec(heads=H, kv_heads=H, dim=D, vdim=Dv, conv=4, head_decay=True)
    qr, kr, rd = _latent_ranks(case)
    return LatentAttentionMixerSpec(heads=H, dim=D, rot_dim=rd, vdim=Dv, q_rank=qr, kv_rank=kr, scale=(D + rd) ** -0.5,
                                    rot=RotarySpec(rd, 10000.0), window=case["window"])


def _ff_weights(case, d):
    W, F, dt = case["width"], case["ff"], _dtype(case)
    if case["ff_kind"] == "dense":
        return {"gate": d.matrix(F, W, dt), "up": d.matrix(F, W, dt), "down": d.matrix(W, F, dt)}
    w = {"router": d.matrix(case["experts"], W, dt)}
    for e in range(case["experts"]):
        w[f"e{e}.gate"], w[f"e{e}.up"], w[f"e{e}.down"] = d.matrix(F, W, dt), d.matrix(F, W, dt), d.matrix(W, F, dt)
    if case["shared"]:
        s = case["shared"]
        w["shared.gate"], w["shared.up"], w["shared.down"] = d.matrix(s, W, dt), d.matrix(s, W, dt), d.matrix(W, s, dt)
    return w


def _attn_inputs(case, d):
    B, nh, nkv, hd = case["B"], case["nh"], case["nkv"], case["hd"]
    bf = torch.bfloat16
    if case["kind"] == "attn_prompt":
        S = case["S"]
        return d.normal(B, S, nh, hd, dtype=bf), d.normal(B, nkv, S, hd, dtype=bf), d.normal(B, nkv, S, hd, dtype=bf)
    kc, vc = d.normal(B, nkv, case["T"], hd, dtype=bf), d.normal(B, nkv, case["T"], hd, dtype=bf)
    return d.normal(B, (nh + 2 * nkv) * hd, dtype=bf), kc, vc


def _linear_inputs(case, d):
    x, w = d.normal(case["M"], case["K"], dtype=torch.bfloat16), d.matrix(case["N"], case["K"])
    gain = d.gain(case["K"]) if case["mode"] != "residual" else None
    res = d.normal(case["M"], case["N"], dtype=torch.bfloat16) if case["mode"] == "residual" else None
    return x, w, gain, res


def prepare(case, seed):
    d, kind = _Draws(seed), case["kind"]
    i32 = dict(dtype=torch.int32, device="cuda")
    if kind == "sample":
        return dict(case=case, logits=d.normal(case["B"], case["V"], scale=2.5), step=torch.full((1,), 3, **i32), seed=int(seed) % 100003)
    if kind == "linear":
        x, w, gain, res = _linear_inputs(case, d)
        return dict(case=case, x=x, w=w, gain=gain, res=res)
    if kind == "attn_prompt":
        q, kc, vc = _attn_inputs(case, d)
        return dict(case=case, q=q, kc=kc, vc=vc, pad=torch.tensor(_pads(case, case["B"]), **i32), filled=torch.zeros(1, **i32))
    if kind == "attn_decode":
        qkv, kc, vc = _attn_inputs(case, d)
        cos, sin = rotary_table(case["hd"], 500000.0, case["T"], torch.device("cuda"))
        splits, scratch = K.decode_attn_fused_plan(case["B"], case["nh"], case["nkv"], case["hd"], case["T"], kc.device)
        return dict(case=case, qkv=qkv, kc=kc, vc=vc, cos=cos, sin=sin, splits=splits, scratch=scratch,
                    filled=torch.full((1,), case["length"], **i32), pad=torch.tensor(_pads(case, case["B"]), **i32))
    if kind in ("llama", "folirax"):
        if kind == "llama":
            cfg = LLaMAConfig(vocab_size=case["vocab"], hidden_size=case["width"], intermediate_size=case["ff"], num_hidden_layers=case["layers"],
                              num_attention_heads=case["heads"], num_key_value_heads=case["kv"], max_sequence_length=1024, rms_norm_eps=EPS,
                              rope_theta=500000.0)
            engine = B200Engine.from_tree(cfg, _llama_tree(case, d))
            engine.mega_write_logits = True            # the caller reads the logits of a step
        else:
            cfg = FoliraxConfig.from_dict({"architecture": "Folirax", "vocab": case["vocab"], "width": case["width"], "norm": {"eps": EPS},
                                           "logit_scale": 0.5, "logit_softcap": 30.0, "layers": _folirax_layers(case)})
            engine = HybridEngine(cfg, _folirax_tensors(case, d))
        ids = d.ints(case["vocab"], case["B"], case["P"])
        mask = torch.ones_like(ids)
        for b, n in enumerate(_request_pads(case)):
            mask[b, :n] = 0
        feed = d.ints(case["vocab"], case["steps"], case["B"]).to(torch.int32).cpu().pin_memory()
        return dict(case=case, engine=engine, ids=ids, mask=mask, feed=feed)
    if kind == "mixer":
        dt, B, S = _dtype(case), case["B"], case["S"]
        mixer = MIXERS[_mixer_spec(case).kind](_mixer_spec(case), _mixer_weights(case, d), EPS)
        kv, dev = mixer.new_cache(B, S, torch.device("cuda")), torch.device("cuda")
        cache = HybridCache(k=torch.zeros(1, device=dev), v=torch.zeros(1, device=dev), index=0, pad_left=torch.zeros(B, **i32),
                            len_dev=torch.zeros(1, **i32), ks=[kv[0] if kv is not None else None], vs=[kv[1] if kv is not None else None],
                            states=[mixer.new_state(B, dev)], length=S)
        rot = getattr(mixer.spec, "rot", None)
        rope = rotary_table(rot.dims, rot.base, S, dev) if rot is not None else rotary_table(2, 1.0, 1, dev)
        return dict(case=case, mixer=mixer, cache=cache, rope=rope, h=d.normal(B * S, case["width"], dtype=dt))
    spec = (DenseMlpSpec(ff=case["ff"], act="gelu_tanh", gated=True) if case["ff_kind"] == "dense" else
            MoeMlpSpec(experts=case["experts"], top=case["top"], ff=case["ff"], act="silu", score="softmax", gated=True, shared_ff=case["shared"],
                       shared_gate=False))
    layer = (DenseFeedForward if case["ff_kind"] == "dense" else MoeFeedForward)(spec, _ff_weights(case, d))
    return dict(case=case, layer=layer, h=d.normal(case["M"], case["width"], dtype=_dtype(case)))


# ------------------------------------------------------------------------------------------ one pass
def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind == "sample":
        return K.sample_full(s["logits"], temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"], seed=s["seed"], step=s["step"])
    if kind == "linear":
        mode = {"swiglu": K.SWIGLU, "residual": K.RESIDUAL, "plain": K.PLAIN}[case["mode"]]
        return K.linear(s["x"], s["w"], norm_w=s["gain"], eps=EPS, residual=s["res"], mode=mode)
    if kind == "attn_prompt":
        return K.prefill_attn(s["q"], s["kc"], s["vc"], 0, case["S"], s["pad"], s["filled"])
    if kind == "attn_decode":
        out = K.decode_attn_fused(s["qkv"], s["kc"], s["vc"], s["cos"], s["sin"], s["filled"], s["pad"], case["nh"], case["nkv"], case["hd"],
                                  s["splits"], s["scratch"])
        at = case["length"]
        return out, s["kc"][:, :, at], s["vc"][:, :, at]
    if kind in ("llama", "folirax"):
        stream = s["engine"].begin_stream(s["ids"], s["mask"], max_length=case["P"] + case["steps"] + 2)
        first = stream.logits().clone()
        for t in range(case["steps"]):
            stream.step(s["feed"][t])
        return first, stream.logits()
    if kind == "mixer":
        cache = s["cache"]
        cache.set_index(0)
        y = s["mixer"].forward(s["h"], case["B"], case["S"], cache, 0, s["rope"])
        kept = cache.ks[0] if case["mixer"] == "latent" else cache.states[0]
        return y, kept
    return s["layer"].run(s["h"])


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def _seen_pairs(S, window):
    """Pairs of a query and a key it sees, per head, over S tokens."""
    if window <= 0 or window >= S:
        return S * (S + 1) // 2
    return window * (window + 1) // 2 + (S - window) * window


def work(case):
    kind = case["kind"]
    if kind == "sample":
        return {"bytes": 4 * case["B"] * case["V"], "flops": 4 * case["B"] * case["V"]}
    if kind == "linear":
        M, N, Kd = case["M"], case["N"], case["K"]
        out = M * N // 2 if case["mode"] == "swiglu" else M * N * (2 if case["mode"] == "residual" else 1)
        return {"bytes": 2 * (M * Kd + N * Kd + out), "flops": 2 * M * N * Kd}
    if kind == "attn_prompt":
        B, S, nh, nkv, hd = case["B"], case["S"], case["nh"], case["nkv"], case["hd"]
        pairs = sum(_seen_pairs(S - p, 0) for p in _pads(case, B))
        return {"bytes": 2 * B * S * hd * (2 * nh + 2 * nkv), "flops": 4 * pairs * nh * hd}
    if kind == "attn_decode":
        B, nh, nkv, hd = case["B"], case["nh"], case["nkv"], case["hd"]
        keys = sum(case["length"] + 1 - p for p in _pads(case, B))
        return {"bytes": 4 * keys * nkv * hd + 2 * B * hd * (2 * nh + 2 * nkv), "flops": 4 * keys * nh * hd}
    if kind in ("llama", "folirax"):
        W, F, V, n = case["width"], case["ff"], case["vocab"], case["layers"]
        hd = case["heads"] * 128
        if kind == "llama":
            weights = n * (2 * W * hd + 2 * W * case["kv"] * 128 + 3 * W * F)
        else:
            gla, own = 2 * W * hd * 2 + 2 * W * case["heads"] * 64 + W * 16, 2 * W * hd + 2 * W * case["kv"] * 128
            weights = n // 4 * (2 * gla + own + 2 * W * hd + 3 * 2 * W * F)
        tokens = case["B"] * (case["P"] + case["steps"])
        return {"bytes": 2 * (case["steps"] + 1) * (weights + W * V), "flops": 2 * tokens * weights + 2 * case["B"] * (case["steps"] + 1) * W * V}
    if kind == "mixer":
        B, S, W, H, D, Dv = (case[k] for k in ("B", "S", "width", "H", "D", "Dv"))
        M, el = B * S, 4 if case["dtype"] == "f32" else 2
        if case["mixer"] == "latent":
            qr, kr, rd = _latent_ranks(case)
            weights = qr * W + H * (D + rd) * qr + (kr + rd) * W + H * (D + Dv) * kr + W * H * Dv
            flops = 2 * M * weights + 2 * B * _seen_pairs(S, case["window"]) * H * (D + rd + Dv)
            kept = M * (kr + rd) * el
        else:
            qk = 2 * D if case["mixer"] == "state_space" else 2 * H * D
            weights = W * (qk + 3 * H * Dv + (H if case["mixer"] in ("state_space", "delta") else 0))
            flops, kept = 2 * M * weights + 4 * M * H * D * Dv, 4 * B * H * D * Dv
        return {"bytes": el * (weights + M * W) + 4 * M * W + kept, "flops": flops}
    M, W, F = case["M"], case["width"], case["ff"]
    el = 4 if case["dtype"] == "f32" else 2
    if case["ff_kind"] == "dense":
        return {"bytes": el * (3 * W * F + M * W) + 4 * M * W, "flops": 6 * M * W * F}
    used = min(case["experts"], M * case["top"])
    return {"bytes": el * (3 * W * F * used + 3 * W * case["shared"] + M * W) + 4 * M * W, "flops": 6 * M * W * (F * case["top"] + case["shared"])}


def tolerance(case):
    """bfloat16 outputs of fp32-accumulated sums round at 2^-9 of a value; what is computed and stored in fp32 from bfloat16 intermediates
    carries their rounding; true float32 paths differ by the order of their sums."""
    kind = case["kind"]
    if kind == "sample":
        return "exact"                                 # integer sums of a fixed-point mass: any order gives the same token
    if kind in ("llama", "folirax"):
        return {"rel": 5e-2}                           # roundings of one layer travel through the rest
    if case.get("dtype") == "f32":
        return {"rel": 2e-5}
    return {"rel": 1e-2}


# ------------------------------------------------------------------------------------------ the results in 64 bits
def _unit(x, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _softplus(z):
    return torch.clamp(z, min=0.0) + torch.log1p(torch.exp(-z.abs()))


def _turn(x, pos, dims, base, layout="interleaved"):
    """x [T, heads, n]: the leading `dims` channels of a head turned in pairs by pos · base^(-2i/dims)."""
    i = torch.arange(dims // 2, dtype=F64, device=x.device)
    ang = pos.to(F64)[:, None] * base ** (-2.0 * i / dims)
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    out = x.clone()
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if layout == "interleaved" else (slice(0, dims // 2), slice(dims // 2, dims))
    u, v = x[..., a], x[..., b]
    out[..., a], out[..., b] = u * c - v * s, v * c + u * s
    return out


def _attend(q, k, v, scale, window=0):
    """q [T, H, D] at the last T of the keys' positions; k [N, G, D], v [N, G, Dv] -> [T, H, Dv], causal."""
    T, H, N, G = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
    i = torch.arange(N - T, N, device=q.device)[:, None]
    j = torch.arange(N, device=q.device)[None, :]
    hidden = (j > i) | (i - j >= window) if window > 0 else j > i
    out = []
    for h in range(H):
        g = h * G // H
        s = (q[:, h] @ k[:, g].T * scale).masked_fill(hidden, -math.inf)
        out.append(torch.softmax(s, -1) @ v[:, g])
    return torch.stack(out, 1)


def _gla(h, w, H, D, Dv, tau=16.0):
    """h [B, T, W] -> (input of the output projection [B, T, H·Dv], state [B, H, D, Dv]); token by token."""
    B, T, _ = h.shape
    q, k = (h @ w["q"].T).view(B, T, H, D) * D ** -0.5, (h @ w["k"].T).view(B, T, H, D)
    v = (h @ w["v"].T).view(B, T, H, Dv)
    alpha = torch.sigmoid((h @ w["a1"].T) @ w["a2"].T + w["a2.b"]).pow(1.0 / tau).view(B, T, H, D)
    o, S = _linear_scan(q, k, v, alpha)
    return (_unit(o) * w["norm"]).reshape(B, T, H * Dv) * _silu(h @ w["g"].T), S


def _linear_scan(q, k, v, alpha):
    """S_t = diag(alpha_t) S_(t-1) + k_t v_tᵀ, o_t = S_tᵀ q_t over [B, T, H, ·]."""
    B, T, H, D = q.shape
    S = torch.zeros(B, H, D, v.shape[-1], dtype=F64, device=q.device)
    o = torch.empty(B, T, H, v.shape[-1], dtype=F64, device=q.device)
    for t in range(T):
        S = alpha[:, t, :, :, None] * S + k[:, t, :, :, None] * v[:, t, :, None]
        o[:, t] = torch.einsum("bhdv,bhd->bhv", S, q[:, t])
    return o, S


def _conv(x, w):
    """Causal convolution over time of x [B, T, C] with w [C, taps], the last tap on the current token."""
    taps = w.shape[1]
    xp = torch.cat([torch.zeros_like(x[:, :taps - 1]) if x.shape[1] >= taps - 1 else x.new_zeros(x.shape[0], taps - 1, x.shape[2]), x], 1)
    return sum(xp[:, j:j + x.shape[1]] * w[:, j] for j in range(taps))


def _conv_state(x, taps=4):
    """The last taps - 1 inputs of every row (zeros before the start)."""
    return torch.cat([x.new_zeros(x.shape[0], taps - 1, x.shape[2]), x], 1)[:, -(taps - 1):]


def _mixer_exact(case, h, w):
    B, S, H, D, Dv, m = (case[k] for k in ("B", "S", "H", "D", "Dv", "mixer"))
    W = case["width"]
    h = h.view(B, S, W)
    pos = torch.arange(S, device=h.device)
    if m == "gla":
        y, state = _gla(h, w, H, D, Dv)
        return (y @ w["o"].T).view(B * S, W), state
    if m == "retention":
        q, k = ((h @ w[n].T).view(B, S, H, D) for n in ("q", "k"))
        q = torch.stack([_turn(r, pos, D, 10000.0, "half") for r in q])
        k = torch.stack([_turn(r, pos, D, 10000.0, "half") for r in k]) * D ** -0.5
        alpha = torch.tensor(_decays(H), dtype=torch.float64, device=h.device)[None, None, :, None].expand(B, S, H, D)
        o, state = _linear_scan(q, k, (h @ w["v"].T).view(B, S, H, Dv), alpha)
        return ((_unit(o).reshape(B, S, H * Dv) * _silu(h @ w["g"].T)) @ w["o"].T).view(B * S, W), state
    if m == "state_space":
        inner = H * Dv
        y = h @ w["in"].T
        z, raw, dt = y[..., :inner], y[..., inner:2 * inner + 2 * D], _softplus(y[..., 2 * inner + 2 * D:] + w["dt_bias"])
        u = _silu(_conv(raw, w["conv"]) + w["conv.b"])
        x = u[..., :inner].reshape(B, S, H, Dv)
        k, q = (u[..., a:a + D][:, :, None].expand(B, S, H, D) for a in (inner, inner + D))
        alpha = torch.exp(-torch.exp(w["A_log"]) * dt)[..., None].expand(B, S, H, D)
        o, state = _linear_scan(q, k, x * dt[..., None], alpha)
        o = (o + w["D"][:, None] * x).reshape(B, S, inner) * _silu(z)
        return ((_unit(o) * w["norm"]) @ w["o"].T).view(B * S, W), (state, _conv_state(raw))
    if m == "delta":
        raw = torch.cat([h @ w[n].T for n in ("q", "k", "v")], -1)
        u = _silu(_conv(raw, torch.cat([w[n + ".conv"] for n in ("q", "k", "v")], 0)))
        q, k, v = u[..., :H * D].reshape(B, S, H, D), u[..., H * D:2 * H * D].reshape(B, S, H, D), u[..., 2 * H * D:].reshape(B, S, H, Dv)
        q, k = (z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
        q = q * D ** -0.5
        beta = torch.sigmoid(h @ w["b"].T)
        decay = torch.exp(-torch.exp(w["A_log"]) * _softplus(h @ w["a"].T + w["dt_bias"]))
        state = torch.zeros(B, H, D, Dv, dtype=F64, device=h.device)
        o = torch.empty(B, S, H, Dv, dtype=F64, device=h.device)
        for t in range(S):
            state = decay[:, t, :, None, None] * state
            e = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhdv,bhd->bhv", state, k[:, t]))
            state = state + k[:, t, :, :, None] * e[:, :, None]
            o[:, t] = torch.einsum("bhdv,bhd->bhv", state, q[:, t])
        o = (_unit(o) * w["norm"]).reshape(B, S, H * Dv) * _silu(h @ w["g"].T)
        return (o @ w["o"].T).view(B * S, W), (state, _conv_state(raw))
    qr, kr, rd = _latent_ranks(case)
    rows, kept = [], []
    for b in range(B):
        q = ((_unit(h[b] @ w["dq"].T) * w["dq.norm"]) @ w["uq"].T).view(S, H, D + rd)
        low = h[b] @ w["dkv"].T
        c = _unit(low[:, :kr]) * w["dkv.norm"]
        shared = _turn(low[:, None, kr:], pos, rd, 10000.0)
        q = torch.cat([q[..., :D], _turn(q[..., D:], pos, rd, 10000.0)], -1)
        k = torch.cat([(c @ w["uk"].T).view(S, H, D), shared.expand(S, H, rd)], -1)
        o = _attend(q, k, (c @ w["uv"].T).view(S, H, Dv), (D + rd) ** -0.5, case["window"])
        rows.append(o.reshape(S, H * Dv) @ w["o"].T)
        kept.append(torch.cat([c, shared[:, 0]], -1))
    return torch.cat(rows), torch.stack(kept)


def _ff_exact(case, h, w):
    if case["ff_kind"] == "dense":
        return (_gelu(h @ w["gate"].T) * (h @ w["up"].T)) @ w["down"].T
    val, idx = torch.softmax(h @ w["router"].T, -1).topk(case["top"], -1)
    val = val / val.sum(-1, keepdim=True)
    out = torch.zeros_like(h)
    for e in range(case["experts"]):
        m, c = torch.nonzero(idx == e, as_tuple=True)
        if m.numel():
            g, u, dn = (w[f"e{e}.{n}"].to(F64) for n in ("gate", "up", "down"))
            out.index_add_(0, m, val[m, c][:, None] * ((_silu(h[m] @ g.T) * (h[m] @ u.T)) @ dn.T))
    if case["shared"]:
        out = out + (_silu(h @ w["shared.gate"].T) * (h @ w["shared.up"].T)) @ w["shared.down"].T
    return out


def _llama_exact(case, tree, tokens):
    """Logits [T, V] of one sequence."""
    W, H, G = case["width"], case["heads"], case["kv"]
    t, pos, T = tree["transformer"], torch.arange(len(tokens), device="cuda"), len(tokens)
    x = t["wte"]["embedding"][tokens].to(F64)
    for i in range(case["layers"]):
        l = t["h"][str(i)]
        a, f = l["attention"], l["feed_forward"]
        k64 = lambda m: m["kernel"].to(F64)            # noqa: E731
        h = _unit(x) * k64(l["attention_norm"])
        q = _turn((h @ k64(a["wq"])).view(T, H, 128), pos, 128, 500000.0)
        k = _turn((h @ k64(a["wk"])).view(T, G, 128), pos, 128, 500000.0)
        x = x + _attend(q, k, (h @ k64(a["wv"])).view(T, G, 128), 128 ** -0.5).reshape(T, H * 128) @ k64(a["wo"])
        h = _unit(x) * k64(l["ffn_norm"])
        x = x + (_silu(h @ k64(f["w1"])) * (h @ k64(f["w3"]))) @ k64(f["w2"])
    return x[[case["_first"], T - 1]], t


def _folirax_exact(case, tensors, tokens):
    """Normed stream of one sequence, the two rows whose logits are read."""
    W, H, G = case["width"], case["heads"], case["kv"]
    T = len(tokens)
    pos = torch.arange(T, device="cuda")
    norm = lambda z, n: _unit(z) * (1.0 + tensors[n].to(F64))         # noqa: E731
    x = tensors["embed"][tokens].to(F64)
    kv = {}
    for i, l in enumerate(_folirax_layers(case)):
        p = f"l{i}."
        w = {k[len(p) + 4:]: v.to(F64) for k, v in tensors.items() if k.startswith(p + "mix.")}
        h = norm(x, p + "norm1")
        if l["type"] == "gla":
            y = _gla(h[None], w, H, 64, 128)[0][0]
        else:
            turned = lambda z, n: _unit(_turn(z.view(T, n, 128), pos, 64, 10000.0))      # noqa: E731
            if l["mixer"].get("kv_from") is None:
                kv[i] = turned(h @ w["k"].T, G), (h @ w["v"].T).view(T, G, 128)
            k, v = kv[i if l["mixer"].get("kv_from") is None else i - 1]
            y = (_attend(turned(h @ w["q"].T, H), k, v, 128 ** -0.5) * torch.sigmoid(h @ w["g"].T)[..., None]).reshape(T, H * 128)
        x = x + norm(y @ w["o"].T, p + "norm1b")
        if l["mlp"] is not None:
            h = norm(x, p + "norm2")
            x = x + norm(torch.relu(h @ tensors[p + "mlp.up"].to(F64).T) ** 2 @ tensors[p + "mlp.down"].to(F64).T, p + "norm2b")
    return norm(x[[case["_first"], T - 1]], "final.norm")


@torch.no_grad()
def exact(case, seed):
    d, kind = _Draws(seed), case["kind"]
    if kind == "sample":
        return None
    if kind == "linear":
        x, w, gain, res = (None if v is None else v.to(F64) for v in _linear_inputs(case, d))
        y = (_unit(x) * gain if gain is not None else x) @ w.T
        if case["mode"] == "swiglu":
            return _silu(y[:, 0::2]) * y[:, 1::2]
        return y + res if res is not None else y
    if kind == "attn_prompt":
        q, kc, vc = (v.to(F64) for v in _attn_inputs(case, d))
        rows = []
        for b, p in enumerate(_pads(case, case["B"])):
            o = _attend(q[b, p:], kc[b, :, p:].transpose(0, 1), vc[b, :, p:].transpose(0, 1), case["hd"] ** -0.5)
            rows.append(torch.cat([torch.zeros((p, *o.shape[1:]), dtype=F64, device=o.device), o]))
        return torch.stack(rows).view(case["B"], case["S"], -1)
    if kind == "attn_decode":
        qkv, kc, vc = (v.to(F64) for v in _attn_inputs(case, d))
        nh, nkv, hd, at = case["nh"], case["nkv"], case["hd"], case["length"]
        outs, keys = [], []
        for b, p in enumerate(_pads(case, case["B"])):
            x = qkv[b].view(1, nh + 2 * nkv, hd)
            qk = _turn(x[:, :nh + nkv], torch.tensor([at - p], device="cuda"), hd, 500000.0)
            k = torch.cat([kc[b, :, p:at].transpose(0, 1), qk[:, nh:]])
            v = torch.cat([vc[b, :, p:at].transpose(0, 1), x[:, nh + nkv:]])
            outs.append(_attend(qk[:, :nh], k, v, hd ** -0.5).reshape(1, nh * hd))
            keys.append(qk[0, nh:])
        return torch.cat(outs), torch.stack(keys), qkv.view(-1, nh + 2 * nkv, hd)[:, nh + nkv:]
    if kind in ("llama", "folirax"):
        weights = _llama_tree(case, d) if kind == "llama" else _folirax_tensors(case, d)
        ids = d.ints(case["vocab"], case["B"], case["P"])
        feed = d.ints(case["vocab"], case["steps"], case["B"])
        rows = []
        for b, p in enumerate(_request_pads(case)):
            tokens = torch.cat([ids[b, p:], feed[:, b]])
            c = dict(case, _first=case["P"] - p - 1)
            if kind == "llama":
                x, t = _llama_exact(c, weights, tokens)
                rows.append((_unit(x) * t["ln_f"]["kernel"].to(F64)) @ weights["lm_head"]["kernel"].to(F64))
            else:
                rows.append(30.0 * torch.tanh(_folirax_exact(c, weights, tokens) @ weights["head"].to(F64).T * (0.5 / 30.0)))
        both = torch.stack(rows)
        return both[:, 0], both[:, 1]
    if kind == "mixer":
        w = {k: v.to(F64) for k, v in _mixer_weights(case, d).items()}
        return _mixer_exact(case, d.normal(case["B"] * case["S"], case["width"], dtype=_dtype(case)).to(F64), w)
    w = _ff_weights(case, d)
    h = d.normal(case["M"], case["width"], dtype=_dtype(case)).to(F64)
    return _ff_exact(case, h, {k: (v if k.startswith("e") else v.to(F64)) for k, v in w.items()})

"""The work this framework is measured on: what its users have it do, through the entry points they call.

Two families are served.  Dia turns text into codec frames: one text pass through the encoder, one pass over the voice prompt and
then a frame per decode step.  The decoder-only language models take prompt portions and decode rows of several requests in one
step; six designs are built from the same mechanisms, so besides whole calls the cases take one mechanism at a time (an attention,
a recurrence, a mixture of experts) at the operator boundary that holds it.

Kinds of a case
  dia_frame     ``Decoder.decode_step``: one codec frame of Dia-1.6B behind ``slot`` cached ones (classifier-free guidance: two rows)
  dia_text      ``Encoder``: the text of one utterance
  dia_prompt    ``Decoder.forward``: a voice prompt fills the caches before the first generated frame
  sink          ``LMEngine.op_mixer``: Pubopel's grouped-query attention (score cap, distance bias, window that keeps the first tokens)
  latent        ``LMEngine.op_mixer``: Fipadra's attention over one cached latent per token, with a turned key part and a window
  talk          ``LMEngine.op_mixer``: Kupelix's attention whose scores are mixed across heads
  delta         ``LMEngine.op_mixer``: Fipadra's gated delta rule (a matrix state per head), several requests of uneven length
  experts       ``LMEngine.op_ff``: Pubopel's routed experts with a shared one
  model_prompt  ``CausalLM.run_step``: whole prompts through a Forilorn model, the logits behind each
  model_decode  ``CausalLM.run_step``: one token for each of several running requests of a Forilorn model

``rows`` of a language-model case are the new tokens of each request ("700,33,1" is three requests in one step); ``past`` is how many
tokens every request's state holds before.  ``dtype`` is the precision a user asks ``CausalLM`` for.
"""

from __future__ import annotations

import math

import torch

from dia_tts_prune_b200.config import DataConfig, DecoderConfig, DiaConfig, EncoderConfig, ModelConfig
from dia_tts_prune_b200.lm_config import FipadraConfig, ForilornConfig, KupelixConfig, PubopelConfig
from dia_tts_prune_b200.lm_model import CausalLM
from dia_tts_prune_b200.model import Dia
from dia_tts_prune_b200.state import DecoderInferenceState, EncoderInferenceState, KVCache

EPS = 1e-5
PAGE = 64

# the two model sizes that the repository's benchmark uses for every language-model design
W2048 = dict(width=2048, heads=16, kv_heads=4, dim=128)
W1024 = dict(width=1024, heads=8, kv_heads=2, dim=128)
LAT2048 = dict(width=2048, heads=16, dim=96, rot_dim=32, vdim=128, q_rank=768, kv_rank=256)
LAT1024 = dict(width=1024, heads=8, dim=96, rot_dim=32, vdim=128, q_rank=384, kv_rank=128)
MODEL2048 = dict(layers=4, ff=6144, vocab=32768, buckets=65521, chunk=2048, window=1024)
MODEL1024 = dict(layers=4, ff=1536, vocab=16384, buckets=65521, chunk=2048, window=512)


def listed():
    return [
        # the frame loop of the text-to-speech model in the middle of an utterance: small work, a chain of weight reads
        dict(name="dia_frame_1500", kind="dia_frame", layers=18, slot=1500, text=117),
        # the text of an utterance (60 to 200 bytes are usual; the model takes 1024)
        dict(name="dia_text_200", kind="dia_text", layers=12, text=200),
        # a ten-second voice prompt (861 codec frames) in front of the utterance
        dict(name="dia_prompt_861", kind="dia_prompt", layers=18, frames=861, text=129),
        # a long prompt through the attention of a window model, one portion of 4096 rows
        dict(name="sink_4096", kind="sink", **W2048, window=1024, keep_first=4, softcap=30.0, rows="4096", past=0, dtype="bfloat16"),
        # the same for attention over a cached latent
        dict(name="latent_4096", kind="latent", **LAT2048, window=1024, rows="4096", past=0, dtype="bfloat16"),
        # three prompts of uneven length in one step through the attention that mixes scores across heads
        dict(name="talk_ragged", kind="talk", **W1024, vdim=128, rows="1500,333,215", past=0, dtype="bfloat16"),
        # a batch of prompts of uneven length through a recurrence
        dict(name="delta_ragged", kind="delta", **W2048, vdim=128, taps=4, rows="1024,700,513,37,1", past=0, dtype="bfloat16"),
        # the mixture of experts on a prompt portion
        dict(name="experts_4096", kind="experts", width=2048, experts=8, top=2, ff=2048, shared=4096, rows="4096", dtype="bfloat16"),
        # time to the first token of a whole model: one long prompt
        dict(name="model_prompt_4096", kind="model_prompt", **LAT2048, kv_heads=4, head_dim=128, **MODEL2048, rows="4096", dtype="bfloat16"),
        # a step of two odd-sized prompts in the precision the parity tools ask for
        dict(name="model_prompt_f32", kind="model_prompt", **LAT1024, kv_heads=2, head_dim=128, **MODEL1024, rows="777,201", dtype="float32"),
        # generation: one running request (latency), and eight (a small server's batch)
        dict(name="model_decode_1", kind="model_decode", **LAT2048, kv_heads=4, head_dim=128, **MODEL2048, requests=1, past=1024, dtype="bfloat16"),
        dict(name="model_decode_8", kind="model_decode", **LAT2048, kv_heads=4, head_dim=128, **MODEL2048, requests=8, past=1024, dtype="bfloat16"),
    ]


def draw(rng):
    def size(lo, hi):                                             # even over the logarithm, odd sizes among them
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def ragged(total, most):                                      # a step of up to `most` requests
        n = rng.randint(1, most)
        cuts = sorted(rng.randint(1, total) for _ in range(n - 1))
        parts = [b - a for a, b in zip([0] + cuts, cuts + [total])]
        return ",".join(str(p) for p in parts if p > 0) or "1"

    def heads(dims=(64, 128)):
        d, kv = rng.choice(dims), rng.choice((1, 2, 4))
        h = kv * rng.choice((1, 2, 4, 8) if kv < 4 else (1, 2, 4))
        return dict(width=rng.choice((512, 1024, 1536, 2048)), heads=h, kv_heads=kv, dim=d)

    def latent():
        return dict(width=rng.choice((512, 1024, 2048)), heads=rng.choice((4, 8, 16)), dim=rng.choice((64, 96, 128)), rot_dim=rng.choice((16, 32, 64)),
                    vdim=rng.choice((64, 128)), q_rank=rng.choice((192, 384, 768)), kv_rank=rng.choice((64, 128, 192, 256)))

    dtype = "float32" if rng.random() < 0.2 else "bfloat16"
    most = 1536 if dtype == "float32" else 4096
    kind = rng.choice(("dia_frame", "dia_text", "dia_prompt", "sink", "latent", "talk", "delta", "experts", "model_prompt", "model_prompt",
                       "model_decode", "model_decode"))
    if kind == "dia_frame":
        return dict(kind=kind, layers=rng.randint(2, 18), slot=size(1, 3000), text=size(10, 1000))
    if kind == "dia_text":
        return dict(kind=kind, layers=12, text=size(10, 1024))
    if kind == "dia_prompt":
        return dict(kind=kind, layers=rng.randint(2, 9), frames=size(20, 1500), text=size(10, 600))
    if kind == "sink":
        win = rng.choice((0, 256, 1024))
        return dict(kind=kind, **heads(), window=win, keep_first=rng.choice((0, 4)) if win else 0, softcap=rng.choice((0.0, 30.0)),
                    rows=ragged(size(1, most), 6), past=rng.choice((0, 0, size(1, 1500))), dtype=dtype)
    if kind == "latent":
        return dict(kind=kind, **latent(), window=rng.choice((0, 512, 1024)), rows=ragged(size(1, most // 2), 6), past=rng.choice((0, 0, size(1, 1500))),
                    dtype=dtype)
    if kind == "talk":
        return dict(kind=kind, **heads(), vdim=rng.choice((64, 128)), rows=ragged(size(1, most // 2), 6), past=rng.choice((0, 0, size(1, 1000))),
                    dtype=dtype)
    if kind == "delta":
        return dict(kind=kind, **heads(), vdim=rng.choice((64, 128)), taps=4, rows=ragged(size(1, most // 2), 8), past=0, dtype=dtype)
    if kind == "experts":
        return dict(kind=kind, width=rng.choice((512, 1024, 2048)), experts=rng.choice((4, 8, 16)), top=rng.choice((1, 2)), ff=rng.choice((256, 512, 2048)),
                    shared=rng.choice((0, 1024, 4096)), rows=str(size(1, most)), dtype=dtype)
    sizes = dict(**latent(), kv_heads=rng.choice((1, 2, 4)), head_dim=rng.choice((64, 128)), layers=rng.choice((2, 4)), ff=rng.choice((1024, 1536, 4096)),
                 vocab=rng.choice((8192, 16384)), buckets=65521, chunk=rng.choice((0, 512, 2048)), window=rng.choice((0, 512, 1024)))
    if kind == "model_prompt":
        return dict(kind=kind, **sizes, rows=ragged(size(16, most // 2), 6), dtype=dtype)
    return dict(kind=kind, **sizes, requests=rng.randint(1, 24), past=size(16, 1500), dtype=dtype)


# ---- inputs ------------------------------------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")


class _Draw:
    """Random tensors of a seed: bfloat16 weights ~ N(0, 1 / fan_in) and vectors around a mean, as checkpoints hold them."""

    def __init__(self, seed):
        self.dev = _device()
        self.g = torch.Generator(device=self.dev).manual_seed(int(seed) * 7919 + 17)

    def normal(self, *shape):
        return torch.randn(shape, generator=self.g, device=self.dev)

    def mat(self, n, k, gain=1.0):
        return (self.normal(n, k) * (gain * k ** -0.5)).to(torch.bfloat16)

    def vec(self, n, mean, spread):
        return (mean + spread * self.normal(n)).to(torch.bfloat16)

    def ints(self, n, high):
        return torch.randint(0, high, (n,), generator=self.g, device=self.dev).tolist()


def _rows(case):
    return [int(v) for v in case["rows"].split(",")]


def _dia_config(case):
    frames = case["frames"] if case["kind"] == "dia_prompt" else 3072
    n = case["layers"]
    return DiaConfig(
        model=ModelConfig(
            encoder=EncoderConfig(n_layer=n if case["kind"] == "dia_text" else 1, n_embd=1024, n_hidden=4096, n_head=16, head_dim=128),
            decoder=DecoderConfig(n_layer=1 if case["kind"] == "dia_text" else n, n_embd=2048, n_hidden=8192, gqa_query_heads=16, kv_heads=4,
                                  gqa_head_dim=128, cross_query_heads=16, cross_head_dim=128),
            src_vocab_size=256, tgt_vocab_size=1028),
        data=DataConfig(text_length=1024, audio_length=max(128, frames), channels=9))


def _dia_weights(case, r):
    """The parameters that the case's pass reads, by name, in the layout of a checkpoint."""
    cfg = _dia_config(case)
    w = {}

    def dense(name, shape, fan_in):
        w[name + ".weight"] = (r.normal(*shape) * fan_in ** -0.5).to(torch.bfloat16)

    def norm(name, n):
        w[name + ".weight"] = r.vec(n, 1.0, 0.05).float()

    def attention(p, dq, dkv, heads, kv, own_kv=True):
        dense(p + "q_proj", (dq, heads, 128), dq)
        if own_kv:
            dense(p + "k_proj", (dkv, kv, 128), dkv)
            dense(p + "v_proj", (dkv, kv, 128), dkv)
        dense(p + "o_proj", (heads, 128, dq), heads * 128)

    if case["kind"] == "dia_text":
        w["encoder.embedding.weight"] = r.normal(256, 1024).to(torch.bfloat16).float()
        for i in range(case["layers"]):
            p = f"encoder.layers.{i}."
            norm(p + "pre_sa_norm", 1024), norm(p + "post_sa_norm", 1024)
            attention(p + "self_attention.", 1024, 1024, 16, 16)
            dense(p + "mlp.wi_fused", (1024, 2, 4096), 1024)
            dense(p + "mlp.wo", (4096, 1024), 4096)
        norm("encoder.norm", 1024)
        return cfg, w
    for c in range(9):
        w[f"decoder.embeddings.{c}.weight"] = r.normal(1028, 2048).to(torch.bfloat16).float()
    for i in range(case["layers"]):
        p = f"decoder.layers.{i}."
        norm(p + "pre_sa_norm", 2048), norm(p + "pre_ca_norm", 2048), norm(p + "pre_mlp_norm", 2048)
        attention(p + "self_attention.", 2048, 2048, 16, 4)
        attention(p + "cross_attention.", 2048, 1024, 16, 16, own_kv=False)
        dense(p + "mlp.wi_fused", (2048, 2, 8192), 2048)
        dense(p + "mlp.wo", (8192, 2048), 8192)
    norm("decoder.norm", 2048)
    dense("decoder.logits_dense", (2048, 9, 1028), 2048)
    return cfg, w


def _dia_inputs(case, r, cfg):
    """Text bytes, or codec tokens with the caches an utterance holds at that point (keys of a turned unit-scale head, values)."""
    if case["kind"] == "dia_text":
        return dict(text=torch.randint(1, 256, (1, case["text"]), generator=r.g, device=r.dev))
    frames = 1 if case["kind"] == "dia_frame" else case["frames"]
    slots = case["slot"] if case["kind"] == "dia_frame" else 0
    length = cfg.data.audio_length
    out = dict(tokens=torch.randint(0, 1024, (frames, 9), generator=r.g, device=r.dev, dtype=torch.int32), own=[], cross=[])
    for _ in range(case["layers"]):
        own = [torch.zeros(2, 4, length, 128, device=r.dev) for _ in range(2)]
        cross = [torch.zeros(2, 16, 1024, 128, device=r.dev) for _ in range(2)]
        for t in own:
            t[:, :, :slots] = r.normal(2, 4, slots, 128)
        for t in cross:                                           # the unconditional row sees no text
            t[1, :, :case["text"]] = r.normal(16, case["text"], 128)
        out["own"].append(own)
        out["cross"].append(cross)
    return out


def _rot_cfg(dims):
    return {"base": 10000.0, "dims": dims}


def _lm(case, r):
    """(configuration class, configuration, weights) of a language-model case."""
    k, D = case["kind"], case["width"]
    norm = {"eps": EPS}
    if k in ("sink", "experts"):
        H, G, d = (case["heads"], case["kv_heads"], case["dim"]) if k == "sink" else (1, 1, 64)
        m = {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "softcap": (case["softcap"] or None) if k == "sink" else None}
        if k == "sink" and case["window"]:
            m["mask"] = {"size": case["window"], "keep_first": case["keep_first"]}
        layer = {"type": "attention", "mixer": m}
        w = {"embed": r.mat(256, D), "head": r.mat(256, D), "l0.mix.q": r.mat(H * d, D), "l0.mix.k": r.mat(G * d, D), "l0.mix.o": r.mat(D, H * d),
             "l0.mix.q.norm": r.vec(H * d, 1.0, 0.05), "l0.mix.k.norm": r.vec(G * d, 1.0, 0.05), "l0.mix.temp": r.vec(H, 1.0, 0.1),
             "l0.mix.sink": r.vec(H, 0.0, 0.5), "l0.canon1": r.mat(D, 4), "l0.canon2": r.mat(D, 4)}
        for n in ("l0.norm1", "l0.norm1b", "l0.norm2", "l0.norm2b", "final.norm"):
            w[n], w[n + ".b"], w[n + ".alpha"] = r.vec(D, 1.0, 0.05), r.vec(D, 0.0, 0.02), torch.tensor(0.7, dtype=torch.bfloat16, device=r.dev)
        if k == "experts":
            E, F, S = case["experts"], case["ff"], case["shared"]
            layer["mlp"] = {"kind": "moe", "expert": {"ff": F}, "router": {"experts": E, "top": case["top"]}, "shared": {"ff": S} if S else None}
            w["l0.mlp.router"] = r.mat(E, D)
            for e in [f"e{e}" for e in range(E)] + (["shared"] if S else []):
                n = S if e == "shared" else F
                w[f"l0.mlp.{e}.gate"], w[f"l0.mlp.{e}.up"], w[f"l0.mlp.{e}.down"] = r.mat(n, D), r.mat(n, D), r.mat(D, n)
        return PubopelConfig, {"architecture": "Pubopel", "vocab": 256, "width": D, "canon": {"taps": 4}, "norm": norm, "layers": [layer]}, w

    def latent(q, gate):
        H, d, rd, dv, rq, R = (case[n] for n in ("heads", "dim", "rot_dim", "vdim", "q_rank", "kv_rank"))
        w.update({q + "dq": r.mat(rq, D), q + "dq.norm": r.vec(rq, 1.0, 0.05), q + "uq": r.mat(H * (d + rd), rq), q + "dkv": r.mat(R + rd, D),
                  q + "dkv.norm": r.vec(R, 1.0, 0.05), q + "uk": r.mat(H * d, R), q + "uv": r.mat(H * dv, R), q + "o": r.mat(D, H * dv)})
        if gate:
            w[q + "g"] = r.mat(H, D)
        m = {"heads": H, "dim": d, "rot_dim": rd, "vdim": dv, "q_rank": rq, "kv_rank": R, "scale": (d + rd) ** -0.5, "rot": _rot_cfg(rd)}
        if case["window"]:
            m["mask"] = {"size": case["window"]}
        return m

    w = {}
    if k == "latent":
        w = {"embed": r.mat(256, D), "embed.norm": r.vec(D, 1.0, 0.05), "final.norm": r.vec(D, 1.0, 0.05), "l0.norm1": r.vec(D, 1.0, 0.05)}
        m = latent("l0.mix.", False)
        return FipadraConfig, {"architecture": "Fipadra", "vocab": 256, "width": D, "norm": norm, "logit_scale": 1.0,
                               "layers": [{"type": "latent_attention", "mixer": m, "mlp": None}]}, w
    if k == "delta":
        H, G, d, dv, T = case["heads"], case["kv_heads"], case["dim"], case["vdim"], case["taps"]
        w = {"embed": r.mat(256, D), "embed.norm": r.vec(D, 1.0, 0.05), "final.norm": r.vec(D, 1.0, 0.05), "l0.norm1": r.vec(D, 1.0, 0.05),
             "l0.mix.b": r.mat(H, D), "l0.mix.a": r.mat(H, D), "l0.mix.A_log": r.vec(H, -1.0, 0.5), "l0.mix.dt_bias": r.vec(H, -2.0, 1.0),
             "l0.mix.norm": r.vec(dv, 1.0, 0.05), "l0.mix.g": r.mat(H * dv, D), "l0.mix.o": r.mat(D, H * dv)}
        for n, rows in (("q", G * d), ("k", G * d), ("v", H * dv)):
            w["l0.mix." + n], w[f"l0.mix.{n}.conv"] = r.mat(rows, D), r.mat(rows, T)
        m = {"heads": H, "kv_heads": G, "dim": d, "vdim": dv, "conv": T}
        return FipadraConfig, {"architecture": "Fipadra", "vocab": 256, "width": D, "norm": norm, "logit_scale": 1.0,
                               "layers": [{"type": "delta", "mixer": m, "mlp": None}]}, w
    if k == "talk":
        H, G, d, dv = case["heads"], case["kv_heads"], case["dim"], case["vdim"]
        w = {"embed": r.mat(256, D), "head": r.mat(256, D), "final.norm": r.vec(D, 1.0, 0.05), "final.norm.b": r.vec(D, 0.0, 0.02),
             "l0.norm1": r.vec(D, 1.0, 0.05), "l0.norm1.b": r.vec(D, 0.0, 0.02), "l0.mix.q": r.mat(H * d, D), "l0.mix.k": r.mat(G * d, D),
             "l0.mix.v": r.mat(G * dv, D), "l0.mix.g": r.mat(H, D), "l0.mix.o": r.mat(D, H * dv), "l0.mix.q.b": r.vec(H * d, 0.0, 0.1),
             "l0.mix.k.b": r.vec(G * d, 0.0, 0.1), "l0.mix.v.b": r.vec(G * dv, 0.0, 0.1), "l0.mix.q.norm": r.vec(d, 1.0, 0.05),
             "l0.mix.k.norm": r.vec(d, 1.0, 0.05), "l0.mix.sink": r.vec(H, 0.0, 0.5),
             "l0.mix.talk": (torch.eye(H, device=r.dev) + 0.3 * H ** -0.5 * r.normal(H, H)).to(torch.bfloat16)}
        m = {"heads": H, "kv_heads": G, "dim": d, "vdim": dv, "scale": d ** -0.5, "rot": _rot_cfg(d // 2)}
        return KupelixConfig, {"architecture": "Kupelix", "vocab": 256, "width": D, "norm": norm, "logit_scale": 1.0,
                               "layers": [{"type": "attention", "mixer": m, "mlp": None}]}, w
    # a whole model: attention and latent attention in turn, a gelu unit behind each, a pair table beside the embedding
    V, F, d, G = case["vocab"], case["ff"], case["head_dim"], case["kv_heads"]
    H = max(G, case["heads"])
    w = {"embed": r.mat(V, D), "bigram": r.mat(case["buckets"] + 1, D), "final.norm": r.vec(D, 0.0, 0.05)}
    layers = []
    for i in range(case["layers"]):
        q = f"l{i}.mix."
        w[f"l{i}.norm1"], w[f"l{i}.norm2"] = r.vec(D, 0.0, 0.05), r.vec(D, 0.0, 0.05)
        if i % 2 == 0:
            w[q + "q"], w[q + "k"], w[q + "g"], w[q + "o"] = r.mat(H * d, D), r.mat(G * d, D), r.mat(H * d, D), r.mat(D, H * d)
            m = {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "rot": _rot_cfg(d)}
            if case["chunk"]:
                m["mask"] = {"size": case["chunk"]}
        else:
            m = latent(q, True)
        w[f"l{i}.mlp.up"], w[f"l{i}.mlp.down"] = r.mat(F, D), r.mat(D, F)
        layers.append({"type": "latent_attention" if i % 2 else "attention", "mixer": m, "mlp": {"kind": "dense", "ff": F}})
    cfg = {"architecture": "Forilorn", "vocab": V, "width": D, "norm": norm, "residual_mult": 1.0, "layers": layers,
           "embedding": {"scale": 1.0, "bigram": {"buckets": case["buckets"], "mul_prev": 40503, "mul_cur": 10007}}}
    return ForilornConfig, cfg, w


def _lm_inputs(case, r):
    if case["kind"] == "model_prompt":
        return [r.ints(n, case["vocab"]) for n in _rows(case)]
    if case["kind"] == "model_decode":
        return [r.ints(case["past"] + 1, case["vocab"]) for _ in range(case["requests"])]
    rows, past = _rows(case), case.get("past", 0)
    return [r.normal(past + n, case["width"]) for n in rows]      # what a norm with weights near one hands the mechanism


# ---- one pass -----------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    r = _Draw(seed)
    if case["kind"].startswith("dia_"):
        return _prepare_dia(case, r)
    conf, cfg, weights = _lm(case, r)
    data = _lm_inputs(case, r)
    n, past = len(data), case.get("past", 0)
    longest = max(len(t) for t in data)
    total = sum(len(t) for t in data)
    model = CausalLM(conf.model_validate(cfg), weights, dtype=case["dtype"], device=r.dev, max_tokens=total + PAGE * n, max_sequences=n, page_size=PAGE,
                     max_rows=max(past, total - n * past, 1), max_sequence_tokens=longest + PAGE)
    s = dict(case=case, model=model)
    if case["kind"] == "model_prompt":
        s["entries"] = [{"id": str(i), "tokens": t, "want": [len(t) - 1]} for i, t in enumerate(data)]
        s["end"] = [e["id"] for e in s["entries"]]
        return s
    if case["kind"] == "model_decode":
        for i, t in enumerate(data):                              # the requests' prompts, a portion each
            model.run_step([{"id": str(i), "tokens": t[:-1], "want": []}])
        s["entries"] = [{"id": str(i), "tokens": t[-1:], "want": [0]} for i, t in enumerate(data)]
        return s
    if case["kind"] == "experts":
        s["h"] = data[0]
        return s
    seqs = [model.state.open(str(i)) for i in range(n)]
    for q, t in zip(seqs, data):
        model.state.reserve(q, len(t))
        if past:
            model.engine.op_mixer(0, t[:past], [(q, past, 0)])
    s["h"] = torch.cat([t[past:] for t in data])
    s["parts"] = [(q, len(t) - past, past) for q, t in zip(seqs, data)]
    return s


def _prepare_dia(case, r):
    cfg, w = _dia_weights(case, r)
    x = _dia_inputs(case, r, cfg)
    with torch.device(r.dev):
        dia = Dia(cfg, "bfloat16", r.dev)
    own = dict(dia.model.named_parameters())
    with torch.no_grad():
        for n, t in w.items():
            own[n].data = t
    dia.model.eval()
    s = dict(case=case, dia=dia, x=x)
    with torch.inference_mode():
        if case["kind"] == "dia_text":
            return s
        enc = EncoderInferenceState(max_seq_len=1024, device=r.dev, positions=torch.arange(1024, dtype=torch.float32, device=r.dev)[None, :].expand(2, -1),
                                    padding_mask=torch.zeros(2, 1024, dtype=torch.bool, device=r.dev), attn_mask=None)
        cross = [KVCache.from_kv(k, v) for k, v in x["cross"]]
        st = DecoderInferenceState.new(cfg, enc, torch.zeros(2, 1024, 1024, device=r.dev), cross, torch.bfloat16)
        st.text_len = case["text"]
        for c, (k, v) in zip(st.self_attn_cache, x["own"]):
            c.k, c.v = k, v
        s["state"] = st
        s["tokens"] = x["tokens"].unsqueeze(0).expand(2, -1, -1)
        dia.model.decoder.engine()                                # the weights as the kernels read them
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind.startswith("dia_"):
        return _run_dia(s)
    model = s["model"]
    if kind == "model_prompt":
        return model.run_step(s["entries"], s["end"])
    if kind == "model_decode":
        out = model.run_step(s["entries"])
        for e in s["entries"]:                                    # another token may follow the same context: take this one back
            model.state.sequences[e["id"]].length -= 1
        return out
    if kind == "experts":
        return model.engine.op_ff(0, s["h"])
    y = model.engine.op_mixer(0, s["h"], s["parts"])
    st = model.state
    if kind == "delta":
        return [y, st.rec_states[0], st.conv_tails[0]]
    return [y, st.latent_pages[0]] if kind == "latent" else [y, st.k_pages[0], st.v_pages[0]]


@torch.inference_mode()
def _run_dia(s):
    case, dia = s["case"], s["dia"]
    if case["kind"] == "dia_text":
        text = s["x"]["text"]
        n, dev = text.shape[1], text.device
        state = EncoderInferenceState(max_seq_len=n, device=dev, positions=torch.arange(n, dtype=torch.float32, device=dev)[None, :],
                                      padding_mask=torch.ones_like(text, dtype=torch.bool), attn_mask=None, valid_lens=[n])
        return dia.model.encoder(text, state)
    st = s["state"]
    if case["kind"] == "dia_frame":
        for c in st.self_attn_cache:
            c.current_idx = case["slot"]
        st.prepare_step(case["slot"])
        return dia.model.decoder.decode_step(s["tokens"], st)
    st.prepare_step(0, case["frames"])
    logits = dia.model.decoder.forward(s["tokens"], st)
    return [logits, [c.k for c in st.self_attn_cache], [c.v for c in st.self_attn_cache]]


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------------
def _pairs(rows, past, window, chunk=0):
    """(query, key) pairs that are seen, over all requests."""
    n = 0
    for m in rows:
        for i in range(past, past + m):
            lo = max(0, i - window + 1) if window else 0
            n += i + 1 - (max(lo, i - i % chunk) if chunk else lo)
    return n


def _keys(rows, past, window):
    """Cached positions behind the new rows that some row sees."""
    return sum(min(past, window - 1) if window else past for _ in rows)


def work(case):
    k = case["kind"]
    if k == "dia_text":
        n, L = case["text"], case["layers"]
        w = L * (4 * 1024 * 2048 + 3 * 1024 * 4096)
        return dict(bytes=2 * w + 4 * n * 1024 * 2, flops=2 * n * w + L * 4 * n * n * 2048)
    if k in ("dia_frame", "dia_prompt"):
        L, text = case["layers"], case["text"]
        T, past = (1, case["slot"]) if k == "dia_frame" else (case["frames"], 0)
        w = L * (2048 * (2048 + 1024) + 2048 * 2048 + 2 * 2048 * 2048 + 3 * 2048 * 8192) + 2048 * 9252
        keys = L * 8 * (2 * 4 * (past + T) * 128 + 16 * text * 128)
        pairs = 2 * _pairs([T], past, 0) + T * text
        return dict(bytes=2 * w + keys + 4 * 2 * T * 9252, flops=2 * 2 * T * w + L * 4 * 2048 * pairs)
    if k == "experts":
        D, n = case["width"], int(case["rows"])
        used = min(case["experts"], n * case["top"])
        active = case["top"] * 3 * D * case["ff"] + 3 * D * case["shared"] + D * case["experts"]
        return dict(bytes=2 * (used * 3 * D * case["ff"] + 3 * D * case["shared"] + D * case["experts"]) + 8 * n * D, flops=2 * n * active)
    D = case["width"]

    def attention(rows, past, H, G, d, dv, extra, window, chunk=0):
        n = sum(rows)
        w = D * (H * d + G * (d + dv)) + D * H * dv + extra
        return 2 * w + 4 * G * (d + dv) * (_keys(rows, past, window or chunk) + n), 2 * n * w + 2 * H * (d + dv) * _pairs(rows, past, window, chunk)

    def latent(rows, past, gate):
        H, d, rd, dv, rq, R = (case[x] for x in ("heads", "dim", "rot_dim", "vdim", "q_rank", "kv_rank"))
        n, seen = sum(rows), _pairs(rows, past, case["window"])
        w = D * (rq + R + rd + gate * H) + rq * H * (d + rd) + H * R * (d + dv) + D * H * dv
        # scores and values either per head from the up-projected keys and values, or against the latent itself
        per_pair = min(2 * (d + rd + dv), 2 * (2 * R + rd))
        return 2 * w + 4 * (R + rd) * (_keys(rows, past, case["window"]) + n), 2 * n * w + H * per_pair * seen

    if k in ("model_prompt", "model_decode"):
        rows, past = (_rows(case), 0) if k == "model_prompt" else ([1] * case["requests"], case["past"])
        n, H, G, d = sum(rows), max(case["kv_heads"], case["heads"]), case["kv_heads"], case["head_dim"]
        b = f = 0
        for i in range(case["layers"]):
            x = latent(rows, past, 1) if i % 2 else attention(rows, past, H, G, d, 0, D * H * d * 2, 0, case["chunk"])
            if i % 2 == 0:                                        # (the values are the projected keys, and still 2 d per pair and cached)
                x = (x[0] + 4 * G * d * n, x[1] + 2 * H * d * _pairs(rows, past, 0, case["chunk"]))
            b, f = b + x[0] + 4 * D * case["ff"], f + x[1] + 4 * n * D * case["ff"]
        return dict(bytes=b + 2 * D * case["vocab"] + 4 * len(rows) * case["vocab"], flops=f + 2 * len(rows) * D * case["vocab"])
    rows, past = _rows(case), case["past"]
    n = sum(rows)
    if k == "sink":
        b, f = attention(rows, past, case["heads"], case["kv_heads"], case["dim"], case["dim"], -D * case["kv_heads"] * case["dim"], case["window"])
    elif k == "talk":
        b, f = attention(rows, past, case["heads"], case["kv_heads"], case["dim"], case["vdim"], D * case["heads"], 0)
        f += 2 * case["heads"] ** 2 * _pairs(rows, past, 0)
    elif k == "latent":
        b, f = latent(rows, past, 0)
    else:
        H, G, d, dv = case["heads"], case["kv_heads"], case["dim"], case["vdim"]
        w = D * (2 * G * d + 3 * H * dv + 2 * H)
        b, f = 2 * w + 4 * len(rows) * H * d * dv, 2 * n * w + 8 * n * H * d * dv
    return dict(bytes=b + 8 * n * D, flops=f)


# ---- how far another correct implementation may be off ---------------------------------------------------------------------------
def tolerance(case):
    if case["kind"].startswith("dia_"):
        return {"rel": 1e-4, "max": 5e-3}                        # float32 operands through up to 18 layers, sums of thousands of terms
    if case["kind"].startswith("model_"):
        return {"rel": 1e-2, "max": 0.4} if case["dtype"] == "bfloat16" else {"rel": 2e-5, "max": 2e-3}
    return {"rel": 5e-3, "max": 0.2} if case["dtype"] == "bfloat16" else {"rel": 1e-5, "max": 1e-3}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------------------
def _rms(x, w=None, eps=EPS):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _turn(x, pos, base, dims):
    """x [T, heads, n]: pairs (2i, 2i + 1) of the first `dims` channels turn with the position."""
    if not dims:
        return x
    f = torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float64, device=x.device)
    a = pos.double()[:, None, None] * f
    y, c, s = x.clone(), torch.cos(a), torch.sin(a)
    y[..., 0:dims:2] = x[..., 0:dims:2] * c - x[..., 1:dims:2] * s
    y[..., 1:dims:2] = x[..., 1:dims:2] * c + x[..., 0:dims:2] * s
    return y


def _turn_half(x, pos):
    """x [T, heads, 128]: channel i turns with channel i + 64."""
    f = torch.tensor([10000.0 ** (-2.0 * i / 128) for i in range(64)], dtype=torch.float64, device=x.device)
    a = pos.double()[:, None, None] * f
    c, s, u, v = torch.cos(a), torch.sin(a), x[..., :64], x[..., 64:]
    return torch.cat([u * c - v * s, u * s + v * c], dim=-1)


def _softmax_sum(s, v, sink=None):
    """softmax of s [T, n] over the keys (with a sink logit that has no value) times v [n, d]."""
    m = s.max(-1, keepdim=True).values
    if sink is not None:
        m = torch.maximum(m, sink)
    e = torch.exp(s - m)
    return (e @ v) / (e.sum(-1, keepdim=True) + (torch.exp(sink - m) if sink is not None else 0.0))


def _seen(n, past, window=0, keep=0, chunk=0, dev=None):
    """[n - past, n]: which keys the rows from position `past` on see."""
    i, j = torch.arange(past, n, device=dev)[:, None], torch.arange(n, device=dev)[None, :]
    ok = j <= i
    if window:
        ok = ok & ((i - j < window) | (j < keep))
    return ok & (torch.div(i, chunk, rounding_mode="floor") == torch.div(j, chunk, rounding_mode="floor")) if chunk else ok


def _paged(per_request, heads, size, pages):
    """[page][head][PAGE][size] of the requests' rows, pages taken in order."""
    out = torch.zeros(pages, heads, PAGE, size, dtype=torch.float64, device=per_request[0].device)
    at = 0
    for t in per_request:
        for p in range(0, t.shape[0], PAGE):
            part = t[p:p + PAGE].reshape(-1, heads, size).transpose(0, 1)
            out[at, :, :part.shape[1]] = part
            at += 1
    return out


def _pages(case, data):
    return -(-(sum(len(t) for t in data) + PAGE * len(data)) // PAGE) + len(data)


def _exact_latent(x, w, case, past, gate):
    H, d, rd, dv, R = (case[n] for n in ("heads", "dim", "rot_dim", "vdim", "kv_rank"))
    n, pos = x.shape[0], torch.arange(x.shape[0], device=x.device)
    q = (_rms(x[past:] @ w["dq"].T, w["dq.norm"]) @ w["uq"].T).reshape(n - past, H, d + rd)
    down = x @ w["dkv"].T
    c, kr = _rms(down[:, :R], w["dkv.norm"]), _turn(down[:, None, R:], pos, 10000.0, rd)[:, 0]
    qr = _turn(q[..., d:], pos[past:], 10000.0, rd)
    k, v = (c @ w["uk"].T).reshape(n, H, d), (c @ w["uv"].T).reshape(n, H, dv)
    ok = _seen(n, past, case["window"], dev=x.device)
    out = []
    for h in range(H):
        s = (q[:, h, :d] @ k[:, h].T + qr[:, h] @ kr.T) * (d + rd) ** -0.5
        out.append(_softmax_sum(s.masked_fill(~ok, -math.inf), v[:, h]))
    o = torch.stack(out, 1)
    if gate:
        o = o * torch.sigmoid(x[past:] @ w["g"].T)[:, :, None]
    return o.reshape(n - past, H * dv) @ w["o"].T, torch.cat([c, kr], 1)


def _exact_mixer(case, x, w):
    """(output rows, state tensors) of one request's rows x."""
    k, past = case["kind"], case["past"]
    n, dev = x.shape[0], x.device
    pos = torch.arange(n, device=dev)
    if k == "latent":
        y, c = _exact_latent(x, w, case, past, False)
        return y, [c]
    H, G, d = case["heads"], case["kv_heads"], case["dim"]
    if k == "sink":
        q, raw = x[past:] @ w["q"].T, x @ w["k"].T
        q, key = _rms(q, w["q.norm"]).reshape(-1, H, d), _rms(raw, w["k.norm"]).reshape(n, G, d)
        v = raw.reshape(n, G, d)
        ok, gap = _seen(n, past, case["window"], case["keep_first"], dev=dev), (pos[past:, None] - pos[None, :]).double()
        out = []
        for h in range(H):
            s = q[:, h] @ key[:, h * G // H].T * (d ** -0.5 * w["temp"][h])
            if case["softcap"]:
                s = case["softcap"] * torch.tanh(s / case["softcap"])
            s = s - 2.0 ** (-8.0 * (h + 1) / H) * gap
            out.append(_softmax_sum(s.masked_fill(~ok, -math.inf), v[:, h * G // H], w["sink"][h]))
        return torch.stack(out, 1).reshape(n - past, H * d) @ w["o"].T, [key.reshape(n, G * d), raw]
    dv = case["vdim"]
    if k == "talk":
        q = _turn(_rms((x[past:] @ w["q"].T + w["q.b"]).reshape(-1, H, d), w["q.norm"]), pos[past:], 10000.0, d // 2)
        key = _turn(_rms((x @ w["k"].T + w["k.b"]).reshape(n, G, d), w["k.norm"]), pos, 10000.0, d // 2)
        v = (x @ w["v"].T + w["v.b"]).reshape(n, G, dv)
        raw = torch.stack([q[:, h] @ key[:, h * G // H].T for h in range(H)]) * d ** -0.5
        ok, gate = _seen(n, past, dev=dev), torch.sigmoid(x[past:] @ w["g"].T)
        out = []
        for h in range(H):
            s = torch.einsum("g,gij->ij", w["talk"][h], raw).masked_fill(~ok, -math.inf)
            out.append(_softmax_sum(s, v[:, h * G // H], w["sink"][h]) * gate[:, h:h + 1])
        return torch.stack(out, 1).reshape(n - past, H * dv) @ w["o"].T, [key.reshape(n, G * d), v.reshape(n, G * dv)]

    u = torch.cat([x @ w[a].T for a in ("q", "k", "v")], 1)       # the delta rule
    cw = torch.cat([w[a + ".conv"] for a in ("q", "k", "v")], 0)
    taps = cw.shape[1]
    pad = torch.cat([torch.zeros(taps - 1, u.shape[1], dtype=u.dtype, device=dev), u])
    z = sum(pad[j:j + n] * cw[:, j] for j in range(taps))
    z = z * torch.sigmoid(z)
    q, key, v = z[:, :G * d].reshape(n, G, d), z[:, G * d:2 * G * d].reshape(n, G, d), z[:, 2 * G * d:].reshape(n, H, dv)
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
    key = key / torch.sqrt((key * key).sum(-1, keepdim=True) + 1e-6)
    q, key = q.repeat_interleave(H // G, 1), key.repeat_interleave(H // G, 1)
    beta = torch.sigmoid(x @ w["b"].T)
    decay = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(x @ w["a"].T + w["dt_bias"]))
    S, out = torch.zeros(H, dv, d, dtype=u.dtype, device=dev), []
    for t in range(n):
        S = S * decay[t][:, None, None]
        S = torch.baddbmm(S, (beta[t][:, None] * (v[t] - torch.bmm(S, key[t][:, :, None])[..., 0]))[:, :, None], key[t][:, None, :])
        out.append(torch.bmm(S, q[t][:, :, None])[..., 0])
    g = x @ w["g"].T
    o = _rms(torch.stack(out), w["norm"]).reshape(n, H * dv) * (g * torch.sigmoid(g))
    return o @ w["o"].T, [S, pad[n:]]


def _exact_model(case, tokens, w, past):
    """Logits of the last token."""
    T, dev = len(tokens), w["embed"].device
    ids = torch.tensor(tokens, device=dev)
    pair = torch.cat([torch.tensor([case["buckets"]], device=dev), (ids[:-1] * 40503 + ids[1:] * 10007) % case["buckets"]])
    x = w["embed"][ids] + w["bigram"][pair]
    pos = torch.arange(T, device=dev)
    for i in range(case["layers"]):
        p = {n[len(f"l{i}.mix."):]: t for n, t in w.items() if n.startswith(f"l{i}.mix.")}
        if i % 2:
            y = _exact_latent(x, p, case, 0, True)[0]
        else:
            d, G = case["head_dim"], case["kv_heads"]
            H = max(G, case["heads"])
            raw = (x @ p["k"].T).reshape(T, G, d)
            q, key = _rms(_turn((x @ p["q"].T).reshape(T, H, d), pos, 10000.0, d)), _rms(_turn(raw, pos, 10000.0, d))
            ok = _seen(T, 0, chunk=case["chunk"], dev=dev)
            o = [_softmax_sum((q[:, h] @ key[:, h * G // H].T * d ** -0.5).masked_fill(~ok, -math.inf), raw[:, h * G // H]) for h in range(H)]
            y = (torch.stack(o, 1).reshape(T, H * d) * torch.sigmoid(x @ p["g"].T)) @ p["o"].T
        x = x + _rms(y, 1.0 + w[f"l{i}.norm1"])
        y = torch.nn.functional.gelu(x @ w[f"l{i}.mlp.up"].T, approximate="tanh") @ w[f"l{i}.mlp.down"].T
        x = x + _rms(y, 1.0 + w[f"l{i}.norm2"])
    return _rms(x[-1:], 1.0 + w["final.norm"]) @ w["embed"].T


def _exact_dia(case, w, x):
    def attention(q, k, v, ok=None):                              # [T, heads, 128], [n, kv heads, 128] twice
        rep, out = q.shape[1] // k.shape[1], []
        for h in range(q.shape[1]):
            s = q[:, h] @ k[:, h // rep].T * 128 ** -0.5
            out.append(_softmax_sum(s if ok is None else s.masked_fill(~ok, -math.inf), v[:, h // rep]))
        return torch.stack(out, 1).reshape(q.shape[0], -1)

    def dense(y, name):
        t = w[name + ".weight"].double()
        n = 2 if name.endswith("o_proj") else 1
        return y @ t.reshape(math.prod(t.shape[:n]), -1)

    def norm(y, name):
        return _rms(y, w[name + ".weight"].double())

    def mlp(y, p):
        gu = dense(y, p + "wi_fused")
        g, u = gu.chunk(2, -1)
        return dense(g * torch.sigmoid(g) * u, p + "wo")

    if case["kind"] == "dia_text":
        y = w["encoder.embedding.weight"].double()[x["text"][0]]
        n = y.shape[0]
        pos = torch.arange(n, device=y.device)
        for i in range(case["layers"]):
            p = f"encoder.layers.{i}."
            h = norm(y, p + "pre_sa_norm")
            q, k, v = (dense(h, p + f"self_attention.{a}_proj").reshape(n, 16, 128) for a in "qkv")
            y = y + dense(attention(_turn_half(q, pos), _turn_half(k, pos), v), p + "self_attention.o_proj")
            y = y + mlp(norm(y, p + "post_sa_norm"), p + "mlp.")
        return norm(y, "encoder.norm")[None]
    T = x["tokens"].shape[0]
    past = case["slot"] if case["kind"] == "dia_frame" else 0
    dev = x["tokens"].device
    pos, ok = torch.arange(past, past + T, device=dev), _seen(past + T, past, dev=dev)
    own = [[t.double().clone() for t in kv] for kv in x["own"]]
    logits = []
    for b in range(2):
        y = sum(w[f"decoder.embeddings.{c}.weight"].double()[x["tokens"][:, c].long()] for c in range(9))
        for i in range(case["layers"]):
            p = f"decoder.layers.{i}."
            h = norm(y, p + "pre_sa_norm")
            q, k, v = (dense(h, p + f"self_attention.{a}_proj").reshape(T, -1, 128) for a in "qkv")
            kc, vc = own[i]
            kc[b, :, past:past + T], vc[b, :, past:past + T] = _turn_half(k, pos).transpose(0, 1), v.transpose(0, 1)
            y = y + dense(attention(_turn_half(q, pos), kc[b, :, :past + T].transpose(0, 1), vc[b, :, :past + T].transpose(0, 1), ok),
                          p + "self_attention.o_proj")
            if b == 1:
                q = _turn_half(dense(norm(y, p + "pre_ca_norm"), p + "cross_attention.q_proj").reshape(T, 16, 128), pos)
                ck, cv = (t[1, :, :case["text"]].double().transpose(0, 1) for t in x["cross"][i])
                y = y + dense(attention(q, ck, cv), p + "cross_attention.o_proj")
            y = y + mlp(norm(y, p + "pre_mlp_norm"), p + "mlp.")
        logits.append(dense(norm(y, "decoder.norm"), "decoder.logits_dense").reshape(T, 9, 1028))
    out = torch.stack(logits)
    return out if case["kind"] == "dia_frame" else [out, [kv[0] for kv in own], [kv[1] for kv in own]]


@torch.no_grad()
def exact(case, seed):
    r = _Draw(seed)
    if case["kind"].startswith("dia_"):
        cfg, w = _dia_weights(case, r)
        return _exact_dia(case, w, _dia_inputs(case, r, cfg))
    _, _, weights = _lm(case, r)
    data = _lm_inputs(case, r)
    w = {n: t.double() for n, t in weights.items()}
    if case["kind"].startswith("model_"):
        return torch.cat([_exact_model(case, t, w, 0) for t in data])
    if case["kind"] == "experts":
        p, h = {n[len("l0.mlp."):]: t for n, t in w.items() if n.startswith("l0.mlp.")}, data[0].double()

        def unit(x, e):
            g = x @ p[e + ".gate"].T
            return (g * torch.sigmoid(g) * (x @ p[e + ".up"].T)) @ p[e + ".down"].T

        score, best = torch.sigmoid(h @ p["router"].T).topk(case["top"], -1)
        out = unit(h, "shared") if case["shared"] else torch.zeros_like(h)
        for e in range(case["experts"]):
            row, place = (best == e).nonzero(as_tuple=True)
            if row.numel():
                out.index_add_(0, row, unit(score[row, place][:, None] * h[row], f"e{e}"))
        return out
    p = {n[len("l0.mix."):]: t for n, t in w.items() if n.startswith("l0.mix.")}
    got = [_exact_mixer(case, t.double(), p) for t in data]
    y = torch.cat([g[0] for g in got])
    if case["kind"] == "delta":
        return [y, torch.stack([g[1][0] for g in got]), torch.stack([g[1][1] for g in got])]
    pages = _pages(case, data)
    if case["kind"] == "latent":
        return [y, _paged([g[1][0] for g in got], 1, case["kv_rank"] + case["rot_dim"], pages)[:, 0]]
    dv = case["dim"] if case["kind"] == "sink" else case["vdim"]
    return [y] + [_paged([g[1][j] for g in got], case["kv_heads"], size, pages) for j, size in ((0, case["dim"]), (1, dv))]

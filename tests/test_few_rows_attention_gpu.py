"""The attention of a handful of rows (few_rows_attention_kernel of csrc/lm_attention.cu) where it can go wrong: every number of heads per CTA with
and without a remainder, one to four key groups per tile, shares of no key, of a part of a tile and of several tiles, windows with kept keys."""

import pytest
import torch

pytestmark = pytest.mark.gpu

PAST = [0, 1, 30, 31, 32, 65, 130, 300]                           # cached keys of the eight rows of one step


@pytest.mark.parametrize("heads,kv_heads,dim,window,keep", [(2, 1, 20, 0, 0), (2, 1, 64, 40, 3), (6, 2, 72, 0, 0), (5, 1, 128, 0, 0), (16, 2, 40, 33, 1),
                                                            (18, 1, 256, 0, 0), (20, 1, 128, 70, 4)])
def test_decoded_rows(heads, kv_heads, dim, window, keep):
    """Sums of up to 300 weighted values and 256 products in fp32, each relative to the row's largest: 1e-5, as for the other kernels."""
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import PubopelConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    from oracle import pubopel_oracle as O
    cfg = SY.pubopel_config(width=64, layers=1, heads=heads, kv_heads=kv_heads, dim=dim, experts=2, top=1, expert_ff=8, shared_ff=None, vocab=32,
                            window=window or None, keep_first=keep, softcap=None if heads == 5 else 20.0)
    w = SY.pubopel_weights(cfg, heads)
    model = CausalLM(PubopelConfig.model_validate(cfg), w, dtype="float32", device="cuda:0", max_tokens=2048, max_sequences=8, page_size=16, max_rows=320)
    p = {k[len("l0.mix."):]: v.double() for k, v in w.items() if k.startswith("l0.mix.")}
    h = [torch.randn((n + 1, 64), generator=torch.Generator().manual_seed(n)) for n in PAST]
    ref = torch.cat([O.sink_attention(t.double(), p, cfg["layers"][0]["mixer"], cfg["norm"]["eps"])[-1:] for t in h])
    decoded(model, h, ref, 1e-5)


def decoded(model, h, ref, bound):
    """The last rows of ``h`` in one step and each in a step of its own, behind cached keys of the others"""
    seqs = []
    for i, (n, t) in enumerate(zip(PAST, h)):
        seqs.append(model.state.open(str(i)))
        model.state.reserve(seqs[-1], n + 1)
        if n:
            model.engine.op_mixer(0, t[:n].cuda(), [(seqs[-1], n, 0)])
    got = model.engine.op_mixer(0, torch.cat([t[-1:] for t in h]).cuda(), [(q, 1, n) for q, n in zip(seqs, PAST)])
    one = torch.cat([model.engine.op_mixer(0, t[-1:].cuda(), [(q, 1, n)]) for q, n, t in zip(seqs, PAST, h)])     # other shares: rows alone
    for y in (got, one):
        assert (y.double().cpu() - ref).abs().max() <= bound * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("heads,kv_rank,rot_dim,window", [(4, 64, 16, 0), (5, 64, 64, 70), (4, 192, 64, 0), (16, 192, 16, 33), (5, 256, 64, 0), (16, 256, 16, 0),
                                                          (18, 132, 20, 0)])
def test_decoded_latent_rows(heads, kv_rank, rot_dim, window):
    """Cached rows of kv_rank + rot_dim channels, of which the first kv_rank are the value: two roundings more per output than above (the queries and
    the outputs go through the latent's up-projections)"""
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import FipadraConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    from oracle import fipadra_oracle as O
    cfg = SY.fipadra_config(width=64, kinds=["latent_attention"], heads=heads, dim=32, rot_dim=rot_dim, vdim=40, q_rank=72, kv_rank=kv_rank, window=window, vocab=32)
    cfg["layers"][0]["mlp"] = None
    w = SY.fipadra_weights(cfg, heads)
    model = CausalLM(FipadraConfig.model_validate(cfg), w, dtype="float32", device="cuda:0", max_tokens=2048, max_sequences=8, page_size=16, max_rows=320)
    p = {k[len("l0.mix."):]: v.double() for k, v in w.items() if k.startswith("l0.mix.")}
    h = [torch.randn((n + 1, 64), generator=torch.Generator().manual_seed(n)) for n in PAST]
    ref = torch.cat([O.latent_attention(t.double(), p, cfg["layers"][0]["mixer"], cfg["norm"]["eps"])[-1:] for t in h])
    decoded(model, h, ref, 2e-5)


@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(6, 2, 32, 64), (16, 1, 64, 24), (10, 2, 48, 128), (4, 2, 96, 200)])
def test_decoded_gated_rows(heads, kv_heads, dim, vdim, monkeypatch):
    """A layer whose scores are not mixed across heads, with a sink in the denominator and a gate per head"""
    from dia_tts_prune_b200 import lm_model, synthetic as SY
    from dia_tts_prune_b200.lm_config import KupelixConfig
    from oracle import kupelix_oracle as O
    cfg = SY.kupelix_config(width=64, kinds=["attention"], heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, ff=8, vocab=32)
    w = SY.kupelix_weights(cfg, heads)
    cfg["layers"][0]["mlp"] = None
    layer = lm_model.TalkingAttention
    monkeypatch.setattr(lm_model, "TalkingAttention", lambda *a, **k: layer(*a, **{**k, "talk": None}))
    model = lm_model.CausalLM(KupelixConfig.model_validate(cfg), w, dtype="float32", device="cuda:0", max_tokens=2048, max_sequences=8, page_size=16, max_rows=320)
    p = {k[len("l0.mix."):]: v.double() for k, v in w.items() if k.startswith("l0.mix.")}
    p["talk"] = torch.eye(heads, dtype=torch.float64)
    h = [torch.randn((n + 1, 64), generator=torch.Generator().manual_seed(n)) for n in PAST]
    ref = torch.cat([O.talking_attention(t.double(), p, cfg["layers"][0]["mixer"], cfg["norm"]["eps"])[-1:] for t in h])
    decoded(model, h, ref, 2e-5)

"""The attention of a handful of rows (few_rows_attention_kernel of csrc/lm_attention.cu) where it can go wrong: every number of heads per CTA with
and without a remainder, one to four key groups per tile, shares of no key, of a part of a tile and of several tiles, windows with kept keys."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dim,window,keep", [(1, 1, 20, 0, 0), (2, 1, 64, 40, 3), (6, 2, 72, 0, 0), (5, 1, 128, 0, 0), (16, 2, 40, 33, 1),
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
    past = [0, 1, 30, 31, 32, 65, 130, 300]                       # cached keys of eight rows of one step
    h = [torch.randn((n + 1, 64), generator=torch.Generator().manual_seed(n)) for n in past]
    ref = torch.cat([O.sink_attention(t.double(), p, cfg["layers"][0]["mixer"], cfg["norm"]["eps"])[-1:] for t in h])
    seqs = []
    for i, (n, t) in enumerate(zip(past, h)):
        seqs.append(model.state.open(str(i)))
        model.state.reserve(seqs[-1], n + 1)
        if n:
            model.engine.op_mixer(0, t[:n].cuda(), [(seqs[-1], n, 0)])
    got = model.engine.op_mixer(0, torch.cat([t[-1:] for t in h]).cuda(), [(q, 1, n) for q, n in zip(seqs, past)])
    one = torch.cat([model.engine.op_mixer(0, t[-1:].cuda(), [(q, 1, n)]) for q, n, t in zip(seqs, past, h)])     # other shares: rows alone
    for y in (got, one):
        assert (y.double().cpu() - ref).abs().max() <= 1e-5 * max(1.0, ref.abs().max().item())

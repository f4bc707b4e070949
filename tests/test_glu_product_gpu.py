"""The product of a gated unit with its gate behind the accumulators (csrc/gemm_tcgen05.cu): against the same product and gate one after the other, which
more weight rows than two of the unit's halves ask for nothing else than."""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def unit(rows, width, ff, shared, experts, top):
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import PubopelConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    cfg = SY.pubopel_config(width=width, layers=1, heads=1, kv_heads=1, dim=64, experts=experts, top=top, expert_ff=ff, shared_ff=shared, vocab=64)
    w = SY.pubopel_weights(cfg, 3)
    return CausalLM(PubopelConfig.model_validate(cfg), w, dtype="bfloat16", device="cuda:0", max_tokens=256, max_sequences=1, max_rows=rows), w


@pytest.mark.parametrize("rows,width,ff,shared,experts,top", [
    (1000, 256, 128, 256, 4, 2),        # one and two tiles of columns; groups of 256 rows, the last of each partly filled
    (257, 192, 384, 128, 2, 1),         # one row more than a tile; three k-blocks
    (2048, 1024, 256, 1152, 8, 2),      # nine tiles of columns
    (600, 256, 160, 96, 4, 2),          # no multiple of 128 columns: one after the other
])
def test_gated_units_against_64_bits(rows, width, ff, shared, experts, top):
    """Operands and hidden values are bf16 (2^-9 each), sums are fp32: hidden values of fan-in sums around one, so an output differs by a few 2^-9 of the largest"""
    model, w = unit(rows, width, ff, shared, experts, top)
    h = torch.randn(rows, width, generator=torch.Generator().manual_seed(rows)).cuda()
    got = model.engine.op_ff(0, h).double().cpu()
    p = {n[len("l0.mlp."):]: t.double() for n, t in w.items() if n.startswith("l0.mlp.")}
    x = h.double().cpu()
    score, pick = (x @ p["router"].T).topk(top, dim=1)

    def one(e, rows_of, scale):
        a = (rows_of * scale).bfloat16().double()
        mid = torch.nn.functional.silu(a @ p[f"{e}.gate"].T) * (a @ p[f"{e}.up"].T)
        return mid.bfloat16().double() @ p[f"{e}.down"].T

    want = one("shared", x, 1.0)
    for k in range(top):
        for e in range(experts):
            sel = pick[:, k] == e
            want[sel] += one(f"e{e}", x[sel], torch.sigmoid(score[sel, k:k + 1]))
    assert (got - want).abs().max() <= 2.0 ** -6 * want.abs().max()
    assert (got - want).norm() <= 2.0 ** -8 * want.norm()

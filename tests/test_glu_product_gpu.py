"""The product of a gated unit with its gate behind the accumulators (csrc/gemm_tcgen05.cu): bit for bit against product and gate one after the other, units of
both routes against 64 bits, and a wait that ran out."""

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


def gated(x, w, F, act, fused, groups=0, row_group=None, n_rows=None):
    """Hidden rows bf16 [M + 16][F]: sixteen rows behind the result stay 7.0"""
    from dia_tts_prune_b200 import _lm_lib
    M, K = x.shape
    y = torch.full((M + 16, F), 7.0, dtype=torch.bfloat16, device="cuda")
    xb, gu = torch.empty((M, K), dtype=torch.bfloat16, device="cuda"), torch.empty((M, 2 * F), device="cuda")
    rc = _lm_lib.load().lm_b200_op_gated_tc(x.data_ptr(), w.data_ptr(), xb.data_ptr(), gu.data_ptr(), y.data_ptr(), M, F, K, act, 3.0, fused, row_group.data_ptr() if groups else None,
                                            groups, n_rows.data_ptr() if groups else None, torch.cuda.current_stream().cuda_stream)
    if rc:
        raise RuntimeError(rc)
    return y


@pytest.mark.parametrize("act", [0, 2, 4])                       # silu, clamped, gelu
@pytest.mark.parametrize("M,F,K,groups", [(2049, 2048, 136, 0), (1501, 1024, 520, 0), (4095, 384, 200, 0), (300, 4096, 512, 0), (1280, 256, 328, 4), (512, 128, 72, 2)])
def test_fused_and_apart_have_the_same_bits(M, F, K, groups, act):
    """One row more than tiles, one less, k-blocks of 8 to 64, groups whose last rows are nothing: every product and every gate is the same operation in either
    form.  Scores up to 30 and rows of zeros are among them."""
    g = torch.Generator(device="cuda").manual_seed(M + act)
    x = torch.randn((M, K), generator=g, device="cuda") * torch.logspace(-3, 1.5, M, device="cuda")[:, None]
    x[5::97] = 0.0
    w = (torch.randn((2 * F * max(groups, 1), K), generator=g, device="cuda") * K ** -0.5).bfloat16()
    more = {}
    if groups:
        more = dict(groups=groups, row_group=(torch.arange(M, device="cuda") // 256).clamp(max=groups - 1).int(), n_rows=torch.tensor([M - 256], dtype=torch.int32, device="cuda"))
    one, two = gated(x, w, F, act, 1, **more), gated(x, w, F, act, 0, **more)
    rows = M - 256 if groups else M
    assert torch.isfinite(two[:rows]).all() and torch.equal(one[:rows], two[:rows]) and (one[rows:] == 7.0).all()


@pytest.mark.parametrize("M,F,K,groups", [(2049, 2048, 136, 0), (512, 128, 72, 2)])
def test_a_wait_that_ran_out(M, F, K, groups):
    """No look at a barrier: all hidden rows are NaN and none behind them, the next launch returns an error, the one after it has the result"""
    from dia_tts_prune_b200 import _lm_lib
    from test_gemm_pair_gpu import ran_out
    x, w = torch.randn((M, K), device="cuda"), (torch.randn((2 * F * max(groups, 1), K), device="cuda") * K ** -0.5).bfloat16()
    more = dict(groups=groups, row_group=(torch.arange(M, device="cuda") // 256).int(), n_rows=torch.tensor([M], dtype=torch.int32, device="cuda")) if groups else {}
    word, polls = ran_out(_lm_lib.load())
    good, kept = gated(x, w, F, 0, 1, **more), polls[0]
    assert word[0] == 0 and kept > 1000000
    polls[0] = 0
    try:
        bad = gated(x, w, F, 0, 1, **more)
        torch.cuda.synchronize()
    finally:
        polls[0] = kept
    assert torch.isnan(bad[:M]).all() and (bad[M:] == 7.0).all() and word[0] == 1
    with pytest.raises(RuntimeError):
        gated(x, w, F, 0, 1, **more)
    assert word[0] == 0 and torch.equal(gated(x, w, F, 0, 1, **more), good)


@pytest.mark.parametrize("rows,width,ff,launches", [(1030, 512, 2048, 2), (3000, 2048, 2048, 1)])
def test_the_shorter_way_is_taken(rows, width, ff, launches):
    """A shared expert's hidden rows: product and gate, or one kernel (the other launches of the layer are counted with a unit that is never fused)"""
    from dia_tts_prune_b200 import _lm_lib

    def count(shared):
        model, _ = unit(rows, width, 96, shared, 2, 1)
        h = torch.randn(rows, width, generator=torch.Generator().manual_seed(rows)).cuda()
        before = _lm_lib.load().lm_b200_launch_count()
        model.engine.op_ff(0, h)
        return _lm_lib.load().lm_b200_launch_count() - before

    assert count(ff) - count(ff + 32) == launches - 2

"""The product on pairs of SMs (dia_gemm_pair_kernel of csrc/gemm_tcgen05.cu) where it can go wrong: edges of its 256-row tiles, of each tile
width, of 64-wide k-blocks, one row tile of a pair without rows, expert groups padded to a pair's rows."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def product(x, w):
    from dia_tts_prune_b200 import _lm_lib
    lib = _lm_lib.load()
    (M, K), N = x.shape, w.shape[0]
    y = torch.full((M, N), float("nan"), device="cuda")
    xb = torch.empty((M, K), dtype=torch.bfloat16, device="cuda")
    rc = lib.lm_b200_op_linear_tc(x.data_ptr(), w.data_ptr(), y.data_ptr(), xb.data_ptr(), M, N, K, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    return y


@pytest.mark.parametrize("M,N,K", [(1153, 2052, 72), (2049, 8192, 64), (1024, 3076, 520), (1300, 16388, 192), (2304, 9476, 136), (129, 18948, 264)])
def test_bf16_rows(M, N, K):
    """Sums of K products of bf16 operands in an fp32 accumulator that cuts off: at most K / 16 additions, a unit of 2^-23 of the sum's
    largest partial value each."""
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn((M, K), generator=g, device="cuda")
    w = (torch.randn((N, K), generator=g, device="cuda") * K ** -0.5).bfloat16()
    ref = x.bfloat16().double() @ w.double().T
    assert (product(x, w) - ref).abs().max() <= 2.0 ** -23 * (K / 16 + 2) * ref.abs().max()


@pytest.mark.parametrize("M,N,K", [(257, 12292, 64), (600, 16384, 192), (1722, 3076, 128), (1722, 9252, 320)])
def test_fp32_rows_and_residual(M, N, K):
    from dia_tts_prune_b200 import engine
    g = torch.Generator(device="cuda").manual_seed(N)
    x, r = torch.randn((M, K), generator=g, device="cuda"), torch.randn((M, N), generator=g, device="cuda")
    w = (torch.randn((K, N), generator=g, device="cuda") * K ** -0.5).bfloat16()
    ref = r.double() + x.double() @ w.double()
    got = engine.dense_forward(x, engine.dense_prepare_weight(w), residual=r.clone())
    assert (got - ref).abs().max() <= 2.0 ** -23 * (3 * K / 16 + 2) * ref.abs().max()


@pytest.mark.parametrize("rows,top", [(193, 1), (700, 2), (2048, 1)])
def test_expert_groups(rows, top):
    """Groups of one pair tile and of several, their last rows padding.  The operands are rounded to bf16 twice (2^-9 each), and a few
    rows change their experts with the rounded scores' order: not here, the scores are fp32."""
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import PubopelConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    from oracle import pubopel_oracle as O
    cfg = SY.pubopel_config(width=128, layers=1, heads=1, kv_heads=1, dim=16, experts=3, top=top, expert_ff=264, shared_ff=136, vocab=64)
    w = SY.pubopel_weights(cfg, 3)
    model = CausalLM(PubopelConfig.model_validate(cfg), w, dtype="bfloat16", device="cuda:0", max_tokens=2 * rows, max_sequences=1, max_rows=rows)
    h = torch.randn(rows, 128, generator=torch.Generator().manual_seed(rows))
    p = {k[len("l0.mlp."):]: v.double() for k, v in w.items() if k.startswith("l0.mlp.")}
    ref = O.routed_experts(h.double(), p, cfg["layers"][0]["mlp"])
    got = model.engine.op_ff(0, h.cuda()).double().cpu()
    assert (got - ref).norm() <= 2.0 ** -7 * ref.norm()

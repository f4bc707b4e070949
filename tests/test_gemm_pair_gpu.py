"""The product on pairs of SMs (dia_gemm_pair_kernel of csrc/gemm_tcgen05.cu) where it can go wrong: edges of its 256-row tiles, of each tile
width, of 64-wide k-blocks, one row tile of a pair without rows, expert groups padded to a pair's rows."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def product(x, w, y=None):
    from dia_tts_prune_b200 import _lm_lib
    lib = _lm_lib.load()
    (M, K), N = x.shape, w.shape[0]
    y = torch.full((M, N), float("nan"), device="cuda") if y is None else y
    xb = torch.empty((M, K), dtype=torch.bfloat16, device="cuda")
    rc = lib.lm_b200_op_linear_tc(x.data_ptr(), w.data_ptr(), y.data_ptr(), xb.data_ptr(), M, N, K, torch.cuda.current_stream().cuda_stream)
    if rc:
        raise RuntimeError(rc)
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


@pytest.mark.parametrize("M,N,K,gated,norm,residual", [(129, 16388, 64, False, False, True), (257, 9252, 320, False, True, False),
                                                       (300, 2052, 8256, False, True, True), (511, 260, 576, True, False, True),
                                                       (1722, 2048, 256, False, False, False), (300, 132, 8256, True, False, False)])
def test_two_fp16_terms(M, N, K, gated, norm, residual):
    """Edges of the row tiles, of every tile width, of chunks of four k-blocks and of the rows that fit a CTA's registers (8192 channels).  Terms and
    weights are exact to 2^-22 of a value, an accumulator takes 32 additions that cut off, and there are K / 256 fp32 additions."""
    from dia_tts_prune_b200 import engine
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn((M, 2 * K if gated else K), generator=g, device="cuda") * torch.exp2(torch.randint(-50, 50, (M, 1), generator=g, device="cuda").float())
    if gated:
        x = x.clamp(-1e9, 1e9)
    w = (torch.randn((K, N), generator=g, device="cuda") * torch.exp2(torch.randint(-20, 20, (1, N), generator=g, device="cuda").float())).bfloat16()
    nw = torch.rand((K,), generator=g, device="cuda") + 0.5 if norm else None
    inexact = torch.zeros((1,), dtype=torch.int32, device="cuda")
    half = engine.dense_prepare_half(w, inexact)
    assert inexact.item() == 0
    xd = x.double()
    if gated:
        xd = torch.nn.functional.silu(xd[:, :K]) * xd[:, K:]
    if norm:
        xd = xd * torch.rsqrt((xd * xd).mean(-1, keepdim=True) + 1e-5) * nw.double()
    ref, size = xd @ w.double(), xd.abs() @ w.double().abs()
    r = torch.randn((M, N), generator=g, device="cuda") * ref.abs().max(1, keepdim=True).values.float() if residual else None
    if residual:
        ref, size = ref + r.double(), size + r.double().abs()
    got = engine.dense_forward_half(x.reshape(M, 2, K) if gated else x, half, nw, 1e-5, r.clone() if residual else None, gated)
    assert ((got - ref).abs() <= 2.0 ** -23 * (8 + 34 + K / 256) * size).all()


@pytest.mark.parametrize("M,N,K", [(600, 16384, 2048), (1722, 2048, 2048), (1722, 2048, 8192), (1000, 8192, 1024)])
@pytest.mark.parametrize("rows", ["normal", "gated", "positive", "outlier"])
def test_two_fp16_terms_beside_three_bf16_terms(M, N, K, rows):
    """The widths of Dia's layers: 22 bits of a row's numbers and sums of 256 products are nowhere further off than 24 bits and one sum of all products
    on the tensor cores (an addition that cuts off per 16 products and term), which these rows would take.  Outlier: a channel 2^16 times the others,
    and columns with a zero weight there, which see the others alone."""
    from dia_tts_prune_b200 import engine
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, w = torch.randn((M, K), generator=g, device="cuda"), (torch.randn((K, N), generator=g, device="cuda") * K ** -0.5).bfloat16()
    if rows == "gated":
        x = torch.nn.functional.silu(2 * x) * torch.randn((M, K), generator=g, device="cuda") * 3
    elif rows == "positive":
        x, w = x.abs(), w.abs()
    elif rows == "outlier":
        x[:, 5], w[5] = 2.0 ** 16, 0.0
    assert engine.dense_half_rows(M, N, K, x.device)
    two = engine.dense_forward_half(x, engine.dense_prepare_half(w, torch.zeros((1,), dtype=torch.int32, device="cuda")))
    three, ref = engine.dense_forward(x, engine.dense_prepare_weight(w)), x.double() @ w.double()
    off, was = (two - ref).norm() / ref.norm(), (three - ref).norm() / ref.norm()
    # 16 additions per accumulator that cut off half a unit of 2^-23 each, as a bias where all numbers are positive; K / 256 rounded ones
    assert off <= was and off <= 2.0 ** -23 * 10


def test_two_fp16_terms_at_the_ends_of_fp32():
    """Rows of the smallest and the largest numbers, zeros, infinities and NaNs beside ordinary ones, against three bf16 terms."""
    from dia_tts_prune_b200 import engine
    g = torch.Generator(device="cuda").manual_seed(1)
    x, w = torch.randn((130, 128), generator=g, device="cuda"), torch.randn((128, 128), generator=g, device="cuda").bfloat16()
    x[0], x[1] = x[0] * 1e-38, x[1].clamp(-3, 3) * 1e36
    x[2] = 0.0
    x[3, 5], x[4, 6] = float("inf"), float("nan")
    inexact = torch.zeros((1,), dtype=torch.int32, device="cuda")
    got, ref = engine.dense_forward_half(x, engine.dense_prepare_half(w, inexact)), x.double() @ w.double()
    assert (got[0] - ref[0]).abs().max() <= 1e-5 * ref[0].abs().max() and (got[1] - ref[1]).abs().max() <= 1e-5 * ref[1].abs().max()
    assert (got[2] == 0).all() and not torch.isfinite(got[3:5]).any() and torch.isnan(got[4]).all()
    assert (torch.isinf(got[3]) & (got[3].double() == ref[3])).sum() == torch.isinf(ref[3]).sum()
    assert (got[5:] - ref[5:]).abs().max() <= 1e-5 * ref[5:].abs().max()


def test_weights_that_fp16_cannot_hold():
    """2^33 between the values of one column, or an infinity: told by the flag, and such a layer keeps its three bf16 terms."""
    from dia_tts_prune_b200 import engine
    from dia_tts_prune_b200.layers import DenseGeneral
    for small, big, fits in ((2.0 ** -31, 1.0, True), (2.0 ** -33 * 1.0078125, 1.0, False), (1.0, float("inf"), False)):
        w = torch.full((64, 4), small, device="cuda").bfloat16()
        w[3, 2] = big
        inexact = torch.zeros((1,), dtype=torch.int32, device="cuda")
        engine.dense_prepare_half(w, inexact)
        assert (inexact.item() == 0) == fits
    d = DenseGeneral((64,), (16384,), weight_dtype=torch.bfloat16, device="cuda")
    with torch.no_grad():
        d.weight.normal_()
        x = torch.randn((600, 64), device="cuda")
        assert engine.dense_half_rows(600, 16384, 64, x.device) and d.kernel_weight_half() is not None
        d.weight[7, 9] = 2.0 ** -40
        assert d.kernel_weight_half() is None
        ref = x.double() @ d.weight.double()
        assert (d(x) - ref).norm() <= 1e-6 * ref.norm()


@pytest.mark.parametrize("M,N,K", [(1024, 2048, 1024), (513, 2048, 1024), (1153, 1024, 1536), (2305, 512, 1024), (768, 3072, 1024), (128, 2048, 1024)])
def test_products_that_keep_fp32_sums(M, N, K):
    """bf16 rows whose 128 x 128 tiles fit one round: pieces of 64 products added in fp32, also where one sum of all products on a pair of SMs is
    the faster one.  All products positive, so that what is cut off adds up: about half a unit of 2^-23 per 16 products of a sum, 2.4e-7 for pieces of 64
    and 3.8e-6 for 1024."""
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = torch.rand((M, K), generator=g, device="cuda"), (torch.rand((N, K), generator=g, device="cuda") * K ** -0.5).bfloat16()
    ref = x.bfloat16().double() @ w.double().T
    assert (product(x, w) - ref).norm() <= 1e-6 * ref.norm()


def ran_out(lib):
    """(the word that a kernel sets when a wait of its ran out, how often the waits of this thread's products look at their barriers)"""
    import ctypes as C
    word_of, polls_of = getattr(lib, "_ZN3dia23split_attention_ran_outEiP11CUstream_st"), getattr(lib, "_ZN3dia15gemm_pair_pollsEv")
    word_of.restype, word_of.argtypes = C.POINTER(C.c_int), [C.c_int, C.c_void_p]
    polls_of.restype, polls_of.argtypes = C.POINTER(C.c_uint), []
    return word_of(torch.cuda.current_device(), None), polls_of()


@pytest.mark.parametrize("M,N,K,half", [(600, 16384, 192, False), (129, 18948, 264, False), (600, 16384, 192, True), (1722, 3076, 576, True)])
def test_a_wait_that_ran_out(M, N, K, half):
    """Waits that run out before anything is issued (no look at a barrier): the whole result is NaN, the next launch returns an error, the one after it
    has the result"""
    from dia_tts_prune_b200 import _lib, _lm_lib, engine
    x, w = torch.randn((M, K), device="cuda"), (torch.randn((N, K), device="cuda") * K ** -0.5).bfloat16()
    if half:
        copy = engine.dense_prepare_half(w.t().contiguous(), torch.zeros((1,), dtype=torch.int32, device="cuda"))
        call = lambda r: engine.dense_forward_half(x, copy, residual=r)
    else:
        call = lambda r: product(x, w, r)
    word, polls = ran_out((_lib if half else _lm_lib).load())
    good, kept = call(torch.zeros((M, N), device="cuda")), polls[0]
    assert word[0] == 0 and kept > 1000000
    polls[0] = 0
    try:
        bad = call(torch.zeros((M, N), device="cuda"))
        torch.cuda.synchronize()
    finally:
        polls[0] = kept
    assert torch.isnan(bad).all() and word[0] == 1
    with pytest.raises(RuntimeError):
        call(torch.zeros((M, N), device="cuda"))
    assert word[0] == 0 and torch.equal(call(torch.zeros((M, N), device="cuda")), good)


def test_a_wait_that_ran_out_reaches_a_step():
    """The word set by hand between a step's launches and the look behind its synchronisation"""
    from dia_tts_prune_b200 import _lm_lib, synthetic as SY
    from dia_tts_prune_b200.lm_config import PubopelConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    cfg = SY.pubopel_config(width=128, layers=1, heads=1, kv_heads=1, dim=16, experts=3, top=1, expert_ff=64, shared_ff=None, vocab=64)
    model = CausalLM(PubopelConfig.model_validate(cfg), SY.pubopel_weights(cfg, 3), dtype="bfloat16", device="cuda:0", max_tokens=64, max_sequences=1, max_rows=32)
    word, _ = ran_out(_lm_lib.load())
    assert model.generate([[1, 2, 3]], max_new_tokens=3)
    model.engine.check()
    word[0] = 1
    with pytest.raises(RuntimeError):
        model.engine.check()
    assert word[0] == 0
    model.engine.check()
    word[0] = 1
    with pytest.raises(RuntimeError):
        model.generate([[1, 2, 3]], max_new_tokens=3)

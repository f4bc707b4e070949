"""The tensor-core product in fp32 arithmetic (gemm_f32 of csrc/gemm_tcgen05.cu) where it can go wrong: edges of its 128 x 128 tiles and
64-wide k-blocks, through the products of a float32 model and the per-head products of latent attention."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def forilorn(width, ff, heads, dim, kv_rank, vdim, rows, seed):
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import ForilornConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    cfg = SY.forilorn_config(width=width, kinds=["latent_attention"], heads=heads, dim=dim, vocab=64, lat_dim=dim, rot_dim=8, lat_vdim=vdim,
                             q_rank=72, kv_rank=kv_rank, ff=ff)
    w = SY.forilorn_weights(cfg, seed)
    return cfg, w, CausalLM(ForilornConfig.model_validate(cfg), w, dtype="float32", device="cuda:0", max_tokens=2 * rows, max_sequences=1, max_rows=rows)


@pytest.mark.parametrize("rows,width,ff", [(9, 64, 72), (128, 136, 128), (129, 128, 132), (200, 264, 1000)])
def test_products_of_a_float32_unit(rows, width, ff):
    """down(gelu(up h)): sums of K fp32 products in 64-product blocks.  Each block is off by at most about 2^-21 of its magnitude, so
    1e-5 of the result's largest magnitude leaves a factor of ten."""
    cfg, w, model = forilorn(width, ff, 2, 16, 24, 16, rows, 3)
    h = torch.randn((rows, width), generator=torch.Generator().manual_seed(4))
    got = model.engine.op_ff(0, h.cuda()).double().cpu()
    up, down = w["l0.mlp.up"].double(), w["l0.mlp.down"].double()
    ref = torch.nn.functional.gelu(h.double() @ up.T, approximate="tanh") @ down.T
    assert (got - ref).abs().max() <= 1e-5 * ref.abs().max()


@pytest.mark.parametrize("heads,dim,kv_rank,vdim,rows", [(1, 8, 8, 8, 9), (3, 40, 72, 136, 130), (4, 96, 256, 128, 128)])
def test_per_head_products(heads, dim, kv_rank, vdim, rows):
    """The latent attention of a float32 model: queries into the latent space and attended latents out of it, with one gate per head."""
    cfg, w, model = forilorn(64, 8, heads, dim, kv_rank, vdim, rows, 5)
    h = torch.randn((rows, 64), generator=torch.Generator().manual_seed(6))
    seq = model.state.open("a")
    model.state.reserve(seq, rows)
    got = model.engine.op_mixer(0, h.cuda(), [(seq, rows, 0)]).double().cpu()
    p, x, n = {k[len("l0.mix."):]: t.double() for k, t in w.items() if k.startswith("l0.mix.")}, h.double(), rows
    rms = lambda t: t / torch.sqrt((t * t).mean(-1, keepdim=True) + cfg["norm"]["eps"])      # noqa: E731

    def turn(t):
        a = torch.arange(n).double()[:, None, None] * torch.tensor([10000.0 ** (-i / 4) for i in range(4)], dtype=torch.float64)
        y = t.clone()
        y[..., 0::2] = t[..., 0::2] * a.cos() - t[..., 1::2] * a.sin()
        y[..., 1::2] = t[..., 1::2] * a.cos() + t[..., 0::2] * a.sin()
        return y

    q = ((rms(x @ p["dq"].T) * p["dq.norm"]) @ p["uq"].T).reshape(n, heads, dim + 8)
    down = x @ p["dkv"].T
    c, kr = rms(down[:, :kv_rank]) * p["dkv.norm"], turn(down[:, None, kv_rank:])[:, 0]
    k, v, qr = (c @ p["uk"].T).reshape(n, heads, dim), (c @ p["uv"].T).reshape(n, heads, vdim), turn(q[..., dim:])
    s = (torch.einsum("ihd,jhd->hij", q[..., :dim], k) + torch.einsum("ihd,jd->hij", qr, kr)) * (dim + 8) ** -0.5
    o = torch.einsum("hij,jhd->ihd", torch.softmax(s.masked_fill(torch.ones(n, n).triu(1).bool(), -torch.inf), -1), v)
    ref = (o * torch.sigmoid(x @ p["g"].T)[:, :, None]).reshape(n, heads * vdim) @ p["o"].T
    assert (got - ref).abs().max() <= 2e-5 * ref.abs().max()


@pytest.mark.parametrize("dtype,rows,width,ff", [("float32", 3, 2056, 2060), ("float32", 8, 4104, 1544), ("bfloat16", 9, 136, 132),
                                                 ("bfloat16", 31, 264, 1000)])
def test_products_of_a_few_rows(dtype, rows, width, ff):
    """The same unit where the few-rows kernel takes it (3 to 8 rows of large matrices; up to 31 rows of bf16 products), with clusters that
    split K, a remainder of K and of N, and up to 8 and up to 32 rows per operand; the bound is the one above."""
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import ForilornConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    cfg = SY.forilorn_config(width=width, kinds=["latent_attention"], heads=2, dim=16, vocab=64, lat_dim=16, rot_dim=8, lat_vdim=16, q_rank=72,
                             kv_rank=24, ff=ff)
    w = SY.forilorn_weights(cfg, 3)
    model = CausalLM(ForilornConfig.model_validate(cfg), w, dtype=dtype, device="cuda:0", max_tokens=64, max_sequences=1, max_rows=64)
    h = torch.randn((rows, width), generator=torch.Generator().manual_seed(4))
    got = model.engine.op_ff(0, h.cuda()).double().cpu()
    up, down = w["l0.mlp.up"].double(), w["l0.mlp.down"].double()
    ref = torch.nn.functional.gelu(h.double() @ up.T, approximate="tanh") @ down.T
    assert (got - ref).abs().max() <= 1e-5 * ref.abs().max()


@pytest.mark.parametrize("M,N,K", [(1, 4, 64), (32, 100, 128), (31, 2048, 4096), (33, 2048, 1024), (129, 260, 192), (200, 1024, 4096),
                                   (128, 128, 8192), (300, 9252, 128)])
def test_dense_rows_of_fp32_sums(M, N, K):
    """The dense layers of the text and prompt passes on the two kernels that add every 64 products in fp32 registers: norm in front and
    residual behind, one CTA per tile and clusters over K.  The bound is the one above, on the product's largest magnitude."""
    from dia_tts_prune_b200 import engine as E
    g = torch.Generator().manual_seed(M + N + K)
    x, nw = torch.randn(M, K, generator=g), torch.rand(K, generator=g) + 0.5
    w, res = (torch.randn(K, N, generator=g) * K ** -0.5).to(torch.bfloat16), torch.randn(M, N, generator=g)
    wt = E.dense_prepare_weight(w.cuda())
    xd = x.double()
    xn = xd * torch.rsqrt((xd * xd).mean(-1, keepdim=True) + 1e-5) * nw.double()
    for norm in (False, True):
        ref = (xn if norm else xd) @ w.double()
        r = res.clone().cuda()
        y = E.dense_forward(x.cuda(), wt, norm_weight=nw.cuda() if norm else None, residual=r)
        assert (y.cpu().double() - (ref + res.double())).abs().max() <= 1e-5 * ref.abs().max()


@pytest.mark.parametrize("rows", [9, 515, 1100])
def test_grouping_of_many_assignments(rows):
    """The expert units of a step with more assignments than the grouping kernel has threads against those of the same rows in short
    steps, where no grouping takes place; both within fp32 rounding of the products."""
    import test_lm_gpu as T
    model, _ = T.build(T.small_config(), 7, max_rows=1100)
    h = torch.randn((rows, 96), generator=torch.Generator().manual_seed(8)).cuda()
    whole = model.engine.op_ff(0, h)
    parts = torch.cat([model.engine.op_ff(0, h[i:i + 8]) for i in range(0, rows, 8)])
    assert (whole - parts).abs().max() <= 1e-5 * parts.abs().max()


@pytest.mark.parametrize("M,N,K", [(32, 2048, 2048), (150, 288, 96), (200, 100, 72), (129, 132, 4104), (1024, 2048, 6144), (1, 8, 8)])
def test_products_of_bf16_rows(M, N, K):
    """A bf16 operand on both sides of the rule between 128 x 256 tiles and 128 x 128 tiles with split sums.  The wider tiles add K products
    in tensor memory, each addition cut off at 2^-23 of the sum: K 2^-23 of its magnitude at most, against 2e-6 + K 2^-24 here (the errors
    do not all add up)."""
    import ctypes as C

    from dia_tts_prune_b200 import _lm_lib
    lib, g = _lm_lib.load(), torch.Generator().manual_seed(M + N + K)
    x, w = torch.randn(M, K, generator=g).cuda(), (torch.randn(N, K, generator=g) * K ** -0.5).to(torch.bfloat16).cuda()
    y, xb = torch.empty(M, N, device="cuda"), torch.empty(M, K, device="cuda", dtype=torch.bfloat16)
    p = lambda t: C.c_void_p(t.data_ptr())                                                       # noqa: E731
    _lm_lib.check(lib.lm_b200_op_linear_tc(p(x), p(w), p(y), p(xb), M, N, K, C.c_void_p(torch.cuda.current_stream().cuda_stream)), "op_linear_tc")
    assert torch.equal(xb, x.to(torch.bfloat16))
    ref = x.to(torch.bfloat16).double() @ w.double().T
    assert (y - ref).abs().max() <= (2e-6 + K * 2.0 ** -24) * ref.abs().max()

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

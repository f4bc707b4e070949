"""One layer over many rows in one native call (dia_b200_rows_layer_forward) against float64, where its dispatch can go wrong: rows of the
few-rows kernel, of one and two attention tiles, of three-term and two-term products; cross-attention; stacked and separate projections."""

import copy

import pytest
import torch

pytestmark = pytest.mark.gpu


def weights(layer, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    with torch.no_grad():
        for n, p in layer.named_parameters():
            if "norm" in n:
                p.copy_(1 + 0.1 * torch.randn(p.shape, generator=g, device="cuda"))
            else:
                fan = p.shape[0] * p.shape[1] if n.endswith("o_proj.weight") else p.shape[0]
                p.copy_(torch.randn(p.shape, generator=g, device="cuda") * fan ** -0.5)
    return g


def dense(y, m):
    w = m.weight.detach().double()
    return y @ w.reshape(y.shape[-1], -1)


def rms(y, n):
    return y * torch.rsqrt((y * y).mean(-1, keepdim=True) + n.eps) * n.weight.detach().double()


def turn(x, pos):
    a = pos.double()[:, None, None] * 10000.0 ** (-2.0 * torch.arange(64, device="cuda").double() / 128)
    u, v = x[..., :64], x[..., 64:]
    return torch.cat([u * a.cos() - v * a.sin(), u * a.sin() + v * a.cos()], -1)


def attend(q, k, v, ok):
    rep = q.shape[1] // k.shape[1]
    k, v = k.repeat_interleave(rep, 1), v.repeat_interleave(rep, 1)
    s = torch.einsum("ihd,jhd->hij", q, k) * 128 ** -0.5
    return torch.einsum("hij,jhd->ihd", torch.softmax(s.masked_fill(~ok, -torch.inf), -1).nan_to_num(0.0), v).flatten(1)


def mlp(y, m):
    gate, up = dense(y, m.wi_fused).chunk(2, -1)
    return dense(torch.nn.functional.silu(gate) * up, m.wo)


def config(hidden=576):
    from dia_tts_prune_b200.config import DataConfig, DecoderConfig, DiaConfig, EncoderConfig, ModelConfig
    return DiaConfig(model=ModelConfig(encoder=EncoderConfig(n_layer=1, n_embd=256, n_hidden=512, n_head=3, head_dim=128),
                                       decoder=DecoderConfig(n_layer=1, n_embd=320, n_hidden=hidden, gqa_query_heads=4, kv_heads=2, gqa_head_dim=128,
                                                             cross_query_heads=3, cross_head_dim=128), src_vocab_size=256, tgt_vocab_size=1028),
                     data=DataConfig(text_length=512, audio_length=2048, channels=9))


def encode(layer, x, valid):
    T = x.shape[1]
    pos, sa, y = torch.arange(T, device="cuda"), layer.self_attention, x[0].double()
    h = rms(y, layer.pre_sa_norm)
    q, k, v = (dense(h, m).reshape(T, -1, 128) for m in (sa.q_proj, sa.k_proj, sa.v_proj))
    y = y + dense(attend(turn(q, pos), turn(k, pos), v, (pos[:, None] < valid) == (pos[None, :] < valid)), sa.o_proj)
    return y + mlp(rms(y, layer.post_sa_norm), layer.mlp)


def text_state(T, valid):
    from dia_tts_prune_b200.state import EncoderInferenceState
    return EncoderInferenceState(max_seq_len=T, device=torch.device("cuda"), positions=torch.arange(T, device="cuda")[None].float(),
                                 padding_mask=torch.ones((1, T), dtype=torch.bool, device="cuda"), attn_mask=None, valid_lens=[valid])


@pytest.mark.parametrize("T,valid", [(5, 5), (31, 20), (70, 70), (200, 133), (300, 300)])
def test_encoder_layer(T, valid):
    from dia_tts_prune_b200.layers import EncoderLayer
    layer = EncoderLayer(config(), torch.bfloat16).cuda()
    g = weights(layer, T)
    x = torch.randn((1, T, 256), generator=g, device="cuda")
    want = encode(layer, x, valid)
    with torch.inference_mode():
        kept = x.clone()
        got, again = layer(x, text_state(T, valid)), layer(x, text_state(T, valid))
    assert torch.equal(x, kept) and torch.equal(got, again)       # the input stays
    assert (got[0] - want).norm() <= 4e-6 * want.norm()           # a few roundings of fp32 per sum and layer part


@pytest.mark.parametrize("width,heads,kv_heads,B,T", [(1024, 16, 16, 1, 300), (1024, 16, 16, 1, 400), (1024, 16, 16, 1, 700), (1024, 16, 16, 1, 1024),
                                                      (2048, 16, 4, 2, 300), (2048, 16, 4, 2, 500), (2048, 16, 4, 2, 861), (2048, 16, 4, 2, 1300)])
def test_projections_keep_their_sums(width, heads, kv_heads, B, T):
    """Widths and heads of Dia's encoder and decoder.  By themselves the values (which every later frame of a prompt reads) are sums of 64 products that are
    added in fp32; one product of q, k and v has so many columns that it would be summed on the tensor cores, from 385 encoder rows and 769 prompt rows on, and one of
    k and v from 2305 prompt rows on.  K / 64 fp32 additions and terms that are exact to 2^-24: 1e-6; all K products in one accumulator that cuts off: 5e-6 and more."""
    from dia_tts_prune_b200 import engine
    from dia_tts_prune_b200.config import DataConfig, DecoderConfig, DiaConfig, EncoderConfig, ModelConfig
    from dia_tts_prune_b200.layers import EncoderLayer, _rows_layer
    cfg = DiaConfig(model=ModelConfig(encoder=EncoderConfig(n_layer=1, n_embd=width, n_hidden=128, n_head=heads, head_dim=128), decoder=DecoderConfig(
        n_layer=1, n_embd=256, n_hidden=256, gqa_query_heads=2, kv_heads=1, gqa_head_dim=128, cross_query_heads=2, cross_head_dim=128),
        src_vocab_size=256, tgt_vocab_size=1028), data=DataConfig(text_length=1024, audio_length=2048, channels=9))
    layer = EncoderLayer(cfg, torch.bfloat16)
    if kv_heads != heads:
        from dia_tts_prune_b200.layers import Attention
        layer.self_attention = Attention(cfg, width, width, heads, kv_heads, 128, torch.bfloat16, out_embed_dim=width)
    layer, sa = layer.cuda(), layer.self_attention
    g = weights(layer, T)
    x = torch.randn((B, T, width), generator=g, device="cuda")
    k, v = torch.zeros((2, B, kv_heads, T, 128), device="cuda")
    with torch.inference_mode():
        _rows_layer(x, sa, layer.pre_sa_norm, layer.mlp, layer.post_sa_norm, 1e-5, lambda: engine.positions_i32(T, B, x.device), engine.rope_tables_device(cfg, x.device),
                    0, None, k, v)
    want = dense(rms(x.double(), layer.pre_sa_norm), sa.v_proj).reshape(B, T, kv_heads, 128).transpose(1, 2)
    assert (v - want).norm() <= 1e-6 * want.norm()


def test_arguments_follow_the_weights():
    """A weight changed in place, replaced by another tensor, a norm replaced, a copied layer, other rows: the next call reads what is there."""
    from dia_tts_prune_b200.layers import EncoderLayer
    layer = EncoderLayer(config(), torch.bfloat16).cuda()
    g = weights(layer, 1)

    def check(m, T=40):
        x = torch.randn((1, T, 256), generator=g, device="cuda")
        want = encode(m, x, T)
        with torch.no_grad():
            got = m(x, text_state(T, T))
        assert (got[0] - want).norm() <= 4e-6 * want.norm()

    check(layer)
    with torch.no_grad():
        layer.mlp.wo.weight.mul_(0.5)
    check(layer)
    for _ in range(3):                                            # (a new tensor may land on the address of the old one)
        layer.self_attention.q_proj.weight = torch.nn.Parameter(torch.randn((256, 3, 128), generator=g, device="cuda").bfloat16() * 0.06)
        check(layer)
    layer.pre_sa_norm.weight = torch.nn.Parameter(torch.rand((256,), generator=g, device="cuda") + 0.5)
    check(layer)
    twin = copy.deepcopy(layer)
    with torch.no_grad():
        twin.self_attention.v_proj.weight.neg_()
    check(twin)
    check(layer, 300)
    check(layer.double().float())


@pytest.mark.parametrize("T,hidden", [(7, 576), (40, 576), (161, 576), (450, 4096), (900, 4096)])
def test_decoder_layer(T, hidden):
    from dia_tts_prune_b200.layers import DecoderLayer
    from dia_tts_prune_b200.state import DecoderInferenceState, EncoderInferenceState, KVCache
    cfg = config(hidden)
    layer = DecoderLayer(cfg, torch.bfloat16).cuda()
    g = weights(layer, T)
    text, slots = 37, T + 3
    x = torch.randn((2, T, 320), generator=g, device="cuda")
    own = KVCache(2, slots, 128, torch.float32, torch.device("cuda"))
    ck, cv = (torch.randn((2, 3, 64, 128), generator=g, device="cuda") for _ in range(2))
    enc = EncoderInferenceState(max_seq_len=64, device=x.device, positions=torch.zeros(2, 64, device="cuda"),
                                padding_mask=torch.zeros((2, 64), dtype=torch.bool, device="cuda"), attn_mask=None)
    st = DecoderInferenceState.new(cfg, enc, torch.zeros(2, 64, 256, device="cuda"), [KVCache.from_kv(ck, cv)], torch.bfloat16)
    st.text_len = text
    st.prepare_step(0, T)
    pos, want, sa, ca = torch.arange(T, device="cuda"), [], layer.self_attention, layer.cross_attention
    for b in range(2):
        y = x[b].double()
        h = rms(y, layer.pre_sa_norm)
        q, k, v = (dense(h, m).reshape(T, -1, 128) for m in (sa.q_proj, sa.k_proj, sa.v_proj))
        y = y + dense(attend(turn(q, pos), turn(k, pos), v, pos[None, :] <= pos[:, None]), sa.o_proj)
        if b == 1:
            q = turn(dense(rms(y, layer.pre_ca_norm), ca.q_proj).reshape(T, 3, 128), pos)
            seen = torch.ones(T, text, dtype=torch.bool, device="cuda")
            y = y + dense(attend(q, ck[1, :, :text].double().transpose(0, 1), cv[1, :, :text].double().transpose(0, 1), seen), ca.o_proj)
        want.append(y + mlp(rms(y, layer.pre_mlp_norm), layer.mlp))
        keys, values = turn(k, pos).transpose(0, 1), v.transpose(0, 1)
    with torch.inference_mode():
        got = layer(x.clone(), st, self_attn_cache=own, cross_attn_cache=KVCache.from_kv(ck, cv), prefill=True)
    for b in range(2):
        assert (got[b] - want[b]).norm() <= 4e-6 * want[b].norm()
    # (the turning angles are fp32: off by up to T 2^-24, about a tenth of that over all channels)
    assert (own.k[1, :, :T] - keys).norm() <= (2e-6 + T * 2.0 ** -27) * keys.norm() and (own.v[1, :, :T] - values).norm() <= 2e-6 * values.norm()
    assert own.current_idx == T - 1 and not own.k[:, :, T:].any() and not own.v[:, :, T:].any()


@pytest.mark.parametrize("rows", [40, 600])
def test_copies_are_read_on_another_stream(rows):
    """A kernel whose copies are first made behind other work of one stream, and read on another at once"""
    from dia_tts_prune_b200.layers import DenseGeneral
    d = DenseGeneral((64,), (16384,), weight_dtype=torch.bfloat16, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(rows)
    with torch.no_grad():
        d.weight.copy_(torch.randn((64, 16384), generator=g, device="cuda"))
        x = torch.randn((rows, 64), generator=g, device="cuda")
        want = x.double() @ d.weight.double()
        one, two = torch.cuda.Stream(), torch.cuda.Stream()
        for s in (one, two):                                      # (whatever a first call asks the device for has been asked for)
            with torch.cuda.stream(s):
                d(x)
        torch.cuda.synchronize()
        d.weight.neg_()                                           # other weights: their copies are made anew
        want = -want
        torch.cuda.synchronize()
        with torch.cuda.stream(one):
            torch.cuda._sleep(200_000_000)
            first = d(x)
        with torch.cuda.stream(two):
            second = d(x)
        torch.cuda.synchronize()
    for y in (first, second):
        assert (y - want).norm() <= 2e-6 * want.norm()

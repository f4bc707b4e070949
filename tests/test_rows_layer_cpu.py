"""What the layers of many rows hand to their native call (dia_b200_rows_layer_forward), with the kernels stubbed: what does not fit is refused here,
because the call takes pointers and sizes as they are."""

import ctypes as C

import pytest
import torch

from dia_tts_prune_b200 import engine
from dia_tts_prune_b200.config import DataConfig, DecoderConfig, DiaConfig, EncoderConfig, ModelConfig
from dia_tts_prune_b200.layers import DecoderLayer, EncoderLayer


@pytest.fixture
def calls(monkeypatch):
    """The arguments of every native call.  Products of more than 128 rows and 1024 columns read fp16 copies, the others bf16 ones."""
    made = []

    def kmajor(w, out=None):
        t = w.detach().t().contiguous().bfloat16()
        return t if out is None else out.copy_(t)

    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(engine, "dense_prepare_weight", kmajor)
    monkeypatch.setattr(engine, "dense_prepare_half", lambda w, inexact: (w.detach().t().contiguous().half(), w.detach().abs().amax(0).float()))
    monkeypatch.setattr(engine, "dense_half_choice", lambda M, sizes, device: [M > 128 and N > 1024 for N, K in sizes])
    monkeypatch.setattr(engine, "rows_layer_work_bytes", lambda a: 0)
    monkeypatch.setattr(engine, "rows_layer_forward", lambda a, n, device: made.append(type(a).from_buffer_copy(a)))
    return made


def config(head_dim=128, cross_head_dim=128, width=256):
    return DiaConfig(model=ModelConfig(encoder=EncoderConfig(n_layer=1, n_embd=width, n_hidden=512, n_head=4, head_dim=head_dim),
                                       decoder=DecoderConfig(n_layer=1, n_embd=width, n_hidden=576, gqa_query_heads=4, kv_heads=2, gqa_head_dim=head_dim,
                                                             cross_query_heads=4, cross_head_dim=cross_head_dim), src_vocab_size=256, tgt_vocab_size=1028),
                     data=DataConfig(text_length=512, audio_length=2048, channels=9))


def filled(layer):
    with torch.no_grad():
        for p in layer.parameters():
            p.copy_(torch.randn(p.shape).bfloat16())
    return layer


def run(layer, T, B=1, k=None, v=None, cross=None, cross_heads=4, valid=None):
    """The layer's native call for ``[B, T]`` rows; ``cross``: the (keys, values) of a decoder layer's cross-attention."""
    from dia_tts_prune_b200.layers import _rows_layer
    from dia_tts_prune_b200.state import KVCache
    D = layer.pre_sa_norm.weight.numel()
    sa = layer.self_attention
    shape = (B, sa.num_kv_heads, T, 128)
    tables = (torch.zeros(2049, 64), torch.zeros(2049, 64))
    pos = torch.arange(T, dtype=torch.int32).repeat(B)
    ca = None
    if isinstance(layer, DecoderLayer):
        ck, cv = cross if cross is not None else (torch.zeros(B, cross_heads, 8, 128), torch.zeros(B, cross_heads, 8, 128))
        ca = (layer.cross_attention, layer.pre_ca_norm, KVCache.from_kv(ck, cv), [8] * B)
    norm, norm_mlp = (layer.pre_sa_norm, layer.pre_mlp_norm) if ca else (layer.pre_sa_norm, layer.post_sa_norm)
    with torch.no_grad():
        return _rows_layer(torch.randn(B, T, D), sa, norm, layer.mlp, norm_mlp, 1e-5, lambda: pos, tables, 0 if ca else 1, None if ca else [T] * B if valid is None else valid,
                           torch.zeros(shape) if k is None else k, torch.zeros(shape) if v is None else v, ca)


@pytest.mark.parametrize("T", [5, 200])
@pytest.mark.parametrize("head_dim,cross_head_dim", [(64, 128), (256, 128), (128, 64), (128, 256)])
def test_heads_of_other_widths_are_refused(calls, head_dim, cross_head_dim, T):
    """The call reads 128 rows of a copy per head"""
    cfg = config(head_dim, cross_head_dim)
    with pytest.raises(NotImplementedError):
        run(filled(DecoderLayer(cfg, torch.bfloat16)), T)
    if cross_head_dim == 128:
        with pytest.raises(NotImplementedError):
            run(filled(EncoderLayer(cfg, torch.bfloat16)), T)
    assert not calls


def test_kernels_of_another_size_are_refused(calls):
    layer, wider = filled(EncoderLayer(config(), torch.bfloat16)), filled(EncoderLayer(config(width=320), torch.bfloat16))
    run(layer, 5)
    assert len(calls) == 1 and calls[0].heads == 4 and calls[0].D == 256 and calls[0].F == 512
    for part, name in (("self_attention", "q_proj"), ("self_attention", "o_proj"), ("mlp", "wi_fused"), ("mlp", "wo")):
        kept = getattr(getattr(layer, part), name)
        setattr(getattr(layer, part), name, getattr(getattr(wider, part), name))
        with pytest.raises(NotImplementedError):
            run(layer, 6)
        setattr(getattr(layer, part), name, kept)
    assert len(calls) == 1


def test_heads_of_the_caches(calls):
    """The self-attention's cache has the layer's key heads; the cross-attention reads as many as its cache has, where they divide its query heads"""
    layer = filled(DecoderLayer(config(), torch.bfloat16))
    for heads in (1, 2, 4):
        run(layer, 5, cross_heads=heads)
        assert calls[-1].cross_heads == 4 and calls[-1].cross_kv_heads == heads
    n = len(calls)
    good = torch.zeros(1, 2, 7, 128)
    for bad in (torch.zeros(1, 1, 7, 128), torch.zeros(1, 4, 7, 128), torch.zeros(1, 2, 4, 128), torch.zeros(2, 2, 7, 128), torch.zeros(1, 2, 7, 64),
                good.double(), torch.zeros(1, 2, 128, 7).transpose(2, 3)):
        with pytest.raises(ValueError):
            run(layer, 5, k=bad, v=bad)
    with pytest.raises(ValueError):
        run(layer, 5, k=good, v=torch.zeros(1, 2, 9, 128))
    for ck, cv in ((3, 3), (4, 2), (8, 8)):
        with pytest.raises(ValueError):
            run(layer, 5, cross=(torch.zeros(1, ck, 8, 128), torch.zeros(1, cv, 8, 128)))
    assert len(calls) == n
    run(layer, 5, k=good, v=good.clone())
    assert calls[-1].slots == 7


def copies(layer):
    import weakref
    return [weakref.ref(t) for m in layer.modules() for name in ("_b200_wt", "_b200_half") if name in m.__dict__
            for t in (m.__dict__[name][1] if name == "_b200_half" else m.__dict__[name][1:])]


@pytest.mark.parametrize("T", [5, 200])
def test_dropped_copies_are_freed(calls, T):
    """Copies of weights that were moved or replaced go with them: the layer holds none by another way"""
    layer = filled(EncoderLayer(config(width=1280), torch.bfloat16))
    run(layer, T)
    old = copies(layer)
    assert len(old) >= 6
    layer.to(torch.float32)
    assert not any(r() is not None for r in old)
    run(layer, T)
    old = copies(layer)
    layer.mlp.wo.weight = torch.nn.Parameter(layer.mlp.wo.weight.detach().clone())
    assert sum(r() is None for r in old) == (1 if T == 5 else 2)


def test_a_replaced_part_is_read(calls):
    """Another kernel, attention or MLP in the layer's place of one: its copies are read, not those of the one before"""
    layer, other = filled(EncoderLayer(config(), torch.bfloat16)), filled(EncoderLayer(config(), torch.bfloat16))
    run(layer, 5)
    kept = layer.mlp.wo, layer.self_attention                     # (their copies' addresses are not given to others)
    layer.mlp.wo = other.mlp.wo
    run(layer, 5)
    assert calls[-1].wo.wt_bf16 == other.mlp.wo.kernel_weight_kmajor().data_ptr() != calls[0].wo.wt_bf16
    layer.self_attention = other.self_attention
    run(layer, 5)
    assert calls[-1].o.wt_bf16 == other.self_attention.o_proj.kernel_weight_kmajor().data_ptr() != calls[0].o.wt_bf16
    assert calls[0].wo.wt_bf16 == kept[0].kernel_weight_kmajor().data_ptr()


def test_numbers_of_rows_share_their_arguments(calls, monkeypatch):
    """Texts of different lengths read the same copies: none is made anew"""
    layer = filled(EncoderLayer(config(), torch.bfloat16))
    run(layer, 40)
    monkeypatch.setattr(engine, "dense_prepare_weight", None)
    for T in (41, 7, 99, 40):
        run(layer, T)
        for name in ("q", "k", "v", "o", "wi", "wo"):
            assert getattr(calls[-1], name).wt_bf16 == getattr(calls[0], name).wt_bf16
        assert calls[-1].T == T and calls[-1].norm_self == calls[0].norm_self


def test_copies_that_are_there_stay(calls):
    """Calls of many rows and of few read different kinds of copies; neither replaces one that another stream or a captured graph may be reading"""
    layer = filled(DecoderLayer(DiaConfig(model=ModelConfig(
        encoder=EncoderConfig(n_layer=1, n_embd=256, n_hidden=512, n_head=4, head_dim=128),
        decoder=DecoderConfig(n_layer=1, n_embd=256, n_hidden=576, gqa_query_heads=12, kv_heads=2, gqa_head_dim=128, cross_query_heads=4, cross_head_dim=128),
        src_vocab_size=256, tgt_vocab_size=1028), data=DataConfig(text_length=512, audio_length=2048, channels=9)), torch.bfloat16))
    sa = layer.self_attention
    run(layer, 200)                                               # (1536 columns of q: an fp16 copy; k and v bf16 ones)
    assert calls[-1].q.wt_half and not calls[-1].q.wt_bf16 and calls[-1].k.wt_bf16
    kept = [m.kernel_weight_kmajor() for m in (sa.q_proj, sa.k_proj, sa.v_proj)] + [sa.q_proj.kernel_weight_half()[0]]
    for T in (5, 200, 7, 300):
        run(layer, T)
        assert all(a is b for a, b in zip(kept, [m.kernel_weight_kmajor() for m in (sa.q_proj, sa.k_proj, sa.v_proj)] + [sa.q_proj.kernel_weight_half()[0]]))
    q, k, v = (calls[-2].q.wt_bf16, calls[-2].k.wt_bf16, calls[-2].v.wt_bf16)
    assert k - q == 2 * 1536 * 256 and v - k == 2 * 256 * 256     # one behind the other
    layer = filled(EncoderLayer(config(), torch.bfloat16))
    sa = layer.self_attention
    kept = [sa.k_proj.kernel_weight_kmajor()]                     # (the product was called by itself before)
    run(layer, 5)
    assert sa.k_proj.kernel_weight_kmajor() is kept[0] and calls[-1].k.wt_bf16 == kept[0].data_ptr()


def test_numbers_of_valid_keys(calls):
    """One per batch row, none for the rows that have no number"""
    layer = filled(EncoderLayer(config(), torch.bfloat16))
    run(layer, 5, B=3, valid=[4])
    assert list(calls[-1].n_valid)[:3] == [4, 0, 0] and calls[-1].B == 3
    with pytest.raises(ValueError):
        run(layer, 5, B=1, valid=[4, 4])
    with pytest.raises(ValueError):
        run(layer, 5, B=17)
    assert len(calls) == 1


@pytest.mark.parametrize("T,mode", [(200, 2), (300, 1), (300, 0)])
def test_the_workspace_does_not_depend_on_the_valid_keys(T, mode):
    """A caller may take it before the numbers of valid keys are set, or once for several calls"""
    from dia_tts_prune_b200 import _lib
    lib, bytes_of = _lib.load(), []
    for valid in (0, 1, T):
        a = _lib.RowsLayer(B=2, T=T, D=1024, F=4096, heads=16, kv_heads=16, slots=T, mode=mode, cross_heads=16, cross_kv_heads=16, cross_slots=1024, n_pos=2048)
        for b in range(2):
            a.n_valid[b], a.cross_valid[b] = valid, 3 * valid
        bytes_of.append(lib.dia_b200_rows_layer_work_bytes(C.byref(a)))
    assert bytes_of[0] == bytes_of[1] == bytes_of[2] > 0


@pytest.mark.parametrize("Tk", [0, 1, 64, 2 ** 31 - 1])
def test_the_room_of_any_number_of_keys(Tk):
    """Whole tiles of 64 keys, 65535 of them at most: what a caller asks for is not yet checked against what there is"""
    from dia_tts_prune_b200 import _lib
    need = _lib.load().dia_b200_attention_rows_work_bytes(16, 200, Tk, 16, 16, 2, None)
    tiles = min(16 * (-(-Tk // 64)), 65535)
    assert need >= tiles * 64 * 16 * 2 * 512 and need <= tiles * 64 * 16 * (2 * 512 + 8) + 1024

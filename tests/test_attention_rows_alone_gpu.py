"""The tensor-core attention (csrc/attention_split.cu) gives a row what the row and the tokens that it sees make of it: magnitudes far apart
inside a tile, and the same bits however a prompt is cut and whatever shares the step."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def reference(q, k, v, see):
    """softmax(q k / sqrt(d)) v in 64 bits; q [T, H, d], k / v [G, T, d], see [T, T]"""
    H, G = q.shape[1], k.shape[0]
    k, v = k.double().repeat_interleave(H // G, 0), v.double().repeat_interleave(H // G, 0)
    s = (torch.einsum("ihd,hjd->hij", q.double(), k) * q.shape[-1] ** -0.5).masked_fill(~see, -torch.inf)
    return torch.einsum("hij,hjd->ihd", torch.softmax(s, -1), v)


def spiked(what, factor, at=200, T=300):
    """One utterance whose token ``at`` is larger by ``factor``; a value's token has a weight of about e^-60 where it is seen."""
    g = torch.Generator().manual_seed(7)
    q, k, v = torch.randn(1, T, 4, 128, generator=g), torch.randn(1, 2, T, 128, generator=g), torch.randn(1, 2, T, 128, generator=g)
    if what == "faint":
        q[..., 0], k[:, :, at, :] = 8.0, 0.0
        k[:, :, at, 0] = -85.0
    plain = [t.clone() for t in (q, k, v)]
    if what == "query":
        q[:, at] *= factor
    elif what == "key":
        k[:, :, at] *= factor
    else:
        v[:, :, at] *= factor
    return (q, k, v), plain


@pytest.mark.parametrize("what,factor", [(w, f) for w in ("query", "key", "value", "faint") for f in (1e6, 1e9, 1e12)])
def test_a_token_far_larger_than_its_neighbours(what, factor):
    """Rows in front of the large token do not see it: the same bits as without it.  Every row's error is measured against the row's own
    largest output: 22-bit factors and fp32 sums, 2^-21 of a score of at most about 8 and of the largest weight x value that it sees, a
    few times over."""
    from dia_tts_prune_b200 import engine as E
    (q, k, v), plain = spiked(what, factor)
    T, see = q.shape[1], torch.ones(q.shape[1], q.shape[1]).tril().bool()
    got = E.attention_rows(q.cuda(), k.cuda(), v.cuda(), T, 0, None).cpu()
    base = E.attention_rows(*[t.cuda() for t in plain], T, 0, None).cpu()
    assert torch.equal(got[:, :200], base[:, :200])
    ref = reference(q[0], k[0], v[0], see)
    top = ref.abs().amax(-1, keepdim=True)
    # (a score of a large query or key has an error of its own size: where it decides between two keys there is nothing to hold the row to)
    rows = torch.ones(T, dtype=torch.bool)
    if what == "query":
        rows[200] = False
    err = ((got[0].double() - ref).abs() / top)[rows]
    assert err.max() <= 2e-5, err.max()


@pytest.mark.parametrize("mode", [0, 2])
def test_one_utterance_does_not_set_the_scale_of_another(mode):
    from dia_tts_prune_b200 import engine as E
    g = torch.Generator().manual_seed(8)
    q, k, v = torch.randn(2, 257, 4, 128, generator=g), torch.randn(2, 2, 257, 128, generator=g), torch.randn(2, 2, 257, 128, generator=g)
    one = E.attention_rows(q.cuda(), k.cuda(), v.cuda(), 257, mode, [130, 257]).cpu()
    q[1], k[1], v[1] = q[1] * 1e9, k[1] * 1e-9, v[1] * 1e9
    two = E.attention_rows(q.cuda(), k.cuda(), v.cuda(), 257, mode, [130, 257]).cpu()
    assert torch.equal(one[0], two[0])


def cuts(n, parts):
    assert sum(parts) == n
    at = [sum(parts[:i]) for i in range(len(parts))]
    return [(a, a + p) for a, p in zip(at, parts)]


def grouped(heads, kv_heads, dim, window, keep, cap, page):
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import PubopelConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    cfg = SY.pubopel_config(width=32, layers=1, heads=heads, kv_heads=kv_heads, dim=dim, experts=1, top=1, expert_ff=8, shared_ff=None, vocab=64,
                            window=window or None, keep_first=keep, softcap=cap or None)
    model = CausalLM(PubopelConfig.model_validate(cfg), SY.pubopel_weights(cfg, 3), dtype="bfloat16", device="cuda:0", max_tokens=4096,
                     max_sequences=6, page_size=page, max_rows=1024)
    return model, (heads + kv_heads) * dim, lambda x, parts: model.engine.op_attention(0, x.clone(), parts)


def mixed(heads, kv_heads, dim, vdim):
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import KupelixConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    cfg = SY.kupelix_config(width=32, kinds=["attention"], heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, ff=8, vocab=64)
    w = SY.kupelix_weights(cfg, 3)
    cfg["layers"][0]["mlp"] = None
    model = CausalLM(KupelixConfig.model_validate(cfg), w, dtype="bfloat16", device="cuda:0", max_tokens=4096, max_sequences=6, max_rows=1024)
    return model, model.layers[0].layer.n_in, lambda x, parts: model.engine.op_mixer_kernels(0, x.clone(), parts)


def latent(heads, dim, kv_rank, rot_dim, vdim, window):
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import FipadraConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    cfg = SY.fipadra_config(width=64, kinds=["latent_attention"], heads=heads, dim=dim, rot_dim=rot_dim, vdim=vdim, q_rank=72, kv_rank=kv_rank,
                            window=window, vocab=64)
    cfg["layers"][0]["mlp"] = None
    w = SY.fipadra_weights(cfg, 3)
    model = CausalLM(FipadraConfig.model_validate(cfg), w, dtype="float32", device="cuda:0", max_tokens=4096, max_sequences=6, max_rows=1024)
    return model, 64, lambda x, parts: model.engine.op_mixer(0, x.clone(), parts)


@pytest.mark.parametrize("make,args", [(grouped, (4, 2, 64, 0, 0, 0.0, 64)), (grouped, (8, 1, 128, 100, 3, 0.0, 16)), (grouped, (2, 1, 200, 0, 0, 0.0, 7)),
                                       (grouped, (4, 2, 64, 0, 0, 4.0, 64)), (grouped, (2, 1, 200, 100, 3, 2.0, 16)),    # scores on both sides of the polynomial's range
                                       (mixed, (8, 2, 64, 128)), (latent, (4, 32, 192, 16, 64, 0)), (latent, (2, 16, 40, 8, 16, 90))])
def test_a_row_has_the_same_bits_in_any_step(make, args):
    """A prompt of 300 rows in one step, in portions of more than 8 rows, and beside other sequences whose tokens are larger: with few rows the
    row tiles split the keys themselves, with many a launch in front does it."""
    model, n_in, op = make(*args)
    g = torch.Generator().manual_seed(9)
    x = (torch.randn(300, n_in, generator=g) * 10.0 ** torch.randint(-2, 3, (300, 1), generator=g)).cuda()
    other = (1000 * torch.randn(400, n_in, generator=g)).cuda()

    def run(parts, beside):
        seq = model.state.open("a")
        model.state.reserve(seq, 300)
        out = []
        for i, (a, b) in enumerate(cuts(300, parts)):
            rows, h = [(seq, b - a, a)], x[a:b]
            if beside:
                o = model.state.open(f"o{i}")
                model.state.reserve(o, beside)
                rows, h = [(o, beside, 0), *rows], torch.cat([other[:beside], h])
            y = op(h, rows)
            out.append((y[0] if isinstance(y, (tuple, list)) else y)[-(b - a):].clone())
            if beside:
                model.state.close(f"o{i}")
        model.state.close("a")
        return torch.cat(out)

    whole = run([300], 0)
    for parts, beside in (([100, 9, 191], 0), ([300], 33), ([9, 9, 60, 222], 400)):
        assert torch.equal(whole, run(parts, beside)), (parts, beside)


def by_rows(q, k, v, see):
    """The same in 64 bits, row by row over the keys that the row sees: an infinity or a NaN elsewhere does not enter"""
    T, H, d = q.shape
    out = torch.zeros(T, H, v.shape[-1], dtype=torch.float64)
    for i in range(T):
        j = see[i].nonzero()[:, 0]
        for h in range(H):
            g = h * k.shape[0] // H
            s = (q[i, h].double() * k[g, j].double()).sum(-1) * d ** -0.5
            out[i, h] = (torch.softmax(s, -1)[:, None] * v[g, j].double()).sum(0)
    return out


@pytest.mark.parametrize("what,x", [("value", torch.inf), ("value", -torch.inf), ("value", torch.nan), ("key", torch.inf), ("key", torch.nan),
                                    ("query", torch.inf), ("query", torch.nan)])
def test_a_number_that_is_not_finite(what, x):
    """One infinity or NaN: rows that do not see it keep their bits, rows that do get what fp32 arithmetic makes of it, channel by channel."""
    from dia_tts_prune_b200 import engine as E
    g, at, T = torch.Generator().manual_seed(11), 200, 257
    q, k, v = torch.randn(2, T, 4, 128, generator=g), torch.randn(2, 2, T, 128, generator=g), torch.randn(2, 2, T, 128, generator=g)
    base = E.attention_rows(q.cuda(), k.cuda(), v.cuda(), T, 0, None).cpu()
    if what == "query":
        q[0, at, 1, 5] = x
        touched = torch.zeros(2, T, 4, dtype=torch.bool)
        touched[0, at, 1] = True
    else:
        (k if what == "key" else v)[0, 1, at, 5] = x
        touched = torch.zeros(2, T, 4, dtype=torch.bool)
        touched[0, at:, 2:] = True
    got = E.attention_rows(q.cuda(), k.cuda(), v.cuda(), T, 0, None).cpu()
    assert torch.equal(got[~touched], base[~touched])
    ref = by_rows(q[0], k[0], v[0], torch.ones(T, T).tril().bool())[touched[0]]
    torch.testing.assert_close(got[touched].double(), ref, rtol=2e-5, atol=2e-5, equal_nan=True)


@pytest.mark.parametrize("rows", [150, 300])
@pytest.mark.parametrize("make,args,window", [(grouped, (4, 2, 64, 33, 3, 20.0, 16), 33), (mixed, (8, 2, 64, 160), 0), (latent, (4, 32, 192, 16, 64, 40), 40)])
def test_a_token_of_a_step_that_is_not_finite(make, args, window, rows):
    """A token of NaN in a step: rows in front of it and rows whose window has left it behind keep their bits.  Keys split by the row tiles and
    in advance."""
    model, n_in, op = make(*args)
    x = torch.randn(rows, n_in, generator=torch.Generator().manual_seed(12)).cuda()

    def run(h):
        seq = model.state.open("a")
        model.state.reserve(seq, rows)
        y = op(h, [(seq, rows, 0)])
        model.state.close("a")
        return (y[0] if isinstance(y, (tuple, list)) else y).clone()

    base, h, at = run(x), x.clone(), 70
    h[at] = torch.nan
    got, after = run(h), at + window if window else rows
    assert torch.equal(got[:at], base[:at]) and torch.equal(got[after:], base[after:])
    assert torch.isfinite(base).all() and got[at:after].isnan().any(-1).all()


def test_more_row_tiles_than_a_grid_is_high():
    """128 heads that share their keys leave one token to a row tile: a step of more than 65535 rows"""
    model_rows, heads, dim, window = 65600, 128, 4, 5
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import PubopelConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    cfg = SY.pubopel_config(width=32, layers=1, heads=heads, kv_heads=1, dim=dim, experts=1, top=1, expert_ff=8, shared_ff=None, vocab=64, window=window,
                            keep_first=0, softcap=None)
    model = CausalLM(PubopelConfig.model_validate(cfg), SY.pubopel_weights(cfg, 3), dtype="bfloat16", device="cuda:0", max_tokens=model_rows + 64,
                     max_sequences=1, page_size=64, max_rows=model_rows)
    x = torch.randn(model_rows, (heads + 1) * dim, generator=torch.Generator().manual_seed(13)).cuda()
    seq = model.state.open("a")
    model.state.reserve(seq, model_rows)
    got = model.engine.op_attention(0, x.clone(), [(seq, model_rows, 0)])
    again = model.engine.op_attention(0, x[65500:].clone(), [(seq, 100, 65500)])
    assert torch.equal(got[65500:], again) and torch.isfinite(got).all() and got.abs().amax(-1).min() > 0


def test_keys_split_in_several_rounds():
    """More tiles of keys than the launch that splits them has CTAs for a part: against the keys that the row tiles split for themselves"""
    model, n_in, op = grouped(32, 32, 16, 0, 0, 0.0, 64)
    x = torch.randn(3000, n_in, generator=torch.Generator().manual_seed(14)).cuda()
    seq = model.state.open("a")
    model.state.reserve(seq, 3000)
    parts = [op(x[a:b], [(seq, b - a, a)]).clone() for a, b in ((0, 1024), (1024, 2048), (2048, 3000))]
    for a in (1900, 2048, 2980):
        assert torch.equal(op(x[a:a + 20], [(seq, 20, a)]), torch.cat(parts)[a:a + 20])


def kernels_of(call):
    """Kernels of a call.  A session of the profiler loses some of its first or last kernels, or all of a few, when seconds have passed since one before (after
    half a minute two of five, or five of five, in two sessions of three); it has lost none of a call between two hundred others on either side."""
    from torch.profiler import ProfilerActivity, profile
    other = torch.zeros(64, device="cuda")
    call()
    best = []
    for _ in range(2):
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            for part in (None, call, None):
                for _ in range(200 if part is None else 1):
                    other.erfinv_() if part is None else part()
                torch.cuda.synchronize()
        names = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA and not any(n in e.name for n in ("emcpy", "emset", "erfinv"))]
        best = max(best, names, key=len)
    return best


@pytest.mark.parametrize("heads", [4, 8, 16])
def test_the_widest_latent_rows(heads):
    """Latent rows of 256 + 64 channels leave the row tile's queries and two slots of keys 3 KB of shared memory for all else, whatever the number
    of heads; against the row kernels of short steps"""
    model, n_in, op = latent(heads, 32, 256, 64, 64, 0)
    x = torch.randn(200, n_in, generator=torch.Generator().manual_seed(15)).cuda()
    seq = model.state.open("a")
    model.state.reserve(seq, 200)
    assert any("split_attention_kernel" in n for n in kernels_of(lambda: op(x, [(seq, 200, 0)])))
    whole = op(x, [(seq, 200, 0)]).clone()
    short = torch.cat([op(x[a:a + 8], [(seq, 8, a)]) for a in range(0, 200, 8)])
    assert (whole - short).abs().max() <= 2e-5 * short.abs().max()


def test_a_wait_that_ran_out_reaches_the_caller():
    """The word that a kernel sets when a wait of its ran out, set by hand: the next launch returns an error, the one after it runs"""
    import ctypes as C

    from dia_tts_prune_b200 import _lib
    from dia_tts_prune_b200 import engine as E
    q, k, v = torch.randn(1, 256, 2, 128).cuda(), torch.randn(1, 1, 256, 128).cuda(), torch.randn(1, 1, 256, 128).cuda()
    good = E.attention_rows(q, k, v, 256, 0, None)
    word_of = getattr(_lib.load(), "_ZN3dia23split_attention_ran_outEiP11CUstream_st")
    word_of.restype, word_of.argtypes = C.POINTER(C.c_int), [C.c_int, C.c_void_p]
    word = word_of(torch.cuda.current_device(), None)
    assert word and word[0] == 0
    word[0] = 1
    with pytest.raises(Exception):
        E.attention_rows(q, k, v, 256, 0, None)
    assert word[0] == 0 and torch.equal(E.attention_rows(q, k, v, 256, 0, None), good)

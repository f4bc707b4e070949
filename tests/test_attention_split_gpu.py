"""The tensor-core attention with split fp32 operands (csrc/attention_split.cu) at the sizes where it can go wrong: edges of its
tiles of 64 keys and 128 (token, head) rows, channel groups, segments of several sequences, windows, magnitudes far from one."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def close(got, ref, scale):
    """fp32 arithmetic: 22-bit terms and fp32 sums.  A score is off by at most about 2^-21 |q| |k| and a weighted sum by 2^-21 of the
    largest value, so 2e-5 of the result's largest magnitude leaves a factor of ten."""
    assert torch.isfinite(got).all()
    err = (got.double().cpu() - ref).abs().max().item()
    assert err <= 2e-5 * scale, (err, scale)


def sink_reference(x, past, H, G, d, p, window, keep, cap, eps):
    n = x.shape[0]
    q, raw = x[past:, :H * d], x[:, H * d:]
    rms = lambda t: t / torch.sqrt((t * t).mean(-1, keepdim=True) + eps)      # noqa: E731
    q, k, v = (rms(q) * p["q"]).reshape(-1, H, d), (rms(raw) * p["k"]).reshape(n, G, d), raw.reshape(n, G, d)
    i, j = torch.arange(past, n)[:, None], torch.arange(n)[None]
    ok = j <= i
    if window:
        ok = ok & ((i - j < window) | (j < keep))
    out = []
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].T * (d ** -0.5 * p["temp"][h])
        if cap:
            s = cap * torch.tanh(s / cap)
        s = (s - 2.0 ** (-8.0 * (h + 1) / H) * (i - j)).masked_fill(~ok, -torch.inf)
        m = torch.maximum(s.max(-1, keepdim=True).values, p["sink"][h])
        e = torch.exp(s - m)
        out.append(e @ v[:, h * G // H] / (e.sum(-1, keepdim=True) + torch.exp(p["sink"][h] - m)))
    return torch.stack(out, 1).reshape(n - past, H * d)


@pytest.mark.parametrize("rows,past,H,G,d,window,keep,cap,amp,page", [
    ([64], 0, 4, 1, 128, 0, 0, 0.0, 1.0, 64),           # one key tile
    ([65], 0, 1, 1, 128, 0, 0, 30.0, 1.0, 16),          # one key more; one head per row tile
    ([32], 33, 8, 2, 64, 0, 0, 0.0, 1e-4, 16),          # a portion behind cached keys; small values
    ([127, 1, 2], 0, 4, 4, 16, 0, 0, 0.0, 1e4, 64),     # 128 tokens of a row tile: the last segments in the next one; large values
    ([40, 90], 70, 6, 2, 96, 33, 3, 30.0, 1.0, 16),     # two heads per tile, a window that keeps the first keys
    ([130], 0, 8, 1, 200, 100, 200, 0.0, 1.0, 64),      # two channel groups, more kept keys than the window starts behind
    ([70], 0, 16, 1, 256, 0, 0, 0.0, 1.0, 64),          # the widest heads
    ([33], 0, 3, 1, 20, 5, 1, 0.0, 1.0, 7),             # channels that are no multiple of 16, odd pages
    # from here on enough rows that the keys are split in advance
    ([128], 0, 4, 1, 128, 0, 0, 0.0, 1.0, 64),
    ([200, 1, 63, 190], 130, 8, 2, 64, 33, 3, 30.0, 1.0, 16),    # the kept keys' tile in front of the window's
    ([150, 90], 200, 8, 1, 40, 50, 100, 0.0, 1e3, 7),   # more kept keys than one tile holds
    ([256], 6100, 4, 2, 64, 0, 0, 0.0, 1.0, 64),        # more cached keys than the room holds
])
def test_grouped_query_attention(rows, past, H, G, d, window, keep, cap, amp, page):
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import PubopelConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    cfg = SY.pubopel_config(width=32, layers=1, heads=H, kv_heads=G, dim=d, experts=1, top=1, expert_ff=8, shared_ff=None, vocab=64,
                            window=window or None, keep_first=keep, softcap=cap or None)
    w = SY.pubopel_weights(cfg, 3)
    model = CausalLM(PubopelConfig.model_validate(cfg), w, dtype="bfloat16", device="cuda:0", max_tokens=8192, max_sequences=4,
                     page_size=page, max_rows=512)
    p = {n: w[f"l0.mix.{t}"].double() for n, t in (("q", "q.norm"), ("k", "k.norm"), ("temp", "temp"), ("sink", "sink"))}
    g = torch.Generator().manual_seed(5)
    x = [torch.randn((past + n, (H + G) * d), generator=g) * amp for n in rows]
    seqs = [model.state.open(str(i)) for i in range(len(rows))]
    for s, t in zip(seqs, x):
        model.state.reserve(s, len(t))
        for a in range(0, past, 512):
            b = min(past, a + 512)
            model.engine.op_attention(0, t[a:b].cuda(), [(s, b - a, a)])
    got = model.engine.op_attention(0, torch.cat([t[past:] for t in x]).cuda(), [(s, n, past) for s, n in zip(seqs, rows)])
    ref = torch.cat([sink_reference(t.double(), past, H, G, d, p, window, keep, cap, cfg["norm"]["eps"]) for t in x])
    close(got, ref, ref.abs().max().item())


@pytest.mark.parametrize("H,G,d,dv,rows", [(8, 2, 128, 128, [70, 1]), (8, 2, 128, 128, [128, 40]), (4, 4, 64, 32, [64]), (12, 3, 40, 24, [33, 5]), (16, 1, 24, 256, [65])])
def test_mixed_scores(H, G, d, dv, rows):
    """Scores mixed across heads: the kernel mixes the queries instead, against the mixer's definition in 64 bits."""
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import KupelixConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    cfg = SY.kupelix_config(width=32, kinds=["attention"], heads=H, kv_heads=G, dim=d, vdim=dv, ff=8, vocab=64)
    cfg["layers"][0]["mixer"]["rot"] = None
    w = SY.kupelix_weights(cfg, 3)
    cfg["layers"][0]["mlp"] = None
    model = CausalLM(KupelixConfig.model_validate(cfg), w, dtype="bfloat16", device="cuda:0", max_tokens=512, max_sequences=2, max_rows=256)
    n_in = model.layers[0].layer.n_in
    g = torch.Generator().manual_seed(6)
    x = [torch.randn((n, n_in), generator=g) for n in rows]
    seqs = [model.state.open(str(i)) for i in range(len(rows))]
    for s, n in zip(seqs, rows):
        model.state.reserve(s, n)
    got = model.engine.op_mixer_kernels(0, torch.cat(x).cuda(), [(s, n, 0) for s, n in zip(seqs, rows)])
    p = {n[len("l0.mix."):]: t.double() for n, t in w.items() if n.startswith("l0.mix.")}
    ref = []
    for t in x:
        t, n = t.double(), t.shape[0]
        nq, nk = H * d, G * d
        rms = lambda a: a / torch.sqrt((a * a).mean(-1, keepdim=True) + cfg["norm"]["eps"])      # noqa: E731
        q = rms((t[:, :nq] + p["q.b"]).reshape(n, H, d)) * p["q.norm"]
        k = rms((t[:, nq:nq + nk] + p["k.b"]).reshape(n, G, d)) * p["k.norm"]
        v = (t[:, nq + nk:nq + nk + G * dv] + p["v.b"]).reshape(n, G, dv)
        raw = torch.stack([q[:, h] @ k[:, h * G // H].T for h in range(H)]) * cfg["layers"][0]["mixer"]["scale"]
        mixed = torch.einsum("hg,gij->hij", p["talk"], raw).masked_fill(torch.ones(n, n).triu(1).bool(), -torch.inf)
        gate = torch.sigmoid(t[:, nq + nk + G * dv:nq + nk + G * dv + H])
        out = []
        for h in range(H):
            m = torch.maximum(mixed[h].max(-1, keepdim=True).values, p["sink"][h])
            e = torch.exp(mixed[h] - m)
            out.append(e @ v[:, h * G // H] / (e.sum(-1, keepdim=True) + torch.exp(p["sink"][h] - m)) * gate[:, h:h + 1])
        ref.append(torch.stack(out, 1).reshape(n, H * dv))
    ref = torch.cat(ref)
    close(got, ref, ref.abs().max().item())


@pytest.mark.parametrize("mode,B,Tq,Tk,Hq,Hkv,n_valid", [(0, 2, 256, 256, 4, 1, None), (1, 2, 300, 300, 2, 2, [37, 257]), (1, 1, 256, 256, 3, 3, [0]),
                                                         (2, 2, 257, 130, 4, 2, [0, 129]), (2, 1, 511, 64, 2, 2, [64])])
def test_row_modes(mode, B, Tq, Tk, Hq, Hkv, n_valid):
    """Dia's causal, pad-partitioned and prefix attention where the split kernel takes them (256 queries and more), against 64 bits.  Both
    factors keep 22 bits: 2^-21 of a score of at most about 6 here and of the value, a few times over."""
    from dia_tts_prune_b200 import engine as E
    g = torch.Generator().manual_seed(Tq + Tk)
    q, k, v = (torch.randn(s, generator=g) for s in ((B, Tq, Hq, 128), (B, Hkv, Tk, 128), (B, Hkv, Tk, 128)))
    got = E.attention_rows(q.cuda(), k.cuda(), v.cuda(), Tk, mode, n_valid).cpu().double()
    i, j = torch.arange(Tq)[:, None], torch.arange(Tk)[None, :]
    for b in range(B):
        n = n_valid[b] if n_valid else Tk
        see = j <= i if mode == 0 else (i < n) == (j < n) if mode == 1 else (j < n).expand(Tq, Tk)
        s = (torch.einsum("ihd,hjd->hij", q[b].double(), k[b].double().repeat_interleave(Hq // Hkv, 0)) * 128 ** -0.5).masked_fill(~see, -torch.inf)
        w = torch.nan_to_num(torch.softmax(s, -1), nan=0.0)
        ref = torch.einsum("hij,hjd->ihd", w, v[b].double().repeat_interleave(Hq // Hkv, 0))
        assert (got[b] - ref).abs().max() <= 2e-5 * max(1.0, ref.abs().max())


@pytest.mark.parametrize("mode,B,Tq,Tk,Hq,Hkv,n_valid", [(0, 2, 192, 192, 4, 1, None), (1, 2, 200, 200, 2, 2, [37, 200]), (1, 1, 256, 256, 3, 3, [0]),
                                                         (2, 3, 257, 130, 4, 2, [0, 129, 64]), (0, 1, 1000, 1000, 4, 2, None)])
def test_row_modes_have_the_same_bits_with_keys_split_in_advance(mode, B, Tq, Tk, Hq, Hkv, n_valid):
    """Keys that a launch in front splits, and keys that every row tile splits for itself: the same terms and scales"""
    from dia_tts_prune_b200 import engine as E
    g = torch.Generator().manual_seed(Tq + Tk)
    q, k, v = (torch.randn(s, generator=g).cuda() for s in ((B, Tq, Hq, 128), (B, Hkv, Tk, 128), (B, Hkv, Tk, 128)))
    assert torch.equal(E.attention_rows(q, k, v, Tk, mode, n_valid), E.attention_rows(q, k, v, Tk, mode, n_valid, room=False))


@pytest.mark.parametrize("H,G,d,window", [(2, 1, 16, 0), (4, 1, 256, 400)])
def test_keys_beyond_the_room(H, G, d, window):
    """A sequence with more keys than the room for split keys holds (twice 64 rows, 32768 and 192 keys): the last tiles are split by the row tiles"""
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import PubopelConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    past, rows, step = 33408, 40, 64
    cfg = SY.pubopel_config(width=32, layers=1, heads=H, kv_heads=G, dim=d, experts=1, top=1, expert_ff=8, shared_ff=None, vocab=64, window=window or None,
                            keep_first=0, softcap=None)
    w = SY.pubopel_weights(cfg, 3)
    model = CausalLM(PubopelConfig.model_validate(cfg), w, dtype="bfloat16", device="cuda:0", max_tokens=33600, max_sequences=1, page_size=64, max_rows=step)
    p = {n: w[f"l0.mix.{t}"].double() for n, t in (("q", "q.norm"), ("k", "k.norm"), ("temp", "temp"), ("sink", "sink"))}
    x = torch.randn((past + rows, (H + G) * d), generator=torch.Generator().manual_seed(5))
    seq = model.state.open("a")
    model.state.reserve(seq, past + rows)
    dev = x.cuda()
    for a in range(0, past, step):
        model.engine.op_attention(0, dev[a:a + step].clone(), [(seq, step, a)])
    got = model.engine.op_attention(0, dev[past:].clone(), [(seq, rows, past)])
    ref = sink_reference(x.double(), past, H, G, d, p, window, 0, 0.0, cfg["norm"]["eps"])
    close(got, ref, ref.abs().max().item())


@pytest.mark.parametrize("kind,window", [("latent", 0), ("latent_narrow", 0), ("latent_widest", 0), ("talk", 0), ("grouped", 0), ("grouped", 700)])
def test_keys_beyond_the_room_have_the_same_bits(kind, window):
    """Keys that the room holds (all, with 1024 rows a step) and keys that it does not (with 64 rows the last seven tiles of 527): split by a launch in front, or by
    the row tiles that walk them; an engine that is told the step's sizes gets room for them.  The caches are filled with numbers, not by steps."""
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import FipadraConfig, KupelixConfig, PubopelConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    if kind == "talk":
        cfg = SY.kupelix_config(width=64, kinds=["attention"], heads=4, kv_heads=2, dim=72, vdim=100, ff=32, vocab=64)
        conf, w = KupelixConfig, SY.kupelix_weights(cfg, 5)
    elif kind == "grouped":
        cfg = SY.pubopel_config(width=64, layers=1, heads=4, kv_heads=2, dim=64, experts=1, top=1, expert_ff=8, shared_ff=None, vocab=64, window=window or None,
                                keep_first=4 if window else 0, softcap=30.0)
        conf, w = PubopelConfig, SY.pubopel_weights(cfg, 5)
    else:
        rank, rot = {"latent": (256, 32), "latent_narrow": (64, 16), "latent_widest": (256, 64)}[kind]
        cfg = SY.fipadra_config(width=64, kinds=["latent_attention"], heads=4, dim=32, vdim=32, vocab=64, q_rank=48, kv_rank=rank, rot_dim=rot)
        conf, w = FipadraConfig, SY.fipadra_weights(cfg, 5)
    past, x = (32900, 700), torch.randn(40, 64, generator=torch.Generator().manual_seed(6)).cuda()
    got, more = [], []
    for rows, told in ((64, False), (64, True), (1024, True)):
        model = CausalLM(conf.model_validate(cfg), w, dtype="float32", device="cuda:0", max_tokens=33800, max_sequences=2, max_sequence_tokens=33024, page_size=64, max_rows=rows)
        seqs = [model.state.open(n) for n in "ab"]
        for q, n in zip(seqs, past):
            model.state.reserve(q, n + 20)
        g = torch.Generator().manual_seed(7)
        for t in (model.state.k_pages[0], model.state.v_pages[0], model.state.latent_pages[0]):
            if t is not None:
                t.copy_(torch.randn(t.shape, generator=g))
        if not told:
            model.engine._say = lambda *sizes: None
        bytes_of = lambda: model.engine.lib.lm_b200_engine_workspace_bytes(model.engine._h)
        before = bytes_of()
        got.append(model.engine.op_mixer(0, x, [(q, 20, n) for q, n in zip(seqs, past)]).clone())
        more.append(bytes_of() - before)
    assert torch.isfinite(got[0]).all() and torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    assert more[0] == 0 and (more[1] > 0) == (window == 0) and more[2] == 0      # (a window's keys fit in any case)


@pytest.mark.parametrize("B,Tq,Hq,Hkv", [(1, 200, 16, 16), (2, 300, 4, 1)])
def test_calls_without_room_borrow_it(B, Tq, Hq, Hkv):
    """Their keys are split by a launch in front like those of calls that bring room; during a capture they go without"""
    from dia_tts_prune_b200 import _lib, engine as E
    lib = _lib.load()
    g = torch.Generator().manual_seed(Tq)
    q, k, v = (torch.randn(s, generator=g).cuda() for s in ((B, Tq, Hq, 128), (B, Hkv, 300, 128), (B, Hkv, 300, 128)))

    def call(out):
        before = lib.dia_b200_launch_count()
        _lib.check(lib.dia_b200_attention_rows(*[t.data_ptr() for t in (q, k, v, out)], B, Tq, 300, Hq, Hkv, 300, 2, None, torch.cuda.current_stream().cuda_stream),
                   "attention_rows")
        return lib.dia_b200_launch_count() - before

    want, out = E.attention_rows(q, k, v, 300, 2, None), torch.zeros_like(q)
    assert call(out) == 2 and torch.equal(out, want)
    side, graph, again = torch.cuda.Stream(), torch.cuda.CUDAGraph(), torch.zeros_like(q)
    with torch.cuda.graph(graph, stream=side):
        assert call(again) == 1
    graph.replay()
    torch.cuda.synchronize()
    assert (again - want).abs().max() <= 2e-5 * want.abs().max()      # (200 rows: the fp32 kernel)
    assert lib.dia_b200_trim() == 0 and call(out) == 2 and torch.equal(out, want)


@pytest.mark.parametrize("place", [3, 20, 45, 63])
def test_denominators_are_summed_per_16_keys(place):
    """One key of weight one and, in every tile of 64, one of 2^-25: half a unit in the last place of a sum with the first, so 64 of them are lost from a sum per
    tile (a denominator 2^-19 too small) and none from a sum per 16 keys, unless they share those 16.  Channel 1, which has the first key's value
    alone, is one over the denominator; four roundings of the score change a weight of 2^-25 by 2^-17 of itself at most, and the result by less than 2^-24."""
    from dia_tts_prune_b200 import engine as E
    tiles, light = 64, 2.0 ** -25
    q, k, v = torch.zeros(1, 192, 1, 128), torch.zeros(1, 1, 64 * tiles, 128), torch.zeros(1, 1, 64 * tiles, 128)
    q[..., 0] = 1.0
    k[..., 0] = -400.0 * 128 ** 0.5                               # (exp of that is zero)
    k[0, 0, place::64, 0] = math.log(light) * 128 ** 0.5
    heavy = 8 if place >= 16 else 40
    k[0, 0, heavy, 0] = 0.0
    v[0, 0, :, 0], v[0, 0, heavy, 0], v[0, 0, heavy, 1] = 1.0, 0.0, 1.0
    got = E.attention_rows(q.cuda(), k.cuda(), v.cuda(), 64 * tiles, 2, None)[0, :, 0, 1].double().cpu()
    assert (got - 1.0 / (1.0 + tiles * light)).abs().max() <= 2.0 ** -22


def test_sizes_are_for_one_call():
    """Sizes said for a call that is refused are gone with it: the call that follows, with as many sequences and rows, is another step"""
    import ctypes as C

    import numpy as np

    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import FipadraConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    cfg = SY.fipadra_config(width=64, kinds=["delta"], heads=2, kv_heads=2, dim=64, vdim=64, vocab=64)
    model = CausalLM(FipadraConfig.model_validate(cfg), SY.fipadra_weights(cfg, 5), dtype="float32", device="cuda:0", max_tokens=1024, max_sequences=2, max_rows=256)
    x = torch.randn(200, 64, generator=torch.Generator().manual_seed(3)).cuda()

    def run(rows):
        seqs = [model.state.open(n) for n in "ab"]
        for q, n in zip(seqs, rows):
            model.state.reserve(q, n)
        y = model.engine.op_mixer(0, x, [(q, n, 0) for q, n in zip(seqs, rows)]).clone()
        for n in "ab":
            model.state.close(n)
        return y

    want = run((190, 10))
    model.engine._say = lambda *sizes: None
    sizes = np.array([100, 100, 0, 0], dtype=np.int32)            # (both long: with these the short one would have no kernel)
    lib, h = model.engine.lib, model.engine._h
    assert lib.lm_b200_step_sizes(h, sizes.ctypes.data, sizes.ctypes.data + 8, 2) == 0
    assert lib.lm_b200_op_mixer(h, 0, None, None, 200, 2, None, C.c_void_p(0)) != 0
    assert torch.equal(run((190, 10)), want)
    assert lib.lm_b200_step_sizes(h, sizes.ctypes.data, sizes.ctypes.data + 8, 0) != 0

"""The delta rule with one decay per head in chunks of 32 tokens (csrc/lm_delta.cu) against the same tokens one after the other (csrc/lm_scan.cu, which
portions of fewer than 96 tokens take): ragged last chunks, heads and columns that do not fill a block, a state that is continued, a token of NaN."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def delta_model(heads, kv_heads, dim, vdim, max_rows=2048):
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import FipadraConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    cfg = SY.fipadra_config(width=64, kinds=["delta"], heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, vocab=64)
    return CausalLM(FipadraConfig.model_validate(cfg), SY.fipadra_weights(cfg, 5), dtype="float32", device="cuda:0", max_tokens=8192, max_sequences=4,
                    max_rows=max_rows)


def run(model, x, cuts):
    """Outputs and the state behind them of sequences x, every one in the portions of its cuts, one step per portion index."""
    seqs = [model.state.open(str(i)) for i in range(len(x))]
    out = [[] for _ in x]
    at = [0] * len(x)
    for q, t in zip(seqs, x):
        model.state.reserve(q, len(t))
    for step in range(max(len(c) for c in cuts)):
        who = [i for i in range(len(x)) if step < len(cuts[i])]
        y = model.engine.op_mixer(0, torch.cat([x[i][at[i]:at[i] + cuts[i][step]] for i in who]), [(seqs[i], cuts[i][step], at[i]) for i in who])
        for i, part in zip(who, y.split([cuts[i][step] for i in who])):
            out[i].append(part.clone())
            at[i] += cuts[i][step]
    state = [model.state.rec_states[0][q.slot].clone() for q in seqs]
    for i in range(len(x)):
        model.state.close(str(i))
    return [torch.cat(o) for o in out], state


def portions(n, most=90):
    return [min(most, n - a) for a in range(0, n, most)]


def close(a, b):
    """Both sum in fp32: a token's state and read-out are sums of up to `dim` and 32 products with factors of at most one, behind up to 1000 tokens that decay;
    64 such sums in another order are off by about 64 x 2^-24 of the largest value."""
    assert torch.isfinite(a).all()
    assert (a - b).abs().max() <= 64 * 2.0 ** -24 * b.abs().max()


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,rows", [
    (2, 1, 128, 128, [96]),                                       # whole chunks, the shortest portion that takes them
    (4, 2, 64, 16, [97]),                                         # one token more; the smallest block of columns
    (3, 3, 72, 20, [351, 5, 320, 1000]),                          # channels and columns that do not fill a block; a short sequence between long ones
    (8, 2, 128, 132, [640, 95]),                                  # the longest portion that stays with the scan
    (4, 2, 64, 64, [90, 40, 95, 3]),                              # rows for chunks, but no sequence
    (4, 1, 4, 4, [330]),                                          # the narrowest heads
])
def test_chunks_against_one_token_after_the_other(heads, kv_heads, dim, vdim, rows):
    model = delta_model(heads, kv_heads, dim, vdim)
    g = torch.Generator().manual_seed(sum(rows))
    x = [torch.randn(n, 64, generator=g).cuda() for n in rows]
    ya, sa = run(model, x, [portions(n) for n in rows])
    yb, sb = run(model, x, [[n] for n in rows])
    for a, b in zip(yb + sb, ya + sa):
        close(a, b)
    # and a state that chunks continue: a portion of 50 tokens in front
    x = [t for t in x if len(t) >= 420]
    if x:
        yc, sc = run(model, x, [[50, len(t) - 50] for t in x])
        for a, b in zip(yc + sc, [y for y in ya if len(y) >= 420] + [s for s, n in zip(sa, rows) if n >= 420]):
            close(a, b)


def test_a_sequence_beside_others_has_the_same_bits():
    model = delta_model(4, 2, 64, 64)
    g = torch.Generator().manual_seed(3)
    x = [torch.randn(n, 64, generator=g).cuda() for n in (400, 700, 33)]
    together, states = run(model, x, [[len(t)] for t in x])
    for i in range(2):
        y, s = run(model, [x[i]], [[len(x[i])]])
        assert torch.equal(y[0], together[i]) and torch.equal(s[0], states[i])


def test_a_token_of_nan_reaches_no_token_in_front():
    model = delta_model(2, 1, 64, 64)
    x = torch.randn(400, 64, generator=torch.Generator().manual_seed(4)).cuda()
    good = run(model, [x], [[400]])[0][0]
    for at in (37, 64, 383):
        bad = x.clone()
        bad[at] = float("nan")
        y = run(model, [bad], [[400]])[0][0]
        assert torch.equal(y[:at], good[:at]) and torch.isnan(y[at:at + 1]).any()


def test_short_sequences_of_a_long_step():
    """Three sequences of 300 rows in one step (four rows of the convolution a block, across the sequences' ends) against each alone (one)"""
    model = delta_model(4, 2, 64, 64)
    g = torch.Generator().manual_seed(6)
    x = [torch.randn(n, 64, generator=g).cuda() for n in (299, 300, 301)]
    for cuts in ([[len(t)] for t in x], [[2, len(t) - 2] for t in x]):
        together, states = run(model, x, cuts)
        for i in range(3):
            y, s = run(model, [x[i]], [cuts[i]])
            close(together[i], y[0])
            close(states[i], s[0])


def test_steps_of_long_and_short_portions_repeat_their_bits():
    """The scan of the short ones runs beside the chunks of the long ones: thirty times the same outputs and states"""
    model = delta_model(4, 2, 128, 128)
    g = torch.Generator().manual_seed(11)
    x = [torch.randn(n, 64, generator=g).cuda() for n in (700, 37, 96, 95)]
    first = None
    for _ in range(30):
        got = run(model, x, [[len(t)] for t in x])
        first = first or got
        for a, b in zip(got[0] + got[1], first[0] + first[1]):
            assert torch.equal(a, b)


def test_only_kernels_with_sequences_are_launched():
    """The same 288 rows: short portions by the scan, long ones by the two kernels of the chunks, both by all three"""
    model = delta_model(2, 2, 64, 64)
    count = model.engine.lib.lm_b200_launch_count
    launches = []
    for rows in ([95, 95, 95, 3], [96, 96, 96], [100, 92, 93, 3]):
        x = [torch.randn(n, 64, generator=torch.Generator().manual_seed(n)).cuda() for n in rows]
        before = count()
        run(model, x, [[n] for n in rows])
        launches.append(count() - before)
    assert launches[1] - launches[0] == 1 and launches[2] - launches[0] == 2

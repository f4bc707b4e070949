"""The products of a few rows (few_rows of csrc/gemm_tcgen05.cu) in chains of launches that start before their predecessors have ended."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("requests", [4, 8])
def test_chains_of_early_launches(requests):
    """Products small enough that an SM could hold four CTAs, each with half of its tensor memory: a step is repeated through its graph, and
    has the same bits each time"""
    from dia_tts_prune_b200 import synthetic as SY
    from dia_tts_prune_b200.lm_config import ForilornConfig
    from dia_tts_prune_b200.lm_model import CausalLM
    cfg = SY.forilorn_config(width=2048, kinds=["latent_attention"] * 6, heads=8, dim=64, vocab=64, lat_dim=64, rot_dim=16, lat_vdim=64, q_rank=512,
                             kv_rank=64, ff=2048)
    model = CausalLM(ForilornConfig.model_validate(cfg), SY.forilorn_weights(cfg, 3), dtype="bfloat16", device="cuda:0", max_tokens=64 * requests,
                     max_sequences=requests, max_rows=64)
    for i in range(requests):
        model.run_step([{"id": str(i), "tokens": [1 + i, 2, 3], "want": []}])
    entries = [{"id": str(i), "tokens": [5 + i], "want": [0]} for i in range(requests)]
    first = None
    for _ in range(300):
        out = model.run_step(entries).clone()
        for e in entries:
            model.state.sequences[e["id"]].length -= 1
        first = out if first is None else first
        assert torch.equal(out, first)
    assert torch.isfinite(first).all()


@pytest.mark.parametrize("M", [4, 200, 2000])
def test_the_largest_numbers(M):
    """Numbers that a bf16 would round up to an infinity, in dense layers of few, some and many rows; an infinity stays one.  The bound on the
    others is that of fp32 sums of 64 products: 2^-21 of the result, a few times over."""
    from dia_tts_prune_b200 import engine as E
    g = torch.Generator().manual_seed(M)
    x, w = torch.randn(M, 128, generator=g), (torch.rand(128, 64, generator=g) * 1e-3 + 1e-4).to(torch.bfloat16)
    x[0, 3], x[1, 7], x[3, 9] = 3.4e38, -3.4028234e38, torch.inf
    y = E.dense_forward(x.cuda(), E.dense_prepare_weight(w.cuda())).cpu().double()
    ref = x.double() @ w.double()
    assert (y[3] == torch.inf).all()
    rows = torch.arange(M) != 3
    assert ((y - ref)[rows].abs() / ref[rows].abs().amax(-1, keepdim=True)).max() <= 1e-5


def test_launches_are_counted_kernel_by_kernel():
    """The launch counters against the kernels that a profiler sees: products that prepare their operand, attention that splits its keys first"""
    import test_attention_rows_alone_gpu as A

    from dia_tts_prune_b200 import engine as E
    from dia_tts_prune_b200.lm_engine import launch_count
    model, n_in, op = A.grouped(8, 1, 64, 0, 0, 0.0, 64)
    x = torch.randn(200, n_in, generator=torch.Generator().manual_seed(1)).cuda()
    seq = model.state.open("a")
    model.state.reserve(seq, 200)
    lat, lat_in, lat_op = A.latent(4, 32, 64, 16, 64, 0)
    h = torch.randn(40, lat_in, generator=torch.Generator().manual_seed(2)).cuda()
    lseq = lat.state.open("a")
    lat.state.reserve(lseq, 40)
    w = E.dense_prepare_weight(torch.randn(128, 256).to(torch.bfloat16).cuda())
    nw = torch.rand(128).cuda()
    own = lambda names: sum("dia::" in n or "lm::" in n or "dia_" in n for n in names)                    # noqa: E731
    for count, call in [(launch_count, lambda: op(x[:200], [(seq, 200, 0)])), (launch_count, lambda: op(x[:12], [(seq, 12, 0)])),
                        (launch_count, lambda: lat_op(h, [(lseq, 40, 0)])),
                        *[(E.launch_count, lambda M=M, n=n: E.dense_forward(torch.randn(M, 128).cuda(), w, norm_weight=n))
                          for M in (4, 40, 4000) for n in (None, nw)]]:
        seen = own(A.kernels_of(call))
        before = count()
        call()
        assert count() - before == seen, seen

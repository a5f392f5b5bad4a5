"""Top-k routing kernel against its PyTorch statement."""

import pytest
import torch

from pplx_garden.ops import topk_route, topk_route_reference


def test_reference_on_cpu():
    logits = torch.tensor([[0.0, 3.0, 1.0, 2.0]])
    idx, w = topk_route_reference(logits, 2)
    assert idx.view(torch.int32).tolist() == [[1, 3]]
    assert torch.allclose(w, torch.softmax(torch.tensor([[3.0, 2.0]]), dim=-1))
    idx, _ = topk_route_reference(logits, 2, bias=torch.tensor([10.0, 0.0, 0.0, 0.0]))
    assert idx.view(torch.int32).tolist() == [[0, 1]]


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,experts,k,dtype,with_bias", [
    (128, 256, 8, torch.float32, False),
    (4096, 256, 8, torch.float32, True),
    (2048, 128, 8, torch.bfloat16, False),
    (77, 60, 6, torch.float32, True),
    (5, 1024, 32, torch.float32, False),
    (33, 8, 8, torch.float32, False),
    (1, 384, 1, torch.bfloat16, True),
])
def test_topk_route_matches_reference(tokens, experts, k, dtype, with_bias):
    dev = torch.device("cuda", 0)
    gen = torch.Generator(device="cpu").manual_seed(tokens * 31 + experts)
    logits = torch.randn((tokens, experts), generator=gen).to(dtype).to(dev)
    bias = (torch.randn(experts, generator=gen) * 0.5).to(dev) if with_bias else None
    idx, w = topk_route(logits, k, bias)
    ref_idx, ref_w = topk_route_reference(logits, k, bias)
    torch.cuda.synchronize()
    got, want = idx.view(torch.int32).cpu(), ref_idx.view(torch.int32).cpu()
    if dtype == torch.bfloat16:
        # bf16 logits tie often; the chosen sets must then agree as sets of (logit) values
        x = logits.float().cpu() + (0 if bias is None else bias.cpu())
        assert torch.equal(torch.gather(x, 1, got.long()), torch.gather(x, 1, want.long()))
    else:
        assert torch.equal(got, want)
    assert torch.allclose(w.cpu(), ref_w.cpu(), rtol=1e-4, atol=1e-6)
    assert torch.allclose(w.sum(dim=-1).cpu(), torch.ones(tokens), atol=1e-5)


@pytest.mark.gpu
def test_ties_go_to_the_lower_index():
    dev = torch.device("cuda", 0)
    logits = torch.zeros((3, 64), device=dev)
    idx, w = topk_route(logits, 4)
    assert idx.view(torch.int32).cpu().tolist() == [[0, 1, 2, 3]] * 3
    assert torch.allclose(w.cpu(), torch.full((3, 4), 0.25))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("experts,k,levels", [
    (8, 8, 3), (31, 5, 4), (64, 6, 1000), (96, 8, 7), (160, 6, 50), (256, 8, 1000), (256, 8, 9), (256, 32, 40),
    (512, 10, 2), (1000, 32, 300), (1024, 1, 5)])
def test_ties_and_row_layouts(experts, k, levels, dtype):
    """Few distinct logits, so that the k-th ties with many others (more than a warp's worth too), on
    rows that can and cannot be read as vectors; the order is the stable one."""
    dev = torch.device("cuda", 0)
    gen = torch.Generator(device="cpu").manual_seed(experts * k + levels)
    for tokens, row in ((1, experts), (700, experts), (9, experts + 1)):
        # whole and half numbers up to 128: exact in bf16
        wide = (torch.randint(0, levels, (tokens, row), generator=gen) % 256 / 2 - 50).to(dtype).to(dev)
        logits = wide[:, :experts]
        for bias in (None, (torch.randint(0, 3, (experts,), generator=gen) / 2).to(dev)):
            idx, w = topk_route(logits, k, bias)
            x = logits.float().cpu()
            want = torch.sort(x if bias is None else x + bias.cpu(), dim=-1, descending=True, stable=True).indices[:, :k]
            assert torch.equal(idx.view(torch.int32).cpu().long(), want)
            # __expf is good to 2 ulp + |x| ulp; differences of logits here are below 200, and what is
            # that far down has no weight
            assert torch.allclose(w.cpu(), torch.softmax(torch.gather(x, 1, want), dim=-1), rtol=1e-4, atol=1e-6)


def _us(fn, n=30):
    for _ in range(3):
        fn()
    best = float("inf")
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(n):
            fn()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3 / n)
    return best


@pytest.mark.gpu
@pytest.mark.parametrize("experts,full,k", [(96, 128, 6), (160, 256, 6), (192, 256, 8), (320, 512, 8), (384, 512, 8)])
def test_expert_counts_that_leave_lanes_empty_cost_no_more(experts, full, k):
    """The same number of keys a lane, fewer lanes: a token must not cost more than with all lanes filled. It
    does, 1.4 to 1.7 times, where the bound is not found and every token takes the rounds."""
    dev = torch.device("cuda", 0)
    some, all_ = torch.randn((32768, experts), device=dev), torch.randn((32768, full), device=dev)
    assert _us(lambda: topk_route(some, k)) < 1.2 * _us(lambda: topk_route(all_, k))


@pytest.mark.gpu
@pytest.mark.parametrize("experts,k", [(96, 24), (96, 25), (160, 20), (160, 21), (160, 32), (384, 24), (384, 25), (33, 32), (32, 32), (30, 20)])
def test_k_at_the_number_of_filled_lanes(experts, k):
    """k at and above what the vector layout fills (24, 20 and 24 lanes), where another layout takes over."""
    dev = torch.device("cuda", 0)
    logits = torch.randn((65, experts), generator=torch.Generator().manual_seed(experts + k)).to(dev)
    idx, w = topk_route(logits, k)
    want = torch.sort(logits.cpu(), dim=-1, descending=True, stable=True).indices[:, :k]
    assert torch.equal(idx.view(torch.int32).cpu().long(), want)
    # __expf: 2 ulp and |x| ulp, |x| below 10 here
    assert torch.allclose(w.cpu(), torch.softmax(torch.gather(logits.cpu(), 1, want), dim=-1), rtol=1e-5, atol=1e-7)


@pytest.mark.gpu
@pytest.mark.parametrize("experts,ranked,rounds", [(128, 3, 2), (160, 14, 17), (256, 3, 1), (256, 19, 22), (320, 14, 16), (384, 16, 18),
                                                   (512, 18, 21), (512, 3, 2), (1000, 19, 24), (1024, 8, 32)])
@pytest.mark.parametrize("tokens", [9, 3000])
def test_ranking_and_rounds_on_both_sides_of_their_rule(experts, ranked, rounds, tokens):
    dev = torch.device("cuda", 0)
    logits = torch.randn((tokens, experts), generator=torch.Generator().manual_seed(experts + ranked)).to(dev)
    x = logits.cpu()
    order = torch.sort(x, dim=-1, descending=True, stable=True).indices
    for k in (ranked, rounds):
        idx, w = topk_route(logits, k)
        assert torch.equal(idx.view(torch.int32).cpu().long(), order[:, :k])
        # __expf: 2 ulp and |x| ulp, |x| below 12 here
        assert torch.allclose(w.cpu(), torch.softmax(torch.gather(x, 1, order[:, :k]), dim=-1), rtol=1e-5, atol=1e-7)

"""tcgen05 grouped SwiGLU runner against a plain PyTorch FP32 statement of the same op."""

import pytest
import torch

from conftest import gpu_count

from ep_xpress_b200.ops import GroupedSwiGLU, swiglu_reference

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(gpu_count() < 1, reason="needs a CUDA device")]


def make_case(rows, topk, experts, hidden, inter, valid, seed, local_fraction=0.6):
    g = torch.Generator(device="cpu").manual_seed(seed)
    x = (torch.randn((rows, hidden), generator=g) * 0.5).to(torch.bfloat16)
    ids = torch.full((rows, topk), -1, dtype=torch.int64)
    for r in range(rows):
        chosen = torch.randperm(experts, generator=g)[:min(topk, experts)]
        keep = torch.rand(len(chosen), generator=g) < local_fraction
        ids[r, :len(chosen)] = torch.where(keep, chosen, torch.full_like(chosen, -1))
    weights = torch.rand((rows, topk), generator=g).to(torch.float32)
    w13 = (torch.randn((experts, 2 * inter, hidden), generator=g) * 0.05).to(torch.bfloat16)
    w2 = (torch.randn((experts, hidden, inter), generator=g) * 0.05).to(torch.bfloat16)
    count = torch.tensor([valid], dtype=torch.int32)
    return [t.cuda() for t in (x, ids, weights, count, w13, w2)]


def assert_elementwise_close(got, want):
    """Every element within 2 % of the reference, plus an absolute allowance of one BF16 step of a
    value four times the tensor's typical magnitude: a row is a sum of per-slot results that are
    rounded to BF16 one by one, a slot result is often several times larger than the sum it
    cancels into, and a different FP32 accumulation order may flip one of those roundings."""
    got, want = got.float(), want.float()
    if not want.numel():
        return
    step = float(want.pow(2).mean().sqrt()) * 2.0 ** -5
    torch.testing.assert_close(got, want, rtol=2e-2, atol=max(step, 1e-6))


@pytest.mark.parametrize("gather_loads", [True, False])
@pytest.mark.parametrize("rows,topk,experts,hidden,inter,valid", [
    (64, 2, 2, 256, 128, 64),
    (300, 4, 3, 512, 256, 257),
    (1000, 8, 8, 1024, 384, 1000),
    (130, 8, 32, 256, 128, 0),
    (5, 2, 2, 256, 128, 3),
    (300, 9, 16, 512, 128, 300),       # more slots than the slot sum keeps in flight
    (10000, 4, 8, 256, 128, 9800),     # more pairs than the align step holds in registers, streaming slot sum
])
def test_matches_fp32_reference(rows, topk, experts, hidden, inter, valid, gather_loads):
    x, ids, weights, count, w13, w2 = make_case(rows, topk, experts, hidden, inter, valid, seed=rows)
    runner = GroupedSwiGLU(w13, w2, max_rows=rows, topk=topk, gather_loads=gather_loads)
    out = torch.full((rows, hidden), 7.0, dtype=torch.bfloat16, device="cuda")
    runner(x, ids, weights, count, out=out)
    runner.check()
    want = swiglu_reference(x, ids, weights, valid, w13, w2)
    assert_elementwise_close(out[:valid], want[:valid])
    assert (out[valid:] == 7.0).all()          # rows at or above valid_count are not touched
    again = torch.empty_like(out)
    runner(x, ids, weights, count, out=again)  # order of pairs inside an expert never changes a result
    assert torch.equal(again[:valid], out[:valid])


def test_benchmarked_shape_matches_fp32_reference():
    """Hidden 7168, intermediate 2048 (112 k-steps, 16 and 28 column tiles): the shape of the layer
    benchmark, on a few experts and a few hundred rows, gathered and pre-gathered activations
    bit-identical to each other."""
    rows, topk, experts, hidden, inter, valid = 520, 8, 4, 7168, 2048, 500
    x, ids, weights, count, w13, w2 = make_case(rows, topk, experts, hidden, inter, valid, seed=11, local_fraction=0.4)
    outs = []
    for gather_loads in (True, False):
        runner = GroupedSwiGLU(w13, w2, max_rows=rows, topk=topk, gather_loads=gather_loads)
        out = torch.full((rows, hidden), 7.0, dtype=torch.bfloat16, device="cuda")
        runner(x, ids, weights, count, out=out)
        runner.check()
        outs.append(out)
    assert torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16))
    want = swiglu_reference(x, ids, weights, valid, w13, w2)
    assert_elementwise_close(outs[0][:valid], want[:valid])
    assert (outs[0][valid:] == 7.0).all()


@pytest.mark.parametrize("valid,topk,experts,hidden,inter", [
    (16, 2, 2, 256, 128),
    (100, 4, 3, 512, 256),
    (250, 8, 8, 1024, 384),
    (650, 4, 3, 512, 256),
])
def test_padding_of_the_batch_does_not_change_its_rows(valid, topk, experts, hidden, inter):
    """The number of rows a batch is padded to bounds the token tiles: other tile widths, ring depths and
    numbers of epilogue warps, the same sums. ``pair_ctas`` is accepted and changes nothing."""
    x, ids, weights, count, w13, w2 = make_case(valid, topk, experts, hidden, inter, valid, seed=valid + 1)
    want = swiglu_reference(x, ids, weights, valid, w13, w2)
    first = None
    for rows, pair_ctas in ((valid, False), (valid, True), (2 * valid, False), (1300, True)):
        padded = [torch.cat([t, torch.full((rows - valid, t.shape[1]), fill, dtype=t.dtype, device=t.device)])
                  for t, fill in ((x, 0), (ids, -1), (weights, 0))]
        runner = GroupedSwiGLU(w13, w2, max_rows=rows, topk=topk, pair_ctas=pair_ctas)
        out = torch.full((rows, hidden), 7.0, dtype=torch.bfloat16, device="cuda")
        runner(*padded, count, out=out)
        runner.check()
        assert (out[valid:] == 7.0).all()
        first = out if first is None else first
        assert torch.equal(out[:valid].view(torch.int16), first[:valid].view(torch.int16))
    assert_elementwise_close(first[:valid], want[:valid])


@pytest.mark.parametrize("counts,pad", [
    ([0, 1, 15, 16, 17, 31, 33, 0], 3),               # one narrow tile each, experts without rows
    ([63, 65, 127, 128, 129, 2], 0),                  # every token-box size
    ([255, 256, 257, 0, 511, 513], 40),               # one, two and three token tiles per expert
    ([2047], 1), ([1, 2047], 0), ([4090, 7], 0),      # one, two and four CTAs in the align step
    ([1], 0),
])
@pytest.mark.parametrize("gather_loads", [True, False])
def test_token_tile_edges_match_fp32_reference(counts, pad, gather_loads):
    """Rows per expert at the edges of the token tiles; rows of one expert are spread over the batch."""
    hidden, inter = 256, 128
    g = torch.Generator().manual_seed(sum(counts))
    experts = torch.repeat_interleave(torch.arange(len(counts)), torch.tensor(counts))
    valid = len(experts)
    ids = torch.full((valid + pad, 2), -1, dtype=torch.int64)
    ids[torch.arange(valid), torch.randint(0, 2, (valid,), generator=g)] = experts[torch.randperm(valid, generator=g)]
    x = (torch.randn((valid + pad, hidden), generator=g) * 0.5).to(torch.bfloat16)
    weights = torch.rand((valid + pad, 2), generator=g)
    w13 = (torch.randn((len(counts), 2 * inter, hidden), generator=g) * 0.05).to(torch.bfloat16)
    w2 = (torch.randn((len(counts), hidden, inter), generator=g) * 0.05).to(torch.bfloat16)
    x, ids, weights, w13, w2 = (t.cuda() for t in (x, ids, weights, w13, w2))
    runner = GroupedSwiGLU(w13, w2, max_rows=valid + pad, topk=2, gather_loads=gather_loads)
    out = torch.full((valid + pad, hidden), 7.0, dtype=torch.bfloat16, device="cuda")
    runner(x, ids, weights, torch.tensor([valid], dtype=torch.int32, device="cuda"), out=out)
    runner.check()
    assert_elementwise_close(out[:valid], swiglu_reference(x, ids, weights, valid, w13, w2)[:valid])
    assert (out[valid:] == 7.0).all()


@pytest.mark.parametrize("count", [-1, -(2 ** 31)])
@pytest.mark.parametrize("rows,gather_loads", [(5, False), (5, True), (10000, False)])     # both forms of the slot sum
def test_negative_count_is_an_empty_batch(rows, gather_loads, count):
    """The count is a device value that no host check sees: nothing is read or written for it."""
    x, ids, weights, _, w13, w2 = make_case(rows, 2, 2, 256, 128, rows, seed=11)
    runner = GroupedSwiGLU(w13, w2, max_rows=rows, topk=2, gather_loads=gather_loads)
    out = torch.full_like(x, 7.0)
    runner(x, ids, weights, torch.tensor([count], dtype=torch.int32, device="cuda"), out=out)
    runner.check()
    assert (out == 7.0).all() and runner.counters.tolist() == [0, 0]


def test_misaligned_rows_are_rejected_on_the_host():
    x, ids, weights, count, w13, w2 = make_case(64, 2, 2, 256, 128, 64, seed=6)
    runner = GroupedSwiGLU(w13, w2, max_rows=64, topk=2)
    skewed = torch.zeros(64 * 256 + 1, dtype=torch.bfloat16, device="cuda")[1:].view(64, 256)
    for hidden, out in ((skewed, torch.empty_like(x)), (x, skewed)):
        with pytest.raises(RuntimeError, match="16-byte aligned"):
            runner(hidden, ids, weights, count, out=out)


def test_pair_bound_overflow_is_reported():
    x, ids, weights, count, w13, w2 = make_case(512, 4, 2, 256, 128, 512, seed=3, local_fraction=1.0)
    runner = GroupedSwiGLU(w13, w2, max_rows=512, topk=4, max_local_pairs=128)
    runner(x, ids, weights, count)
    with pytest.raises(RuntimeError, match="max_local_pairs"):
        runner.check()

"""MoE exchange kernels: routing with the plan in its last block, the quantising dispatch, the conversion of received rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def group():
    import dataclasses

    from parallelkernelbench_b200.parallel import init_context
    from parallelkernelbench_b200.parallel.symm_heap import SymmetricHeap

    base = init_context()
    ctx = dataclasses.replace(base, owns_group=False, _heap=None)
    ctx._heap = SymmetricHeap.create(ctx, nbytes=1 << 30)
    yield ctx.heap().world_group
    ctx.finalize()
    base.finalize()


@pytest.mark.parametrize("T,hidden,E,k,cap", [(1, 128, 8, 1, 2.0), (7, 384, 8, 2, 2.0), (149, 640, 16, 8, 2.0), (300, 2048, 8, 2, 0.6),
                                              (1500, 256, 64, 4, 1.2)])
def test_quantising_dispatch_matches_quantise_then_copy(group, T, hidden, E, k, cap):
    from parallelkernelbench_b200.ops import fp8_dequantize_1x128, fp8_quantize_1x128
    from parallelkernelbench_b200.ops.moe import MoEExchange, route_topk

    mark = group.heap.mark()
    g = torch.Generator(device="cuda").manual_seed(T + hidden)
    x = (torch.randn(T, hidden, device="cuda", generator=g) * torch.rand(T, 1, device="cuda", generator=g)).to(torch.bfloat16)
    x[T // 2, :128] = 0                                                   # an all-zero block
    logits = torch.randn(T, E, device="cuda", generator=g)
    ex = MoEExchange(group, E, hidden, T, k, cap, True)
    ref_gates, ref_idx, ref_counts = route_topk(logits, None, k)
    for _ in range(2):                                                    # the work words are zero again after a call
        gates, idx = ex.route(logits, None, None)
        assert torch.equal(gates, ref_gates) and torch.equal(idx, ref_idx) and torch.equal(ex.counts, ref_counts)
        off = torch.zeros(E + 1, dtype=torch.int32, device="cuda")
        off[1:] = ref_counts.cumsum(0)
        assert torch.equal(ex.offsets, off) and torch.equal(ex.seg_base, off[:E]) and (ex.cursor == 0).all() and (ex.route_work == 0).all()
    y, s = fp8_quantize_1x128(x)
    token = torch.arange(T * k, device="cuda") // k
    for dequantize in (True, False):
        ex.plan(idx.view(-1), None, counts_ready=True)
        got = ex.dispatch(x, idx.view(-1), dequantize=dequantize)
        slots = ex.slots.long()
        fits = slots >= 0
        assert int((~fits).sum()) == max(0, T * k - ex.capacity) and slots[fits].unique().numel() == int(fits.sum())
        e = idx.view(-1)[fits].long()
        assert ((slots[fits] >= off[e]) & (slots[fits] < off[e + 1])).all()
        if dequantize:
            assert torch.equal(got[slots[fits]], fp8_dequantize_1x128(y, s)[token[fits]])
        else:
            assert torch.equal(got[0][slots[fits]], y[token[fits]])
            assert torch.equal(got[1][slots[fits]][:, :hidden // 128], s[token[fits]])
    group.heap.release(mark)


@pytest.mark.parametrize("E,k", [(8, 2), (40, 8), (256, 8)])
def test_routing_of_logits_that_are_not_numbers(E, k):
    """Every assignment goes to an expert that exists, k different ones a token; rows without such logits are as they were."""
    from parallelkernelbench_b200.ops.moe import route_topk

    logits = torch.randn(9, E, device="cuda", generator=torch.Generator(device="cuda").manual_seed(E))
    want = route_topk(logits, None, k)
    bad = logits.clone()
    bad[1] = float("nan")
    bad[2, :E - 1] = float("nan")                                         # one number is left
    bad[3, 5] = float("nan")
    bad[4, 3] = float("inf")
    bad[5] = float("-inf")
    gates, idx, counts = route_topk(bad, None, k)
    assert ((idx >= 0) & (idx < E)).all() and int(counts.sum()) == 9 * k
    assert all(row.unique().numel() == k for row in idx)
    assert torch.equal(counts, torch.bincount(idx.view(-1).long(), minlength=E).int())
    for r in (0, 6, 7, 8):
        assert torch.equal(idx[r], want[1][r]) and torch.equal(gates[r], want[0][r])
    assert gates[1].isnan().all() and idx[1].tolist() == list(range(k)) and int(idx[2, 0]) == E - 1


def test_conversion_of_received_rows_leaves_own_rows_alone():
    """What a rank of a larger group does after the dispatch: rows of its own segment are bf16 already."""
    from parallelkernelbench_b200 import _native as nv
    from parallelkernelbench_b200.ops import fp8_dequantize_1x128, fp8_quantize_1x128

    hidden, cap = 640, 200
    offsets = torch.tensor([0, 50, 50, 130, 170], dtype=torch.int32, device="cuda")
    seg_base = torch.tensor([10, 50, 50, 169], dtype=torch.int32, device="cuda")
    counts = torch.tensor([20, 0, 80, 1], dtype=torch.int32, device="cuda")
    y, s = fp8_quantize_1x128(torch.randn(cap, hidden, device="cuda", dtype=torch.bfloat16))
    pitch = 32                                                            # 5 scales padded to a multiple of 16 bytes
    scales = torch.zeros(cap, pitch // 4, device="cuda")
    scales[:, :5] = s
    out = torch.full((cap, hidden), 7.0, device="cuda", dtype=torch.bfloat16)
    nv.check(nv.cuda_lib().pkb_moe_dequant(nv.ptr(y), nv.ptr(scales), hidden, pitch, nv.ptr(offsets), nv.ptr(seg_base), nv.ptr(counts), 4,
                                           cap, nv.ptr(out), nv.current_stream()))
    own = torch.zeros(cap, dtype=torch.bool, device="cuda")
    for b, c in zip(seg_base.tolist(), counts.tolist()):
        own[b:b + c] = True
    own[170:] = True
    assert (out[own] == 7).all() and torch.equal(out[~own], fp8_dequantize_1x128(y, s)[~own])

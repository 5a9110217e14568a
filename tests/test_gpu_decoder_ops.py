"""Row-wise and elementwise kernels of the decoder step at the edges of their loops, against fp64 restatements."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


# one element; one 16-byte load; a row that is no multiple of it (scalar form); the end of one pass of four loads per thread
# (512 x 8 x 4), one load more, and a row of several passes
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("vocab", [1, 8, 1001, 16384, 16392, 50008])
def test_ce_stats_edges(vocab, dtype):
    from parallelkernelbench_b200.ops import ce_local_stats

    rows = 5
    x = (torch.randn(rows, vocab, device="cuda", generator=_gen(vocab)) * 6).to(dtype)
    x[1] = -50.0                                         # a row far below zero
    x[2, -1] = 80.0                                      # the maximum sits in the last column
    tgt = torch.tensor([0, vocab - 1, vocab // 2, 7 + vocab, -1], device="cuda") + 7
    st = ce_local_stats(x, tgt, 7).double()
    xd = x.double()
    assert torch.equal(st[:, 0], xd.max(-1).values)
    ref = torch.exp(xd - xd.max(-1, keepdim=True).values).sum(-1)
    # ex2.approx is within 2 ulp, its argument within |x| * 2^-23 of exact, and the terms add up in fp32 over a few hundred per thread
    torch.testing.assert_close(st[:, 1], ref, rtol=5e-5, atol=0)
    inside = ((tgt - 7) >= 0) & ((tgt - 7) < vocab)
    want = torch.where(inside, xd.gather(1, (tgt - 7).clamp(0, vocab - 1)[:, None])[:, 0], torch.zeros(rows, device="cuda", dtype=torch.float64))
    assert torch.equal(st[:, 2], want)


# columns: one load, the end of a block's 8192 columns, one load more
@pytest.mark.parametrize("rows,vocab", [(1, 8), (3, 8192), (3, 8200), (130, 1000)])
def test_ce_backward_edges(rows, vocab):
    from parallelkernelbench_b200.ops import ce_backward

    x = torch.randn(rows, vocab, device="cuda", generator=_gen(rows)).to(torch.bfloat16)
    tgt = torch.randint(0, vocab, (rows,), device="cuda", generator=_gen(1))
    lse = torch.logsumexp(x.double(), -1)
    got = ce_backward(x, lse.float(), tgt, 0, 0.25, upstream=torch.tensor(2.0, device="cuda"))
    ref = torch.exp(x.double() - lse[:, None])
    ref[torch.arange(rows, device="cuda"), tgt] -= 1.0
    # one bf16 rounding of a value of at most 0.5
    torch.testing.assert_close(got.double(), ref * 0.5, rtol=2 ** -8, atol=1e-6)


# hidden sizes at the edges of the one-, two- and four-chunk forms and the scalar form (no multiple of 8); rows below, at and
# beyond one per block
@pytest.mark.parametrize("rows,H", [(1, 8), (297, 2048), (296, 2056), (593, 4096), (40, 4104), (700, 8192), (33, 100)])
def test_rmsnorm_backward_edges(rows, H):
    from parallelkernelbench_b200.ops import rmsnorm_bwd

    x = torch.randn(rows, H, device="cuda", generator=_gen(H)).to(torch.bfloat16)
    dy = torch.randn(rows, H, device="cuda", generator=_gen(H + 1)).to(torch.bfloat16)
    g = (1 + 0.2 * torch.randn(H, device="cuda", generator=_gen(H + 2))).to(torch.bfloat16)
    dx, dg = rmsnorm_bwd(x, g, dy, 1e-5)
    xd, gd = x.double().requires_grad_(), g.double().requires_grad_()
    (xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5) * gd).backward(dy.double())
    scale = float(xd.grad.abs().max())
    torch.testing.assert_close(dx.double(), xd.grad, rtol=2 ** -8, atol=scale * 1e-5)      # one bf16 rounding
    torch.testing.assert_close(dg.double(), gd.grad, rtol=1e-5, atol=1e-5 * rows ** 0.5 * 4)   # fp32 sums over the rows


# counts around the four elements of an access, more than one sweep of the grid, and tensors off the 16-byte boundary (scalar form)
@pytest.mark.parametrize("n", [1, 3, 4, 7, 4099, 148 * 16 * 256 * 8 + 5])
@pytest.mark.parametrize("offset", [0, 1])
def test_adam_vector_and_scalar_forms(n, offset):
    from parallelkernelbench_b200.ops import adam_step

    mk = lambda s: torch.randn(n + offset, device="cuda", generator=_gen(s))[offset:]      # noqa: E731
    p, m, v, g = mk(1), mk(2) * 0.1, mk(3).abs() * 0.01, mk(4).to(torch.bfloat16)
    pb = torch.empty(n + offset, device="cuda", dtype=torch.bfloat16)[offset:]
    pd, gd = p.double(), g.double() * 0.5
    md, vd = 0.9 * m.double() + 0.1 * gd, 0.95 * v.double() + 0.05 * gd * gd
    step = 3
    want = pd * (1 - 1e-3 * 0.1) - 1e-3 * (md / (1 - 0.9 ** step)) / ((vd / (1 - 0.95 ** step)).sqrt() + 1e-8)
    adam_step(p, m, v, g, lr=1e-3, beta1=0.9, beta2=0.95, eps=1e-8, step=step, weight_decay=0.1, grad_scale=0.5, p_bf16=pb)
    torch.testing.assert_close(m.double(), md, rtol=1e-5, atol=1e-7)
    torch.testing.assert_close(v.double(), vd, rtol=1e-5, atol=1e-8)
    torch.testing.assert_close(p.double(), want, rtol=1e-6, atol=1e-6)
    assert torch.equal(pb, p.to(torch.bfloat16))

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
    # ex2.approx is within 2 ulp (2^-22), its argument d within |d| * 2^-23 of exact for a term exp(d) <= 1; a thread adds up to 98
    # terms in fp32 (half an ulp each), then the lanes and warps another 21
    torch.testing.assert_close(st[:, 1], ref, rtol=1e-5, atol=0)
    inside = ((tgt - 7) >= 0) & ((tgt - 7) < vocab)
    want = torch.where(inside, xd.gather(1, (tgt - 7).clamp(0, vocab - 1)[:, None])[:, 0], torch.zeros(rows, device="cuda", dtype=torch.float64))
    assert torch.equal(st[:, 2], want)


# a warp per row: up to two of its passes (bf16 2048, fp32 1024, scalar 256 elements) at any number of rows, up to eight where the rows
# fill the GPU; one element more; more rows than the grid takes at a time
@pytest.mark.parametrize("rows,vocab,dtype", [(7, 2048, torch.bfloat16), (7, 2056, torch.bfloat16), (2400, 8192, torch.bfloat16), (2400, 8200, torch.bfloat16),
                                              (5, 1024, torch.float32), (2400, 4096, torch.float32), (2400, 1023, torch.bfloat16), (2400, 1025, torch.bfloat16),
                                              (3, 255, torch.float32), (9999, 24, torch.bfloat16)])
def test_ce_stats_of_short_rows(rows, vocab, dtype):
    from parallelkernelbench_b200.ops import ce_local_stats

    x = (torch.randn(rows, vocab, device="cuda", generator=_gen(rows)) * 5).to(dtype)
    x[1] = float("-inf")
    x[2, :-1] = float("-inf")
    tgt = torch.randint(0, vocab, (rows,), device="cuda", generator=_gen(1))
    st = ce_local_stats(x, tgt, 0).double()
    xd = x.double()
    mx = xd.max(-1).values
    assert torch.equal(st[:, 0], mx) and torch.equal(st[:, 2], xd.gather(1, tgt[:, None])[:, 0])
    ref = torch.exp(xd - mx[:, None].clamp(min=-1e30)).sum(-1)
    # as above, with up to 256 terms per thread (half an ulp each, and they do not all fall to the same side)
    torch.testing.assert_close(st[:, 1], ref, rtol=1e-5, atol=0)


@pytest.mark.parametrize("vocab,dtype", [(1001, torch.float32), (4096, torch.float32), (4096, torch.bfloat16)])
def test_ce_stats_of_large_logits(vocab, dtype):
    """Large maxima: the exponent is the difference from the maximum, whose rounding must not scale with the maximum itself."""
    from parallelkernelbench_b200.ops import ce_local_stats

    top = torch.tensor([80.3, 300.7, 400.9, 511.3, 777.1, -650.9], device="cuda")
    x = torch.randn(6, vocab, device="cuda", generator=_gen(3)) + top[:, None] - 4
    x[::2] -= 200                                        # every other row: one peak, the rest far below it
    x[:, 17] = top + 4
    x = x.to(dtype)
    st = ce_local_stats(x, torch.zeros(6, dtype=torch.int64, device="cuda"), 0).double()
    ref = torch.exp(x.double() - x.double().max(-1, keepdim=True).values).sum(-1)
    # 2^-22 of the exponential, |d| exp(d) 2^-23 of its argument, half an ulp for each of at most 32 + 21 additions
    torch.testing.assert_close(st[:, 1], ref, rtol=4e-6, atol=0)


# columns: one load, the end of a block's 8192 columns, one load more
@pytest.mark.parametrize("rows,vocab", [(1, 8), (3, 8192), (3, 8200), (130, 1000), (5, 8184), (3000, 64)])
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


# hidden sizes at the edges of the one-, two- and four-chunk forms, of the forms with several rows per block and of the scalar form
# (no multiple of 8); rows below, at and beyond one step of the grid, and of a single block
@pytest.mark.parametrize("rows,H", [(1, 8), (297, 2048), (296, 2056), (593, 4096), (40, 4104), (700, 8192), (33, 100), (2369, 256), (8, 256), (9, 248),
                                    (1185, 512), (4, 264), (2000, 520), (593, 1024), (2, 1000), (3, 1032), (4, 8192), (5, 4096), (32, 64), (33, 64)])
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


@pytest.mark.parametrize("moved", ["x", "dy", "gamma"])
def test_rmsnorm_backward_of_tensors_off_the_16_byte_boundary(moved):
    from parallelkernelbench_b200.ops import rmsnorm_bwd

    rows, H = 37, 256
    t = {"x": torch.randn(rows, H, device="cuda", generator=_gen(1)).to(torch.bfloat16), "dy": torch.randn(rows, H, device="cuda", generator=_gen(2)).to(torch.bfloat16),
         "gamma": torch.randn(H, device="cuda", generator=_gen(3)).to(torch.bfloat16)}
    dx, dg = rmsnorm_bwd(t["x"], t["gamma"], t["dy"], 1e-5)
    off = torch.empty(t[moved].numel() + 1, device="cuda", dtype=torch.bfloat16)[1:].view(t[moved].shape).copy_(t[moved])
    assert off.is_contiguous() and off.data_ptr() % 16 == 2
    t[moved] = off
    dx2, dg2 = rmsnorm_bwd(t["x"], t["gamma"], t["dy"], 1e-5)
    # fp32 sums in another order: one step of bf16, and the bound of the gain's gradient above
    torch.testing.assert_close(dx2.float(), dx.float(), rtol=2 ** -7, atol=1e-5)
    torch.testing.assert_close(dg2, dg, rtol=1e-5, atol=1e-5 * rows ** 0.5 * 4)


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


# columns at the edges of the one-, two- and four-chunk forms
@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 2048), (5, 2056), (5, 4096), (2, 4104), (1300, 8192)])
def test_add_rmsnorm_equals_the_separate_passes(rows, cols):
    import ctypes

    from parallelkernelbench_b200 import _native as nv
    from parallelkernelbench_b200.ops import rmsnorm

    x, y = (torch.randn(rows, cols, device="cuda", generator=_gen(s)).to(torch.bfloat16) for s in (1, 2))
    g = torch.randn(cols, device="cuda", generator=_gen(3)).to(torch.bfloat16)
    total, out = torch.empty_like(x), torch.empty_like(x)
    nv.check(nv.cuda_lib().pkb_add_rmsnorm_bf16(nv.ptr(x), nv.ptr(y), nv.ptr(g), nv.ptr(total), nv.ptr(out), rows, cols,
                                                ctypes.c_float(1e-5), nv.current_stream()))
    assert torch.equal(total, x + y)
    # the same sum of squares in the same order of threads; the order inside a thread may differ: one ulp of bf16
    torch.testing.assert_close(out.float(), rmsnorm(x + y, g, 1e-5).float(), rtol=2 ** -7, atol=1e-6)


@pytest.mark.parametrize("tokens,hq,hkv,d", [(1, 1, 1, 64), (37, 4, 2, 128), (130, 8, 8, 64)])
def test_qkv_rope_split_and_merge(tokens, hq, hkv, d):
    from parallelkernelbench_b200 import _native as nv
    from parallelkernelbench_b200.ops import rope

    lib, st = nv.cuda_lib(), nv.current_stream()
    qkv = torch.randn(tokens, (hq + 2 * hkv) * d, device="cuda", generator=_gen(1)).to(torch.bfloat16)
    ang = torch.rand(tokens, d // 2, device="cuda", generator=_gen(2)) * 6.28
    cos, sin = torch.cat([ang.cos(), ang.cos()], -1).to(torch.bfloat16), torch.cat([ang.sin(), ang.sin()], -1).to(torch.bfloat16)
    q = torch.empty(tokens, hq, d, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.empty(tokens, hkv, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    nv.check(lib.pkb_qkv_rope_split(nv.ptr(qkv), nv.ptr(cos), nv.ptr(sin), nv.ptr(q), nv.ptr(k), nv.ptr(v), tokens, hq, hkv, d, st))
    parts = qkv.view(tokens, hq + 2 * hkv, d)
    assert torch.equal(q, rope(parts[:, :hq], cos, sin))
    assert torch.equal(k, rope(parts[:, hq:hq + hkv], cos, sin))
    assert torch.equal(v, parts[:, hq + hkv:])
    dq, dk, dv = (torch.randn(tokens, h, d, device="cuda", generator=_gen(h + 5)) for h in (hq, hkv, hkv))
    got = torch.empty_like(qkv)
    nv.check(lib.pkb_qkv_rope_merge(nv.ptr(dq), nv.ptr(dk), nv.ptr(dv), nv.ptr(cos), nv.ptr(sin), nv.ptr(got), tokens, hq, hkv, d, st))
    back = lambda g: rope(g, cos.float(), -sin.float())      # noqa: E731  fp32 rotation, rounded once below
    want = torch.cat([back(dq), back(dk), dv], 1).reshape(tokens, -1)
    torch.testing.assert_close(got.float(), want, rtol=2 ** -8, atol=1e-6)


# repeated tokens (first, last and middle positions), more positions than one mask word and than 32 of them, tokens repeated less,
# as often and more often than rows are in flight, the two ends of the table
@pytest.mark.parametrize("n,vocab,H", [(1, 5, 128), (33, 7, 256), (257, 1000, 640), (257, 3, 2176), (16, 2, 128), (1100, 2, 256), (16384, 5000, 128)])
def test_embedding_wire_format(n, vocab, H):
    from parallelkernelbench_b200.ops import fp8_dequantize_1x128, fp8_quantize_1x128
    from parallelkernelbench_b200.ops.decoder import embed_fp8, embed_grad_fp8

    table = torch.randn(vocab, H, device="cuda", generator=_gen(1))
    q, s = fp8_quantize_1x128(table)
    tok = torch.randint(0, vocab, (n,), device="cuda", generator=_gen(2))
    tok[0] = vocab - 1
    if n > 2:
        tok[1], tok[-1] = 0, vocab - 1 if n == 257 else 0
    x = embed_fp8(q.view(-1), s.view(-1), tok, vocab, H)
    assert torch.equal(x, fp8_dequantize_1x128(q, s)[tok])
    dx = torch.randn(n, H, device="cuda", generator=_gen(3)).to(torch.bfloat16)
    padded = vocab * H + 256
    gq, gs = embed_grad_fp8(dx, tok, vocab, H, padded)
    dense = torch.zeros(vocab, H)
    for i, row in zip(tok.tolist(), dx.float().cpu()):    # fp32 sums in position order
        dense[i] += row
    dense = dense.cuda()
    wq, ws = fp8_quantize_1x128(torch.nn.functional.pad(dense.to(torch.bfloat16).reshape(-1), (0, 256)).view(-1, 128))
    assert torch.equal(gq, wq.view(-1)) and torch.equal(gs, ws.view(-1))


@pytest.mark.parametrize("bad", [-1, 7, 1 << 40])
def test_tokens_outside_the_table_are_reported(bad):
    from parallelkernelbench_b200 import _native as nv
    from parallelkernelbench_b200.ops import fp8_quantize_1x128
    from parallelkernelbench_b200.ops.decoder import embed_fp8, embed_grad_fp8

    vocab, H = 7, 256
    q, s = fp8_quantize_1x128(torch.randn(vocab, H, device="cuda", generator=_gen(1)))
    tok = torch.tensor([0, bad, 6], device="cuda")
    x = embed_fp8(q.view(-1), s.view(-1), tok, vocab, H)
    with pytest.raises(nv.KernelStatusError, match="BAD_ARGUMENT.*tile=1"):
        nv.raise_on_status()
    assert (x[1] == 0).all() and (x[0] != 0).any()
    embed_grad_fp8(x, tok, vocab, H, vocab * H)
    with pytest.raises(nv.KernelStatusError, match="BAD_ARGUMENT.*tile=1"):
        nv.raise_on_status()


def test_a_step_on_a_token_outside_the_vocabulary_is_reported():
    from parallelkernelbench_b200 import _native as nv
    from parallelkernelbench_b200.models.llama import FSDPLlama, LlamaConfig
    from parallelkernelbench_b200.parallel import init_context

    ctx = init_context()
    try:
        m = FSDPLlama(ctx, LlamaConfig(layers=1, hidden=256, ffn=256, heads=2, kv_heads=1, vocab=512, seq=64))
        tok = torch.arange(64, device="cuda")
        m.step(tok, tok)
        m.step(tok, tok)
        bad = tok.clone()
        bad[9] = 512
        m.step(bad, tok)
        torch.cuda.synchronize()
        with pytest.raises(nv.KernelStatusError, match="BAD_ARGUMENT"):
            m.step(tok, tok)
        assert m.steps == 3
        m.step(tok, tok)
    finally:
        ctx.finalize()


@pytest.mark.parametrize("rows,W", [(1, 1), (1025, 3)])
def test_ce_loss_of_several_shards(rows, W):
    from parallelkernelbench_b200.ops.decoder import ce_loss

    lg = torch.randn(W, rows, 50, device="cuda", generator=_gen(1)) * 5
    mx = lg.max(-1).values
    st = torch.stack([mx, torch.exp(lg - mx[..., None]).sum(-1), torch.zeros_like(mx)], -1)
    st[0, :, 2] = lg[0, :, 7]
    loss, lse = ce_loss(st.contiguous())
    ref = torch.logsumexp(lg.double().permute(1, 0, 2).reshape(rows, -1), -1)
    torch.testing.assert_close(lse.double(), ref, rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(loss.double(), (ref - lg[0, :, 7].double()).mean(), rtol=1e-5, atol=1e-5)


# below and above the row count at which the forward GEMMs change form; a ragged number of tokens; both head dimensions
@pytest.mark.parametrize("S,H,Fn,hq,hkv,d", [(65, 256, 384, 4, 2, 64), (700, 512, 640, 4, 4, 128)])
def test_decoder_layer_against_autograd(S, H, Fn, hq, hkv, d):
    from parallelkernelbench_b200.models.llama import LlamaConfig, layer_forward, rope_tables, split_layer_params
    from parallelkernelbench_b200.ops.decoder import DecoderLayer

    cfg = LlamaConfig(layers=1, hidden=H, ffn=Fn, heads=hq, kv_heads=hkv, vocab=64, seq=S)
    assert cfg.head_dim == d
    flat = torch.randn(cfg.layer_numel(), device="cuda", generator=_gen(1)) * 0.05
    flat[-2 * H:] = 1 + 0.1 * flat[-2 * H:]
    flat = flat.to(torch.bfloat16)
    x, dout = (torch.randn(S, H, device="cuda", generator=_gen(s)).to(torch.bfloat16) for s in (2, 3))
    cos, sin = rope_tables(cfg, "cuda")
    L = DecoderLayer(S, H, Fn, hq, hkv, d, cfg.eps, d ** -0.5)
    scratch = torch.empty(max(L.fwd_scratch_bytes, L.bwd_scratch_bytes), dtype=torch.uint8, device="cuda")
    out, saved = L.forward(x, flat, cos, sin, scratch)
    dflat = torch.full_like(flat, float("nan"))
    dx = L.backward(x, flat, cos, sin, saved, dout, dflat, scratch)
    xr, fr = x.double().requires_grad_(), flat.double().requires_grad_()
    with torch.nn.attention.sdpa_kernel(torch.nn.attention.SDPBackend.MATH):
        ref = layer_forward(cfg, split_layer_params(cfg, fr), xr, cos.double(), sin.double())
        ref.backward(dout.double())
    # every intermediate tensor is rounded to bf16 (2^-9 each); a dozen of them lie between input and result
    for got, want in ((out, ref.detach()), (dx, xr.grad), (dflat, fr.grad)):
        assert torch.isfinite(got).all()
        assert float((got.double() - want).norm() / want.norm()) < 1.5e-2


def test_layer_forward_on_the_native_layer():
    """Both implementations behind the one entry point, with gradients to the separate parameters."""
    from parallelkernelbench_b200.models.llama import LlamaConfig, layer_forward, rope_tables, split_layer_params

    cfg = LlamaConfig(layers=1, hidden=256, ffn=384, heads=4, kv_heads=2, vocab=64, seq=70)
    flat = torch.randn(cfg.layer_numel(), device="cuda", generator=_gen(1)) * 0.05
    flat[-512:] = 1 + flat[-512:]
    x, dout = (torch.randn(70, 256, device="cuda", generator=_gen(s)).to(torch.bfloat16) for s in (2, 3))
    cos, sin = rope_tables(cfg, "cuda")
    res = []
    for impl, dtype in (("ours", torch.bfloat16), ("torch", torch.float64)):
        p = {k: v.detach().clone().requires_grad_() for k, v in split_layer_params(cfg, flat.to(torch.bfloat16).to(dtype)).items()}
        xi = x.detach().to(dtype).requires_grad_()
        with torch.nn.attention.sdpa_kernel(torch.nn.attention.SDPBackend.MATH):
            out = layer_forward(cfg, p, xi, cos.to(dtype), sin.to(dtype), impl)
            out.backward(dout.to(dtype))
        res.append([out.detach(), xi.grad, *(p[k].grad for k in p)])
    for got, want in zip(*res):
        assert got.shape == want.shape
        assert float((got.double() - want).norm() / want.norm()) < 1.5e-2      # as for the layer itself

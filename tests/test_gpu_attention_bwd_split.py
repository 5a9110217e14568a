"""Attention backward whose KV tiles are shared by several CTAs, and what it writes where no query looks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,sq,skv,hq,hkv,D,causal", [(1, 130, 130, 8, 1, 64, True), (2, 1000, 1000, 4, 1, 128, True), (1, 64, 700, 2, 2, 128, False),
                                                      (1, 2000, 129, 6, 3, 64, False), (1, 100, 900, 1, 1, 64, True), (1, 300, 2000, 16, 16, 128, True),
                                                      (4, 257, 257, 16, 8, 128, True)])
def test_attention_backward_shared_between_ctas(B, sq, skv, hq, hkv, D, causal):
    """Every row of dK / dV is written by one CTA or another: stale values in the buffers would show, they are filled with NaN first."""
    from parallelkernelbench_b200.ops.attention import flash_attn_bwd, flash_attn_fwd
    from parallelkernelbench_b200.refs.attention import attention_bwd_positions_ref

    torch.manual_seed(5)
    q, dout = (torch.randn(B, sq, hq, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(B, skv, hkv, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    out, lse = flash_attn_fwd(q, k, v, causal=causal)
    dk_buf, dv_buf = (torch.full(k.shape, float("nan"), device="cuda") for _ in range(2))
    dq, dk, dv = flash_attn_bwd(q, k, v, out, lse, dout, causal=causal, dk_out=dk_buf, dv_out=dv_buf)
    q_pos, kv_pos = torch.arange(sq, device="cuda"), torch.arange(skv, device="cuda")
    for b in range(B):
        ref = attention_bwd_positions_ref(q[b], k[b], v[b], out[b], lse[b], dout[b], q_pos, kv_pos, causal, D ** -0.5)
        for name, got, r in zip(("dq", "dk", "dv"), (dq[b], dk[b], dv[b]), ref):
            err = (got - r).abs().max().item()
            assert err <= 2e-2 * max(r.abs().max().item(), 1.0), f"{name}: {err}"      # bf16 P and dS, as in test_gpu_attention


@pytest.mark.parametrize("splits", [False, True])
def test_attention_backward_zeroes_rows_outside_all_segments(splits):
    from parallelkernelbench_b200.ops.attention import flash_attn_bwd, flash_attn_fwd

    hq, hkv, D, C = (8, 1, 64, 128) if splits else (8, 8, 64, 2560)
    q = torch.randn(1, C, hq, D, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.randn(1, 3 * C, hkv, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    seg = [(C, 0, C)]                                                     # the middle third of the buffer
    out, lse = flash_attn_fwd(q, k, v, causal=True, kv_segments=seg)
    bufs = [torch.full(k.shape, float("nan"), device="cuda") for _ in range(2)]
    _, dk, dv = flash_attn_bwd(q, k, v, out, lse, torch.randn_like(q), causal=True, kv_segments=seg, dk_out=bufs[0], dv_out=bufs[1])
    for g in (dk, dv):
        assert (g[:, :C] == 0).all() and (g[:, 2 * C:] == 0).all() and torch.isfinite(g).all() and (g[:, C:2 * C] != 0).any()


def test_attention_backward_takes_an_output_off_the_16_byte_boundary():
    from parallelkernelbench_b200.ops.attention import flash_attn_bwd, flash_attn_fwd

    q, k, v, dout = (torch.randn(1, 200, 2, 64, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    out, lse = flash_attn_fwd(q, k, v, causal=True)
    moved = torch.empty(out.numel() + 1, device="cuda", dtype=torch.bfloat16)[1:].view(out.shape).copy_(out)
    assert moved.is_contiguous() and moved.data_ptr() % 16 == 2
    for a, b in zip(flash_attn_bwd(q, k, v, out, lse, dout, causal=True), flash_attn_bwd(q, k, v, moved, lse, dout, causal=True)):
        assert torch.equal(a, b)


def test_attention_backward_zeroes_uncovered_rows_beside_overlapping_segments():
    """Two segments over the same rows: their lengths add up to more than the buffer, and a third of it lies outside."""
    from parallelkernelbench_b200.ops.attention import flash_attn_bwd

    H, D, C = 8, 64, 1280                                                 # 320 tiles: one CTA each
    q, out, dout = (torch.randn(1, 2 * C, H, D, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    k, v = (torch.randn(1, 3 * C, H, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    lse = torch.full((1, H, 2 * C), 8.0, device="cuda")
    bufs = [torch.full(k.shape, float("nan"), device="cuda") for _ in range(2)]
    _, dk, dv = flash_attn_bwd(q, k, v, out, lse, dout, causal=False, kv_segments=[(C, 0, 2 * C), (C, 0, 2 * C)], dk_out=bufs[0], dv_out=bufs[1])
    for g in (dk, dv):
        assert (g[:, :C] == 0).all() and torch.isfinite(g).all() and (g[:, C:] != 0).any()


# walks shared by two, four and eight CTAs; tiles whose walk is shorter than the cluster; a last tile with few rows
@pytest.mark.parametrize("B,S,hq,hkv,D,causal", [(2, 1024, 8, 2, 128, True), (1, 1024, 2, 1, 128, True), (1, 700, 16, 4, 128, False), (1, 1500, 4, 1, 64, True),
                                                 (1, 1100, 8, 4, 64, True), (1, 129, 8, 1, 128, True)])
def test_attention_backward_repeats_dk_and_dv_bit_for_bit(B, S, hq, hkv, D, causal):
    """The partial sums of a shared tile are added in the order of the CTAs, not of their arrival. (dQ is summed in no fixed order.)"""
    from parallelkernelbench_b200.ops.attention import flash_attn_bwd, flash_attn_fwd

    g = torch.Generator(device="cuda").manual_seed(S)
    q, dout = (torch.randn(B, S, hq, D, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(B, S, hkv, D, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    out, lse = flash_attn_fwd(q, k, v, causal=causal)
    _, dk, dv = flash_attn_bwd(q, k, v, out, lse, dout, causal=causal)
    for _ in range(12):
        _, dk2, dv2 = flash_attn_bwd(q, k, v, out, lse, dout, causal=causal)
        assert torch.equal(dk, dk2) and torch.equal(dv, dv2)

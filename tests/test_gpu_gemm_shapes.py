"""The GEMM that shares a tile's K range between the CTAs of a cluster and the tile widths of the CTA-pair GEMM, at the sizes
where their rules switch and their edges lie.

Bound: the fp32 sum of K products of bf16 values is off by at most K * 2^-24 * sum|a||w| (here far less), a bf16 result by
another 2^-9 of its value; 2^-8 covers the value, K * 2^-24 * (|a| @ |w|) the sum."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check_gemm(y, a, w, bias=None, act="none"):
    ref = a.double() @ w.double().t()
    bound = a.shape[1] * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t()) + 1e-30
    if bias is not None:
        ref = ref + bias.double()
    if act == "silu":
        ref = torch.nn.functional.silu(ref)
        bound = bound * 1.1 + 1e-5 * ref.abs()        # |silu'| <= 1.1; the fast exponential of the epilogue
    if y.dtype == torch.bfloat16:
        bound = bound + 2.0 ** -8 * ref.abs()
    err = (y.double() - ref).abs()
    assert (err <= bound).all(), f"{(err - bound).max().item():.3g} beyond the bound"


# among them K just below and above the limit of 24 blocks, and tiles at and beyond one wave of clusters of 8 (15), 4 (33) and 2 (74)
@pytest.mark.parametrize("M,N,K", [(40, 1024, 1472), (40, 1024, 1480), (9, 1920, 2048), (64, 2048, 2048), (20, 4224, 1544), (20, 4232, 1544), (3, 9472, 1544),
                                    (3, 9480, 1544), (1, 264, 64), (16, 128, 4096), (17, 8192, 520), (33, 1024, 1032), (65, 136, 264),
                                    (48, 18944, 64), (2, 18952, 136), (31, 72, 16384), (64, 8200, 8)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_with_few_rows(M, N, K, out_dtype):
    from parallelkernelbench_b200.ops import gemm_bf16, gemm_bf16_kn

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16, generator=g)
    w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16, generator=g) * 0.05
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16, generator=g)
    buf = torch.full((M + 2, N + 8), 7.0, device="cuda", dtype=out_dtype)
    _check_gemm(gemm_bf16(a, w, out=buf[1:M + 1, :N]), a, w)
    assert (buf[0] == 7).all() and (buf[M + 1] == 7).all() and (buf[:, N:] == 7).all()
    _check_gemm(gemm_bf16(a, w, bias=bias, epilogue="silu", out_dtype=out_dtype), a, w, bias, "silu")
    _check_gemm(gemm_bf16_kn(a, w.t().contiguous(), out_dtype=out_dtype), a, w)
    first = gemm_bf16(a, w, out_dtype=out_dtype)
    assert all(torch.equal(first, gemm_bf16(a, w, out_dtype=out_dtype)) for _ in range(3))


@pytest.mark.parametrize("M,N,K", [(1333, 4104, 136), (1500, 4096, 72), (4104, 2944, 264), (2560, 1048, 520), (520, 5000, 64), (3000, 3000, 200)])
def test_pair_gemm_tile_widths_on_ragged_problems(M, N, K):
    from parallelkernelbench_b200.ops import gemm_bf16, gemm_bf16_kn, gemm_bf16_tn

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16, generator=g)
    w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16, generator=g) * 0.05
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16, generator=g)
    buf = torch.full((M + 2, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    _check_gemm(gemm_bf16(a, w, out=buf[1:M + 1, :N]), a, w)
    assert (buf[0] == 7).all() and (buf[M + 1] == 7).all() and (buf[:, N:] == 7).all()
    for dt in (torch.bfloat16, torch.float32):
        _check_gemm(gemm_bf16(a, w, bias=bias, out_dtype=dt), a, w, bias)
        _check_gemm(gemm_bf16_kn(a, w.t().contiguous(), out_dtype=dt), a, w)
        if M % 8 == 0:
            _check_gemm(gemm_bf16_tn(a.t().contiguous(), w.t().contiguous(), out_dtype=dt), a, w)

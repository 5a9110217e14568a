"""One decoder layer per native call (csrc/kernels/decoder.cu), and the embedding and loss ends of the decoder step.

``DecoderLayer`` issues all launches of a layer's forward or backward from C++: the host writes one descriptor per shape and
passes pointers. The backward writes the weight gradients into one flat buffer laid out like the parameters.
Reference ancestors: reference/47_fsdp_step_e2e.py, reference/17_rope_allgather.py, reference/18_tp_rms_norm.py,
reference/73_vocab_parallel_cross_entropy_loss.py.
"""
from __future__ import annotations

import ctypes

import torch

from .. import _native as nv


class _LayerDesc(ctypes.Structure):
    _fields_ = [(n, ctypes.c_int32) for n in ("tokens", "hidden", "ffn", "hq", "hkv", "head_dim")] + [("eps", ctypes.c_float), ("scale", ctypes.c_float)]


_P, _I, _LL, _F = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
_ARGS = {"pkb_decoder_layer_fwd": [_P] * 9, "pkb_decoder_layer_bwd": [_P] * 11, "pkb_embed_fp8": [_P] * 4 + [_I] * 3 + [_P],
         "pkb_embed_grad_fp8": [_P, _P, _I, _I, _I, _P, _P, _P], "pkb_ce_loss": [_P, _I, _I, _P, _P, _P]}
_fns: dict = {}


def _fn(name: str):
    f = _fns.get(name)
    if f is None:
        f = getattr(nv.cuda_lib(), name)
        f.argtypes = _ARGS[name]
        _fns[name] = f
    return f


class DecoderLayer:
    """Forward and backward of one layer shape; holds no tensors."""

    FWD_LAUNCHES, BWD_LAUNCHES = 10, 16

    def __init__(self, tokens: int, hidden: int, ffn: int, heads: int, kv_heads: int, head_dim: int, eps: float, scale: float):
        self.desc = _LayerDesc(tokens, hidden, ffn, heads, kv_heads, head_dim, eps, scale)
        sizes = [ctypes.c_longlong() for _ in range(3)]
        nv.check(nv.cuda_lib().pkb_decoder_layer_sizes(ctypes.byref(self.desc), *(ctypes.byref(s) for s in sizes)), "pkb_decoder_layer_sizes")
        self.saved_bytes, self.fwd_scratch_bytes, self.bwd_scratch_bytes = (s.value for s in sizes)
        self.ref = ctypes.byref(self.desc)

    def forward(self, x, flat, cos, sin, scratch):
        """``x`` bf16 [tokens, hidden], ``flat`` the bf16 parameters, ``scratch`` uint8. Returns ``(out, saved)``."""
        out = torch.empty_like(x)
        saved = torch.empty(self.saved_bytes, dtype=torch.uint8, device=x.device)
        nv.check(_fn("pkb_decoder_layer_fwd")(self.ref, x.data_ptr(), flat.data_ptr(), cos.data_ptr(), sin.data_ptr(), out.data_ptr(),
                                              saved.data_ptr(), scratch.data_ptr(), nv.raw_stream(x)), "pkb_decoder_layer_fwd")
        nv.count_launch(self.FWD_LAUNCHES)
        return out, saved

    def backward(self, x, flat, cos, sin, saved, dout, dflat, scratch):
        """Returns ``dx``; ``dflat`` (bf16, laid out like ``flat``) receives the parameter gradients."""
        dx = torch.empty_like(x)
        nv.check(_fn("pkb_decoder_layer_bwd")(self.ref, x.data_ptr(), flat.data_ptr(), cos.data_ptr(), sin.data_ptr(), saved.data_ptr(),
                                              dout.data_ptr(), dx.data_ptr(), dflat.data_ptr(), scratch.data_ptr(), nv.raw_stream(x)),
                 "pkb_decoder_layer_bwd")
        nv.count_launch(self.BWD_LAUNCHES)
        return dx


def embed_fp8(table: torch.Tensor, scales: torch.Tensor, tokens: torch.Tensor, vocab: int, hidden: int) -> torch.Tensor:
    """Rows ``tokens`` of an e4m3 table with 1x128 scales (flat buffers) as bf16 [n, hidden]; ``hidden % 16 == 0``. A token
    outside the table gives a zero row and records a status (``_native.raise_on_status``)."""
    n = tokens.numel()
    out = torch.empty((n, hidden), dtype=torch.bfloat16, device=table.device)
    nv.check(_fn("pkb_embed_fp8")(table.data_ptr(), scales.data_ptr(), tokens.data_ptr(), out.data_ptr(), n, vocab, hidden, nv.raw_stream(table)),
             "pkb_embed_fp8")
    nv.count_launch()
    return out


def embed_grad_fp8_supported(n: int, hidden: int) -> bool:
    return hidden % 128 == 0 and n <= nv.cuda_lib().pkb_embed_grad_max_tokens()


def embed_grad_fp8(dx: torch.Tensor, tokens: torch.Tensor, vocab: int, hidden: int, padded: int):
    """Gradient of :func:`embed_fp8` in the wire format of the gradient exchange: e4m3 bytes [padded] and fp32 scales
    [padded / 128] of the dense [vocab, hidden] gradient (bf16-rounded sums over a token's positions; zero rows have scale 1)."""
    dx = dx if dx.data_ptr() % 16 == 0 else dx.clone()
    q = torch.zeros(padded, dtype=torch.uint8, device=dx.device)
    s = torch.ones(padded // 128, dtype=torch.float32, device=dx.device)
    nv.check(_fn("pkb_embed_grad_fp8")(dx.data_ptr(), tokens.data_ptr(), tokens.numel(), vocab, hidden, q.data_ptr(), s.data_ptr(),
                                       nv.raw_stream(dx)), "pkb_embed_grad_fp8")
    nv.count_launch()
    return q, s


def ce_loss(stats_all: torch.Tensor):
    """``stats_all`` fp32 [W, rows, 3] (see ``ce_local_stats``) -> (mean loss, log-sum-exp per row), one launch."""
    W, rows, _ = stats_all.shape
    lse = torch.empty(rows, dtype=torch.float32, device=stats_all.device)
    loss = torch.empty((), dtype=torch.float32, device=stats_all.device)
    nv.check(_fn("pkb_ce_loss")(stats_all.data_ptr(), rows, W, lse.data_ptr(), loss.data_ptr(), nv.raw_stream(stats_all)), "pkb_ce_loss")
    nv.count_launch()
    return loss, lse

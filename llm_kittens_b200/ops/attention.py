"""Causal flash attention on packed QKV (``csrc/attention.cu``). Reference jobs:
llmc/attention.cuh:261-338, 481-604 and llmc/attention_gqa.cuh:415-572."""
from __future__ import annotations

import torch

from . import _native as N


import os

# "tc" = tcgen05/TMEM kernels (csrc/attention_tc.cu) where the shape allows, "warp" = warp-level MMA kernels
IMPL = os.environ.get("LLMK_ATTENTION", "tc")


def _tc_length(T: int) -> bool:
    """Whether the tcgen05 kernels take sequences of this length. They work on 128-row tiles; a ragged last tile costs them
    half a tile, which the warp-level kernels (64-row tiles) undercut in the backward pass only when it is most of the
    sequence: us at B7 T448 12 heads of 64 38 against 59, at B1 T320 32/8 heads 37 against 50 and with heads of 128 57 against
    91, but at B64 T192 12 heads 98 against 104 with 50 against 32 in front of it, and at B32 T64 24 against 17."""
    return T % 128 == 0 or (T % 64 == 0 and T > 256)


_SMS: dict[int, int] = {}


def _sms() -> int:
    dev = torch._C._cuda_getDevice()
    if dev not in _SMS:
        _SMS[dev] = int(N.lib().llmk_num_sms())
    return _SMS[dev]


def _tc_forward(B: int, T: int, NH: int, HS: int) -> bool:
    """Whether the forward of these sequences is faster on the tcgen05 kernels. Lengths that are multiples of 128 are, except
    for a few sequences of 128 or 256 with heads of 64, where a launch lasts as long as its longest tile and the warp-level
    kernel's 64-row tiles are shorter (B1 T128 12 heads 4.4 / 5.9, B2 T128 25 heads 4.6 / 6.0, B1 T256 12 heads 6.5 / 7.1, but B2 T256 25
    heads 6.9 / 7.2, B16 T128 32 heads 14.4 / 12.5).
    With a ragged last tile they are too, except for heads of 64 and the shortest such length, 320, while the warp-level launch
    is 1.2 waves of 64-row tiles (us, warp level / tcgen05, heads in all: 12 7.7 / 8.4, 24 7.5 / 8.6, 30 8.4 / 9.0, 34 8.9 / 9.0, but 36 9.6 /
    9.1, 48 9.8 / 9.3, 400 38 / 30; 448 4 heads 9.2 / 9.2, 12 9.8 / 9.7, 36 12.6 / 10.4; 576 12 heads 11.9 / 10.9; 1088 4 heads 20.5 / 15.7; heads of
    128: 320 4 heads 11.2 / 8.7, 64 17.5 / 12.9, 448 112 heads 40 / 23, 600 167 / 100)."""
    if not _tc_length(T):
        return False
    if T % 128 == 0:
        return HS != 64 or T > 256 or T // 128 * B * NH > _sms() // 2
    return HS != 64 or T > 320 or 5 * (T // 64) * B * NH > 6 * _sms()


def forward_is_tc(B: int, T: int, NH: int, HS: int) -> bool:
    """Whether :func:`attention_fwd` without ``impl`` runs on the tcgen05 kernels."""
    return IMPL == "tc" and _tc_forward(B, T, NH, HS)


def attention_fwd(qkv, B, T, NH, NKVH, HS, out=None, lse=None, impl=None):
    """``qkv``: [B, T, (NH+2*NKVH)*HS] -> ``out`` [B, T, NH*HS], ``lse`` [B, NH, T] fp32. ``impl`` "warp" / "tc" asks for the
    warp-level kernels / for the tcgen05 kernels wherever they take the length; both leave what either backward needs."""
    out = torch.empty(B, T, NH * HS, dtype=qkv.dtype, device=qkv.device) if out is None else out
    lse = torch.empty(B, NH, T, dtype=torch.float32, device=qkv.device) if lse is None else lse
    if _tc_length(T) if impl == "tc" else (impl or IMPL) == "tc" and _tc_forward(B, T, NH, HS):
        N.call("llmk_attention_fwd_tc", out, lse, qkv, B, T, NH, NKVH, HS, N.status_word())
    else:
        N.call("llmk_attention_fwd", out, lse, qkv, B, T, NH, NKVH, HS)
    return out, lse


def fused_rope_available(T: int) -> bool:
    """Whether the tcgen05 backward runs for this sequence length, i.e. whether RoPE can live in the QKV GEMM's epilogue
    and its backward in the output tiles of the attention backward kernels."""
    return IMPL == "tc" and _tc_length(T)


def attention_bwd_prep(dout, out, dvec, B, T, NH, HS) -> bool:
    """D = rowsum(dO * O) into ``dvec`` [B, NH, T], the bandwidth-shaped first pass of the tcgen05 backward. A caller that
    runs it itself (e.g. on a side stream, beside a GEMM) passes ``prep_done=True`` to :func:`attention_bwd`. Returns
    False (and does nothing) when the warp-level fallback will run, which computes D inside its own entry point."""
    if IMPL == "tc" and _tc_length(T):
        N.call("llmk_attention_bwd_prep", dvec, dout, out, B, T, NH, HS)
        return True
    return False


def attention_bwd(dout, qkv, out, lse, B, T, NH, NKVH, HS, dqkv=None, dvec=None, impl=None, rope=None, prep_done=False):
    """``rope`` ([T, HS/2, 2] table, tcgen05 path only): ``qkv`` holds rotated q / k and the dq / dk columns of ``dqkv``
    are returned as gradients of the un-rotated projections (the inverse rotation happens in the kernels' output tiles)."""
    dqkv = torch.empty_like(qkv) if dqkv is None else dqkv
    dvec = torch.empty(B, NH, T, dtype=torch.float32, device=qkv.device) if dvec is None else dvec
    if (impl or IMPL) == "tc" and _tc_length(T):
        if not prep_done:
            N.call("llmk_attention_bwd_prep", dvec, dout, out, B, T, NH, HS)
        if rope is not None:
            N.call("llmk_attention_bwd_tc_rope", dqkv, dvec, dout, qkv, lse, B, T, NH, NKVH, HS, N.status_word(), rope)
        else:
            N.call("llmk_attention_bwd_tc", dqkv, dvec, dout, qkv, lse, B, T, NH, NKVH, HS, N.status_word())
    elif rope is not None:
        raise N.NativeError("attention_bwd: the fused RoPE backward needs the tcgen05 path")
    else:
        N.call("llmk_attention_bwd", dqkv, dvec, dout, qkv, out, lse, B, T, NH, NKVH, HS)
    return dqkv

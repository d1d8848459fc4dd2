"""piecewise_attention: host side of the B200 kernels.

Mirrors src/flag_attn/piecewise.py:25-191: score(m, n) = q2.k2 when the
bottom-right-aligned distance (m + N - M) - n is at least `dist_threshold`,
else q1.k1; returns the output only; gradients for the five tensors.
"""
import math

import torch

from . import _C, _native
from .flash import use_one_pass_backward

__all__ = ["attention"]


class PiecewiseAttention(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q1, k1, q2, k2, v, w, causal, sm_scale):
        Dq1, Dk1, Dq2, Dk2, Dv = q1.shape[-1], k1.shape[-1], q2.shape[-1], k2.shape[-1], v.shape[-1]
        assert Dq1 == Dk1 == Dq2 == Dk2 == Dv
        assert Dk1 in {16, 32, 64, 128}
        assert q1.shape == q2.shape and k1.shape == k2.shape == v.shape
        assert q1.shape[1] == k1.shape[1], "piecewise attention has no grouped-query mode"
        assert q1.is_cuda, "inputs must be CUDA tensors"
        assert all(x.device == q1.device for x in (k1, q2, k2, v)), "inputs must share a device"
        assert q1.dtype == k1.dtype == q2.dtype == k2.dtype == v.dtype

        B, H, M, D = q1.shape
        N = k1.shape[2]
        if sm_scale is None:
            sm_scale = 1. / math.sqrt(D)
        q1, k1, q2, k2, v = (_C.kernel_ready(x) for x in (q1, k1, q2, k2, v))
        with _C.device_guard(q1.device):
            o = torch.empty(q1.shape, dtype=q1.dtype, device=q1.device)
            L = torch.empty((B, H, M), device=q1.device, dtype=torch.float32)
            st = _C.call("fa_piecewise_fwd")(
                _C.pack_shape(q1.dtype, B, H, H, M, N, D, causal, sm_scale), int(w),
                *[_C.pack4(x) for x in (q1, k1, q2, k2, v, o)], L.data_ptr(), _C.raw_stream(q1.device))
            _C.check(st, "fa_piecewise_fwd")

        ctx.save_for_backward(q1, k1, q2, k2, v, o, L)
        ctx.sm_scale = sm_scale
        ctx.causal = causal
        ctx.w = int(w)
        return o

    @staticmethod
    def backward(ctx, do):
        q1, k1, q2, k2, v, o, L = ctx.saved_tensors
        w, causal, sm_scale = ctx.w, ctx.causal, ctx.sm_scale
        B, H, M, D = q1.shape
        N = k1.shape[2]
        do = _C.kernel_ready(do)

        with _C.device_guard(q1.device):
            raw = _C.raw_stream(q1.device)
            packed = _C.pack_shape(q1.dtype, B, H, H, M, N, D, causal, sm_scale)
            delta = torch.empty_like(L)
            tdo = _C.pack4(do)
            _C.check(_C.call("fa_flash_bwd_delta")(packed, _C.pack4(o), tdo, delta.data_ptr(), raw), "fa_flash_bwd_delta")

            dk1 = torch.empty(k1.shape, dtype=k1.dtype, device=k1.device)
            dk2 = torch.empty(k2.shape, dtype=k2.dtype, device=k2.device)
            dv = torch.empty(v.shape, dtype=v.dtype, device=v.device)
            dq1 = torch.empty(q1.shape, dtype=q1.dtype, device=q1.device)
            dq2 = torch.empty(q2.shape, dtype=q2.dtype, device=q2.device)
            ins = (packed, w, *[_C.pack4(x) for x in (q1, k1, q2, k2, v)], tdo, L.data_ptr(), delta.data_ptr())
            tq1, tq2, tk1, tk2, tv = (_C.pack4(x) for x in (dq1, dq2, dk1, dk2, dv))
            ws_bytes = (_C.call("fa_piecewise_bwd_fused_workspace_bytes")(packed)
                        if use_one_pass_backward() else 0)
            if ws_bytes > 0:
                # one launch: every key block walks its near tiles, then its far tiles; dq1 / dq2
                # accumulate in two fp32 workspaces, dV in TMEM across both walks
                ws = torch.empty(ws_bytes, dtype=torch.uint8, device=q1.device)
                st = _C.call("fa_piecewise_bwd_fused")(*ins, tq1, tq2, tk1, tk2, tv, ws.data_ptr(), ws_bytes, raw)
                # a layout the one-pass kernel cannot map (a broadcast stride) goes to the pair below
                if st != _C.FA_ERR_UNSUPPORTED:
                    _C.check(st, "fa_piecewise_bwd_fused")
                    return dq1, dk1, dq2, dk2, dv, None, None, None
            _C.check(_C.call("fa_piecewise_bwd_dkdv")(*ins, tk1, tk2, tv, raw), "fa_piecewise_bwd_dkdv")
            _C.check(_C.call("fa_piecewise_bwd_dq")(*ins, tq1, tq2, raw), "fa_piecewise_bwd_dq")
        return dq1, dk1, dq2, dk2, dv, None, None, None


def attention(q1, k1, q2, k2, v, dist_threshold, causal=False, sm_scale=None):
    """Piecewise attention (for NLPE): the attention score of (q_i, k_j) is
    q1_i.k1_j when their distance is below `dist_threshold` and q2_i.k2_j
    otherwise.  All tensors are (batch, heads, seqlen, headdim); returns the
    output, shaped like q1."""
    if _native.usable(q1):
        o = _native.load().piecewise(q1, k1, q2, k2, v, dist_threshold, causal, sm_scale)
        if o is not None:
            return o
    return PiecewiseAttention.apply(q1, k1, q2, k2, v, dist_threshold, causal, sm_scale)

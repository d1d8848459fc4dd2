"""flash_attention: host side of the B200 kernels.

Mirrors the operator interface of the reference (src/flag_attn/flash.py:23-286):
same argument names, same return structure (the output alone, or the 5-tuple
when any return_* flag is set), same AssertionErrors on bad shapes, autograd
through q, k, v only.  The kernels run on the current CUDA stream of the
inputs' device.
"""
import functools
import math

import torch

from . import _C, _native
from .dropout import philox_cuda_seed_offset
from .paged import coarsen_partition, partition_workspace
from .split_kv import get_fwd_config as get_fwd_config_kv_split
from .split_kv import num_splits_herustic, _splitkv_forward

__all__ = ["attention", "set_backward_mode", "get_backward_mode", "backward_mode"]

# Which kernels compute the gradients:
#   "one_pass"   one kernel for dq, dk, dv (five matrix products per tile); dq is summed with fp32
#                reductions in global memory, so it is reproducible to fp32 rounding only;
#   "two_kernel" a dK/dV kernel and a dQ kernel without any global reduction or atomic (seven
#                products per tile), the split of the reference (src/flag_attn/flash.py:204-249):
#                every gradient is bitwise reproducible;
#   "auto"       (default) "two_kernel" while torch.are_deterministic_algorithms_enabled(),
#                else "one_pass".
_BACKWARD_MODES = ("auto", "one_pass", "two_kernel")
_backward_mode = "auto"


def set_backward_mode(mode):
    """Selects the backward kernels of flash_attention and piecewise_attention (see above);
    returns the previous mode."""
    global _backward_mode
    assert mode in _BACKWARD_MODES, f"mode must be one of {_BACKWARD_MODES}"
    previous, _backward_mode = _backward_mode, mode
    _native.set_backward_mode(_BACKWARD_MODES.index(mode))
    return previous


def get_backward_mode():
    return _backward_mode


class backward_mode:
    """`with backward_mode("two_kernel"): loss.backward()`"""

    def __init__(self, mode):
        assert mode in _BACKWARD_MODES, f"mode must be one of {_BACKWARD_MODES}"
        self.mode = mode

    def __enter__(self):
        self.previous = set_backward_mode(self.mode)
        return self

    def __exit__(self, *exc):
        set_backward_mode(self.previous)
        return False


def use_one_pass_backward():
    if _backward_mode == "auto":
        return not torch.are_deterministic_algorithms_enabled()
    return _backward_mode == "one_pass"


def get_fwd_config(B, H, M, N, D, causal):
    """Tile shape used by the one-pass forward kernel: (BLOCK_M, BLOCK_N, stages, warps).
    Kept for interface compatibility (src/flag_attn/flash.py:290-322); the tile
    shape is compiled into the kernels, so overriding this has no effect."""
    return (128, 64, 2, 6)


def get_bwd_config(B, H, M, N, D, causal):
    """Counterpart of src/flag_attn/flash.py:493-519, for the one-pass kernel; informational only."""
    return (128, 128, 2 if D == 128 else 3, 24)


def _forward(q, k, v, causal, sm_scale, dropout_p=0.0, seed=0, offset=0, keep=False):
    """(o, log-normaliser), and with `keep` the buffer of dropout decisions for the backward, or None where the kernels
    keep none."""
    B, H, M, D = q.shape
    N, Hk = k.shape[2], k.shape[1]
    o = torch.empty((B, H, M, D), dtype=q.dtype, device=q.device)
    L = torch.empty((B, H, M), device=q.device, dtype=torch.float32)
    shape = _C.pack_shape(q.dtype, B, H, Hk, M, N, D, causal, sm_scale, dropout_p, seed, offset)
    args = (shape, _C.pack4(q), _C.pack4(k), _C.pack4(v), _C.pack4(o), L.data_ptr())
    stream = _C.raw_stream(q.device)
    bits_bytes = _C.call("fa_flash_keep_bits_bytes")(shape) if keep else 0
    bits = None
    if bits_bytes:
        try:
            bits = torch.empty(bits_bytes, dtype=torch.uint8, device=q.device)
        except torch.OutOfMemoryError:   # the backward draws them again
            pass
    if bits is not None:
        st = _C.call("fa_flash_fwd_keep")(*args, bits.data_ptr(), bits_bytes, stream)
        if st != _C.FA_ERR_UNSUPPORTED:   # a layout for the kernels below
            _C.check(st, "fa_flash_fwd_keep")
            return o, L, bits
        del bits
    st = _C.call("fa_flash_fwd")(*args, stream)
    _C.check(st, "fa_flash_fwd")
    return (o, L, None) if keep else (o, L)


@functools.lru_cache(maxsize=1024)
def _few_rows_pay(B, H, M, N, D, causal, num_sms):
    """Whether a call that splits its keys is faster by clusters of CTAs than by the split-KV kernels."""
    return bool(_C.call("fa_flash_few_rows_pays")(_C.pack_shape(torch.float16, B, H, H, M, N, D, causal, 1.0), num_sms))


def _few_rows_forward(q, k, v, causal, sm_scale):
    """(o, log-normaliser) of a call that splits its keys, by clusters of CTAs; None for what only the split-KV kernels
    take."""
    B, H, M, D = q.shape
    N, Hk = k.shape[2], k.shape[1]
    o = torch.empty((B, H, M, D), dtype=q.dtype, device=q.device)
    L = torch.empty((B, H, M), device=q.device, dtype=torch.float32)
    st = _C.call("fa_flash_fwd_few_rows")(
        _C.pack_shape(q.dtype, B, H, Hk, M, N, D, causal, sm_scale), _C.pack4(q), _C.pack4(k), _C.pack4(v), _C.pack4(o),
        L.data_ptr(), _C.raw_stream(q.device))
    if st == _C.FA_ERR_UNSUPPORTED:
        return None
    _C.check(st, "fa_flash_fwd_few_rows")
    return o, L


def _identity_block_table(B, blocks_per_batch, id_stride, device):
    """(block_tables, context_lens) with block_tables[b, c] = b * id_stride + c: what FA_BLOCK_TABLE_IN_PLACE
    stands for, under which a (B, Hk, N, D) key tensor is a paged cache of 16-token blocks.  The kernel works
    the entries out itself; the tests hold it to this table."""
    tab = (torch.arange(B, device=device, dtype=torch.int32)[:, None] * id_stride +
           torch.arange(blocks_per_batch, device=device, dtype=torch.int32)[None, :]).contiguous()
    return tab, torch.full((B,), blocks_per_batch * 16, dtype=torch.int32, device=device)


# Elements of the attention matrix from which the forward keeps its dropout decisions for the backward.  On the GPU keeping
# is the faster at every size (4 M 55 us kept and 70 drawn, 16.8 M 110 and 140, forward and backward at D=64, p = 0.1, not
# causal), but it takes 5 to 8 us of host work, which bounds a call up to about 20 M, causal 40 M.  A call in a loop, us
# kept / drawn: 8.4 M 187 / 179, 16.8 M 183 / 182, 25 M 185 / 209, 33.6 M 192 / 217, 67 M 281 / 370; causal at D=128
# 16.8 M 186 / 182, 33.5 M 182 / 177, 67 M 207 / 263.  The line lies between the two crossings.
_KEEP_BITS_FROM = 1 << 25

_DECODE_MAX_ROWS = 64   # query rows (group x queries) per kv head the gather kernel is given


def _decode_covered(q, k, v, causal=False):
    """Decode-shaped forward (a few queries per head, at most _DECODE_MAX_ROWS rows per kv head)
    that the paged-decode kernels can run directly on k and v: the keys of a batch element are then
    16-token blocks that follow one another in memory."""
    B, H, M, D = q.shape
    N, Hk = k.shape[2], k.shape[1]
    if M < 1 or N % 16 != 0 or N == 0 or (H // Hk) * M > _DECODE_MAX_ROWS:
        return False
    if causal and M > 1 and N < M:
        return False      # rows that see no key at all: the tile kernels give them their zeros
    if k.stride() != v.stride() or k.stride(3) != 1 or k.data_ptr() % 16 or v.data_ptr() % 16:
        return False
    sb, sh, sl, _ = k.stride()
    # (one row broadcast over the length has stride 0: no block of it follows another)
    return sl > 0 and not (sl % 8 or sh % 8 or sb % (16 * sl))


def _decode_forward(q, k, v, sm_scale, causal=False):
    """o for a few queries per head through fa_paged_decode / fa_paged_reduce (an HBM-bound gather
    kernel that streams K and V once per 16 query rows of a kv head), instead of the split-KV tile
    kernels.  The M queries of a head go in as M consecutive "query heads" of its kv head."""
    B, H, M, D = q.shape
    Hk, N = k.shape[1], k.shape[2]
    BS = 16
    sb, sh, sl, _ = k.stride()
    num_sms = _C.sm_count(q.device)
    # Partitions of the key axis, long enough to amortise a CTA's pipeline fill and the reduction (one block a
    # row goes through the row's partitions): about one wave of CTAs, up to 4096 keys.  Every context is N long
    # here, so that the rule may count CTAs at the bound.  fp16, 2048 / 4096 / 8192 keys: B=32 H=32 N=8192 D=128
    # 619 / 625 / 654 us, B=8 H=32 N=32768 633 / 630 / 645, B=2 H=32 N=131072 D=64 336 / 333 / 345, B=2 H=16
    # N=131072 340 / 326 / 311; by the rule 1024 of N=8192 B=4 H=32 Hk=4 M=6 D=64 22.9 (2048: 28.4, 512: 27.2).
    partition_size = coarsen_partition(256, B * Hk, N, num_sms, 4096)
    if N <= partition_size:
        partition_size = 0   # one pass, no reduction kernel
    q2 = q.reshape(B, H * M, D)
    if q2.stride(-1) != 1 or q2.data_ptr() % 16 or q2.stride(0) % 8 or q2.stride(1) % 8:
        q2 = q2.contiguous()
    o = torch.empty((B, H, M, D), dtype=q.dtype, device=q.device)
    part_out = part_max = part_sum = 0
    if partition_size:
        P = (N + partition_size - 1) // partition_size
        ws, part_out, part_max, part_sum = partition_workspace(B * H * M, P, D, q.device)
    args = _C.PAGED_ARGS.pack(
        _C.dtype_code(q.dtype), B, H * M, Hk, D, BS, N, _C.FA_BLOCK_TABLE_IN_PLACE, partition_size, sm_scale,
        q2.data_ptr(), q2.stride(0), q2.stride(1), k.data_ptr(), v.data_ptr(),
        BS * sl, sh if Hk > 1 else 0, sl, 0, 0, sb // (BS * sl),
        o.data_ptr(), H * M * D, D, part_out, part_max, part_sum, M if (causal and M > 1) else 0)
    stream = _C.raw_stream(q.device)
    _C.check(_C.call("fa_paged_decode")(args, stream), "fa_paged_decode")
    if partition_size:
        _C.check(_C.call("fa_paged_reduce")(args, stream), "fa_paged_reduce")
    return o


def _total_attention(q, k, L, causal, sm_scale):
    B, H, M, D = q.shape
    N, Hk = k.shape[2], k.shape[1]
    tot = torch.empty((B, H, N), device=q.device, dtype=torch.float32)
    st = _C.call("fa_total_attention")(
        _C.pack_shape(q.dtype, B, H, Hk, M, N, D, causal, sm_scale), _C.pack4(q), _C.pack4(k), L.data_ptr(),
        tot.data_ptr(), _C.raw_stream(q.device))
    _C.check(st, "fa_total_attention")
    return tot


def _backward(q, k, v, o, L, do, causal, sm_scale, mark=None, dropout_p=0.0, seed=0, offset=0, bits=None):
    """Launches delta, dK/dV and dQ. `mark(name)`, when given, is called before the first launch
    and after each one (the benchmark records CUDA events there)."""
    B, H, M, D = q.shape
    N, Hk = k.shape[2], k.shape[1]
    do = _C.kernel_ready(do)
    with _C.device_guard(q.device):
        # dk / dv come out with Hk heads: the group sum is done in the kernel
        dk = torch.empty((B, Hk, N, D), dtype=k.dtype, device=q.device)
        dv = torch.empty((B, Hk, N, D), dtype=v.dtype, device=q.device)
        dq = torch.empty((B, H, M, D), dtype=q.dtype, device=q.device)
        shape, stream = (_C.pack_shape(q.dtype, B, H, Hk, M, N, D, causal, sm_scale, dropout_p, seed, offset),
                         _C.raw_stream(q.device))
        tq, tk, tv, to, tdo, tdq, tdk, tdv = (_C.pack4(x) for x in (q, k, v, o, do, dq, dk, dv))
        if mark is None and use_one_pass_backward():
            # everything in one call: one workspace, one trip through the binding
            ws_bytes = _C.call("fa_flash_bwd_workspace_bytes")(shape)
            if ws_bytes > 0:
                try:
                    ws = torch.empty(ws_bytes, dtype=torch.uint8, device=q.device)
                except torch.OutOfMemoryError:   # without room for shared walks, if that is less
                    least = _C.call("fa_flash_bwd_least_workspace_bytes")(shape)
                    if least >= ws_bytes:
                        raise
                    ws_bytes = least
                    ws = torch.empty(ws_bytes, dtype=torch.uint8, device=q.device)
                args = (shape, tq, tk, tv, to, tdo, L.data_ptr(), tdq, tdk, tdv)
                if bits is None:
                    st = _C.call("fa_flash_bwd")(*args, ws.data_ptr(), ws_bytes, stream)
                else:   # the forward kept its dropout decisions
                    st = _C.call("fa_flash_bwd_keep")(*args, bits.data_ptr(), bits.numel(), ws.data_ptr(), ws_bytes, stream)
                # a layout the one-pass kernel cannot map (a broadcast stride) goes to the pair below
                if st != _C.FA_ERR_UNSUPPORTED:
                    _C.check(st, "fa_flash_bwd")
                    return dq, dk, dv
                del ws
        # the parts one by one
        delta = torch.empty_like(L)
        if mark:
            mark("start")
        ws_bytes = (_C.call("fa_flash_bwd_fused_workspace_bytes")(shape) if mark and use_one_pass_backward() else 0)
        if ws_bytes > 0:
            # one pass over the score tiles; dq is accumulated in an fp32 workspace, which the
            # delta kernel fills with zeros on its way (two memory-bound passes in one launch)
            ws = torch.empty(ws_bytes, dtype=torch.uint8, device=q.device)
            st = _C.call("fa_flash_bwd_delta_zero")(shape, to, tdo, delta.data_ptr(), ws.data_ptr(), ws_bytes, stream)
            _C.check(st, "fa_flash_bwd_delta_zero")
        else:
            _C.check(_C.call("fa_flash_bwd_delta")(shape, to, tdo, delta.data_ptr(), stream), "fa_flash_bwd_delta")
        if mark:
            mark("delta")
        ins = (shape, tq, tk, tv, tdo, L.data_ptr(), delta.data_ptr())
        if ws_bytes > 0:
            st = 0
            for stage, name in ((2, "dkdvdq"), (4, "dq_convert")):
                st = _C.call("fa_flash_bwd_fused_stages")(*ins, tdq, tdk, tdv, ws.data_ptr(), ws_bytes, stage, stream)
                if st != 0:
                    break
                mark(name)
            # a layout the one-pass kernel cannot map (a broadcast stride) goes to the pair below
            if st != _C.FA_ERR_UNSUPPORTED:
                _C.check(st, "fa_flash_bwd_fused")
                return dq, dk, dv
        _C.check(_C.call("fa_flash_bwd_dkdv")(*ins, tdk, tdv, stream), "fa_flash_bwd_dkdv")
        if mark:
            mark("dkdv")
        _C.check(_C.call("fa_flash_bwd_dq")(*ins, tdq, stream), "fa_flash_bwd_dq")
        if mark:
            mark("dq")
    return dq, dk, dv


class FlashAttention(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, causal, sm_scale, dropout_p, return_log_normalizer,
                return_total_attention, return_seed_offset):
        Dq, Dk, Dv = q.shape[-1], k.shape[-1], v.shape[-1]
        assert Dq == Dk == Dv, "feature size of q, k, v should be equal"
        assert Dk in {16, 32, 64, 128}
        assert 0.0 <= dropout_p < 1.0, f"dropout_p={dropout_p}"
        assert q.is_cuda and k.is_cuda and v.is_cuda, "inputs must be CUDA tensors"
        assert q.dtype == k.dtype == v.dtype

        B, H, M, D = q.shape
        N = k.shape[2]
        Hk, Hv = k.shape[1], v.shape[1]
        assert Hk == Hv, "num of heads in k and v should be equal"
        assert H % Hk == 0, "number of heads in q must be a multiple of that in k & v"

        if sm_scale is None:
            sm_scale = 1. / math.sqrt(D)

        q, k, v = _C.kernel_ready(q), _C.kernel_ready(k), _C.kernel_ready(v)

        has_extra_return = True in (return_log_normalizer, return_total_attention, return_seed_offset)
        if (M <= 16 and dropout_p == 0 and not has_extra_return and not any(ctx.needs_input_grad[:3])
                and _decode_covered(q, k, v, causal)):
            # decode step without gradients: nothing but o is needed.  One query always goes to the
            # gather kernel, which streams K and V once; a few queries go there when the reference
            # would split the keys (src/flag_attn/flash.py:59-61), i.e. when the tile grid alone
            # would leave most of the GPU idle.
            with _C.device_guard(q.device):
                take = M == 1
                if not take:
                    cfg = get_fwd_config_kv_split(B, H, M, N, D, causal)
                    take = num_splits_herustic(B, H, M, N, cfg[0], cfg[1], _C.sm_count(q.device), 128) > 1
                if take:
                    return _decode_forward(q, k, v, sm_scale, causal)

        with _C.device_guard(q.device):
            # dropout: one Philox counter per element of the (B, H, M, N) attention matrix
            is_dropout = dropout_p > 0
            if is_dropout:
                seed, offset = philox_cuda_seed_offset(B * H * M * N, q.device)
            else:
                seed, offset = 0, 0

            bits = None
            cfg = get_fwd_config_kv_split(B, H, M, N, D, causal)
            S = num_splits_herustic(B, H, M, N, cfg[0], cfg[1], _C.sm_count(q.device), 128)
            if S > 1:
                assert not is_dropout, "Cannot apply dropout with splitkv."
                pays = _few_rows_pay(B, H, M, N, D, bool(causal), _C.sm_count(q.device))
                o, L = ((pays and _few_rows_forward(q, k, v, causal, sm_scale))
                        or _splitkv_forward(q, k, v, causal, sm_scale, S))
            elif (is_dropout and B * H * M * N >= _KEEP_BITS_FROM and any(ctx.needs_input_grad[:3])
                  and use_one_pass_backward()):
                o, L, bits = _forward(q, k, v, causal, sm_scale, dropout_p, seed, offset, True)
            else:
                o, L = _forward(q, k, v, causal, sm_scale, dropout_p, seed, offset)
            tot_attn = None
            if return_total_attention:
                tot_attn = _total_attention(q, k, L, causal, sm_scale)

        ctx.save_for_backward(q, k, v, o, L, *([] if bits is None else [bits]))
        ctx.sm_scale = sm_scale
        ctx.causal = causal
        ctx.dropout_p = dropout_p
        ctx.seed = seed
        ctx.offset = offset

        if has_extra_return:
            return (o, L if return_log_normalizer else None, tot_attn,
                    seed if is_dropout and return_seed_offset else None,
                    offset if is_dropout and return_seed_offset else None)
        return o

    @staticmethod
    def backward(ctx, do, *ignored):
        q, k, v, o, L, *bits = ctx.saved_tensors
        dq, dk, dv = _backward(q, k, v, o, L, do, ctx.causal, ctx.sm_scale, None, ctx.dropout_p,
                               ctx.seed, ctx.offset, *bits)
        return dq, dk, dv, None, None, None, None, None, None


def attention(q, k, v, causal=False, sm_scale=None, dropout_p=0.0,
              return_log_normalizer=False, return_total_attention=False, return_seed_offset=False):
    """FlashAttention forward/backward on B200.

    Arguments:
        q: (batch, heads_q, seqlen_q, headdim); k, v: (batch, heads_k, seqlen_k, headdim),
           fp16 or bf16 CUDA tensors, heads_q a multiple of heads_k, headdim in {16,32,64,128}.
        causal: bottom-right aligned causal mask.
        sm_scale: softmax scale, default 1/sqrt(headdim).
        dropout_p: dropout probability on the attention weights.
        return_log_normalizer / return_total_attention / return_seed_offset: when any is set,
           returns (out, log_normalizer | None, total_attention | None, seed | None, offset | None);
           seed and offset are the Philox seed and starting offset used by dropout (None without).

    Returns out, shape of q; log_normalizer (batch, heads_q, seqlen_q) fp32;
    total_attention (batch, heads_q, seqlen_k) fp32.
    """
    if (dropout_p == 0 and not (return_log_normalizer or return_total_attention or return_seed_offset)
            and _native.usable(q)):
        native = _native.load()
        o = native.flash(q, k, v, causal, sm_scale)
        if o is None:   # a view that needs a copy, or keys for the split-KV kernels; else the form below
            o = native.flash_rest(q, k, v, causal, sm_scale)
        if o is False:   # 2 to 16 queries a head, for the decode kernels
            return _decode_forward(_C.kernel_ready(q), _C.kernel_ready(k), _C.kernel_ready(v),
                                   1. / math.sqrt(q.shape[-1]) if sm_scale is None else sm_scale, causal)
        if o is not None:
            return o
    return FlashAttention.apply(q, k, v, causal, sm_scale, dropout_p, return_log_normalizer,
                                return_total_attention, return_seed_offset)

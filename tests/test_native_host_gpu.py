"""The native form of the operators' usual calls against the Python form: the same bits, the same gradients, the same
errors; and what it must leave to the Python form."""
import pytest
import torch

import flagattention_b200 as fa
from flagattention_b200 import _native, flash, paged, piecewise, rotary
from helpers import make_qkv

pytestmark = pytest.mark.gpu


@pytest.fixture
def python_form(monkeypatch):
    """Calls `f` through the Python form."""
    def run(f):
        with monkeypatch.context() as m:
            m.setattr(_native, "usable", lambda x: False)
            return f()
    return run


def _same(a, b):
    for x, y in zip(a, b):
        assert x.shape == y.shape and x.stride() == y.stride() and x.dtype == y.dtype and x.device == y.device
        assert torch.equal(x, y)


@pytest.mark.parametrize("B,H,Hk,M,N,D,causal,layout", [
    (2, 8, 8, 256, 256, 64, True, "BHTD"), (2, 16, 4, 300, 333, 128, True, "BTHD"), (4, 8, 2, 160, 160, 32, False, "BHTD"),
    (1, 8, 8, 1, 4096, 128, False, "BHTD"), (2, 8, 2, 1, 1024, 64, True, "BTHD"), (1, 4, 1, 4, 8192, 128, True, "BHTD"),
    (3, 2, 2, 1, 1000, 64, False, "BHTD"), (1, 2, 2, 40, 40, 64, True, "BHTD")])
def test_flash_calls(python_form, B, H, Hk, M, N, D, causal, layout):
    q, k, v, do = make_qkv(B, H, Hk, M, N, D, torch.bfloat16, "cuda", layout=layout, seed=N)
    call = lambda *a, **kw: fa.flash_attention(q, k, v, *a, **kw)
    _same([call(causal)], [python_form(lambda: call(causal))])
    _same([call(causal, 0.3)], [python_form(lambda: call(causal, 0.3))])
    for x in (q, k, v):
        x.requires_grad_()
    grads = lambda: (lambda o: (o,) + torch.autograd.grad(o, (q, k, v), do))(call(causal))
    with flash.backward_mode("two_kernel"):   # bitwise reproducible
        _same(grads(), python_form(grads))
    got, want = grads(), python_form(grads)
    _same(got[2:], want[2:])   # dk, dv; dq is summed in any order: one rounding to 16 bits apart at most
    _same(got[:1], want[:1])
    assert (got[1].float() - want[1].float()).abs().max() <= 2 ** -7 * want[1].float().abs().max()
    with torch.no_grad():
        _same([call(causal)], [python_form(lambda: call(causal))])


@pytest.mark.parametrize("B,H,Hk,M,N,D,causal", [
    (1, 8, 8, 4, 1024, 64, True), (2, 8, 2, 16, 2048, 128, True), (2, 8, 2, 3, 512, 32, False), (1, 4, 4, 16, 16, 64, True),
    (1, 8, 8, 1, 1000, 64, False), (1, 4, 1, 5, 1001, 128, True), (1, 8, 8, 20, 1024, 64, True), (1, 2, 1, 31, 700, 128, True),
    (1, 4, 4, 40, 300, 32, True), (2, 2, 2, 20, 10, 64, True), (1, 4, 2, 60, 90, 16, False)])
@pytest.mark.parametrize("layout", ["BHTD", "BTHD"])
def test_few_queries_and_split_keys(python_form, B, H, Hk, M, N, D, causal, layout):
    """Decoding of several queries, and calls that the split-KV kernels take."""
    q, k, v, do = make_qkv(B, H, Hk, M, N, D, torch.bfloat16, "cuda", layout=layout, seed=N + M)
    call = lambda: fa.flash_attention(q, k, v, causal)
    assert any(f(q, k, v, causal, None) is not None for f in (_native.load().flash, _native.load().flash_rest))
    _same([call()], [python_form(call)])
    for x in (q, k, v):
        x.requires_grad_()
    with flash.backward_mode("two_kernel"):
        grads = lambda: (lambda o: (o,) + torch.autograd.grad(o, (q, k, v), do))(call())
        _same(grads(), python_form(grads))


def test_views_that_need_a_copy(python_form):
    gen = torch.Generator().manual_seed(4)
    mk = lambda *s: torch.randn(s, generator=gen).half().cuda()
    inner = [mk(2, 4, 64, 200).transpose(2, 3).requires_grad_() for _ in range(5)]
    rows = [mk(2, 4, 200, 68)[..., :64].requires_grad_() for _ in range(5)]     # rows 136 bytes apart
    off = [mk(2, 4, 200, 72)[..., 4:68].requires_grad_() for _ in range(5)]     # rows that start off 16 bytes
    do = mk(2, 4, 200, 64)
    n = _native.load()
    for x in (inner, rows, off):
        assert n.flash(*x[:3], True, None) is None and n.flash_rest(*x[:3], True, None) is not None
        with flash.backward_mode("two_kernel"):
            one = lambda: (lambda o: (o,) + torch.autograd.grad(o, x[:3], do))(fa.flash_attention(*x[:3], True))
            _same(one(), python_form(one))
            five = lambda: (lambda o: (o,) + torch.autograd.grad(o, x, do))(fa.piecewise_attention(*x, 60, True))
            _same(five(), python_form(five))
        assert n.piecewise(*x, 60, True, None) is not None
        with torch.no_grad():
            _same([fa.flash_attention(x[0][:, :, :1], x[1], x[2])], [python_form(lambda: fa.flash_attention(x[0][:, :, :1], x[1], x[2]))])
    # the copies are saved, not the views: what becomes of these afterwards does not matter, in either form
    o = fa.flash_attention(*inner[:3], True)
    with torch.no_grad():
        inner[0].zero_()
    torch.autograd.grad(o, inner[:3], do)
    # a contiguous tensor off the alignment is refused as before
    bad = mk(2 * 4 * 200 * 64 + 4)[4:].view(2, 4, 200, 64)
    assert n.flash_rest(bad, bad, bad, True, None) is None and n.piecewise(bad, bad, bad, bad, bad, 3, True, None) is None
    with pytest.raises(RuntimeError):
        fa.flash_attention(bad, bad, bad, True)


def test_paged_operands_that_are_converted(python_form):
    gen = torch.Generator(device="cuda").manual_seed(11)
    rnd = lambda *s: torch.randn(s, generator=gen, device="cuda", dtype=torch.float16)
    kc, vc, key, value = rnd(400, 2, 16, 128), rnd(400, 2, 16, 128), rnd(3, 128, 2), rnd(3, 2, 128)
    most = 700
    table = torch.randint(0, 400, (3, 44), generator=gen, device="cuda", dtype=torch.int32)
    lens = torch.tensor([most, 1, 250], device="cuda")
    wide = torch.stack([lens.int(), lens.int()], 1)
    n = _native.load()
    for q, l, t in ((rnd(3, 8, 128), lens, table), (rnd(3, 128, 8).transpose(1, 2), lens.int(), table),
                    (rnd(3, 8, 132)[..., 4:], wide[:, 0], table.t().contiguous().t()), (rnd(8, 3, 128).transpose(0, 1), lens, table.long())):
        assert n.paged(q, kc, vc, l, t, 0.1, most, 0, 0, 0, 0, 0, 0, 0, 0) is not None
        call = lambda: fa.paged_attention(q, kc, vc, l, t, 0.1, most)
        _same([call()], [python_form(call)])
    q, column = rnd(3, 8, 128), table[:, 3:4]   # (contiguous, whatever its last stride)
    assert n.paged(q, kc, vc, lens.clamp(max=16), column.t().contiguous().t(), 0.1, 16, 0, 0, 0, 0, 0, 0, 0, 0) is not None
    call = lambda: fa.paged_attention(q, kc, vc, lens.clamp(max=16), torch.stack([column[:, 0]] * 2, 1)[:, ::2], 0.1, 16)
    _same([call()], [python_form(call)])
    # neither form can help a contiguous operand off the alignment
    assert n.append(rnd(3 * 256 + 4)[4:].view(3, 2, 128), value, kc, vc, torch.zeros(3, dtype=torch.int64, device="cuda")) is False
    assert n.paged(rnd(3 * 1024 + 4)[4:].view(3, 8, 128), kc, vc, lens, table, 0.1, most, 0, 0, 0, 0, 0, 0, 0, 0) is None
    slots = torch.tensor([5, -1, 400 * 16 - 1], device="cuda")

    def write(k, v, s):
        caches = kc.clone(), vc.clone()
        paged.reshape_and_cache(k, v, *caches, s)
        return caches
    for k, v, s in ((key.transpose(1, 2), value, slots), (value, value + 1, slots.int()),
                    (value, value, torch.stack([slots, slots], 1)[:, 0]), (rnd(3, 2, 132)[..., 4:], rnd(3, 2, 132)[..., 4:], slots)):
        assert n.append(k, v, kc.clone(), vc.clone(), s)
        _same(write(k, v, s), python_form(lambda: write(k, v, s)))


def test_piecewise_and_rotary_calls(python_form):
    B, H, L, D = 2, 4, 300, 64
    gen = torch.Generator().manual_seed(1)
    x, y, v, do = (torch.randn((B, H, L, D), generator=gen).half().cuda().requires_grad_() for _ in range(4))
    tables = rotary.rotary_tables(L, D, device="cuda") + rotary.rotary_tables(L, D, position_scale=0.25, device="cuda")

    def run():
        q1, q2 = rotary.rotary_pair(x, *tables)
        k1, k2 = rotary.rotary_pair(y, *tables, interleaved=True)
        o = fa.piecewise_attention(q1, k1, q2, k2, v, 100, True)
        return (q1, q2, k1, k2, o) + torch.autograd.grad(o, (x, y, v), do.detach())

    with flash.backward_mode("two_kernel"):
        _same(run(), python_form(run))


@pytest.mark.parametrize("index", [torch.int32, torch.int64])
@pytest.mark.parametrize("most", [300, 5000])
def test_paged_calls(python_form, index, most):
    gen = torch.Generator(device="cuda").manual_seed(most)
    rnd = lambda *s: torch.randn(s, generator=gen, device="cuda", dtype=torch.float16)
    q, kc, vc, key, value = rnd(3, 8, 128), rnd(400, 2, 16, 128), rnd(400, 2, 16, 128), rnd(3, 2, 128), rnd(3, 2, 128)
    lens = torch.tensor([most, 1, 250], dtype=torch.int32, device="cuda")
    table = torch.randint(0, 400, (3, -(-most // 16)), generator=gen, device="cuda").to(index)
    slots = torch.tensor([5, -1, 400 * 16 - 1], device="cuda")
    call = lambda: fa.paged_attention(q, kc, vc, lens, table, 128 ** -0.5, most)
    _same([call()], [python_form(call)])

    def write():
        caches = kc.clone(), vc.clone()
        paged.reshape_and_cache(key, value, *caches, slots)
        return caches
    _same(write(), python_form(write))


def test_the_usual_calls_are_taken():
    """A check that went wrong would send every call to the Python form, unnoticed."""
    n, x = _native.load(), torch.randn(2, 4, 256, 64, device="cuda", dtype=torch.float16)
    t = rotary.rotary_tables(256, 64, device="cuda")
    assert n.flash(x, x, x, True, None) is not None
    assert n.flash(x[:, :, :1], x, x, False, 0.1) is not None
    assert n.flash(x, x.requires_grad_(), torch.nn.Parameter(x.detach()), True, None).requires_grad
    assert n.piecewise(x, x, x, x, x, 10, True, None) is not None
    assert n.rotary_pair(x, *t, *t, False) is not None
    q, cache, lens = x[0, :2, 0].detach()[:, None].contiguous(), x.detach()[..., :16, :].contiguous(), torch.ones(2, dtype=torch.int32, device="cuda")
    assert n.paged(q.expand(2, 4, 64).contiguous(), cache, cache, lens, lens[:, None], 1.0, 16, 0, 0, 0, 0, 0, 0, 0, 0) is not None
    assert n.append(x[:, :, 0].detach(), x[:, :, 0].detach(), cache, cache.clone(), torch.zeros(2, dtype=torch.int64, device="cuda"))


def test_what_is_left_to_the_python_form():
    """Transforms, modes, views that need a copy and errors."""
    n, x = _native.load(), torch.randn(2, 4, 256, 64, device="cuda", dtype=torch.float16)
    for q, k, v in ((x.cpu(), x, x), (x, x.float(), x), (x, x[:, :3], x[:, :3]), (x, x[:, :, :9], x), (x[..., ::2], x[..., ::2], x[..., ::2]),
                    (x.transpose(2, 3), x, x), (x[0], x, x), (x[..., :48], x[..., :48], x[..., :48]), (x[:, :0], x, x),
                    (x[:, :1, :20], x[:, :1], x[:, :1]), (None, x, x), (1, 2, 3)):
        assert n.flash(q, k, v, True, None) is None
    assert n.flash(x, x, x, 1, None) is None and n.flash(x, x, x, True, "no") is None and n.flash(x, x) is None

    from torch.autograd import forward_ad
    from torch.utils._python_dispatch import TorchDispatchMode

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))
    with Mode():
        assert n.flash(x, x, x, True, None) is None
    with forward_ad.dual_level():
        dual = forward_ad.make_dual(x, torch.ones_like(x))
        assert n.flash(dual, x, x, True, None) is None
        with pytest.raises(Exception):
            fa.flash_attention(dual, x, x, True)
    with pytest.raises(Exception):   # no vmap rule, in either form
        torch.func.vmap(lambda y: fa.flash_attention(y, x, x, True))(torch.stack([x, x]))
    with pytest.raises(Exception):
        torch.func.grad(lambda y: fa.flash_attention(y, x, x, True).float().sum())(x)
    with pytest.raises(AssertionError, match="multiple"):
        fa.flash_attention(x, x[:, :3], x[:, :3])
    with pytest.raises(AssertionError):
        fa.flash_attention(x.cpu(), x.cpu(), x.cpu())


def test_saved_tensors_obey_hooks_and_versions():
    q, k, v, do = make_qkv(1, 8, 8, 200, 200, 64, torch.float16, "cuda", seed=5)
    for x in (q, k, v):
        x.requires_grad_()
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t.cpu(), lambda t: t.cuda()):
        o = fa.flash_attention(q, k, v, True)
    assert len(packed) == 5
    with flash.backward_mode("two_kernel"):
        got = torch.autograd.grad(o, (q, k, v), do)
        _same(got, torch.autograd.grad(fa.flash_attention(q, k, v, True), (q, k, v), do))
    o = fa.flash_attention(q, k, v, True)
    with torch.no_grad():
        k.mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(o, (q, k, v), do)
    o = fa.flash_attention(q, k, v, True)
    torch.autograd.grad(o, q, do)
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(o, q, do)


def test_deterministic_switch_reaches_the_native_backward():
    q, k, v, do = make_qkv(2, 8, 8, 700, 700, 64, torch.float16, "cuda", seed=6)
    for x in (q, k, v):
        x.requires_grad_()
    run = lambda: torch.autograd.grad(fa.flash_attention(q, k, v, True), (q, k, v), do)
    with flash.backward_mode("two_kernel"):
        want = run()
    torch.use_deterministic_algorithms(True)
    try:
        _same(run(), want)
    finally:
        torch.use_deterministic_algorithms(False)


def test_several_threads_and_streams():
    import threading
    q, k, v, do = make_qkv(2, 8, 8, 300, 300, 64, torch.float16, "cuda", seed=7)
    for x in (q, k, v):
        x.requires_grad_()
    want = fa.flash_attention(q, k, v, True)
    torch.cuda.synchronize()
    bad = []

    def work():
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                o = fa.flash_attention(q, k, v, True)
                torch.autograd.grad(o, (q, k, v), do)
                if not torch.equal(o, want):
                    bad.append(1)
            torch.cuda.current_stream().synchronize()
    threads = [threading.Thread(target=work) for _ in range(3)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not bad


@pytest.mark.parametrize("B,H,Hk,L,D", [(2, 8, 8, 300, 64), (1, 16, 2, 500, 128)])   # the second: shared walks
def test_gradients_from_several_threads_and_streams(B, H, Hk, L, D):
    """Each call has its own workspace and work-item counter, and its backward runs on the stream of its forward."""
    import threading
    q, k, v, do = make_qkv(B, H, Hk, L, L, D, torch.float16, "cuda", seed=8)
    for x in (q, k, v):
        x.requires_grad_()
    want = torch.autograd.grad(fa.flash_attention(q, k, v, True), (q, k, v), do)
    torch.cuda.synchronize()
    bad = []

    def work():
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                got = torch.autograd.grad(fa.flash_attention(q, k, v, True), (q, k, v), do)
                # dk, dv bitwise; dq is summed in any order: a rounding to 16 bits apart at most
                if not (torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
                        and (got[0].float() - want[0].float()).abs().max() <= 2 ** -10 * want[0].float().abs().max()):
                    bad.append(1)
            torch.cuda.current_stream().synchronize()
    threads = [threading.Thread(target=work) for _ in range(3)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not bad

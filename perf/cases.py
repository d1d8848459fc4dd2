"""The attention work whose speed this framework answers for.

`listed()` names twelve calls a user's program makes; `draw()` gives more of the same ranges.  A case is a dict of
plain values with a "kind":

  train      flash_attention forward + backward to q, k, v
  piecewise  piecewise_attention forward + backward to q1, k1, q2, k2, v
  nlpe       an NLPE layer's attention: rotary_pair of q and of k, piecewise_attention, backward to q, k, v
  prefill    flash_attention forward without gradients: a block of new queries over the keys so far
  score      the same with the log-normaliser and the total attention every key received
  decode     flash_attention with one query per head over a dense KV cache
  paged      one serving step over a paged KV cache: paged_attention, with `append` the new tokens' keys and values
             are written into their slots first

Lengths, heads and head sizes are those of the repository's tests and benchmark, or lie between them; lengths are as
often odd as even, since batches are cut by tokens and not by tiles.  Activations, caches and output gradients are
N(0, 1), as in the tests, scaled by 0.5 where the configuration says so.
"""
import math

import torch

import flagattention_b200 as fa
from flagattention_b200 import paged, rotary

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # a training step's attention at the headline configuration
        dict(name="train_hd128", kind="train", dtype="bf16", B=4, H=32, Hk=32, M=4096, N=4096, D=128, causal=True,
             scale=1.0, dropout=0.0, lse=False, layout="bhld"),
        # the same step of a grouped-query model on packed sequences of no round length, q, k, v as the projections
        # leave them: (batch, length, heads, head_dim) in memory
        dict(name="train_gqa_ragged", kind="train", dtype="bf16", B=3, H=32, Hk=8, M=1867, N=1867, D=128, causal=True,
             scale=1.0, dropout=0.0, lse=False, layout="blhd"),
        # long bidirectional training at head_dim 64, with the log-normaliser a caller may want beside the output
        dict(name="train_hd64_long", kind="train", dtype="fp16", B=2, H=16, Hk=16, M=8192, N=8192, D=64, causal=False,
             scale=0.5, dropout=0.0, lse=True, layout="bhld"),
        # an encoder's short sequences with dropout on the attention weights
        dict(name="train_dropout", kind="train", dtype="bf16", B=16, H=16, Hk=16, M=512, N=512, D=64, causal=False,
             scale=1.0, dropout=0.1, lse=False, layout="bhld"),
        # the smallest training call: launches and host work count here
        dict(name="train_small", kind="train", dtype="bf16", B=2, H=4, Hk=4, M=256, N=256, D=64, causal=True,
             scale=1.0, dropout=0.0, lse=False, layout="bhld"),
        # piecewise attention at the size of an Aquila-2-34B layer
        dict(name="piecewise_long", kind="piecewise", dtype="bf16", B=1, H=48, L=16384, D=128, w=4096, causal=True),
        # a whole NLPE layer on a sequence of ordinary length
        dict(name="nlpe_layer", kind="nlpe", dtype="fp16", B=2, H=16, L=2048, D=128, w=700, causal=True),
        # chunked prefill of one request: the next 512 tokens over 7300 keys
        dict(name="prefill_chunk", kind="prefill", dtype="bf16", B=1, H=32, Hk=8, M=512, N=7300, D=128, causal=True),
        # which keys of a prompt receive attention (cache eviction, analysis)
        dict(name="score_prompt", kind="score", dtype="fp16", B=1, H=16, Hk=16, M=6144, N=6144, D=128, causal=True),
        # decoding over a long dense cache
        dict(name="decode_dense", kind="decode", dtype="fp16", B=2, H=16, Hk=16, M=1, N=131072, D=128, causal=False),
        # decoding for a full batch of requests over a paged cache
        dict(name="paged_batch", kind="paged", dtype="fp16", seqs=64, H=32, Hk=8, D=128, block=16, lo=1024, hi=32768,
             append=False),
        # decoding for a few short requests: the smallest step of a serving loop
        dict(name="paged_few", kind="paged", dtype="bf16", seqs=4, H=32, Hk=8, D=128, block=16, lo=200, hi=1500,
             append=True),
    ]


# ---------------------------------------------------------------------------------------------
# drawn cases
# ---------------------------------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    n = _log_int(rng, lo, hi)
    return n if rng.random() < 0.6 else max(lo, n // 64 * 64)


def _head_dim(rng):
    return rng.choice([128, 128, 128, 64, 64, 32])


def _heads(rng, D):
    return rng.choice([4, 8, 16, 32]) if D >= 64 else rng.choice([8, 16])


def _kv_heads(rng, H):
    return rng.choice([h for h in (H, H, H // 4, 1 if H < 16 else H // 8) if h >= 1])


def draw(rng):
    kind = rng.choice(["train", "train", "train", "piecewise", "nlpe", "prefill", "prefill", "score", "decode", "paged",
                       "paged"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "train":
        D = _head_dim(rng)
        H = _heads(rng, D)
        L = _length(rng, 64, 8192)
        B = max(1, min(64, _log_int(rng, 256, 16384) // L))
        # (calls of fewer rows split the keys over CTAs, where dropout is refused)
        dropout = rng.choice([0.0, 0.0, 0.0, 0.1]) if L <= 4096 and B * H * (L // 16) >= 128 else 0.0
        return dict(kind=kind, dtype=dtype, B=B, H=H, Hk=_kv_heads(rng, H), M=L, N=L, D=D, causal=rng.random() < 0.7,
                    scale=rng.choice([1.0, 1.0, 0.5]), dropout=dropout, lse=rng.random() < 0.2,
                    layout=rng.choice(["bhld", "blhd"]))
    if kind in ("piecewise", "nlpe"):
        D = rng.choice([128, 128, 64])
        L = _length(rng, 256, 8192)
        return dict(kind=kind, dtype=dtype, B=max(1, min(8, 8192 // L)), H=rng.choice([8, 16, 24]), L=L, D=D,
                    w=max(1, int(L * rng.uniform(0.1, 0.7))), causal=rng.random() < 0.8)
    if kind in ("prefill", "score"):
        D = _head_dim(rng)
        H = _heads(rng, D)
        N = _length(rng, 256, 16384)
        M = N if kind == "score" or rng.random() < 0.3 else _length(rng, 32, min(N, 2048))
        return dict(kind=kind, dtype=dtype, B=max(1, min(8, 8192 // N)), H=H, Hk=_kv_heads(rng, H), M=M, N=N, D=D,
                    causal=rng.random() < 0.85)
    if kind == "decode":
        D = rng.choice([128, 128, 64])
        H = rng.choice([8, 16, 32])
        N = _length(rng, 512, 131072)
        return dict(kind=kind, dtype=dtype, B=max(1, min(16, _log_int(rng, 1, 262144 // N))), H=H, Hk=_kv_heads(rng, H),
                    M=1, N=N, D=D, causal=False)
    H = rng.choice([16, 32])
    hi = _length(rng, 256, 32768)
    seqs = max(1, min(64, _log_int(rng, 1, max(2, 524288 // hi))))
    return dict(kind="paged", dtype=dtype, seqs=seqs, H=H,
                Hk=rng.choice([H, H // 4, H // 8]), D=rng.choice([128, 128, 64]), block=rng.choice([16, 16, 32]),
                lo=max(1, hi // 8), hi=hi, append=seqs * hi <= 32768 and rng.random() < 0.6)


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _normal(gen, dtype, shape, layout="bhld", scale=1.0):
    B, H, L, D = shape
    x = torch.randn((B, L, H, D) if layout == "blhd" else shape, generator=gen, device="cuda", dtype=dtype)
    if scale != 1.0:
        x *= scale
    return x.transpose(1, 2) if layout == "blhd" else x


def _leaves(*ts):
    return [t.requires_grad_() for t in ts]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = _DTYPES[case["dtype"]]
    kind, s = case["kind"], dict(case=case)
    if kind == "train":
        B, H, Hk, M, N, D = (case[k] for k in ("B", "H", "Hk", "M", "N", "D"))
        lay, sc = case["layout"], case["scale"]
        s["q"], s["k"], s["v"] = _leaves(_normal(gen, dt, (B, H, M, D), lay, sc), _normal(gen, dt, (B, Hk, N, D), lay, sc),
                                         _normal(gen, dt, (B, Hk, N, D), lay, sc))
        s["do"] = _normal(gen, dt, (B, H, M, D), lay)
        if case["dropout"]:
            torch.cuda.manual_seed(seed)   # the masks come from torch's CUDA generator
    elif kind == "piecewise":
        shape = tuple(case[k] for k in ("B", "H", "L", "D"))
        s["x"] = _leaves(*[_normal(gen, dt, shape) for _ in range(5)])
        s["do"] = _normal(gen, dt, shape)
    elif kind == "nlpe":
        shape = tuple(case[k] for k in ("B", "H", "L", "D"))
        s["q"], s["k"], s["v"] = _leaves(*[_normal(gen, dt, shape) for _ in range(3)])
        s["do"] = _normal(gen, dt, shape)
        # near pairs keep their positions, far pairs see them compressed
        s["tables"] = (rotary.rotary_tables(case["L"], case["D"], device="cuda") +
                       rotary.rotary_tables(case["L"], case["D"], position_scale=0.25, device="cuda"))
    elif kind in ("prefill", "score", "decode"):
        B, H, Hk, M, N, D = (case[k] for k in ("B", "H", "Hk", "M", "N", "D"))
        s["q"], s["k"], s["v"] = (_normal(gen, dt, (B, H, M, D)), _normal(gen, dt, (B, Hk, N, D)),
                                  _normal(gen, dt, (B, Hk, N, D)))
    else:
        seqs, H, Hk, D, bs = (case[k] for k in ("seqs", "H", "Hk", "D", "block"))
        lens = torch.randint(case["lo"], case["hi"] + 1, (seqs,), generator=torch.Generator().manual_seed(seed))
        lens[0] = case["hi"]
        blocks = [(int(n) + bs - 1) // bs for n in lens]
        pool = seqs * max(blocks)   # room for every sequence at its longest
        order = torch.randperm(pool, generator=gen, device="cuda", dtype=torch.int32)
        table = torch.zeros((seqs, max(blocks)), dtype=torch.int32, device="cuda")
        at = 0
        for i, n in enumerate(blocks):
            table[i, :n] = order[at:at + n]
            at += n
        s["cache"] = [_normal(gen, dt, (pool, Hk, bs, D)) for _ in range(2)]
        s["q"] = torch.randn((seqs, H, D), generator=gen, device="cuda", dtype=dt)
        s["table"], s["lens"], s["max_len"] = table, lens.to(torch.int32).cuda(), case["hi"]
        if case["append"]:
            s["new"] = [torch.randn((seqs, Hk, D), generator=gen, device="cuda", dtype=dt) for _ in range(2)]
            last = lens.cuda() - 1
            s["slots"] = table.gather(1, (last // bs)[:, None]).squeeze(1).long() * bs + last % bs
    return s


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "train":
        q, k, v = s["q"], s["k"], s["v"]
        if c["lse"]:
            o, lse = fa.flash_attention(q, k, v, causal=c["causal"], dropout_p=c["dropout"], return_log_normalizer=True)[:2]
            return (o, lse) + torch.autograd.grad(o, (q, k, v), s["do"])
        o = fa.flash_attention(q, k, v, causal=c["causal"], dropout_p=c["dropout"])
        return (o,) + torch.autograd.grad(o, (q, k, v), s["do"])
    if kind == "piecewise":
        o = fa.piecewise_attention(*s["x"], c["w"], causal=c["causal"])
        return (o,) + torch.autograd.grad(o, s["x"], s["do"])
    if kind == "nlpe":
        q1, q2 = rotary.rotary_pair(s["q"], *s["tables"])
        k1, k2 = rotary.rotary_pair(s["k"], *s["tables"])
        o = fa.piecewise_attention(q1, k1, q2, k2, s["v"], c["w"], causal=c["causal"])
        return (o,) + torch.autograd.grad(o, (s["q"], s["k"], s["v"]), s["do"])
    if kind in ("prefill", "decode"):
        return fa.flash_attention(s["q"], s["k"], s["v"], causal=c["causal"])
    if kind == "score":
        return fa.flash_attention(s["q"], s["k"], s["v"], causal=c["causal"], return_log_normalizer=True,
                                  return_total_attention=True)[:3]
    kc, vc = s["cache"]
    if c["append"]:
        paged.reshape_and_cache(*s["new"], kc, vc, s["slots"])
    out = fa.paged_attention(s["q"], kc, vc, s["lens"], s["table"], c["D"] ** -0.5, s["max_len"])
    return (out, kc, vc) if c["append"] else out


# ---------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------
def _exact_head(near, far, v, do, w, causal, aux):
    """One head in float64: (o, lse, total, near gradients, far gradients, dv).  `near` and `far` are (q, k) pairs, `far`
    None for plain attention; query rows are taken 2048 at a time, and `v` may carry no gradient (do None)."""
    M, N, D = near[0].shape[0], near[1].shape[0], v.shape[1]
    pairs = [near] if far is None else [near, far]
    cols = torch.arange(N, device=v.device)
    outs, lses, total = [], [], torch.zeros(N, dtype=torch.float64, device=v.device)
    dqs, dks, dv = [[] for _ in pairs], [torch.zeros_like(k) for _, k in pairs], torch.zeros_like(v)
    for a in range(0, M, 2048):
        b = min(M, a + 2048)
        at = torch.arange(a, b, device=v.device)[:, None] + (N - M)
        n = min(N, b + N - M) if causal else N        # later keys are seen by none of these rows
        s = near[0][a:b] @ near[1][:n].T
        is_far = (at - cols[:n]) >= w
        if far is not None:
            s = torch.where(is_far, far[0][a:b] @ far[1][:n].T, s)
        s *= D ** -0.5
        if causal:
            s.masked_fill_(cols[:n] > at, -math.inf)
        lse = torch.logsumexp(s, 1, keepdim=True)
        p = torch.exp_(s - lse)
        del s
        o = p @ v[:n]
        outs.append(o)
        lses.append(lse.squeeze(1))
        if aux:
            total[:n] += p.sum(0)
        if do is None:
            continue
        dv[:n] += p.T @ do[a:b]
        ds = do[a:b] @ v[:n].T
        ds -= (do[a:b] * o).sum(1, keepdim=True)
        ds *= p
        ds *= D ** -0.5
        del p
        for i, (q, k) in enumerate(pairs):
            d = ds if far is None else ds.masked_fill(is_far if i == 0 else ~is_far, 0.0)
            dqs[i].append(d @ k[:n])
            dks[i][:n] += d.T @ q[a:b]
    grads = [(torch.cat(dq), dk) for dq, dk in zip(dqs, dks)] if do is not None else None
    return torch.cat(outs), torch.cat(lses), total, grads, dv


def _exact_heads(near, far, v, do, w, causal, aux=False):
    """`_exact_head` over (batch, head), the gradients of keys and values summed over the heads of a group."""
    q, k = near
    B, H, Hk = q.shape[0], q.shape[1], k.shape[1]
    new = lambda *shape: torch.zeros(shape, dtype=torch.float64, device=q.device)
    o, lse, total = new(*q.shape), new(*q.shape[:3]), new(B, H, k.shape[2])
    grads = [(new(*x.shape), new(*y.shape)) for x, y in ([near] if far is None else [near, far])] if do is not None else []
    dv = new(*v.shape) if do is not None else None
    for b in range(B):
        for h in range(H):
            g = h // (H // Hk)
            at = lambda pair: None if pair is None else (pair[0][b, h].double(), pair[1][b, g].double())
            o[b, h], lse[b, h], total[b, h], gs, gv = _exact_head(
                at(near), at(far), v[b, g].double(), None if do is None else do[b, h].double(), w, causal, aux)
            for (dq, dk), (x, y) in zip(grads, gs or ()):
                dq[b, h] = x
                dk[b, g] += y
            if do is not None:
                dv[b, g] += gv
    return o, lse, total, grads, dv


def _rotate(x, cos, sin, back=False):
    lo, hi = x.double().chunk(2, -1)
    c, s = cos.double(), -sin.double() if back else sin.double()
    return torch.cat((lo * c - hi * s, hi * c + lo * s), -1)


@torch.no_grad()
def exact(case, seed):
    """What `run` returns, in 64 bits.  None with dropout: its mask is a matter of the random stream, not of precision."""
    c, kind = case, case["kind"]
    if kind == "train" and c["dropout"]:
        return None
    s = prepare(case, seed)
    if kind == "train":
        o, lse, _, [(dq, dk)], dv = _exact_heads((s["q"], s["k"]), None, s["v"], s["do"], 0, c["causal"])
        return (o, lse, dq, dk, dv) if c["lse"] else (o, dq, dk, dv)
    if kind == "piecewise":
        q1, k1, q2, k2, v = s["x"]
        o, _, _, [(dq1, dk1), (dq2, dk2)], dv = _exact_heads((q1, k1), (q2, k2), v, s["do"], c["w"], c["causal"])
        return o, dq1, dk1, dq2, dk2, dv
    if kind == "nlpe":
        cos1, sin1, cos2, sin2 = s["tables"]
        near, far = ([_rotate(s[x], cos, sin) for x in "qk"] for cos, sin in ((cos1, sin1), (cos2, sin2)))
        o, _, _, (g1, g2), dv = _exact_heads(near, far, s["v"], s["do"], c["w"], c["causal"])
        dq, dk = (_rotate(x, cos1, sin1, True) + _rotate(y, cos2, sin2, True) for x, y in zip(g1, g2))
        return o, dq, dk, dv
    if kind in ("prefill", "score", "decode"):
        o, lse, total, _, _ = _exact_heads((s["q"], s["k"]), None, s["v"], None, 0, c["causal"], kind == "score")
        return (o, lse, total) if kind == "score" else o
    kc, vc = s["cache"]
    if c["append"]:
        for cache, new in zip((kc, vc), s["new"]):
            cache[s["slots"] // c["block"], :, s["slots"] % c["block"]] = new
    out = torch.empty(s["q"].shape, dtype=torch.float64, device="cuda")
    for i, n in enumerate(s["lens"].tolist()):
        blocks = s["table"][i, :(n + c["block"] - 1) // c["block"]].long()
        k, v = (x[blocks].double().transpose(0, 1).flatten(1, 2)[:, :n] for x in (kc, vc))
        q = s["q"][i].double().unflatten(0, (c["Hk"], -1))
        out[i] = (torch.softmax(q @ k.transpose(1, 2) * c["D"] ** -0.5, -1) @ v).flatten(0, 1)
    return (out, kc, vc) if c["append"] else out


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _pairs(M, N, causal):
    """Query-key pairs a (batch, head) has: the causal mask is aligned to the last query and key (N >= M here)."""
    return M * N - M * (M - 1) // 2 if causal else M * N


def work(case):
    kind, c = case["kind"], case
    if kind == "train":
        rows = c["B"] * (c["H"] * c["M"] + c["Hk"] * c["N"]) * c["D"]
        gemm = 2.0 * c["B"] * c["H"] * c["D"] * _pairs(c["M"], c["N"], c["causal"])
        # q, k, v, do in; o, dq, dk, dv out
        return {"bytes": 2.0 * 4 * rows + (4.0 * c["B"] * c["H"] * c["M"] if c["lse"] else 0.0), "flops": 7 * gemm}
    if kind in ("piecewise", "nlpe"):
        x = 2.0 * c["B"] * c["H"] * c["L"] * c["D"]
        gemm = 2.0 * c["B"] * c["H"] * c["D"] * _pairs(c["L"], c["L"], c["causal"])
        # five operands and do in, o and five gradients out; the layer: q, k, v, do in, o, dq, dk, dv out, four tables
        tables = 4 * 4.0 * c["L"] * (c["D"] // 2) if kind == "nlpe" else 0.0
        return {"bytes": (12 if kind == "piecewise" else 8) * x + tables, "flops": 7 * gemm}
    if kind in ("prefill", "score", "decode"):
        gemm = 2.0 * c["B"] * c["H"] * c["D"] * _pairs(c["M"], c["N"], c["causal"])
        aux = 4.0 * c["B"] * c["H"] * (c["M"] + c["N"]) if kind == "score" else 0.0
        return {"bytes": 2.0 * 2 * c["B"] * (c["H"] * c["M"] + c["Hk"] * c["N"]) * c["D"] + aux,
                "flops": (3 if kind == "score" else 2) * gemm}
    # contexts are uniform in [lo, hi], the first one is hi
    tokens = c["hi"] + (c["seqs"] - 1) * 0.5 * (c["lo"] + c["hi"])
    new = 2 * 2 * 2.0 * c["seqs"] * c["Hk"] * c["D"] if c["append"] else 0.0
    return {"bytes": tokens * (2 * 2.0 * c["Hk"] * c["D"] + 4.0 / c["block"]) + 2 * 2.0 * c["seqs"] * c["H"] * c["D"] + new,
            "flops": 4.0 * tokens * c["H"] * c["D"]}


def tolerance(case):
    # Four times what was measured, over these ranges, between the outputs and the same formulas in 64 bits: the 16-bit
    # rounding of the probabilities, of dS and of the results (bf16: 2.4e-3 forward, 2.7e-3 with gradients, 4.1e-3 where
    # rotated operands are rounded too; fp16: eight times less).
    backward = case["kind"] in ("train", "piecewise", "nlpe")
    rel, most = (4e-3, 0.11) if case["kind"] == "nlpe" else (2.7e-3, 0.12) if backward else (2.4e-3, 0.02)
    ulps = 4.0 if case["dtype"] == "bf16" else 0.5
    return {"rel": rel * ulps, "max": most * ulps}

"""The work this library is used for, as cases that can be timed and compared.

Every case goes through the public entry points, the way a program that prefills, decodes or
trains with them does.  Sizes are this repository's benchmark configurations, their ragged and
small relatives, and generic serving and training shapes; `draw` gives further cases of the same
ranges.  Lengths, page tables and block lists that shape the work come from the case itself (its
`lens_seed`), tensors and block scores from the seed given to `prepare`."""
import math
import random

import torch

from tritonops_b200 import ops
from tritonops_b200.common.rms import RMSNormTritonFunction
from tritonops_b200.flash_attn_triton.flash_attn_decoding import flash_attention_decoding
from tritonops_b200.flash_attn_triton.flash_attn_decoding_sparse import (
    flash_attention_block_sparse_decoding, flash_attention_sparse_decoding)
from tritonops_b200.flash_attn_triton.flash_attn_sparse_attn_triton import (
    flash_attn_block_sparse, flash_attn_sparse_triton)
from tritonops_b200.flash_attn_triton.flash_attn_triton import flash_attention, flash_attn_triton

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
BLOCK = 64      # block-list granularity of the sparse paths


def listed():
    return [
        # The library's smallest attention call (one CTA): what a caller pays for a launch.
        dict(name="prefill_tiny", kind="prefill", batch=1, seq=128, hq=2, hkv=2, d=64, dtype="fp16", causal=False),
        # The headline configuration: a prompt batch of equal lengths, O and LSE.
        dict(name="prefill_batch", kind="prefill", batch=4, seq=4096, hq=32, hkv=32, d=128, dtype="bf16", causal=True),
        # A serving prefill: sequences of unequal, odd lengths packed together, grouped-query heads.
        dict(name="prefill_packed", kind="packed", batch=12, lo=37, hi=3000, lens_seed=1, hq=32, hkv=8, d=128,
             dtype="bf16"),
        # A training step's attention, forward and backward through autograd, at the headline shape.
        dict(name="train_batch", kind="train", batch=4, lo=4096, hi=4096, lens_seed=0, hq=32, hkv=32, d=128,
             dtype="bf16"),
        # The same over packed documents of odd lengths with narrow heads in fp16.
        dict(name="train_packed", kind="train", batch=9, lo=100, hi=2500, lens_seed=2, hq=16, hkv=4, d=64,
             dtype="fp16"),
        # Sliding window with a global prefix over long packed prompts.
        dict(name="prefill_window", kind="window", batch=2, lo=6000, hi=9000, lens_seed=3, hq=16, hkv=16, d=128,
             dtype="bf16", local=1024, glob=128),
        # Block-list sparse prefill of long prompts: local blocks plus a tenth of the earlier ones.
        dict(name="prefill_blocks", kind="blocks", batch=2, seq=16384, hq=16, hkv=16, d=128, dtype="bf16",
             local_blocks=8, density=0.1, lens_seed=4),
        # A decoding step of a full serving batch over a padded cache, lengths as they come.
        dict(name="decode_batch", kind="decode", batch=64, capacity=8192, lo=1024, hi=8192, lens_seed=5, hq=32, hkv=8,
             d=128, dtype="bf16"),
        # The latency of one user: the new key and value appended, then one token attended.
        dict(name="decode_single", kind="decode_step", batch=1, capacity=4096, lo=3001, hi=3001, lens_seed=0, hq=32,
             hkv=8, d=128, dtype="bf16"),
        # A serving batch over a page pool.
        dict(name="decode_paged", kind="paged", batch=24, page=64, lo=300, hi=6000, lens_seed=6, hq=32, hkv=8, d=128,
             dtype="bf16"),
        # Top-k block decoding of long contexts: selection from block scores, then the gather.
        dict(name="decode_topk", kind="topk", batch=8, seq=32768, hq=32, hkv=32, d=128, dtype="bf16", top_k=64),
        # The normalisation of a training step, forward and backward.
        dict(name="rmsnorm_train", kind="rmsnorm", rows=16384, dim=4096, dtype="bf16"),
    ]


# ---------------------------------------------------------------------------- drawing
def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


_HEADS = [(8, 8), (16, 4), (32, 8), (12, 12), (32, 32), (16, 1), (28, 4), (64, 8)]


def draw(rng):
    """A case of the ranges `listed` stands for; none costs more than the largest listed one."""
    for _ in range(200):
        c = _draw(rng)
        w = work(c)
        if w["bytes"] <= 1.2e9 and w["flops"] <= 5e11 and _held(c) <= 8e9:
            return c
    return dict(kind="prefill", batch=1, seq=_log_int(rng, 64, 4096), hq=8, hkv=8, d=128, dtype="bf16", causal=True)


def _held(c):
    """Bytes of the caches a decoding case keeps."""
    if c["kind"] in ("decode", "decode_step", "window_decode", "topk"):
        return 4.0 * c["batch"] * c.get("capacity", c.get("seq")) * c["hkv"] * c["d"]
    return 0.0


def _draw(rng):
    kind = rng.choice(["prefill", "packed", "packed", "train", "train", "window", "blocks", "decode", "decode_step",
                       "window_decode", "paged", "topk", "rmsnorm"])
    hq, hkv = rng.choice(_HEADS)
    c = dict(kind=kind, hq=hq, hkv=hkv, d=rng.choice([64, 96, 128, 128]), dtype=rng.choice(["bf16", "bf16", "fp16"]))
    if kind == "prefill":
        c.update(batch=_log_int(rng, 1, 16), seq=_log_int(rng, 64, 16384), causal=rng.random() < 0.7)
    elif kind in ("packed", "train"):
        hi = _log_int(rng, 64, 8192)
        c.update(batch=_log_int(rng, 1, 24), lo=max(1, hi // rng.choice([1, 2, 8, 64])), hi=hi,
                 lens_seed=rng.randrange(1 << 20))
    elif kind == "window":
        hi = _log_int(rng, 500, 16384)
        c.update(batch=_log_int(rng, 1, 8), lo=max(1, hi // rng.choice([1, 2, 4])), hi=hi,
                 lens_seed=rng.randrange(1 << 20), local=_log_int(rng, 64, 4096), glob=rng.choice([0, 16, 64, 128, 500]))
    elif kind == "blocks":
        c.update(hkv=hq, batch=_log_int(rng, 1, 4), seq=_log_int(rng, 500, 16384), local_blocks=rng.randint(1, 16),
                 density=round(rng.uniform(0.02, 0.4), 3), lens_seed=rng.randrange(1 << 20))
    elif kind in ("decode", "decode_step", "window_decode"):
        cap = _log_int(rng, 256, 32768)
        hi = max(1, cap - rng.randrange(0, cap // 4))
        c.update(batch=_log_int(rng, 1, 128), capacity=cap, lo=max(1, hi // rng.choice([1, 2, 8])), hi=hi,
                 lens_seed=rng.randrange(1 << 20))
        if kind == "decode_step":
            c.update(hi=min(c["hi"], cap - 1), lo=min(c["lo"], cap - 1))
        if kind == "window_decode":
            c.update(glob=rng.choice([64, 128, 256]), local=_log_int(rng, 64, 4096))
    elif kind == "paged":
        hi = _log_int(rng, 100, 32768)
        c.update(batch=_log_int(rng, 1, 64), page=rng.choice([16, 64, 128]), lo=max(1, hi // rng.choice([1, 2, 8])),
                 hi=hi, lens_seed=rng.randrange(1 << 20))
    elif kind == "topk":
        nb = _log_int(rng, 16, 512)
        c.update(hkv=hq if rng.random() < 0.5 else hkv, batch=_log_int(rng, 1, 32), seq=nb * BLOCK,
                 top_k=min(nb, _log_int(rng, 4, 128)))
    else:
        c = dict(kind="rmsnorm", rows=_log_int(rng, 1, 65536), dim=rng.choice([512, 1000, 2048, 3072, 4096, 5120, 8192]),
                 dtype=rng.choice(["bf16", "fp16", "fp32"]))
    return c


# ---------------------------------------------------------------------------- preparing
def _lens(c):
    r = random.Random(c["lens_seed"])
    return [r.randint(c["lo"], c["hi"]) for _ in range(c["batch"])]


def _normal(g, dtype, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=DTYPES[dtype])


def _cu(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return torch.tensor(cu, dtype=torch.int32, device="cuda")


def _block_lists(c):
    """Per (sequence, head, query block) the ascending KV blocks it attends to: a local band and a
    random share of the earlier blocks, -1 padded, and their number."""
    n = -(-c["seq"] // BLOCK)
    g = torch.Generator(device="cuda").manual_seed(c["lens_seed"])
    i = torch.arange(n, device="cuda")
    near = (i[None, :] <= i[:, None]) & (i[None, :] > i[:, None] - c["local_blocks"])
    far = torch.rand(c["batch"], c["hq"], n, n, generator=g, device="cuda") < c["density"]
    mask = (far & (i[None, :] < i[:, None])) | near
    cnt = mask.sum(-1)
    key = torch.where(mask, i.expand_as(mask), n).sort(-1).values[..., :int(cnt.max())]
    return torch.where(key >= n, -1, key).to(torch.int32).contiguous(), cnt.to(torch.int32).contiguous()


def prepare(case, seed):
    c = case
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = c["kind"]
    s = {"case": dict(c)}
    if kind == "rmsnorm":
        s["x"] = _normal(g, c["dtype"], c["rows"], c["dim"]).requires_grad_()
        s["w"] = (1 + 0.1 * _normal(g, "fp32", c["dim"])).to(DTYPES[c["dtype"]]).requires_grad_()
        s["dy"] = _normal(g, c["dtype"], c["rows"], c["dim"])
        return s
    hq, hkv, d, dt = c["hq"], c["hkv"], c["d"], c["dtype"]
    if kind in ("prefill", "blocks"):
        b, t = (c["batch"], c["seq"]) if kind == "prefill" else (1, c["batch"] * c["seq"])
        s["q"], s["k"], s["v"] = (_normal(g, dt, b, t, h, d) for h in (hq, hkv, hkv))
        if kind == "blocks":
            s["cu"] = _cu([c["seq"]] * c["batch"])
            s["idx"], s["cnt"] = _block_lists(c)
    elif kind in ("packed", "train", "window"):
        lens = _lens(c)
        s["cu"], s["max"] = _cu(lens), max(lens)
        s["q"], s["k"], s["v"] = (_normal(g, dt, 1, sum(lens), h, d) for h in (hq, hkv, hkv))
        if kind == "train":
            for n in "qkv":
                s[n].requires_grad_()
            s["do"] = _normal(g, dt, 1, sum(lens), hq, d)
    elif kind == "paged":
        lens = _lens(c)
        page = c["page"]
        per = -(-max(lens) // page)
        used = [-(-n // page) for n in lens]
        pages = sum(used)
        order = list(range(pages))
        random.Random(c["lens_seed"] + 1).shuffle(order)
        table, at = [], 0
        for n in used:
            table.append(order[at:at + n] + [0] * (per - n))
            at += n
        s["table"] = torch.tensor(table, dtype=torch.int32, device="cuda")
        s["lens"] = torch.tensor(lens, dtype=torch.int32, device="cuda")
        s["q"] = _normal(g, dt, c["batch"], hq, d)
        s["k"], s["v"] = (_normal(g, dt, pages, page, hkv, d) for _ in range(2))
    else:
        cap = c["seq"] if kind == "topk" else c["capacity"]
        lens = [c["seq"]] * c["batch"] if kind == "topk" else _lens(c)
        s["q"] = _normal(g, dt, c["batch"], hq, d)
        s["k"], s["v"] = (_normal(g, dt, c["batch"], cap, hkv, d) for _ in range(2))
        if kind == "topk":
            s["scores"] = torch.randn(c["batch"], hkv, cap // BLOCK, generator=g, device="cuda")
            s["cu"] = _cu(lens)
        elif kind == "decode_step":
            s["before"] = torch.tensor(lens, dtype=torch.int32, device="cuda")
            s["lens"] = s["before"] + 1
            s["new_k"], s["new_v"] = (_normal(g, dt, c["batch"], hkv, d) for _ in range(2))
        else:
            s["cu"] = _cu(lens)
    return s


# ---------------------------------------------------------------------------- one pass
def run(state):
    s = state
    c = s["case"]
    kind = c["kind"]
    if kind == "prefill":
        return flash_attention(s["q"], s["k"], s["v"], causal=c["causal"], return_lse=True)
    if kind == "packed":
        return flash_attention(s["q"], s["k"], s["v"], s["cu"], return_lse=True, max_seqlen=s["max"])
    if kind == "train":
        o = flash_attn_triton.apply(s["q"], s["k"], s["v"], s["cu"])
        return (o.detach(), *torch.autograd.grad(o, (s["q"], s["k"], s["v"]), s["do"]))
    if kind == "window":
        return flash_attn_sparse_triton(s["q"], s["k"], s["v"], s["cu"], c["local"], c["glob"])
    if kind == "blocks":
        return flash_attn_block_sparse(s["q"], s["k"], s["v"], s["cu"], s["idx"], s["cnt"], max_seqlen=c["seq"])
    if kind == "decode":
        return flash_attention_decoding(s["q"], s["k"], s["v"], s["cu"])
    if kind == "decode_step":
        ops.append_kv(s["k"], s["v"], s["new_k"], s["new_v"], s["before"])
        return ops.decode(s["q"], s["k"], s["v"], seqlens=s["lens"]), s["k"], s["v"]
    if kind == "window_decode":
        return flash_attention_sparse_decoding(s["q"], s["k"], s["v"], s["cu"], c["glob"], c["local"])
    if kind == "paged":
        return ops.paged_decode(s["q"], s["k"], s["v"], s["table"], s["lens"])
    if kind == "topk":
        idx, cnt = ops.topk_blocks(s["scores"], c["top_k"], force_last=1)
        return flash_attention_block_sparse_decoding(s["q"], s["k"], s["v"], s["cu"], idx, cnt), idx, cnt
    y = RMSNormTritonFunction.apply(s["x"], s["w"], 1e-6)
    return (y.detach(), *torch.autograd.grad(y, (s["x"], s["w"]), s["dy"]))


# ---------------------------------------------------------------------------- what a pass cannot do without
def _pairs_causal(n):
    return n * (n + 1) // 2


def _pairs_window(n, local, glob):
    """Visible (query, key) pairs: j <= i and (i - j < local or j < glob)."""
    def lower(m):       # sum over i < n of min(i + 1, m)
        m = min(m, n)
        return m * (m + 1) // 2 + (n - m) * m
    # keys of the prefix that the window has left behind: min(glob, i + 1 - local), where positive
    rest = max(n - local, 0)
    g = min(glob, rest)
    return lower(local) + g * (g + 1) // 2 + (rest - g) * g


def work(case):
    c = case
    kind = c["kind"]
    if kind == "rmsnorm":
        e = 4 if c["dtype"] == "fp32" else 2
        return {"bytes": 5.0 * c["rows"] * c["dim"] * e + 2.0 * c["dim"] * e, "flops": 12.0 * c["rows"] * c["dim"]}
    hq, hkv, d, b = c["hq"], c["hkv"], c["d"], c["batch"]
    if kind in ("prefill", "blocks"):
        n = c["seq"]
        if kind == "prefill":
            pairs = b * hq * (_pairs_causal(n) if c["causal"] else n * n)
            lists = 0
        else:
            nb = -(-n // BLOCK)
            m = min(c["local_blocks"], nb)
            near = m * (m + 1) // 2 + (nb - m) * m
            blocks = near + c["density"] * (_pairs_causal(nb) - near)
            pairs = b * hq * (blocks * BLOCK * BLOCK - nb * BLOCK * (BLOCK - 1) / 2)
            lists = 4.0 * b * hq * blocks
        return {"bytes": 2.0 * b * n * d * (2 * hq + 2 * hkv) + 4.0 * b * n * hq + lists, "flops": 4.0 * d * pairs}
    if kind in ("packed", "train", "window"):
        lens = _lens(c)
        t = sum(lens)
        pairs = hq * sum(_pairs_window(n, c["local"], c["glob"]) if kind == "window" else _pairs_causal(n)
                         for n in lens)
        if kind == "train":     # forward and backward: Q, K, V, dO in; O, dQ, dK, dV out; 2 + 5 products
            return {"bytes": 2.0 * t * d * (4 * hq + 4 * hkv), "flops": 14.0 * d * pairs}
        return {"bytes": 2.0 * t * d * (2 * hq + 2 * hkv) + 4.0 * t * hq, "flops": 4.0 * d * pairs}
    if kind == "topk":
        keys = b * c["top_k"] * BLOCK
        return {"bytes": 4.0 * keys * hkv * d + 4.0 * b * hq * d + 4.0 * b * hkv * (c["seq"] // BLOCK + c["top_k"] + 1),
                "flops": 4.0 * keys * hq * d}
    lens = _lens(c)
    if kind == "decode_step":
        lens = [n + 1 for n in lens]
    if kind == "window_decode":
        lens = [min(n, c["glob"] + c["local"]) for n in lens]
    keys = sum(lens)
    extra = 4.0 * b * hkv * d * 2 if kind == "decode_step" else 0.0
    return {"bytes": 4.0 * keys * hkv * d + 4.0 * b * hq * d + extra, "flops": 4.0 * keys * hq * d}


def tolerance(case):
    """About four times the largest errors measured against 64-bit math on the same inputs, over every
    kind of case (relative 2-norm / largest): bf16 3.2e-3 / 7.5e-2, fp16 3.2e-4 / 5.4e-3, fp32 4.3e-7 /
    1.9e-6.  The bf16 and fp16 figures are the rounding of P, dS and the results."""
    return {"bf16": {"rel": 1e-2, "max": 0.3}, "fp16": {"rel": 1.3e-3, "max": 2.2e-2},
            "fp32": {"rel": 1.7e-6, "max": 8e-6}}[case["dtype"]]


# ---------------------------------------------------------------------------- the same in 64 bits
def _attend(q, k, v, visible, scale, do=None):
    """Softmax attention of q [T, G, D] over k, v [N, D] in float64, `visible(r0, r1)` being the
    [1 or G, r1 - r0, N] mask of the rows: (o, natural-log lse), and with `do` also (dq, dk, dv)."""
    t, g, d = q.shape
    n = k.shape[0]
    q, k, v = q.double().transpose(0, 1), k.double(), v.double()
    o, lse = torch.empty_like(q), q.new_empty(g, t)
    if do is not None:
        do = do.double().transpose(0, 1)
        dq, dk, dv = torch.empty_like(q), torch.zeros_like(k), torch.zeros_like(v)
    step = max(1, (1 << 26) // (g * n))
    for r0 in range(0, t, step):
        r1 = min(t, r0 + step)
        s = (q[:, r0:r1] @ k.T).mul_(scale).masked_fill_(~visible(r0, r1), -math.inf)
        lse[:, r0:r1] = s.logsumexp(-1)
        p = s.sub_(lse[:, r0:r1, None]).exp_()
        o[:, r0:r1] = p @ v
        if do is not None:
            g_o = do[:, r0:r1]
            ds = (g_o @ v.T).sub_((g_o * o[:, r0:r1]).sum(-1, keepdim=True)).mul_(p).mul_(scale)
            dq[:, r0:r1] = ds @ k
            dk += (ds.transpose(1, 2) @ q[:, r0:r1]).sum(0)
            dv += (p.transpose(1, 2) @ g_o).sum(0)
    out = (o.transpose(0, 1), lse.T)
    return out + (dq.transpose(0, 1), dk, dv) if do is not None else out


def _visible(c, n, b, h):
    """Mask of the rows [r0, r1) of sequence b, head h, over its n keys."""
    j = torch.arange(n, device="cuda")
    if c["kind"] == "blocks":
        lists = c["idx"][b, h].long()
        nb = lists.shape[0]
        blocks = torch.zeros(nb, nb + 1, dtype=torch.bool, device="cuda")     # the last column takes the padding
        blocks.scatter_(1, torch.where(lists < 0, nb, lists), True)

    def mask(r0, r1):
        i = torch.arange(r0, r1, device="cuda")[:, None]
        if c["kind"] == "prefill" and not c["causal"]:
            return torch.ones(1, r1 - r0, n, dtype=torch.bool, device="cuda")
        m = j <= i
        if c["kind"] == "window":
            m = m & ((i - j < c["local"]) | (j < c["glob"]))
        elif c["kind"] == "blocks":
            m = m & blocks[i // BLOCK, j // BLOCK]
        return m[None]
    return mask


def exact(case, seed):
    """What `run(prepare(case, seed))` returns, computed by plain torch in 64 bits."""
    s = prepare(case, seed)
    c = s["case"]
    kind = c["kind"]
    if kind == "rmsnorm":
        x, w = (s[n].detach().double() for n in "xw")
        dy = s["dy"].double()
        r = (x.square().mean(-1, keepdim=True) + 1e-6).rsqrt()
        gw = dy * w
        return x * r * w, r * (gw - x * r * r * (gw * x).mean(-1, keepdim=True)), (dy * x * r).sum(0)
    g, scale = c["hq"] // c["hkv"], c["d"] ** -0.5
    if kind in ("prefill", "blocks", "packed", "train", "window"):
        q, k, v = (s[n].detach() for n in "qkv")
        do = s.get("do")
        if kind == "prefill":
            spans = [(b, 0, c["seq"]) for b in range(c["batch"])]
        else:
            at = s["cu"].tolist()
            spans = [(0, at[b], at[b + 1]) for b in range(c["batch"])]
        o, lse = q.new_empty(q.shape, dtype=torch.float64), q.new_empty(q.shape[:3], dtype=torch.float64)
        grads = [t.new_empty(t.shape, dtype=torch.float64) for t in (q, k, v)] if do is not None else []
        each = 1 if kind == "blocks" else g     # a block list belongs to one query head
        for b, (row, lo, hi) in enumerate(spans):
            for h in range(0, c["hq"], each):
                hs, hk = slice(h, h + each), h // g
                mask = _visible(dict(c, idx=s.get("idx")), hi - lo, b, h)
                r = _attend(q[row, lo:hi, hs], k[row, lo:hi, hk], v[row, lo:hi, hk], mask, scale,
                            do[row, lo:hi, hs] if do is not None else None)
                o[row, lo:hi, hs], lse[row, lo:hi, hs] = r[:2]
                if do is not None:
                    grads[0][row, lo:hi, hs], grads[1][row, lo:hi, hk], grads[2][row, lo:hi, hk] = r[2:]
        if kind == "train":
            return (o, *grads)
        return o, lse / math.log(2) if kind == "window" else lse
    k, v = s["k"], s["v"]
    if kind == "decode_step":
        lens = [n + 1 for n in _lens(c)]
        for b, n in enumerate(lens):
            k[b, n - 1], v[b, n - 1] = s["new_k"][b], s["new_v"][b]
    elif kind == "topk":
        lens = [c["seq"]] * c["batch"]
        scores = s["scores"].clone()
        scores[..., -1] = math.inf
        idx = scores.topk(c["top_k"], -1).indices.sort(-1).values
    else:
        lens = _lens(c)
    o = s["q"].new_empty(s["q"].shape, dtype=torch.float64)
    for b, n in enumerate(lens):
        if kind == "paged":
            at = s["table"][b, :-(-n // c["page"])].long()
            kb, vb = (t[at].flatten(0, 1)[:n] for t in (k, v))
        else:
            kb, vb = k[b, :n], v[b, :n]
        j = torch.arange(n, device="cuda")
        m = torch.ones(1, 1, n, dtype=torch.bool, device="cuda")
        if kind == "window_decode":
            m = ((j < c["glob"]) | (j >= n - c["local"]))[None, None]
        for h in range(c["hkv"]):
            if kind == "topk":
                listed_ = torch.zeros(n // BLOCK, dtype=torch.bool, device="cuda")
                listed_[idx[b, h]] = True
                m = listed_[j // BLOCK][None, None]
            o[b, h * g:(h + 1) * g] = _attend(s["q"][b:b + 1, h * g:(h + 1) * g], kb[:, h], vb[:, h],
                                              lambda r0, r1: m, scale)[0][0]
    if kind == "decode_step":
        return o, k.double(), v.double()
    if kind == "topk":
        return o, idx.int(), torch.full(idx.shape[:2], c["top_k"], dtype=torch.int32, device="cuda")
    return o

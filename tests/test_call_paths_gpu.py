"""The native call path against the Python one it stands before, the device-side schedule of packed
launches against single-sequence calls, and one-chunk decoding against split decoding."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ops():
    from tritonops_b200 import ops
    return ops


def _packed(lens, hq, hkv, d, dtype, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    q, k, v, do = (torch.randn(1, sum(lens), h, d, generator=g, device="cuda").to(dtype) for h in (hq, hkv, hkv, hq))
    return q, k, v, do, cu


# ragged batches on both sides of the schedule's limits: one lane per sequence (32), several chunks
# of sequences, more sequences than are handed out on the device (256), heads that do not fill a
# group of 8, tiles of exactly one, just under and just over 128 / 256 rows, empty sequences
@pytest.mark.parametrize("lens,hq,hkv,d", [
    ([256, 1, 0, 255, 257, 700, 128], 12, 12, 128),
    ([(37 * i) % 300 for i in range(45)], 4, 2, 64),
    ([1 + (91 * i) % 140 for i in range(260)], 2, 1, 64),
    ([3000, 17], 9, 3, 96),
])
def test_packed_schedule_equals_single_sequences(lens, hq, hkv, d):
    """Every tile of every sequence is computed exactly once: bit-equal to calls that hold one
    sequence each (a tile's arithmetic does not depend on which CTA runs it)."""
    ops = _ops()
    q, k, v, do, cu = _packed(lens, hq, hkv, d, torch.bfloat16)
    o, lse = ops.prefill(q, k, v, cu_seqlens=cu)
    om, lsem = ops.prefill(q, k, v, cu_seqlens=cu, max_seqlen=max(lens))
    assert torch.equal(o, om) and torch.equal(lse, lsem)
    dq, dk, dv = ops.prefill_bwd(q, k, v, o, do, lse, cu_seqlens=cu)
    at = cu.tolist()
    for b, n in enumerate(lens):
        if n == 0 or (len(lens) > 60 and b % 37):
            continue
        s = slice(at[b], at[b + 1])
        one = [t[:, s].contiguous() for t in (q, k, v, do)]
        o1, l1 = ops.prefill(*one[:3])
        assert torch.equal(o[:, s], o1) and torch.equal(lse[:, s], l1), (b, n)
        dq1, dk1, dv1 = ops.prefill_bwd(*one[:3], o1, one[3], l1)
        assert torch.equal(dk[:, s], dk1) and torch.equal(dv[:, s], dv1), (b, n)
        # dq is summed by reduce-adds in arrival order: one rounding of the 16-bit result
        assert (dq[:, s].float() - dq1.float()).abs().max() <= 2 ** -7 * dq1.float().abs().max()


# More tiles than two to an SM, so that CTAs take over a second and further items: whole and cut tiles in
# turn, empty sequences between them, both widths the kernel is built for (128: P over S; 64: P beside it)
# and both that are padded into one of them, causal and not, without and with the longest length; the last
# three of one length each, in CTAs that take over items and one to a CTA.
MANY = [256, 1, 0, 255, 257, 700, 128, 511, 30, 513, 384]


@pytest.mark.parametrize("lens,h,d,causal", [
    (MANY, 40, 128, True), (MANY, 40, 64, True), (MANY, 36, 96, False), (MANY, 36, 32, False), (MANY[::-1], 36, 128, False),
    ([300, 256, 129] * 5, 20, 128, True), ([300, 256, 129] * 5, 20, 64, False), ([300] * 15, 12, 128, True),
    ([300] * 15, 12, 96, False), ([700] * 5, 12, 64, True),
])
def test_taken_over_items_equal_single_sequences(lens, h, d, causal):
    ops = _ops()
    q, k, v, _, cu = _packed(lens, h, h // 4, d, torch.bfloat16, seed=2)
    at = cu.tolist()
    for kw in ({}, {"max_seqlen": max(lens)}):
        for _ in range(2):
            o, lse = ops.prefill(q, k, v, cu_seqlens=cu, causal=causal, **kw)
            for b, n in enumerate(lens):
                if n:
                    s = slice(at[b], at[b + 1])
                    o1, l1 = ops.prefill(*(t[:, s].contiguous() for t in (q, k, v)), causal=causal)
                    assert torch.equal(o[:, s], o1) and torch.equal(lse[:, s], l1), (b, n, kw)


@pytest.mark.parametrize("lens,causal", [([700, 129, 1, 0, 640], True), ([300] * 7, True), ([300, 256, 129] * 5, False),
                                         ([900] + [40] * 9, True)])
def test_backward_with_and_without_the_longest_length(lens, causal):
    """Handed out on the device, or by the grid of batch x longest where that is given and tight."""
    ops = _ops()
    q, k, v, do, cu = _packed(lens, 12, 6, 64, torch.float16, seed=5)
    o, lse = ops.prefill(q, k, v, cu_seqlens=cu, causal=causal)
    dq, dk, dv = ops.prefill_bwd(q, k, v, o, do, lse, cu_seqlens=cu, causal=causal)
    dqm, dkm, dvm = ops.prefill_bwd(q, k, v, o, do, lse, cu_seqlens=cu, causal=causal, max_seqlen=max(lens))
    assert torch.equal(dk, dkm) and torch.equal(dv, dvm)
    # dq is summed by reduce-adds in arrival order: one rounding of the 16-bit result
    assert (dq.float() - dqm.float()).abs().max() <= 2 ** -10 * dq.float().abs().max()


@pytest.mark.parametrize("d", [128, 64, 32])
@pytest.mark.parametrize("local,glob", [(64, 0), (100, 200), (1, 130), (0, 64), (300, 5), (0, 0)])
def test_taken_over_window_items_equal_single_sequences(d, local, glob):
    """Walks with a gap behind the global prefix, tiles that take no part in some steps, packed and of
    one length."""
    ops = _ops()
    win = dict(sparsity=ops.WINDOW, window_local=local, window_global=glob)
    lens, h = [700, 129, 1, 0, 513, 256, 900, 300, 64, 1025, 640, 333], 16
    q, k, v, _, cu = _packed(lens, h, h // 2, d, torch.bfloat16, seed=4)
    o, lse = ops.prefill(q, k, v, cu_seqlens=cu, **win)
    om, lsem = ops.prefill(q, k, v, cu_seqlens=cu, max_seqlen=max(lens), **win)
    assert torch.equal(o, om) and torch.equal(lse, lsem)
    at = cu.tolist()
    for b, n in enumerate(lens):
        if n:
            s = slice(at[b], at[b + 1])
            o1, l1 = ops.prefill(*(t[:, s].contiguous() for t in (q, k, v)), **win)
            assert torch.equal(o[:, s], o1) and torch.equal(lse[:, s], l1), (b, n)
    n, rows = 330, 11
    q, k, v = (t[:, :n * rows].reshape(rows, n, -1, d) for t in (q, k, v))
    o, lse = ops.prefill(q, k, v, **win)
    for b in range(rows):
        o1, l1 = ops.prefill(*(t[b:b + 1].contiguous() for t in (q, k, v)), **win)
        assert torch.equal(o[b:b + 1], o1) and torch.equal(lse[b:b + 1], l1), b


def test_packed_call_without_lengths_can_be_captured():
    """No length goes back to the host any more: the call fits into a CUDA graph."""
    ops = _ops()
    q, k, v, _, cu = _packed([100, 300], 4, 2, 128, torch.float16)
    want = ops.prefill(q, k, v, cu_seqlens=cu)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = ops.prefill(q, k, v, cu_seqlens=cu)
    graph.replay()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_native_calls_equal_python_calls(monkeypatch):
    """Same bits from both paths over the argument forms the native one takes, and the forms it
    leaves to Python (strided, other integer types, lengths on the CPU) still work."""
    ops = _ops()
    q, k, v, do, cu = _packed([70, 200, 33], 8, 2, 128, torch.bfloat16)
    wide = torch.cat([q, q], 3)[..., :128]                       # strided rows
    odd = torch.cat([q.new_zeros(1, q.shape[1], 8, 1), q], 3)[..., 1:]   # rows that are not 16-byte addressable
    kc, vc = (torch.randn(3, 300, 2, 128, device="cuda").bfloat16() for _ in range(2))
    qd, lens = q[0, :3].contiguous(), torch.tensor([300, 5, 64], dtype=torch.int32, device="cuda")
    table = torch.arange(15, device="cuda", dtype=torch.int32).view(3, 5).flip(1).contiguous()
    x, w = torch.randn(40, 512, device="cuda"), torch.rand(512, device="cuda")
    scores = torch.randn(2, 3, 40, device="cuda")

    def results():
        out = []
        for qq in (q, wide, odd):
            for c in (cu, cu.long(), cu.cpu()):
                out += ops.prefill(qq, k, v, cu_seqlens=c)
        o, lse = ops.prefill(q, k, v, cu_seqlens=cu, window_local=50, window_global=3, sparsity=ops.WINDOW)
        out += [o, lse, *ops.prefill_bwd(q, k, v, *[out[0]], do, out[1], cu_seqlens=cu)[1:]]
        out += ops.prefill(kc, kc, vc, causal=False, scale=0.2)
        out += [ops.decode(qd, kc, vc, seqlens=lens), ops.decode(qd, kc, vc, cu_seqlens=cu[:4].contiguous())]
        out.append(ops.paged_decode(qd, kc[:, :256].reshape(12, 64, 2, 128)[:12].repeat(2, 1, 1, 1)[:15],
                                    vc[:, :256].reshape(12, 64, 2, 128)[:12].repeat(2, 1, 1, 1)[:15], table, lens))
        k2, v2 = kc.clone(), vc.clone()
        ops.append_kv(k2, v2, k[0, :3].contiguous(), v[0, :3].contiguous(), lens)
        out += [k2, v2, *ops.topk_blocks(scores, 7, force_last=1), *ops.topk_blocks(scores[0, 0], 7)]
        for xx in (x, x.view(4, 10, 512), x[::2], x.bfloat16()):
            y, r = ops.rmsnorm_fwd(xx, w, 1e-6)
            out += [y, r, *ops.rmsnorm_bwd(y, xx, w, r)]
        return out

    real, answered = ops._native, {}

    def spy(name, *args):
        r = real(name, *args)
        answered.setdefault(name, []).append(r is not None)
        return r
    monkeypatch.setattr(ops, "_native", spy)
    native = results()
    n = ops.launch_counter
    ops.prefill(q, k, v, cu_seqlens=cu)
    assert ops.launch_counter == n + 1
    # who answered: plain arguments are taken natively, the other forms are not
    take = lambda name, *args, **kw: (answered.clear(), getattr(ops, name)(*args, **kw), answered[name] == [True])[2]
    idx = torch.zeros(3, 2, 1, dtype=torch.int32, device="cuda")
    nb = torch.zeros(1, 4, 5, 1, dtype=torch.int32, device="cuda")
    one = torch.tensor([0, 300], dtype=torch.int32, device="cuda")
    q1, k1, v1 = (t[:, :300].contiguous() for t in (q[:, :, :4], k, v))
    pages = kc[:, :256].reshape(12, 64, 2, 128)
    o, lse = ops.prefill(q, k, v, cu_seqlens=cu)
    y, r = ops.rmsnorm_fwd(x, w, 1e-6)
    assert take("prefill", q, k, v, cu_seqlens=cu) and take("prefill", q, k, v)
    assert take("prefill", wide, k, v, cu_seqlens=cu)           # strided rows the kernels can address
    assert take("prefill", q, k, v, cu_seqlens=cu, window_local=5, sparsity=ops.WINDOW)
    assert take("prefill", q1, k1, v1, cu_seqlens=one, max_seqlen=300, sparsity=ops.BLOCK_LIST, block_idx=nb,
                block_cnt=torch.ones_like(nb[..., 0]))
    assert take("prefill_bwd", q, k, v, o, do, lse, cu_seqlens=cu)
    assert take("decode", qd, kc, vc, seqlens=lens) and take("decode", qd, kc, vc, cu_seqlens=cu[:4].contiguous())
    assert take("decode", qd, kc, vc, seqlens=lens, sparsity=ops.BLOCK_LIST, block_idx=idx)
    assert take("paged_decode", qd, pages, pages, (table % 12), lens)
    assert take("append_kv", kc.clone(), vc.clone(), k[0, :3].contiguous(), v[0, :3].contiguous(), lens)
    assert take("topk_blocks", scores, 7) and take("rmsnorm_fwd", x, w, 1e-6) and take("rmsnorm_bwd", y, x, w, r)
    assert not take("prefill", odd, k, v, cu_seqlens=cu)        # rows that have to be copied first
    assert not take("prefill", q, k, v, cu_seqlens=cu.long()) and not take("prefill", q, k, v, cu_seqlens=cu.cpu())
    assert not take("decode", qd, kc, vc, seqlens=lens.long()) and not take("decode", qd, kc, vc, seqlens=lens.cpu())
    assert not take("rmsnorm_fwd", x.T, torch.rand(40, device="cuda"), 1e-6)
    monkeypatch.setattr(ops, "_native", lambda *a: None)
    python = results()
    assert len(native) == len(python)
    for i, (a, b) in enumerate(zip(native, python)):
        assert a.shape == b.shape and a.dtype == b.dtype and a.stride() == b.stride() and torch.equal(a, b), i


def test_native_calls_raise_what_python_calls_raise():
    ops = _ops()
    q, k, v, _, cu = _packed([64], 4, 4, 64, torch.float16)
    for bad, exc in [((q, k[..., :32], v), ValueError), ((q.float(), k, v), ValueError), ((q.cpu(), k, v), RuntimeError),
                     ((q, k[:, :, :3], v[:, :, :3]), ValueError)]:
        with pytest.raises(exc):
            ops.prefill(*bad, cu_seqlens=cu)
    with pytest.raises(ValueError):
        ops.prefill(q.repeat(2, 1, 1, 1), k, v, cu_seqlens=cu)


def test_first_call_of_a_thread_with_cached_memory():
    """A thread that has made no CUDA call yet, all of whose allocations come from the cache."""
    ops = _ops()
    q, k, v, do, cu = _packed([64], 2, 2, 64, torch.float16)
    o, lse = ops.prefill(q, k, v, cu_seqlens=cu)
    ops.prefill_bwd(q, k, v, o, do, lse, cu_seqlens=cu)
    torch.cuda.synchronize()
    for call in (lambda: ops.prefill(q, k, v, cu_seqlens=cu), lambda: ops.prefill_bwd(q, k, v, o, do, lse, cu_seqlens=cu),
                 lambda: ops.decode(q[0, :1], k, v, seqlens=cu[1:].contiguous())):
        failed = []

        def run():
            try:
                call()
            except Exception as e:      # noqa: BLE001 - whatever it is, the test reports it
                failed.append(e)
        t = threading.Thread(target=run)
        t.start()
        t.join()
        assert not failed, failed


@pytest.mark.parametrize("d,dtype", [(128, torch.bfloat16), (64, torch.float16)])
@pytest.mark.parametrize("lens", [[4096, 0, 1, 63, 64, 65, 4095], [130]])
def test_one_chunk_decoding_equals_split_decoding(d, dtype, lens):
    """max_seqlen within one chunk: the split kernel writes the output itself.  Against chunks of 64
    keys: fp32 partial sums in another order, one rounding of the result (values below 4)."""
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(1)
    B, cap = len(lens), max(lens)
    q = torch.randn(B, 8, d, generator=g, device="cuda").to(dtype)
    k, v = (torch.randn(B, cap, 2, d, generator=g, device="cuda").to(dtype) for _ in range(2))
    sl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    one = ops.decode(q, k, v, seqlens=sl, chunk=4096)
    many = ops.decode(q, k, v, seqlens=sl, chunk=64)
    tol = 2 ** (-7 if dtype == torch.bfloat16 else -10) * 4
    assert (one.float() - many.float()).abs().max() <= tol
    if 0 in lens:
        assert one[lens.index(0)].abs().max() == 0
    # more items than fit the chip at once: the CTAs take over those that have not started
    rep = 40
    big = ops.decode(q.repeat(rep, 1, 1), k.repeat(rep, 1, 1, 1), v.repeat(rep, 1, 1, 1), seqlens=sl.repeat(rep), chunk=64)
    assert torch.equal(big, many.repeat(rep, 1, 1))


@pytest.mark.parametrize("d,page", [(128, 16), (128, 64), (64, 64), (96, 48)])
def test_taken_over_paged_items_equal_a_small_batch(d, page):
    """More items than fit the chip at once, whole pages that lie in order or not: bit-equal to a batch
    that takes one item per CTA at the same split."""
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(7)
    lens = [1, 0, 1000, 63, 512, 999, 64, 700]
    B, per, rep = len(lens), -(-1024 // page), 12
    pool = B * per
    k, v = (torch.randn(pool, page, 2, d, generator=g, device="cuda").bfloat16() for _ in range(2))
    table = torch.arange(pool, dtype=torch.int32, device="cuda").view(B, per).clone()
    table[::2] = table[::2].flip(1)
    q, sl = torch.randn(B, 8, d, generator=g, device="cuda").bfloat16(), torch.tensor(lens, dtype=torch.int32, device="cuda")
    small = ops.paged_decode(q, k, v, table, sl, chunk=128)
    big = ops.paged_decode(q.repeat(rep, 1, 1), k, v, table.repeat(rep, 1), sl.repeat(rep), chunk=128)
    assert torch.equal(big, small.repeat(rep, 1, 1))


@pytest.mark.parametrize("glob,local", [(64, 300), (0, 129), (128, 64)])
@pytest.mark.parametrize("d", [128, 64])
def test_taken_over_window_decoding_equals_a_small_batch(d, glob, local):
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(8)
    lens, rep = [1, 0, 1000, 63, 512, 999, 130, 700], 24
    q = torch.randn(len(lens), 8, d, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(len(lens), 1000, 2, d, generator=g, device="cuda").bfloat16() for _ in range(2))
    sl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    kw = dict(sparsity=ops.WINDOW, window_global=glob, window_local=local, chunk=64)
    small = ops.decode(q, k, v, seqlens=sl, **kw)
    big = ops.decode(q.repeat(rep, 1, 1), k.repeat(rep, 1, 1, 1), v.repeat(rep, 1, 1, 1), seqlens=sl.repeat(rep), **kw)
    assert torch.equal(big, small.repeat(rep, 1, 1))

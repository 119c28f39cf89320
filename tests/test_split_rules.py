"""The automatic split of decoding, seen through the scratch it asks for (no GPU)."""
import ctypes as C
import random

import pytest


@pytest.fixture(scope="module")
def lib():
    from tritonops_b200 import _lib
    return _lib.lib()


def _chunks(lib, **kw):
    """Number of chunks the library splits the longest sequence into."""
    from tritonops_b200._lib import DecodeArgs
    a = DecodeArgs(head_dim=128, **kw)
    return lib.b200attn_decode_workspace_bytes(C.byref(a)) // (kw["batch"] * kw["heads_q"] * (128 * 4 + 4))


def _longest_chunk_filling_the_chip(units, visible):
    for c in (8192, 4096, 2048, 1024, 512, 256, 128):
        if units * -(-visible // c) >= 148:
            return c
    return 128


def test_fixed_scratch_takes_what_long_chunks_would_fit(lib):
    """b200attn_decode_fwd_noalloc has a fixed array: a dense problem whose partials fit it with the
    longest chunks that fill the chip still fits with the chunks chosen for balance."""
    from tritonops_b200 import _lib
    rng = random.Random(0)
    seen = 0
    for _ in range(3000):
        hkv = rng.choice([1, 2, 4, 8, 16, 32])
        hq = hkv * rng.choice([1, 2, 4, 8, 16, 32])
        batch, visible = rng.randint(1, 300), int(2 ** rng.uniform(5, 20))
        units = batch * hkv * -(-(hq // hkv) // 16)
        chunk = 2048 if units >= 256 else _longest_chunk_filling_the_chip(units, visible)
        row = batch * hq * (128 * 4 + 4)
        if row * -(-visible // chunk) > _lib.NOALLOC_SCRATCH_BYTES:
            continue
        n = _chunks(lib, batch=batch, heads_q=hq, heads_kv=hkv, max_seqlen=visible)
        assert n * row <= _lib.NOALLOC_SCRATCH_BYTES, (batch, hq, hkv, visible, n)
        seen += 64 <= units < 256
    assert seen > 100


@pytest.mark.parametrize("batch,hkv,blocks,want", [
    (8, 32, 64, 1),      # 256 units of 64 stages fill most of one wave: no split
    (16, 32, 33, 1),     # two waves of whole units beat four of halves
    (2, 8, 40, 14),      # 16 units: 14 chunks of 3 stages are one wave
    (1, 1, 1, 1),
    (1, 300, 64, None),  # 300 units would be two waves of whole units: more, shorter waves
])
def test_block_lists_are_split_by_waves(lib, batch, hkv, blocks, want):
    n = _chunks(lib, batch=batch, heads_q=hkv, heads_kv=hkv, max_seqlen=1 << 20, sparsity=2, block_size=64,
                max_sel=blocks)
    if want is not None:
        assert n == want
    slots, stages, units = 296, blocks, batch * hkv
    cost = lambda c: -(-units * c // slots) * (-(-stages // c) + 3)
    assert cost(n) == min(cost(c) for c in range(1, min(stages, 128) + 1))


@pytest.mark.parametrize("batch,hkv,visible,want", [
    (8, 8, 1024, 1), (8, 8, 2048, 4),        # 64 units: one chunk, then 4 x 64 = 256 items in one wave
    (12, 8, 4096, 3), (24, 8, 2048, 3),      # 96 x 3 = 288 items, not 384; 576 items in two waves, not 384
    (24, 8, 5900, 6), (16, 8, 32768, 16),    # 1024 keys; 2048 beyond 8192
])
def test_splits_of_a_medium_batch_fill_their_waves(lib, batch, hkv, visible, want):
    assert _chunks(lib, batch=batch, heads_q=4 * hkv, heads_kv=hkv, max_seqlen=visible) == want


def test_short_block_lists_are_not_split(lib):
    """A second kernel costs more than two or three stages of the first save."""
    for batch, blocks in [(16, 4), (8, 8)]:
        assert _chunks(lib, batch=batch, heads_q=32, heads_kv=8, max_seqlen=1 << 20, sparsity=2, block_size=64,
                       max_sel=blocks) == 1

"""Inputs of up to 8 blocks per head run as a thread-block cluster per head, longer ones as a look-back chain: both sides of
the line, alone and as appends behind what the other one left, bit for bit against the oracle."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
HEADS = 3


def bits16(a):
    return np.ascontiguousarray(a).view(np.uint16)


def source(blocks, kind, seed):
    x = oracle.make_kv(HEADS, 64 * blocks, seed=seed)[kind]
    x[0, :5] = 0                                # empty tiles
    return x, oracle.prune_ref(x, 0.7)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("parts", [(1,), (7,), (8,), (9,), (1, 8, 9), (9, 8, 10, 1)])
def test_fp16(parts, kind):
    from mustafar_b200 import compression as c
    x, pruned = source(sum(parts), kind, 20 + kind)
    store = c.SparseStore(HEADS, x.shape[1], kind, "cuda")
    t = 0
    for n in parts:
        store.append(x[:, t:t + 64 * n].cuda(), c.keep_rank(0.7))
        t += 64 * n
    store.check()
    bm, acc, packed = (oracle.compress_value_ref if kind else oracle.compress_key_ref)(pruned)
    assert np.array_equal(store.bitmaps.cpu().numpy(), bm) and np.array_equal(store.accum.cpu().numpy(), acc)
    for h in range(HEADS):
        assert np.array_equal(bits16(store.nz[h, :len(packed[h])].cpu().numpy()), bits16(packed[h]))


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("bits,group", [(2, 64), (2, 32), (4, 64), (4, 32)])
@pytest.mark.parametrize("parts", [(1,), (7,), (8,), (9,), (1, 8, 9), (9, 8, 10, 1)])
def test_quantised(parts, bits, group, kind):
    from mustafar_b200 import compression as c, compression_quant as cq
    x, pruned = source(sum(parts), kind, 30 + kind)
    ref = (oracle.quant_compress_value_ref if kind else oracle.quant_compress_key_ref)(pruned, bits, group)
    T = 2 * x.shape[1]
    offsets, words = np.asarray(ref["tile_offsets"]).reshape(HEADS, T), np.asarray(ref["packed"])
    n = np.asarray(ref["units"]).reshape(HEADS, T)
    store = cq.QuantStore(HEADS, x.shape[1], kind, "cuda", bits, group)
    t = 0
    for b in parts:
        store.append(x[:, t:t + 64 * b].cuda(), c.keep_rank(0.7))
        t += 64 * b
    store.check()
    got = store.as_dict()
    for name in ("bitmaps", "counts", "units", "scales", "zeros"):
        a, b = got[name].cpu().numpy().reshape(-1), np.asarray(ref[name]).reshape(-1)
        assert np.array_equal(bits16(a) if a.dtype == np.float16 else a, bits16(b) if b.dtype == np.float16 else b), name
    assert np.array_equal(store.head_tail.cpu().numpy(), n.sum(1))
    flat, at = got["packed"].cpu().numpy(), got["tile_offsets"].cpu().numpy()
    start = flat.size // HEADS
    for h in range(HEADS):      # a head's tiles follow one another from its part of the arena on
        assert np.array_equal(at[h], h * start + np.concatenate([[0], np.cumsum(n[h])[:-1]]))
        lo = offsets[h, 0]
        assert np.array_equal(flat[h * start:h * start + n[h].sum()], words[lo:lo + n[h].sum()])
    # one head alone takes the same two routes in the compact layout
    one = cq.compress_quant(x[:1].cuda(), kind, c.keep_rank(0.7), bits, group)
    assert np.array_equal(one["packed"].cpu().numpy()[:n[0].sum()], words[offsets[0, 0]:offsets[0, 0] + n[0].sum()])
    assert np.array_equal(one["tile_offsets"].cpu().numpy().reshape(-1), at[0])

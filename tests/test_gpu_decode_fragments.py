"""Decoded tiles as tensor-core fragments, at the tile fills where the expansion can go wrong: empty and full tiles, one
value more or less than a byte, a code word or a scale group holds, and zero-points far outside the code range.
2e-3 rel L2: results, probabilities and dequantised values are fp16 (half an ulp is 2^-12 each), sums are fp32."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
TOL = 2e-3
FILLS = [0, 1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 34, 40, 47, 48, 63, 64]


def tiles_with_fills(heads, tokens, kind, offset, seed):
    """[heads, tokens, 128] fp16 whose tiles hold FILLS nonzeros at random positions, values around `offset`."""
    rng = np.random.default_rng(seed)
    n_tiles = heads * 2 * tokens
    x = np.zeros((n_tiles, 64), np.float16)
    for t in range(n_tiles):
        n = FILLS[(t * 5 + t // 31) % len(FILLS)]
        x[t, rng.permutation(64)[:n]] = (rng.standard_normal(n) + offset).astype(np.float16)
    if kind == "key":       # tile = channel down 64 tokens
        x = x.reshape(heads, tokens // 64, 128, 64).transpose(0, 1, 3, 2)
    else:                   # tile = (half, token), 64 channels
        x = x.reshape(heads, tokens // 64, 2, 64, 64).transpose(0, 1, 3, 2, 4)
    return torch.from_numpy(np.ascontiguousarray(x).reshape(heads, tokens, 128))


@pytest.mark.parametrize("offset", [0.0, 300.0])     # 300: zero-points in the hundreds and beyond
@pytest.mark.parametrize("bits,group", [(2, 64), (2, 32), (4, 64), (4, 32)])
@pytest.mark.parametrize("G", [1, 2, 4, 8])
def test_quantised_tiles(G, bits, group, offset):
    from mustafar_b200 import compression as c, compression_quant as cq, ops, ops_quant
    heads, L = 2, 320
    k, v = tiles_with_fills(heads, L, "key", offset, 1), tiles_with_fills(heads, L, "value", offset, 2)
    kq, vq = (cq.compress_quant(x.cuda(), kind, 0, bits, group) for x, kind in ((k, c.KEY), (v, c.VALUE)))
    kd = oracle.dequant_key_ref(oracle.quant_compress_key_ref(k, bits, group), L, bits=bits, group=group)
    vd = oracle.dequant_value_ref(oracle.quant_compress_value_ref(v, bits, group), L, bits=bits, group=group)
    q = oracle.make_query(heads * G, seed=3) * (0.05 if offset else 0.5)    # scores spread over many tokens
    win = torch.zeros(heads, 0, 128)
    want = oracle.decode_attention_ref(q, kd, vd, win, win, G)
    got = ops_quant.decode_attention_quant(q.half().cuda(), kq, vq, L, None, None, G, bits)
    ops.check_device_status()
    assert oracle.rel_l2(got.float().cpu(), want) < TOL


@pytest.mark.parametrize("G", [1, 2, 4, 8])
@pytest.mark.parametrize("L", [64, 320])
def test_fp16_tiles(G, L):
    from mustafar_b200 import compression as c, ops
    heads = 2
    k, v = tiles_with_fills(heads, L, "key", 0.0, 4), tiles_with_fills(heads, L, "value", 0.0, 5)
    ks, vs = (c.SparseStore(heads, L, kind, "cuda") for kind in (c.KEY, c.VALUE))
    ks.append(k.cuda()), vs.append(v.cuda())
    q = (oracle.make_query(heads * G, seed=6) * 0.5).half()
    win = torch.zeros(heads, 0, 128)
    got = ops.decode_attention(q.cuda(), ks, vs, None, None, G)
    assert oracle.rel_l2(got.float().cpu(), oracle.decode_attention_ref(q, k, v, win, win, G)) < TOL
    # the two products by themselves, over the compact layout
    bm, acc, packed = c.convert_key_batched(k.cuda())
    off = torch.tensor(np.cumsum([0] + [p.numel() // 8 for p in packed[:-1]]), dtype=torch.int32, device="cuda")
    q8 = torch.nn.functional.pad(q.cuda().view(heads * G, 1, 128), (0, 0, 0, 7))
    s = ops.mustafar_key_formulation(bm, torch.cat(packed), acc, off, q8, L, 128, heads * G, G)
    assert oracle.rel_l2(s[:, 0].cpu(), oracle.key_formulation_ref(k, q, G)) < TOL
    assert not s[:, 1:].any()
    bm, acc, packed = c.convert_value_batched(v.cuda())
    off = torch.tensor(np.cumsum([0] + [p.numel() // 8 for p in packed[:-1]]), dtype=torch.int32, device="cuda")
    pr = torch.softmax(torch.randn(heads * G, L, generator=torch.Generator().manual_seed(7)), -1).half()
    p8 = torch.nn.functional.pad(pr.cuda().view(heads * G, 1, L), (0, 0, 0, 7))
    o = ops.mustafar_value_formulation(bm, torch.cat(packed), acc, off, p8, torch.zeros(1).half().cuda(), 128, L, heads * G, G)
    assert oracle.rel_l2(o[:, 0].cpu(), oracle.value_formulation_ref(v, pr, G)) < TOL
    assert not o[:, 1:].any()
    ops.check_device_status()


# window CTAs of one block; of several only at W = 1100 and in the smallest workspace (test_gpu_window_split.py has the rest)
@pytest.mark.parametrize("heads,L", [(2, 0), (2, 192), (300, 64)])
@pytest.mark.parametrize("W", [1, 63, 64, 65, 129, 300, 1100])
@pytest.mark.parametrize("bits", [16, 2])
def test_window_split(heads, L, W, bits):
    from mustafar_b200 import compression as c, compression_quant as cq, ops, ops_quant
    G = 4
    k, v = oracle.make_kv(heads, max(L, 64) + W, seed=8)
    q = oracle.make_query(heads * G, seed=9)
    kc, vc, kw, vw = k[:, :L].contiguous(), v[:, :L].contiguous(), k[:, max(L, 64):].contiguous(), v[:, max(L, 64):].contiguous()
    capacity = W + 70                       # a window buffer longer than the valid part, its length on the device
    kb, vb = (torch.full((heads, capacity, 128), float("nan"), dtype=torch.float16) for _ in range(2))
    kb[:, :W], vb[:, :W] = kw, vw
    wl = torch.tensor([W], dtype=torch.int32, device="cuda")
    sample = [0, heads // 2, heads - 1]
    rows = [h * G + g for h in sample for g in range(G)]
    if bits == 16:
        ks, vs = (c.SparseStore(heads, max(L, 64), kind, "cuda") for kind in (c.KEY, c.VALUE))
        if L:
            ks.append(kc.cuda()), vs.append(vc.cuda())
        least = ops.plan(heads, L, 0, G)[1]
        small = ops.new_workspace(torch.device("cuda", 0), least)[:least]
        got = [ops.decode_attention(q.cuda(), ks, vs, kw.cuda(), vw.cuda(), G),
               ops.decode_attention(q.cuda(), ks, vs, kb.cuda(), vb.cuda(), G, window_len=wl),
               ops.decode_attention(q.cuda(), ks, vs, kw.cuda(), vw.cuda(), G, workspace=small)]
        want = oracle.decode_attention_ref(q[rows], kc[sample], vc[sample], kw[sample], vw[sample], G)
    else:
        if not L:
            pytest.skip("covered with the fp16 cache")
        kq, vq = cq.compress_quant(kc.cuda(), c.KEY), cq.compress_quant(vc.cuda(), c.VALUE)
        kd = oracle.dequant_key_ref(oracle.quant_compress_key_ref(kc[sample]), L)
        vd = oracle.dequant_value_ref(oracle.quant_compress_value_ref(vc[sample]), L)
        got = [ops_quant.decode_attention_quant(q.cuda(), kq, vq, L, kw.cuda(), vw.cuda(), G),
               ops_quant.decode_attention_quant(q.cuda(), kq, vq, L, kb.cuda(), vb.cuda(), G, window_len=wl)]
        want = oracle.decode_attention_ref(q[rows], kd, vd, kw[sample], vw[sample], G)
    ops.check_device_status()
    for out in got:
        assert oracle.rel_l2(out[rows].float().cpu(), want) < TOL

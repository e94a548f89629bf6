"""An infinity or a NaN in the cache, the window, the query or the probabilities reaches its own row of a product (token of
S = K q, channel of O = V^T p) and no other.  The expected results come from dense fp32 products of the same tensors; the
single products of the fp16 cache multiply the values that are there and nothing else.
2e-3 rel L2 over the finite part: results and probabilities are fp16 (half an ulp is 2^-12 each), sums are fp32."""
import math

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
TOL = 2e-3
INF, NAN = math.inf, math.nan
HEADS, L, W = 2, 192, 70


def same(got, want):
    """Every non-finite entry in its place, the others within the tolerance."""
    got, want = got.float().cpu(), want.float()
    ok = torch.isfinite(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(got[~ok & ~torch.isnan(want)], want[~ok & ~torch.isnan(want)])
    assert ok.any() and oracle.rel_l2(got[ok], want[ok]) < TOL


def inputs(group, seed=0):
    k, v = (x[:, :L + W].clone() for x in oracle.make_kv(HEADS, L + W, seed=seed))
    k, v = (oracle.prune_ref(x, 0.5) for x in (k, v))
    return k, v, (oracle.make_query(HEADS * group, seed=seed + 1) * 0.5).half()


def stores(k, v):
    from mustafar_b200 import compression as c
    ks, vs = c.SparseStore(HEADS, L, c.KEY, "cuda"), c.SparseStore(HEADS, L, c.VALUE, "cuda")
    ks.append(k[:, :L].contiguous().cuda()), vs.append(v[:, :L].contiguous().cuda())
    return ks, vs


@pytest.mark.parametrize("group", [1, 2, 4, 8])
@pytest.mark.parametrize("bad", [INF, -INF, NAN])
@pytest.mark.parametrize("where", ["k", "v", "window k", "window v", "q"])
def test_fused_fp16(where, bad, group):
    from mustafar_b200 import ops
    k, v, q = inputs(group)
    q[:, 9] = 1.0                              # the score of a token with -inf in channel 9 is -inf for every head
    for i, t in enumerate((3, 68, 131) if "window" not in where else (L + 5, L + 66)):
        if "k" in where:
            k[0, t, 9] = bad
        elif "v" in where:
            v[0, t, (9, 20, 127)[i]] = bad
    if where == "q":
        q[0, 9] = bad
    ks, vs = stores(k, v)
    got = ops.decode_attention(q.cuda(), ks, vs, k[:, L:].cuda(), v[:, L:].cuda(), group)
    ops.check_device_status()
    same(got, oracle.decode_attention_ref(q, k[:, :L], v[:, :L], k[:, L:], v[:, L:], group))


@pytest.mark.parametrize("group", [1, 2, 4, 8])
@pytest.mark.parametrize("bits,qgroup", [(2, 64), (2, 32), (4, 64), (4, 32)])
@pytest.mark.parametrize("where", ["k", "v", "window v"])
def test_fused_quantised(where, bits, qgroup, group):
    """A tile whose scale is infinite: its values are +inf (the zero-point lies below the codes)."""
    from mustafar_b200 import compression as c, compression_quant as cq, ops, ops_quant
    k, v, q = inputs(group, seed=3)
    q[:, 9] = -1.0                             # +inf in channel 9 of K gives scores of -inf
    kc, vc = k[:, :L].contiguous(), v[:, :L].contiguous()
    kq, vq = cq.compress_quant(kc.cuda(), c.KEY, 0, bits, qgroup), cq.compress_quant(vc.cuda(), c.VALUE, 0, bits, qgroup)
    kr, vr = oracle.quant_compress_key_ref(kc, bits, qgroup), oracle.quant_compress_value_ref(vc, bits, qgroup)
    if where == "window v":
        v[0, L + 3, 17] = v[0, L + 69, 100] = INF
    else:
        # K: channel 9 of the second block; V: channels 64.. of token 5 of the third
        tile = 128 + 9 if where == "k" else 256 + 64 + 5
        for t, r in ((kq, kr),) if where == "k" else ((vq, vr),):
            t["scales"].view(HEADS, 2 * L, -1)[0, tile] = INF
            t["zeros"].view(HEADS, 2 * L, -1)[0, tile] = -1
            r["scales"].reshape(HEADS, 2 * L, -1)[0, tile] = np.inf
            r["zeros"].reshape(HEADS, 2 * L, -1)[0, tile] = -1
    kd, vd = oracle.dequant_key_ref(kr, L, bits=bits, group=qgroup), oracle.dequant_value_ref(vr, L, bits=bits, group=qgroup)
    want = oracle.decode_attention_ref(q, kd, vd, k[:, L:], v[:, L:], group)
    assert torch.isfinite(want[0]).any() and (where == "k" or torch.isinf(want[0]).any())
    got = ops_quant.decode_attention_quant(q.cuda(), kq, vq, L, k[:, L:].cuda(), v[:, L:].cuda(), group, bits)
    ops.check_device_status()
    same(got, want)


@pytest.mark.parametrize("group", [1, 2, 4, 8])
@pytest.mark.parametrize("bad", [INF, -INF, NAN])
@pytest.mark.parametrize("where", ["cache", "operand"])
def test_fp16_products(where, bad, group):
    from mustafar_b200 import compression as c, ops
    k, v, q = inputs(group, seed=5)
    k, v = k[:, :L].contiguous(), v[:, :L].contiguous()
    p = torch.softmax(torch.randn(HEADS * group, L, generator=torch.Generator().manual_seed(7)), -1).half()
    if where == "cache":
        k[0, 3, 9] = k[0, 68, 9] = v[0, 131, 20] = v[0, 4, 127] = bad
    else:
        q[0, 9] = p[0, 131] = bad

    def product(a, b):    # [heads, rows, n] x [heads * group, n], absent positions take no part
        a, b = a.float()[:, None], b.float().view(HEADS, group, 1, -1)
        return torch.where(a != 0, a * b, torch.zeros(())).sum(-1).view(HEADS * group, -1)

    def compact(converted):
        bm, acc, packed = converted
        off = torch.tensor(np.cumsum([0] + [x.numel() // 8 for x in packed[:-1]]), dtype=torch.int32, device="cuda")
        return bm, torch.cat(packed), acc, off

    q8 = torch.nn.functional.pad(q.cuda().view(-1, 1, 128), (0, 0, 0, 7))
    s = ops.mustafar_key_formulation(*compact(c.convert_key_batched(k.cuda())), q8, L, 128, HEADS * group, group)
    same(s[:, 0], product(k, q))
    assert not s[:, 1:].any()
    p8 = torch.nn.functional.pad(p.cuda().view(-1, 1, L), (0, 0, 0, 7))
    o = ops.mustafar_value_formulation(*compact(c.convert_value_batched(v.cuda())), p8, torch.zeros(1).half().cuda(), 128, L,
                                       HEADS * group, group)
    same(o[:, 0], product(v.transpose(1, 2), p))
    assert not o[:, 1:].any()
    ops.check_device_status()

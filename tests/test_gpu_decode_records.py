"""Split counts at the ends of their range: more records than the fused kernel's merge has room for, and hints beyond the
largest count."""
import math

import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [496, 512, 700])       # of 256 blocks; one window record more
def test_one_head_so_long_that_its_records_are_merged_by_a_second_launch(splits):
    """An empty cache (no value is kept, every score is 0) in front of a window: 700 splits are 11.5 million tokens."""
    from mustafar_b200 import compression as c, ops
    G, W, L = 8, 64, 64 * 256 * splits
    ks, vs = (c.SparseStore(1, L, kind, "cuda", nz_capacity=8) for kind in (c.KEY, c.VALUE))
    for s in (ks, vs):
        s.bitmaps.zero_(), s.nz.zero_()
        s.tokens = L
    assert ops.plan(1, L, W, G, 1)[0] == splits
    kw, vw = oracle.make_kv(1, W, seed=1, outliers=False)
    kw[..., 0] = 14.0
    q = oracle.make_query(G, seed=2)
    q[:, 0] = 12.0                                        # scores around 15: as much weight as the empty tokens together
    out = ops.decode_attention(q.cuda(), ks, vs, kw.cuda(), vw.cuda(), G, nsplit=1)
    ops.check_device_status()
    w = torch.exp(q.double() @ kw[0].double().T / math.sqrt(128))
    want = w @ vw[0].double() / (L + w.sum(1, keepdim=True))
    assert oracle.rel_l2(out.cpu(), want) < 2e-3         # fp16 result and probabilities, fp32 sums


@pytest.mark.parametrize("blocks,hint", [(480, 480), (600, 600), (960, 4096)])
@pytest.mark.parametrize("bits", [16, 2])
def test_split_hints_beyond_the_largest_count(bits, blocks, hint):
    from mustafar_b200 import compression as c, compression_quant as cq, ops, ops_quant
    G, W, L = 4, 200, 64 * blocks
    k, v = oracle.make_kv(1, L + W, seed=3)
    q = oracle.make_query(G, seed=4).cuda()
    kw, vw = k[:, L:].cuda(), v[:, L:].cuda()
    kc, vc = k[:, :L].contiguous().cuda(), v[:, :L].contiguous().cuda()
    rank = c.keep_rank(0.7)
    if bits == 16:
        ks, vs = (c.SparseStore(1, L, kind, "cuda") for kind in (c.KEY, c.VALUE))
        ks.append(kc, rank), vs.append(vc, rank)
        call = lambda n: ops.decode_attention(q, ks, vs, kw, vw, G, nsplit=n)  # noqa: E731
    else:
        kq, vq = cq.compress_quant(kc, c.KEY, rank), cq.compress_quant(vc, c.VALUE, rank)
        call = lambda n: ops_quant.decode_attention_quant(q, kq, vq, L, kw, vw, G, nsplit=n)  # noqa: E731
    got, want = call(hint), call(0)
    ops.check_device_status()
    assert ops.plan(1, L, W, G, hint)[0] <= 480
    assert oracle.rel_l2(got.cpu(), want.cpu()) < 1e-3   # other partial sums, rounded to fp16 once

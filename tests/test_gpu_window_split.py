"""How many CTAs share the dense window (read off the records a call writes), and its result where they have several blocks
each, a short one at the end, or none because the window is shorter than its buffer.  2e-3 rel L2 as everywhere: fp16 results
and probabilities, fp32 sums."""
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
TOL = 2e-3


def calls(heads, G, L, capacity, bits, nsplit, seed):
    """Inputs on the host and call(window_len, workspace) over a window buffer of `capacity` tokens."""
    from mustafar_b200 import compression as c, compression_quant as cq, ops, ops_quant
    k, v = oracle.make_kv(heads, L + capacity, seed=seed, outliers=False)
    q = oracle.make_query(heads * G, seed=seed + 1)
    kc, vc, kw, vw = k[:, :L].contiguous(), v[:, :L].contiguous(), k[:, L:].contiguous(), v[:, L:].contiguous()
    dev = [x.cuda() for x in (q, kw, vw)]
    if bits == 16:
        ks, vs = (c.SparseStore(heads, L, kind, "cuda") for kind in (c.KEY, c.VALUE))
        ks.append(kc.cuda()), vs.append(vc.cuda())
        call = lambda wl, ws: ops.decode_attention(dev[0], ks, vs, *dev[1:], G, nsplit=nsplit, window_len=wl, workspace=ws)  # noqa: E731
    else:
        kq, vq = cq.compress_quant(kc.cuda(), c.KEY, 0, bits), cq.compress_quant(vc.cuda(), c.VALUE, 0, bits)
        call = lambda wl, ws: ops_quant.decode_attention_quant(dev[0], kq, vq, L, *dev[1:], G, bits, nsplit=nsplit,  # noqa: E731
                                                               window_len=wl, workspace=ws)
    return call, (q, kc, vc, kw, vw)


def expected(inputs, G, L, bits, W, sample):
    q, kc, vc, kw, vw = inputs
    kc, vc = kc[sample], vc[sample]
    if bits != 16:
        kc = oracle.dequant_key_ref(oracle.quant_compress_key_ref(kc, bits), L, bits=bits)
        vc = oracle.dequant_value_ref(oracle.quant_compress_value_ref(vc, bits), L, bits=bits)
    rows = [h * G + g for h in sample for g in range(G)]
    return rows, oracle.decode_attention_ref(q[rows], kc, vc, kw[sample, :W], vw[sample, :W], G)


def records(heads, G, call):
    from mustafar_b200 import ops
    room = 65536 + heads * 520 * G * 132 * 4
    ws = ops.new_workspace(torch.device("cuda", 0), room)
    ws[65536:] = 0xff                                                    # NaN
    call(None, ws)
    ops.check_device_status()
    written = ~torch.isnan(ws[65536:room].view(torch.float32).view(-1, 132)[:, 128])    # a record's running maximum
    n = int(written.sum())
    assert n % (heads * G) == 0 and written[:n].all()
    return n // (heads * G)


# (kv heads, tokens, window, splits): window CTAs on 148 SMs
@pytest.mark.parametrize("heads,L,W,nsplit,want", [
    (8, 10240, 128, 54, 1),     # 440 CTAs are 3 per SM; one more per head would leave a few SMs with 4
    (8, 1024, 200, 16, 4),      # 136 CTAs are one per SM, but a window in one CTA would outlast the splits by far
    (8, 1024, 384, 16, 6),
    (16, 1536, 200, 6, 2),      # 128 CTAs are one per SM still: half of a split's 4 blocks each
    (16, 2048, 200, 8, 1),      # 144 are, 160 are not, and one window CTA is no longer than a split
    (600, 512, 300, 1, 2),      # beyond 4 per SM: half a split's 8 blocks each, the last one short
    (8, 0, 300, 0, 5),
])
def test_ctas(heads, L, W, nsplit, want):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the rule depends on the number of SMs")
    from mustafar_b200 import compression as c, ops
    G = 1
    ks, vs = (c.SparseStore(heads, max(L, 64), kind, "cuda", nz_capacity=8) for kind in (c.KEY, c.VALUE))
    for s in (ks, vs):
        s.bitmaps.zero_(), s.nz.zero_()
        s.tokens = L
    q = torch.zeros(heads, 128, dtype=torch.float16, device="cuda")
    w = torch.zeros(heads, W, 128, dtype=torch.float16, device="cuda")
    n = records(heads, G, lambda wl, ws: ops.decode_attention(q, ks, vs, w, w, G, nsplit=nsplit, workspace=ws))
    assert n - nsplit == want


@pytest.mark.parametrize("bits", [16, 2])
@pytest.mark.parametrize("capacity", [300, 383])
def test_several_blocks_per_cta(capacity, bits):
    from mustafar_b200 import ops
    heads, G, L, nsplit = 600, 1, 512, 1
    call, inputs = calls(heads, G, L, capacity, bits, nsplit, seed=11)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert records(heads, G, call) == 1 + 2
    sample = [0, 299, 599]
    for W in (None, 1, 64, 255, 256, 257, capacity):                     # 256 tokens fill the first CTA, the second is empty
        wl = None if W is None else torch.tensor([W], dtype=torch.int32, device="cuda")
        rows, want = expected(inputs, G, L, bits, W or capacity, sample)
        assert oracle.rel_l2(call(wl, None)[rows].float().cpu(), want) < TOL
    ops.check_device_status()


@pytest.mark.parametrize("bits", [16, 2, 4])
def test_smallest_workspace(bits):
    """A workspace with room for one window record: one CTA takes the whole window."""
    from mustafar_b200 import ops
    heads, G, L, W, nsplit = 3, 4, 256, 300, 4
    call, inputs = calls(heads, G, L, W, bits, nsplit, seed=13)
    least = 65536 + heads * (nsplit + 1) * G * 132 * 4 + 16
    ws = ops.new_workspace(torch.device("cuda", 0), least)
    ws[least:] = 0x5a
    rows, want = expected(inputs, G, L, bits, W, list(range(heads)))
    assert oracle.rel_l2(call(None, ws[:least])[rows].float().cpu(), want) < TOL
    assert (ws[least:] == 0x5a).all()
    ops.check_device_status()

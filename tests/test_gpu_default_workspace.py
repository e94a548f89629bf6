"""The default workspace depends on the heads and the compressed length alone: a window of any length, on either cache and
through the single value product, finds room in what a call with a short window left, also under graph capture."""
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
HEADS, L, G = 64, 1024, 4


@pytest.mark.parametrize("first", ["fused", "product"])
@pytest.mark.parametrize("bits", [16, 2])
def test_longer_window_needs_no_new_buffer(bits, first):
    from mustafar_b200 import compression as c, compression_quant as cq, ops, ops_quant
    k, v = (x.cuda() for x in oracle.make_kv(HEADS, L + 300, seed=1))
    q = oracle.make_query(HEADS * G, seed=2).cuda()
    kc, vc = k[:, :L].contiguous(), v[:, :L].contiguous()
    rank = c.keep_rank(0.7)
    if bits == 16:
        ks, vs = c.SparseStore(HEADS, L, c.KEY, "cuda"), c.SparseStore(HEADS, L, c.VALUE, "cuda")
        ks.append(kc, rank), vs.append(vc, rank)
        ks.stage_hint(), vs.stage_hint()
        call = lambda w: ops.decode_attention(q, ks, vs, k[:, L:L + w], v[:, L:L + w], G)  # noqa: E731
    else:
        kq, vq = cq.compress_quant(kc, c.KEY, rank), cq.compress_quant(vc, c.VALUE, rank)
        call = lambda w: ops_quant.decode_attention_quant(q, kq, vq, L, k[:, L:L + w], v[:, L:L + w], G)  # noqa: E731
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        if first == "fused":
            call(1)
        else:
            p8 = torch.zeros(HEADS * G, 8, L, dtype=torch.float16, device="cuda")
            if bits == 16:
                bm, acc, packed = c.convert_value_batched(c.prune(vc, 0.7))
                off = torch.tensor([0] + [x.numel() // 8 for x in packed[:-1]], device="cuda").cumsum(0).int()
                ops.mustafar_value_formulation(bm, torch.cat(packed), acc, off, p8, p8, 128, L, HEADS * G, G)
            else:
                ops_quant.mustafar_value_formulation_quant(vq["bitmaps"], vq["packed"], vq["tile_offsets"], vq["counts"], vq["units"],
                                                           vq["scales"], vq["zeros"], p8, p8, 128, L, HEADS * G, G, 2, 16)
        key = (q.device, side.cuda_stream)
        before = ops._workspaces[key].data_ptr()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin()
        out = call(300)
        graph.capture_end()
        graph.replay()
        eager = call(300)
    torch.cuda.synchronize()
    assert ops._workspaces[key].data_ptr() == before
    assert torch.equal(out, eager) and torch.isfinite(out).all()
    ops._workspaces.pop(key)

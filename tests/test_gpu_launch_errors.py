"""An entry point whose launch fails reports it and leaves no error behind for the next call.  The launch is made to fail
on the host: the legacy stream may not be used while another blocking stream is being captured."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quantised", [False, True])
@pytest.mark.parametrize("tokens", [256, 1024])          # a cluster per head; the look-back with its memset
def test_no_error_left_behind(tokens, quantised):
    from mustafar_b200 import _lib
    lib, cudart = _lib.lib(), C.CDLL("libcudart.so.12")
    T = 2 * tokens
    x = torch.zeros(tokens, 128, dtype=torch.float16, device="cuda")
    bitmaps, (accum, counts, units), (scales, zeros) = (torch.zeros(*n, dtype=d, device="cuda") for n, d in (
        ((T,), torch.int64), ((3, T + 1), torch.int32), ((2, T), torch.float16)))
    values, scratch = torch.zeros(tokens * 128, dtype=torch.float16, device="cuda"), torch.zeros(1 << 16, dtype=torch.uint8, device="cuda")
    tail, status = torch.zeros(2, dtype=torch.int32, device="cuda")
    ptr = torch.Tensor.data_ptr

    def compress():
        source = (ptr(x), tokens * 128, 128, 0, 0, 1, tokens, 0, 0)
        if quantised:
            return lib.mfar_compress_quant(*source, 2, 64, ptr(bitmaps), T, ptr(accum), ptr(counts), ptr(units), ptr(scales), ptr(zeros),
                                           T, 0, ptr(values), tokens * 64, tokens * 64, ptr(tail), ptr(scratch), scratch.numel(), ptr(status),
                                           None)
        return lib.mfar_compress_fp16(*source, ptr(bitmaps), T, ptr(accum), T + 1, 0, ptr(values), None, tokens * 128, tokens * 128,
                                      ptr(scratch), scratch.numel(), ptr(status), None, None)

    torch.cuda.synchronize()
    stream, graph = C.c_void_p(), C.c_void_p()
    assert cudart.cudaStreamCreate(C.byref(stream)) == 0
    assert cudart.cudaStreamBeginCapture(stream, 0) == 0
    refused = compress()
    left = cudart.cudaGetLastError()
    cudart.cudaStreamEndCapture(stream, C.byref(graph))     # (the capture has become invalid)
    cudart.cudaGetLastError()
    assert cudart.cudaStreamDestroy(stream) == 0
    assert refused == 4 and left == 0
    assert compress() == 0
    torch.cuda.synchronize()

"""``plan`` remembers its answers by the values of whole numbers, and by nothing else."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_plan_takes_whole_numbers_only_and_reads_them_every_time():
    from mustafar_b200 import ops
    torch.zeros(1, device="cuda")
    assert ops.plan(8, 4096, 128, 4, 2) == ops.plan(8, 4096, 128, 4, 2)
    for args in ((8, 4096, 128, 4, 2.0), (8, 4096.0, 128, 4, 2), (8, 4096, 128, "4", 2)):
        with pytest.raises((TypeError, ctypes.ArgumentError)):
            ops.plan(*args)
    tokens = torch.tensor(4096)
    short = ops.plan(8, tokens, 128, 4)
    tokens += 28672
    assert ops.plan(8, tokens, 128, 4) == ops.plan(8, 32768, 128, 4) != short

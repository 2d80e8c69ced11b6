"""256-bit reads of memory that the same kernel writes see the writes before them (a path slot is read and then
overwritten by one thread)."""
import ctypes
import os

import numpy as np
import pytest

KAT = os.path.join(os.path.dirname(os.path.abspath(__file__)), "kat", "libwide_kat.so")


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 127, 128, 1025])
def test_reads_see_the_writes_before_them(n):
    import torch
    lib = ctypes.CDLL(KAT)
    records = torch.arange(8 * n, dtype=torch.float32, device="cuda").reshape(n, 8)
    before, between, after = (torch.empty_like(records) for _ in range(3))
    first = records.cpu().numpy().copy()
    arguments = [ctypes.c_void_p(t.data_ptr()) for t in (records, before, between, after)]
    assert lib.wide_rewrite(*arguments, n, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    second = first + np.float32(1)
    third = second.copy()
    third[:, 4:] += np.float32(2)
    assert np.array_equal(before.cpu().numpy(), first)
    assert np.array_equal(between.cpu().numpy(), second)
    assert np.array_equal(after.cpu().numpy(), third)
    assert np.array_equal(records.cpu().numpy(), third)

"""Alias tables whose weights lie in the bins' memory (at its start, in the middle, at its end): such weights are copied
before the first bin is written, so the table is that of weights elsewhere. Sizes at the edges of a block of 1,024
threads and of the one-launch form (8,192 lights)."""
import ctypes

import numpy as np
import pytest

import pathtracer
from test_alias_windows import sequential_pairing, weights_of


@pytest.mark.gpu
@pytest.mark.parametrize("place", ["start", "middle", "end"])
@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 4096, 8192, 8193])
def test_weights_in_the_memory_of_the_bins(n, place):
    import torch
    w = weights_of("uniform", n)
    memory = torch.full((4 * n,), -1, dtype=torch.int32, device="cuda")
    at = {"start": 0, "middle": (3 * n) // 2, "end": 3 * n}[place]
    memory[at:at + n] = torch.from_numpy(w.view(np.int32)).cuda()
    stream = torch.cuda.current_stream().cuda_stream
    assert pathtracer.lib().gpt_build_alias_table_noalloc(ctypes.c_void_p(memory.data_ptr() + 4 * at), n, ctypes.c_void_p(memory.data_ptr()),
                                                          ctypes.c_void_p(stream)) == 0
    assert np.array_equal(memory.cpu().numpy().view(np.uint32).reshape(n, 4), sequential_pairing(w))

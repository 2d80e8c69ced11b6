"""The alias pairing, predicted window by window: sizes around the block and window sizes, bit for bit
against the reference's pairing in float32."""
import math

import numpy as np
import pytest

import pathtracer


def sequential_pairing(weights):
    """AliasTable.hpp:22-84 restated: float32 values, stacks popped from their ends."""
    f32 = np.float32
    n = len(weights)
    total = f32(math.fsum(weights))
    p = weights / total
    hat = p * f32(n)
    bins = np.zeros((n, 4), dtype=np.uint32)
    bins[:, 1] = p.view(np.uint32)
    bins[:, 3] = np.arange(n)
    under = [(i, hat[i]) for i in range(n) if hat[i] < 1]
    over = [(i, hat[i]) for i in range(n) if not hat[i] < 1]
    q = np.ones(n, dtype=np.float32)
    bins[:, 2] = pathtracer.INVALID
    while under and over:
        (u, uv), (o, ov) = under.pop(), over.pop()
        q[u], bins[u, 2] = uv, o
        excess = f32(f32(uv + ov) - f32(1))
        (under if excess < 1 else over).append((o, excess))
    bins[:, 0] = q.view(np.uint32)
    return bins


def weights_of(kind, n):
    rng = np.random.default_rng(n)
    if kind == "spread":    # a few heavy outcomes
        return (2.0 ** rng.integers(-8, 8, n)).astype(np.float32)
    if kind == "equal":     # no light outcome
        return np.ones(n, dtype=np.float32)
    if kind == "one":       # one outcome takes nearly everything
        w = np.full(n, 2.0 ** -20, dtype=np.float32)
        w[n // 3] = 1.0
        return w
    if kind == "thirds":    # the excess comes back to about 1 all the time: its rounding decides
        return np.where(np.arange(n) % 3 == 0, np.float32(0.7), np.float32(0.1)).astype(np.float32)
    if kind == "uniform":
        return rng.random(n).astype(np.float32)
    w = np.full(n, 0.75, dtype=np.float32)   # "halves": long runs of either list
    w[n // 2:] = 1.25
    return w


# float weights of these sizes sum to the same float from any FP64 order
@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["spread", "equal", "one", "halves", "thirds", "uniform"])
@pytest.mark.parametrize("n", [1, 2, 31, 1023, 1024, 1025, 2047, 2048, 2049, 4096, 6145, 8192, 8193, 65536])
def test_alias_table_equals_the_sequential_pairing(kind, n):
    import torch
    w = weights_of(kind, n)
    bins = torch.full((n, 4), -1, dtype=torch.int32, device="cuda")
    assert pathtracer.build_alias_table_noalloc(torch.from_numpy(w).cuda(), bins) == 0
    assert np.array_equal(bins.cpu().numpy().view(np.uint32), sequential_pairing(w))

"""The launches bench.py counts for a step of squarings, against the kernels that
run, at state counts on both sides of the L2 size."""
import numpy as np
import pytest
import torch

import bench
from kernel_names import kernel_counts, launched

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r,n,k", [(136279841, 2, 16), (136279841, 4, 6), (999961, 3, 16),
                                   (999961, 64, 7), (4423, 16, 1), (4423, 1, 2), (4423, 1, 5)])
def test_counted_passes_are_the_launched_ones(engine, r, n, k):
    nw = (r + 63) // 64
    stride = nw + (nw & 1)
    a = torch.zeros(stride * n, dtype=torch.int64, device="cuda")
    b = torch.zeros_like(a)
    s = torch.from_numpy(np.arange(1, n + 1)).cuda()
    engine.trin_square_batch(a, b, stride, n, r, s, k)
    torch.cuda.synchronize()
    names = kernel_counts(lambda: engine.trin_square_batch(a, b, stride, n, r, s, k))
    got = tuple(launched(names, x) for x in ("k_frob4_batch", "k_square_batch", "Memcpy DtoD"))
    assert got == bench.squaring_passes(engine, r, stride, n, k)

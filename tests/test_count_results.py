"""count_SEIRP's results are tensors of their own: each with its own aligned
storage, which is all that keeping or saving one of them keeps."""

import io

import numpy as np
import pytest

from laser_polio_gb300 import ops


@pytest.mark.gpu
@pytest.mark.parametrize("G,ns", [(1, 1), (13, 3), (775, 2)])
def test_gpu_results_are_tensors_of_their_own(G, ns):
    import torch

    rng = np.random.default_rng(G)
    n = 5000
    cols = [torch.from_numpy(c).cuda() for c in (
        rng.integers(0, G, n).astype(np.int16), rng.integers(-1, 4, n).astype(np.int8), rng.integers(0, ns, n).astype(np.int8),
        rng.integers(-1, 2, n).astype(np.int8), rng.integers(0, 2, n).astype(np.int8))]
    out = ops.count_SEIRP(*cols, G, ns, n)
    shapes = [(G,)] * 4 + [(G, ns)] * 2 + [(G,)] * 2
    assert [tuple(t.shape) for t in out] == shapes
    assert len({t.untyped_storage().data_ptr() for t in out}) == 8
    for t in out:
        assert t.is_contiguous() and t.data_ptr() % 16 == 0
        assert t.untyped_storage().nbytes() == t.numel() * 4
        b = io.BytesIO()
        torch.save(t, b)
        assert len(b.getvalue()) < 4 * t.numel() + 4096

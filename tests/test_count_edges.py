"""count_SEIRP about the kernel's edges (csrc/lpg_ops.cu): steps of 16 slots,
one CTA up to 32768 slots, warps' tiles of 4096, node changes inside and
between steps, byte values outside the states, against the oracle."""

import numpy as np
import pytest

from oracle.oracle import count_seirp
from test_count_seirp import NAMES
from test_count_seirp import _gpu_count


def _columns(n, G, ns, seed, run):
    rng = np.random.default_rng(seed)
    node = (np.arange(n) // run % G).astype(np.int16)
    ds = rng.integers(-2, 6, n).astype(np.int8)  # dead, the four states and values no state has
    ds[rng.random(n) < 0.01] = 127
    strain = rng.integers(-1, ns + 1, n).astype(np.int8)
    strain[rng.random(n) < 0.01] = -128
    pp = rng.integers(-1, 3, n).astype(np.int8)
    par = rng.integers(-1, 3, n).astype(np.int8)
    node[rng.random(n) < 0.001] = G
    node[rng.random(n) < 0.001] = -1
    return node, ds, strain, pp, par


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 15, 16, 17, 511, 32767, 32768, 32769, 65536 + 7, 300_007, 5_000_011])
@pytest.mark.parametrize("G,ns,run", [(1, 1, 10**9), (5, 4, 16), (300, 3, 1000), (774, 2, 7)])
def test_gpu_counts_about_the_edges(n, G, ns, run):
    cols = _columns(n, G, ns, seed=n % 1000 + G, run=run)
    want = count_seirp(*cols, G, ns, n)
    got = _gpu_count("lpg_count_seirp", cols, G, ns, n, 0)
    for name, x, y in zip(NAMES + ("n_invalid",), got, want):
        np.testing.assert_array_equal(x, y, err_msg=name)

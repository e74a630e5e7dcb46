"""The coarsest graph comes down with its rows sorted on the device; the initial partitioner sees the same graph as with
rows sorted on the host. Checked through partitions whose coarsest level has rows of every length up to all vertices, a
bitmap that ends within and at a word, and no coarsening at all (an input with parallel edges keeps the host sort)."""
import numpy as np
import pytest

import gpu_heipa as H
import oracle as O
from helpers import star, to_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("g,k", [(H.Graph.rmat(11, 16, seed=3), 16), (H.Graph.rmat(13, 30, seed=4), 40),
                                 (star(4000), 2), (H.Graph.grid(64, 32, 1, 9, seed=2), 4),
                                 (H.Graph.rgg3d(2048, 30.0, 1, 9, seed=6), 33),
                                 (H.Graph([0, 3, 6, 8], [1, 1, 2, 0, 0, 2, 0, 1], [2, 3, 4, 2, 3, 5, 4, 5]), 2)],
                         ids=["rmat11", "rmat13", "star", "grid", "rgg", "parallel"])
def test_partitions_equal_oracle(ctx, g, k):
    part, cut = ctx.partition(g, k, 0.03, "default", 3)
    want, want_cut = O.partition(to_oracle(g), k, 0.03, False, 3)
    assert cut == want_cut
    np.testing.assert_array_equal(part, want)

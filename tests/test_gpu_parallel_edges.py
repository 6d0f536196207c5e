"""Triangle counts of rows longer than a simple graph's: the 32-bit counts carry what does not fit them."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_clustering_of_a_vertex_with_many_loops():
    """d loops at vertex 0: every one of its d entries is found for every one of its d edges, 2^32 times (some
    seconds).  Vertex 1 has 32 parallel edges to vertex 2 and back, each with one loop."""
    from cugal_b200 import cuda_kernels
    d = 65536
    rows = [[0] * d, [1] + [2] * 32, [1] * 32 + [2], []]
    col = torch.tensor(np.concatenate([np.asarray(r, dtype=np.int32) for r in rows]), device="cuda")
    rp = torch.tensor(np.cumsum([0] + [len(r) for r in rows]), dtype=torch.int32, device="cuda")
    # edge (1, 1): 33 of 33 entries; (1, 2): of the 33 entries of either list all are in the other
    t = np.array([d * d, 33 * 33, 33 * 33, 0], dtype=np.int64)
    deg = np.array([d, 33, 33, 0], dtype=np.int64)
    expected = np.zeros(4, dtype=np.float32)
    expected[:3] = t[:3].astype(np.float32) / (deg * (deg - 1))[:3].astype(np.float32)
    clustering, degrees = torch.empty(4, device="cuda"), torch.empty(4, device="cuda")
    cuda_kernels.graph_features(col, rp, clustering, degrees)
    assert np.array_equal(clustering.cpu().numpy(), expected) and np.array_equal(degrees.cpu().numpy(), deg)

"""Grouping of small edge lists in one block against stable sorts: at the limits of its shared memory (8,192 edges, 4,096 nodes)
and past them, one node, one edge."""
import numpy as np
import pytest
import torch

from openequivariance_b200 import CoordGraph, prepare_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.int64, np.int32])
@pytest.mark.parametrize("nodes,edges", [(1, 1), (1, 700), (31, 1023), (105, 1680), (4096, 8192), (4097, 8192), (4096, 8193), (1025, 1)])
def test_order_matches_stable_sorts(nodes, edges, dtype):
    rng = np.random.default_rng(nodes + edges)
    rows, cols = (rng.integers(0, nodes, edges).astype(dtype) for _ in range(2))
    want = CoordGraph(np.zeros((nodes, 3)), rows, cols, "t")
    got = prepare_graph(torch.tensor(rows, device="cuda"), torch.tensor(cols, device="cuda"), nodes)
    for name, ref in (("rows", want.rows), ("cols", want.cols), ("transpose_perm", want.transpose_perm), ("order", want.edge_order)):
        assert np.array_equal(got[name].cpu().numpy(), ref), name

"""BlockSystem's node coordinates go to the library as a bare pointer: what is
not n_rows x 3 contiguous float64 beside the matrix is refused."""

import pytest
import torch

from cloudfem_b200.device import BlockSystem


def _make(nodes):
    return BlockSystem(None, 4, 3, None, None, torch.zeros(36, dtype=torch.float64), None, None, nodes=nodes)


def test_nodes_as_the_library_reads_them():
    nodes = torch.zeros((4, 3), dtype=torch.float64)
    assert _make(nodes).nodes is nodes
    assert _make(None).nodes is None


@pytest.mark.parametrize("nodes", [
    torch.zeros((4, 3), dtype=torch.float32),
    torch.zeros((3, 3), dtype=torch.float64),
    torch.zeros(12, dtype=torch.float64),
    torch.zeros((3, 4), dtype=torch.float64).t(),
    torch.zeros((4, 3), dtype=torch.float64, device="meta"),
], ids=["float32", "short", "flat", "transposed", "elsewhere"])
def test_other_nodes_are_refused(nodes):
    with pytest.raises(ValueError, match="nodes must be"):
        _make(nodes)

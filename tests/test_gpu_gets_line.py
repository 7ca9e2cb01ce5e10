"""Batched gets on both sides of the size from which they start from a table of upper nodes: the trees' dense voxels,
for trees of several depths in one call and more trees than a deep table has room for."""
import pytest
from test_gpu_gets_table import test_gets_equal_the_dense_trees as gets_equal_the_dense_trees


@pytest.mark.gpu
@pytest.mark.parametrize("bits,depths,n", [
    (8, (1, 2, 3, 4, 5, 6), 1 << 20), (16, (8,), 1 << 20), (8, (5,) * 300, (1 << 20) + 3), (16, (4, 2), (1 << 20) - 1),
    (8, (7, 0, 3), 1 << 21),
])
def test_gets_around_the_line(gpu_lib, bits, depths, n):
    gets_equal_the_dense_trees(gpu_lib, bits, depths, n)

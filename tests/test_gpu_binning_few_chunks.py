"""GPU tests of the lists at the edges of the rule that writes them from primitive
masks where there are few chunks of 512 primitives (three to seven) and at the
largest number of cells that a marking CTA's shared memory holds: bit-exact with the
oracle's, alone and as a batch, on both sides of each edge."""
import pytest
import test_gpu_binning_chain as chain

pytestmark = pytest.mark.gpu

CASES = [  # tile rows, tile columns (cells: rows x ceil(columns / 32)), N, largest radius
    (284, 66, 1025, 60.0),      # 852 cells, 3 chunks: below
    (285, 66, 1025, 60.0),      # 855
    (285, 66, 1024, 60.0),      # two chunks: below
    (121, 66, 3584, 900.0),     # 363 cells, 7 chunks: below
    (122, 66, 3584, 900.0),     # 366
    (66, 66, 3585, 40.0),       # 198 cells, 8 chunks: below
    (67, 66, 3585, 40.0),       # 201
    (1066, 66, 1300, 300.0),    # 3198 cells: the marks fit
    (1067, 66, 1300, 300.0),    # 3201: they do not
]


@pytest.mark.parametrize("rows,cols,N,rmax", CASES)
def test_lists_at_the_edges_of_the_mask_rule_gpu(rows, cols, N, rmax):
    chain.test_lists_match_oracle_alone_and_in_a_batch_gpu(16 * rows, 16 * cols - 5, 16, N, rmax)

"""The direct solve's substitutions at the edges of their blocks: fewer unknowns than the band or two
blocks of 32 columns, orders that are no multiple of 32, a band narrower than a block, and one whose
window takes two elements per thread; psi bit-identical to the oracle's direct solve."""
import pytest

from tests.test_direct_gpu import test_direct_solve_matches_oracle_on_larger_grids as same_bits

pytestmark = pytest.mark.gpu


# band 3 (nz + 1): 27, 51, 39, 963 (two elements per thread)
@pytest.mark.parametrize("nx,nz", [(8, 8), (24, 16), (8, 12), (32, 320)])
def test_direct_solve_matches_oracle_at_block_edges(nx, nz):
    same_bits(nx, nz)

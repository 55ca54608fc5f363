"""The grid stage's forces where warps change between the list of contacts and the sum at once: cells of
one to dozens of particles side by side in a warp, a last warp of a few lanes, one particle.  Against the
oracle, bit for bit (the checks of test_gpu_stage_walks)."""
import pytest

from test_gpu_stage_walks import test_grid_forces_and_contacts as forces_and_contacts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spread,dims", [(3, 0.01, 8), (33, 0.05, 8), (35, 0.4, 4), (500, 0.2, 8),
                                           (1001, 0.5, 8), (4003, 0.5, 16), (6000, 1.0, 16),
                                           (3000, 0.12, 2)])
def test_crowded_cells(ctx, n, spread, dims):
    forces_and_contacts(ctx, n, spread, dims)

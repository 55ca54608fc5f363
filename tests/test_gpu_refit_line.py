"""ar_lbvh_refit on both sides of the size from which subtrees merge in tiles (7 x 2^17 leaves)."""
import pytest

from test_gpu_refit_tiles import test_refit_forms as refit_forms

pytestmark = pytest.mark.gpu

LINE = 7 << 17


@pytest.mark.parametrize("n,codes,renumber", [
    (LINE - 1, "spread", False), (LINE - 1, "equal", True), (LINE, "spread", False),
    (LINE, "spread", True), (LINE + 1, "equal", False)])
def test_refit_line(ctx, n, codes, renumber):
    refit_forms(ctx, n, codes, renumber)

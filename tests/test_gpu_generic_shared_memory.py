"""Run-time sizes whose row pass comes to the last bytes of a block's shared memory, by the
number of histogram bins (up to the largest), against the FP64 oracle."""
import pytest

from tests.search_cases import make_case
from tests.search_check import search_and_check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("X,bins", [(7200, 495), (7200, 496), (7200, 497), (7168, 752), (7150, 908), (7260, 24), (7203, 487),
                                    (7203, 488), (7200, 1024), (2700, 1024)])
def test_rows_at_the_limit_of_shared_memory(X, bins):
    search_and_check(make_case(T=32, X=X, Y=66, n_particles=1, n_orient=3), bins=bins)

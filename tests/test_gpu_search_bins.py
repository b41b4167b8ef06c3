"""The histogram bin by bin, and planes after planes, at the batches, parts and sizes where the row
pass changes its form: an orientation of a pair counted twice or not at all, a wrong bin of the second
of a pair, or a part that takes another's orientation keeps the total and fails here.  Two planes: maxima of
the first that the second does not exceed keep their orientation and defocus."""
import pytest

from tests.search_cases import make_case
from tests.search_check import search_and_check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,X,Y,n,batch", [(32, 256, 256, 7, 0), (32, 256, 256, 8, 0), (32, 256, 256, 41, 19),
                                           (32, 256, 288, 32, 0), (32, 256, 512, 37, 0), (32, 512, 256, 70, 64),
                                           (64, 512, 512, 15, 0), (64, 512, 512, 27, 0), (64, 512, 512, 27, 3)])
def test_divided_batches(T, X, Y, n, batch):
    search_and_check(make_case(T=T, X=X, Y=Y, n_particles=1, n_orient=n), batch=batch, planes=2)


@pytest.mark.parametrize("T,X,Y,n,batch", [(32, 256, 256, 1, 1), (32, 256, 288, 7, 4), (32, 512, 512, 11, 3),
                                           (64, 1024, 1024, 3, 2), (128, 2048, 2916, 3, 2), (256, 2048, 1944, 1, 0)])
def test_odd_and_even_batches(T, X, Y, n, batch):
    search_and_check(make_case(T=T, X=X, Y=Y, n_particles=1, n_orient=n), batch=batch, planes=2)


@pytest.mark.parametrize("X,Y,n", [(130, 154, 3), (286, 98, 1), (729, 66, 2), (3584, 66, 5), (6561, 66, 3), (7280, 66, 2),
                                   (8125, 66, 1), (66, 3528, 3), (66, 7280, 1)])
def test_run_time_sizes(X, Y, n):
    search_and_check(make_case(T=32, X=X, Y=Y, n_particles=1, n_orient=n), planes=2)

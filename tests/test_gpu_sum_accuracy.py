"""The per-pixel sums of the search at the widths and sizes whose row passes add every value by
itself: at least as accurate as FP32 sums compensated at each orientation."""
import numpy as np
import pytest

from cistem_downstream_bah_b200 import core
from tests.search_cases import make_case

pytestmark = pytest.mark.gpu


def _compensated(x):
    """Kahan sums of x (orientations first) and of its squares, one orientation at a time in FP32."""
    f32 = np.float32
    s, c, q, d = (np.zeros(x.shape[1], f32) for _ in range(4))
    for v in x:
        y = v - c
        t = s + y
        c, s = (t - s) - y, t
        y = (v.astype(np.float64) ** 2 - d).astype(f32)   # a multiply-add
        t = q + y
        d, q = (t - q) - y, t
    return s.astype(np.float64) - c, q.astype(np.float64) - d


# compiled widths below 2048, undivided and divided batches; run-time sizes of each row pass on pairs
# (even and odd rows, up to 2048 pixels and above, with and without the tables in shared memory)
@pytest.mark.parametrize("T,X,Y,n", [(32, 256, 256, 6), (32, 256, 256, 33), (64, 512, 512, 40), (64, 1024, 1024, 33),
                                     (32, 130, 154, 33), (32, 729, 66, 33), (32, 2700, 66, 24), (32, 2187, 66, 17),
                                     (32, 3584, 66, 17), (32, 6561, 66, 17), (32, 7280, 66, 17)])
def test_sums_are_no_less_accurate_than_compensated_ones(T, X, Y, n):
    case = make_case(T=T, X=X, Y=Y, n_particles=1, n_orient=n)
    with core.SearchCore(X, Y, T, histogram_min_scaled=case["hmin"], histogram_step_scaled=case["hstep"]) as sc:
        sc.set_template(case["tspec"])
        sc.set_image(case["ispec"])
        values = []
        for k in range(n):   # one value per pixel: the sum is that value
            sc.reset()
            sc.run_plane(case["filt"], case["angles"][k:k + 1])
            values.append(sc.results()["sum"].astype(np.float32))
        sc.reset()
        sc.run_plane(case["filt"], case["angles"])
        r = sc.results()
    x = np.stack(values)
    cs, cq = _compensated(x)
    x = x.astype(np.float64)
    exact, exact2 = x.sum(0), (x * x).sum(0)

    def rms(e):
        return np.sqrt(np.mean(e * e))

    # a tenth for the order of additions
    assert rms(r["sum"] - exact) <= 1.1 * rms(cs - exact)
    assert rms(r["sumsq"] - exact2) <= 1.1 * rms(cq - exact2)

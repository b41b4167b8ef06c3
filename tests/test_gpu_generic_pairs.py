"""The run-time-length kernels on pairs of lines and their one-line forms, against the
FP64 oracle, at the sizes where the choice between them turns: rows and
columns that fit shared memory twice as pairs or not, with and without the
twiddle table beside them, odd rows, every prime radix, and odd orientation
counts."""
import numpy as np
import pytest

from cistem_downstream_bah_b200 import core
from oracle import oracle as O
from tests.search_cases import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("X,Y,n", [(130, 154, 3), (286, 98, 1), (729, 66, 2), (3584, 66, 2), (6561, 66, 3), (7280, 66, 2),
                                   (8125, 66, 1), (66, 3528, 3), (70, 5832, 2), (66, 7280, 1)])
def test_line_pairs_match_oracle(X, Y, n):
    T = 32
    case = make_case(T=T, X=X, Y=Y, n_particles=1, n_orient=n)
    with core.SearchCore(X, Y, T, histogram_min_scaled=case["hmin"], histogram_step_scaled=case["hstep"]) as sc:
        sc.set_template(case["tspec"])
        sc.set_image(case["ispec"])
        sc.run_plane(case["filt"], case["angles"])
        r = sc.results()
    st = O.SearchState(X, Y)
    O.search(st, case["tspec"], case["ispec"], case["filt"], case["angles"], hist_min_scaled=case["hmin"],
             hist_step_scaled=case["hstep"])
    scale = np.abs(st.mip).max()
    # FP32 transforms against FP64: 2e-5 of the map's scale, as the correlation maps' bound
    assert np.abs(r["mip"] - st.mip).max() <= 2e-5 * scale
    assert np.abs(r["sum"] - st.sum).max() <= 2e-5 * scale * n
    assert np.abs(r["sumsq"] - st.sumsq).max() <= 4e-5 * scale * scale * n
    assert r["hist"].sum() == st.hist[:512].sum()
    decided = st.mip - st.second > 1e-4 * scale
    for k in ("psi", "theta", "phi"):
        assert np.array_equal(r[k][decided], getattr(st, k)[decided]), k

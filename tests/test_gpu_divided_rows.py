"""The row pass of small images, whose blocks share a batch of orientations (k_pass_c's divided
form), against the FP64 oracle: orientation counts around the smallest divided batches, odd ones,
several batches, parts of unequal length, and the same search with batches too small to divide."""
import numpy as np
import pytest

from cistem_downstream_bah_b200 import core
from oracle import oracle as O
from tests.search_cases import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,X,Y,n,batch", [(32, 256, 256, 7, 0), (32, 256, 256, 8, 0), (32, 256, 256, 33, 0),
                                           (32, 256, 256, 41, 19), (32, 256, 288, 32, 0), (32, 256, 512, 37, 0),
                                           (32, 512, 256, 70, 64), (64, 512, 512, 15, 0), (64, 512, 512, 16, 0),
                                           (64, 512, 512, 27, 0), (64, 512, 512, 27, 3)])
def test_divided_batches_match_oracle(T, X, Y, n, batch):
    case = make_case(T=T, X=X, Y=Y, n_particles=1, n_orient=n)
    with core.SearchCore(X, Y, T, histogram_min_scaled=case["hmin"], histogram_step_scaled=case["hstep"],
                         orientation_batch=batch) as sc:
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

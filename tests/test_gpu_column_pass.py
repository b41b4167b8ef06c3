"""The column pass on column pairs (k_pass_b) against the FP64 oracle, at the heights where its
layout turns: two and four column pairs per block, one or several blocks per SM, padding
lanes (pairs of threads that do not fill a warp), radix 16 and 18 with short last stages,
pruned lengths above the template, one and two staging buffers, and batches whose left-over
column groups are shared out evenly."""
import numpy as np
import pytest

from cistem_downstream_bah_b200 import core
from oracle import oracle as O
from tests.search_cases import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,X,Y,n", [(32, 256, 288, 3), (48, 256, 288, 1), (128, 256, 256, 5), (256, 512, 512, 3),
                                     (64, 1024, 1024, 9), (256, 2048, 1944, 2), (256, 2048, 2592, 1),
                                     (128, 2048, 2916, 2), (384, 4096, 5832, 1)])
def test_column_pairs_match_oracle(T, X, Y, n):
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

"""The row pass's pairing of orientations (k_pass_c) against the FP64 oracle:
odd and even orientation counts and batches, so that a batch ends with a single
orientation or a whole pair, at widths whose rows share a warp (256), fill one
(512) and span several (1024)."""
import numpy as np
import pytest

from cistem_downstream_bah_b200 import core
from oracle import oracle as O
from tests.search_cases import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,X,Y,n,batch", [(32, 256, 256, 1, 1), (32, 256, 288, 7, 4), (32, 256, 256, 9, 9),
                                           (32, 512, 256, 5, 5), (32, 512, 512, 11, 3), (64, 1024, 1024, 3, 2)])
def test_odd_and_even_batches(T, X, Y, n, batch):
    case = make_case(T=T, X=X, Y=Y, n_orient=n)
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
    # best orientation wherever the two best values are apart
    decided = st.mip - st.second > 1e-4 * scale
    for k in ("psi", "theta", "phi"):
        assert np.array_equal(r[k][decided], getattr(st, k)[decided]), k

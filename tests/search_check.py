"""A search on the GPU against the FP64 oracle, every output and the histogram bin by bin."""
import numpy as np

from cistem_downstream_bah_b200 import core
from oracle import oracle as O


def search_and_check(case, bins=512, batch=0, planes=1):
    """Runs the case's plane, then `planes` - 1 more with other filters and defocus values."""
    T, X, Y, n = case["T"], case["X"], case["Y"], len(case["angles"])
    step = case["hstep"] * 512 / bins   # the same range
    st = O.SearchState(X, Y, hist_bins=bins)
    with core.SearchCore(X, Y, T, histogram_min_scaled=case["hmin"], histogram_step_scaled=step, histogram_bins=bins,
                         orientation_batch=batch) as sc:
        sc.set_template(case["tspec"])
        sc.set_image(case["ispec"])
        for k in range(planes):
            filt = _plane_filter(case, k)
            sc.run_plane(filt, case["angles"], defocus_offset=100.0 * k)
            O.search(st, case["tspec"], case["ispec"], filt, case["angles"], hist_min_scaled=case["hmin"],
                     hist_step_scaled=step, defocus_value=100.0 * k)
        r = sc.results()
    total = n * planes
    scale = np.abs(st.mip).max()
    # FP32 transforms against FP64: 2e-5 of the map's scale, as the correlation maps' bound
    assert np.abs(r["mip"] - st.mip).max() <= 2e-5 * scale
    assert np.abs(r["sum"] - st.sum).max() <= 2e-5 * scale * total
    assert np.abs(r["sumsq"] - st.sumsq).max() <= 4e-5 * scale * scale * total
    # a value within rounding of an edge may fall into the bin next to its own
    assert np.all(np.abs(r["hist"] - st.hist[:bins]) <= 1e-3 * st.hist[:bins] + 2)
    decided = st.mip - st.second > 1e-4 * scale
    for k in ("psi", "theta", "phi", "defocus"):
        assert np.array_equal(r[k][decided], getattr(st, k)[decided]), k


def _plane_filter(case, k):
    """The projection filter of plane k: its CTF rows shifted, so that the planes' maps differ."""
    return case["filt"] if k == 0 else np.ascontiguousarray(np.roll(case["filt"], k, axis=1), dtype=np.float32)

"""The server's top-K at the sizes where its passes change: rows shorter than K and than a warp group, one column past a
batch, rows of ties (thresholded to zero), and K at its limits, against a stable sort of the same coefficients."""
import numpy as np
import pytest

from seismic_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 40, 1024, 4097, 9001])
@pytest.mark.parametrize("topk,threshold", [(1, 0.0), (16, 0.0), (64, 0.0), (64, 0.6), (16, 2.0)])
def test_topk_is_a_stable_sort(cuda_ok, n, topk, threshold):
    from seismic_gb300.serving import Server
    base = synth.family_catalog(700, 1, 64, n_families=9, seed=5)
    cat = np.tile(base, (n // 700 + 1, 1, 1))[:n]  # whole rows repeat: equal coefficients at many columns
    with_srv = Server(cat, shift=20, threshold=threshold, form="fp32", n_slots=2, max_query_events=4, topk=topk)
    query = synth.family_catalog(3, 1, 64, n_families=2, seed=6)
    for begin in (0, n // 3):
        res = with_srv.wait(with_srv.submit(query, subset=(begin, n)))
        for q in range(3):
            order = np.argsort(-res.vals_pos[q], kind="stable")[:topk]
            m = order.size
            np.testing.assert_array_equal(res.topk_index[q][:m], begin + order)
            np.testing.assert_array_equal(res.topk_vals[q][:m], res.vals_pos[q][order])
            np.testing.assert_array_equal(res.topk_index[q][m:], -1)
            np.testing.assert_array_equal(res.topk_vals[q][m:], 0)
    with_srv.close()

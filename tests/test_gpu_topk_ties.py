"""The server's top-K where many values equal the bound of its first pass: rows cut to zero by the threshold, identical
events, and ties that begin before, at and behind the first batch of 4096 columns; against a stable sort."""
import numpy as np
import pytest

from seismic_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("topk", [1, 16, 64])
@pytest.mark.parametrize("n,first", [(20, 0), (1023, 0), (1500, 900), (5000, 0), (4200, 4095), (9000, 4090), (9000, 4096),
                                     (9000, 8900)])
@pytest.mark.parametrize("threshold", [0.0, 0.9])
def test_topk_of_rows_of_ties(cuda_ok, topk, n, first, threshold):
    """Columns from `first` on repeat the query's event, the others are noise (0 above the threshold 0.9)."""
    from seismic_gb300.serving import Server
    rng = np.random.default_rng(n + first)
    event = synth.family_catalog(1, 1, 64, n_families=1, seed=6)
    cat = rng.standard_normal((n, 1, 64)).astype(np.float32)
    cat[first:] = event
    cat[first + 7::11] = 0.0  # some of them silent: zeros among the ties
    srv = Server(cat, shift=20, threshold=threshold, form="fp32", n_slots=1, max_query_events=2, topk=topk)
    res = srv.wait(srv.submit(np.concatenate((event, -event))))
    for q in range(2):
        order = np.argsort(-res.vals_pos[q], kind="stable")[:topk]
        np.testing.assert_array_equal(res.topk_index[q][:order.size], order)
        np.testing.assert_array_equal(res.topk_vals[q][:order.size], res.vals_pos[q][order])
        np.testing.assert_array_equal(res.topk_index[q][order.size:], -1)
    srv.close()

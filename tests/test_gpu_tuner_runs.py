"""The launch-shape report says what was run: candidates that differ only in the CTAs per SM, which the
tuned kernel does not vary, are one run with one time, and none of them is reported as a choice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_candidates_of_one_run_have_one_time(lib):
    from mld_gb300 import _lib, synth
    ds = synth.fe_bcc_batched(n_struct=70, nmin=100, nmax=300, seed=51)
    nat, pos, cell, types = ds.arrays()
    E, F, S, has = ds.labels()
    c = _lib.default_config()
    c.j_max, c.r_cut, c.lambda_krr, c.precision = 2.0, 4.7, 1e-8, _lib.MIXED
    with _lib.Handle(c) as h:
        h.set_structures(nat, pos, cell, types)
        h.set_labels(E, F, S, has, np.ones((len(nat), 3)))
        h.fit()
        t = h.tuning(0)
    ms = np.array(t["candidate_ms"]).reshape(2, 2, 2)  # column tile, CTAs per SM, queue
    assert t["tuned"] and np.array_equal(ms[:, 0], ms[:, 1]) and t["ctas_per_sm"] == 0
    assert ms[[4, 2].index(t["col_tile"]), 0, 1 - t["sorted_queue"]] == ms.min()

"""The conjugate-gradient solve of the mixed method starts from its preconditioned residual and
reads no memory that it has not written: fits in memory that held NaN before are finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_mixed_fit_in_memory_that_held_nan(lib):
    torch = pytest.importorskip("torch")
    from mld_gb300 import _lib, synth
    ds = synth.fe_bcc_batched(n_struct=4, nmin=16, nmax=60, seed=23)
    nat, pos, cell, types = ds.arrays()
    E, F, S, has = ds.labels()
    c = _lib.default_config()
    c.j_max, c.r_cut, c.lambda_krr, c.precision = 2.0, 4.7, 1e-8, _lib.MIXED
    for _ in range(3):
        held = [torch.full((n,), float("nan"), dtype=torch.float64, device="cuda") for n in (1 << 16, 1 << 20)]
        torch.cuda.synchronize()
        del held
        torch.cuda.empty_cache()
        with _lib.Handle(c) as h:
            h.set_structures(nat, pos, cell, types)
            h.set_labels(E, F, S, has, np.ones((len(nat), 3)))
            w, rmse = h.fit()
        assert np.isfinite(w).all() and np.isfinite(rmse).all()

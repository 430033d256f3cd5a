"""mld_gpu_gram_rows after a call that found no memory: the failed allocation is reported once and does
not fail the next call.  2^40 rows ask for 8 TB of workspace before anything is launched or read."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from test_gpu_gram_rows import _call, _rows  # noqa: E402


@pytest.mark.parametrize("method", [0, 1])
def test_next_call_after_no_memory(lib, method):
    import torch
    from mld_gb300 import _lib
    X, w, y = _rows(1000, 65, 3, torch.float32)
    want, _ = _call(X, w, y, 65, 0)
    G = torch.zeros(65, 65, device="cuda", dtype=torch.float64)
    with pytest.raises(_lib.MldError) as ei:
        _lib.gram_rows(method, X.data_ptr(), True, 1 << 40, 65, X.shape[1], w.data_ptr(), y.data_ptr() if method else 0,
                       G.data_ptr(), G.data_ptr() if method else 0, 0)
    assert ei.value.code == 4  # MLD_ERR_OOM
    got, _ = _call(X, w, y, 65, 0)
    assert np.array_equal(got, want)

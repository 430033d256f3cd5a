"""The workspace that mld_gpu_gram_rows keeps between calls is bounded and given back without a handle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from test_gpu_gram_rows import _call, _rows  # noqa: E402


@pytest.mark.parametrize("M,given_back", [(20000, 80_000_000), (160000, 0)])
def test_workspace_is_given_back(lib, M, given_back):
    """82 MB of bf16 planes, kept and given back; 655 MB, more than may stay mapped."""
    import torch
    D = 1024
    X, w, y = _rows(M, D, 3, torch.float32)
    G, _ = _call(X, w, y, D, 0)  # kernels loaded, torch's blocks for the results cached
    lib.mld_gpu_destroy(None)
    before = torch.cuda.mem_get_info()[0]
    assert np.array_equal(_call(X, w, y, D, 0)[0], G)
    kept = torch.cuda.mem_get_info()[0]
    lib.mld_gpu_destroy(None)
    after = torch.cuda.mem_get_info()[0]
    assert before - kept <= 512 << 20
    assert after >= before and after - kept >= given_back

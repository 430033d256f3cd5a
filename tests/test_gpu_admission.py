"""Admission of a large quadratic request: its Z terms are formed pass by pass, so the bytes that the
server charges for them stop growing with the request.

101,306 atoms at j_max 4 with two FP32 channels: 0.36 GB of pairs (56 bytes of 63 a priori neighbours each),
0.40 GB of buffers per atom and at most 1.1 GB of Z terms (2 GB of terms and rows, the terms 48 % of them).
All terms at once would be 3.6 GB, above the budget of 4.0 GB with the rest.  The memory that the batch
really takes stays within the estimate, up to the eighth that buffers are larger than asked for.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from test_gpu_j_range import _config  # noqa: E402

BUDGET = 4.0e9


def test_large_quadratic_request_is_admitted(lib):
    torch = pytest.importorskip("torch")
    from mld_gb300 import _lib, synth
    rng = np.random.default_rng(3)
    pos, cell = synth.bcc(37, 37, 37, synth.FE_A)
    pos = pos + rng.normal(0.0, 0.05, size=pos.shape)
    types = rng.integers(0, 2, size=len(pos)).astype(np.int32)
    cfg = _config(4.0, 4.7, 2, 1, 2)
    with _lib.Handle(cfg) as h:
        w = rng.normal(0.0, 1e-3, h.dim_design_line)
        w[1 + h.dim_desc:] *= 1e-3
    torch.cuda.empty_cache()
    with _lib.Server(cfg, w, n_slots=1, max_batch_atoms=1 << 20, hbm_fraction=0.5) as srv:
        free = srv.stats()["budget_bytes"] / 0.5
    with _lib.Server(cfg, w, n_slots=1, max_batch_atoms=1 << 20, hbm_fraction=BUDGET / free) as srv:
        before = torch.cuda.mem_get_info()[0]
        E, F, S, _ = srv.wait(srv.submit(pos, cell, types))
        taken = before - torch.cuda.mem_get_info()[0]
        estimate = srv.admission()["largest_batch_bytes"]
    assert np.isfinite(E) and np.isfinite(F).all() and np.isfinite(S).all()
    assert estimate <= 2.2e9
    assert taken <= 1.125 * estimate + 2 ** 26

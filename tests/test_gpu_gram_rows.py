"""Normal matrix of design rows on the device (mld_gpu_gram_rows): tile and slice edges of the
bf16-split tensor-core path, the number of row splits it picks, and calls from several threads.

The split keeps x' = hi + lo with |x' - hi - lo| <= 2^-18 |x'| and drops lo_i lo_j (2^-18), so an
element is off by at most 3 * 2^-18 sum w |x_i x_j| plus the FP32 accumulation of 64-row slices
(sixteen MMA steps, 2^-19): 2^-16 sum w |x_i x_j| bounds it.  The right-hand side is summed in
double-FP32 (2^-44 per step over at most 5000 rows): 1e-9 sum |w y x|.
"""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from mld_gb300 import _lib

pytestmark = pytest.mark.gpu


def _rows(M, D, seed, dtype):
    g = torch.Generator(device="cuda").manual_seed(seed)
    ld = (D + 3) // 4 * 4
    X = torch.zeros(M, ld, device="cuda", dtype=dtype)
    X[:, :D] = torch.randn(M, D, device="cuda", generator=g).to(dtype)
    w = torch.rand(M, device="cuda", generator=g, dtype=torch.float64) + 0.1
    y = torch.randn(M, device="cuda", generator=g, dtype=torch.float64)
    return X, w, y


def _call(X, w, y, D, stream):
    G = torch.zeros(D, D, device="cuda", dtype=torch.float64)
    h = torch.zeros(D, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    _lib.gram_rows(_lib.MIXED, X.data_ptr(), X.dtype == torch.float32, X.shape[0], D, X.shape[1], w.data_ptr(),
                   y.data_ptr(), G.data_ptr(), h.data_ptr(), stream)
    return G.cpu().numpy(), h.cpu().numpy()


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("M,D", [(1, 1), (63, 5), (64, 128), (65, 129), (200, 64), (127, 65), (1000, 257),
                                 (4999, 320), (3001, 1153)])
def test_gram_rows_edges(M, D, dtype):
    X, w, y = _rows(M, D, 17 * M + D, getattr(torch, dtype))
    G, h = _call(X, w, y, D, 0)
    x = X[:, :D].double().cpu().numpy()
    wn, yn = w.cpu().numpy(), y.cpu().numpy()
    want, scale = x.T @ (wn[:, None] * x), np.abs(x).T @ (wn[:, None] * np.abs(x))
    assert np.all(np.abs(G - want) <= 2.0**-16 * scale)
    assert np.array_equal(G, G.T)
    assert np.all(np.abs(h - x.T @ (wn * yn)) <= 1e-9 * (np.abs(x).T @ np.abs(wn * yn)))


def test_gram_rows_threads():
    """Workspaces come from one pool: calls on several streams at a time give what they give alone."""
    jobs = [_rows(M, D, i, torch.float32) + (D,) for i, (M, D) in enumerate([(3000, 200), (500, 600), (2500, 97), (64, 33)])]
    alone = [_call(X, w, y, D, 0) for X, w, y, D in jobs]
    got = [[] for _ in jobs]

    def work(i):
        X, w, y, D = jobs[i]
        st = torch.cuda.Stream()
        for _ in range(5):
            got[i].append(_call(X, w, y, D, st.cuda_stream))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i, want in enumerate(alone):
        assert len(got[i]) == 5
        for G, h in got[i]:
            assert np.array_equal(G, want[0]) and np.array_equal(h, want[1])

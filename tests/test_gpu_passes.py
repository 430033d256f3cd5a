"""Z terms and Y rows in several passes, and with less memory than one pass asks for: rows, derivatives and
quadratic evaluation give bitwise what one pass gives (an atom's sums do not depend on its pass).

400 atoms at j_max 3 take 2.6 MB of terms and 3.1 MB of rows in FP32 (4.8 and 5.7 in FP64), 0.8 MB per
tile of 64 (FP32) or 32 (FP64) atoms; 1 MB makes passes of one tile with a remainder.  The derivatives of
12,554 pairs take 4.5 MB (9.0), the lists, rows and other buffers 2.3 (3.5), an eighth more each: 11 MB (20)
hold them with a part of a pass, but not with a whole one.  In 3 MB the derivatives fail as on a full
device, and the handle stays usable.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from test_gpu_j_range import _cell, _config  # noqa: E402


def _all(h, structs, w):
    h.set_structures([len(s[0]) for s in structs], np.concatenate([s[0] for s in structs]),
                     np.stack([s[1] for s in structs]), np.concatenate([s[2] for s in structs]))
    B, nn = h.descriptors()
    _, _, dB = h.descriptor_derivatives(int(nn.sum()))
    return (B, dB) + tuple(h.predict(w)) + tuple(h.evaluate(w))


def _handle(precision, order):
    from mld_gb300 import _lib
    h = _lib.Handle(_config(3.0 if order == 1 else 2.0, 4.7, 1, precision, order))
    w = np.random.default_rng(1).normal(0.0, 1e-3, h.dim_design_line)
    w[1 + h.dim_desc:] *= 1e-3
    return h, w


STRUCTS = [(70, 1), (3, 2), (61, 3), (66, 4), (64, 5), (40, 6), (54, 7), (42, 8)]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("order", [1, 2])
def test_passes_give_what_one_pass_gives(lib, precision, order):
    structs = [_cell(n, s) for n, s in STRUCTS]
    h, w = _handle(precision, order)
    with h:
        want = _all(h, structs, w)
        for pass_bytes in (1, 1 << 20):
            assert lib.mld_gpu_test_memory(h._h, pass_bytes, 0) == 0
            for a, b in zip(_all(h, structs, w), want):
                assert np.array_equal(a, b)


@pytest.mark.parametrize("precision,limit", [(1, 11_000_000), (0, 20_000_000)])
def test_passes_shrink_to_the_memory(lib, precision, limit):
    from mld_gb300 import _lib
    structs = [_cell(n, s) for n, s in STRUCTS]
    h, w = _handle(precision, 1)
    with h:
        want = _all(h, structs, w)
    h, w = _handle(precision, 1)
    with h:
        assert lib.mld_gpu_test_memory(h._h, 0, limit) == 0
        for a, b in zip(_all(h, structs, w), want):
            assert np.array_equal(a, b)
    h, w = _handle(precision, 1)
    with h:
        assert lib.mld_gpu_test_memory(h._h, 0, 3_000_000) == 0
        with pytest.raises(_lib.MldError) as ei:
            _all(h, structs, w)
        assert ei.value.code == 4  # MLD_ERR_OOM
        assert lib.mld_gpu_test_memory(h._h, 0, 0) == 0
        for a, b in zip(_all(h, structs, w), want):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", [0, 1])
def test_a_fit_replays_its_rows_after_smaller_passes(lib, precision):
    """Rows of a batch in whole passes, in smaller ones and in whole ones again, through one handle whose
    later calls replay a captured graph of them."""
    from mld_gb300 import _lib, synth
    ds = synth.fe_bcc_batched(n_struct=70, nmin=100, nmax=300, seed=51)
    nat, pos, cell, types = ds.arrays()
    E, F, S, has = ds.labels()
    c = _lib.default_config()
    c.j_max, c.r_cut, c.lambda_krr, c.precision = 2.0, 4.7, 1e-8, precision
    with _lib.Handle(c) as h:
        got = []
        for pass_bytes in (0, 1 << 20, 0):
            assert lib.mld_gpu_test_memory(h._h, pass_bytes, 0) == 0
            h.set_structures(nat, pos, cell, types)
            h.set_labels(E, F, S, has, np.ones((len(nat), 3)))
            got += [h.design_matrix()[0] for _ in range(3)]  # tuned, captured, replayed
    for a in got[1:]:
        assert np.array_equal(a, got[0])

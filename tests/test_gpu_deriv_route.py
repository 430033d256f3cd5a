"""Descriptors with derivatives of batches of more atoms than SMs (atoms on lanes, Y rows, k_deriv) against
the same structures one by one (one kernel, a CTA per atom; checked against the oracle elsewhere).

Sizes: an isolated atom, chunks of neighbours that just fit and that are split (r_cut), tiles of atoms with
a remainder, one and several channels, the smallest and largest j_max.  Both routes sum the same products in
different orders: FP64 1e-11, FP32 2e-5 of the largest derivative of a structure (up to 250 products of
relative error 6e-8 per sum, three sums each).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from test_gpu_j_range import _cell, _config  # noqa: E402

TOL = {0: 1e-11, 1: 2e-5}


@pytest.fixture(scope="module")
def lib():
    from mld_gb300 import _lib
    return _lib.load()


def _run(h, structs):
    """dB of all pairs and the energies and forces that the design rows give with some weights."""
    h.set_structures([len(s[0]) for s in structs], np.concatenate([s[0] for s in structs]),
                     np.stack([s[1] for s in structs]), np.concatenate([s[2] for s in structs]))
    _, nn = h.descriptors()
    _, _, dB = h.descriptor_derivatives(int(nn.sum()))
    w = np.random.default_rng(1).normal(0.0, 1e-2, h.dim_design_line)
    E, F, S = h.predict(w)
    return dB, E, F.reshape(-1), S.reshape(-1)


@pytest.mark.parametrize("precision,j_max,channels,r_cut", [
    (p, *c) for p in (0, 1) for c in ((0.5, 1, 4.7), (1.0, 2, 4.7), (2.0, 1, 4.7), (2.5, 3, 6.5), (4.0, 1, 4.7),
                                      (4.0, 1, 6.5), (4.0, 3, 5.2), (4.5, 1, 4.7))
] + [(1, 4.5, 2, 4.7), (1, 5.0, 3, 4.7)])
def test_batch_equals_single_structures(lib, precision, j_max, channels, r_cut):
    from mld_gb300 import _lib
    structs = [_cell(n, n) for n in (54, 37, 70, 61)]
    lone = _cell(2, 3)
    structs.append((lone[0][:1], np.eye(3) * 40.0, lone[2][:1]))  # an atom without neighbours
    with _lib.Handle(_config(j_max, r_cut, channels, precision, 1)) as h:
        batch = _run(h, structs)
        single = [_run(h, [s]) for s in structs]
    for got, parts in zip(batch, zip(*single)):
        assert len(got) == sum(len(x) for x in parts)
        o = 0
        for x in parts:
            if len(x):
                assert np.abs(got[o:o + len(x)] - x).max() <= TOL[precision] * np.abs(x).max()
            o += len(x)

"""Descriptors, derivatives and evaluation over the whole range of j_max and neighbour counts, where
the kernels change shape: no recursion (j_max 0), odd and even top layers, tiles of 16 lanes and
coefficients outside shared memory (j_max 4.5 and 5), and atoms with more neighbours than one pass
of the U store holds.  Bars as elsewhere: 1e-10 (FP64) and 2e-5 (mixed), max-norm relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {0: 1e-10, 1: 2e-5}


def _cell(n, seed):
    from mld_gb300 import synth
    rng = np.random.default_rng(seed)
    pos, cell = synth.bcc(3, 3, 4, synth.FE_A)
    pos = pos[np.sort(rng.choice(len(pos), size=n, replace=False))] + rng.normal(0.0, 0.1, size=(n, 3))
    return pos, cell, rng.integers(0, 2, size=n).astype(np.int32)


def _config(j_max, r_cut, channels, precision, order=1):
    from mld_gb300 import _lib
    c = _lib.default_config()
    c.j_max, c.r_cut, c.precision, c.mld_order, c.n_elements = j_max, r_cut, precision, order, 2
    c.weighted, c.weighted_3ch = int(channels > 1), int(channels > 2)
    for i, (a, b) in enumerate(((0.4, 0.9), (0.7, 1.3))):
        c.weight_per_element[i], c.weight_per_element_3ch[i] = a, b
    return c


def _rel(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("j_max,channels", [(0.0, 1), (0.5, 3), (1.0, 2), (3.5, 2), (4.5, 1), (5.0, 3)])
@pytest.mark.parametrize("n", [1, 33, 65])
def test_descriptors(lib, precision, j_max, channels, n):
    import oracle
    from mld_gb300 import _lib
    pos, cell, types = _cell(n, 3 * n + 1)
    with _lib.Handle(_config(j_max, 4.7, channels, precision)) as h:
        h.set_structures([n], pos, cell[None], types)
        B, nn = h.descriptors()
    chw = np.array([[1.0, 1.0], [0.4, 0.7], [0.9, 1.3]])[:channels]
    d = oracle.bispectrum(pos, cell, types, 4.7, j_max, channel_weights=chw, want_deriv=False)
    assert np.array_equal(nn, d["nn"])
    assert _rel(B, d["B"]) <= TOL[precision]


@pytest.mark.parametrize("precision,j_max", [(0, 0.5), (0, 4.5), (1, 3.5), (1, 4.5), (1, 5.0)])
def test_derivatives(lib, precision, j_max):
    import oracle
    from mld_gb300 import _lib
    pos, cell, types = _cell(40, 7)
    with _lib.Handle(_config(j_max, 6.5, 1, precision)) as h:  # about 100 neighbours
        h.set_structures([40], pos, cell[None], types)
        _, nn = h.descriptors()
        _, _, dB = h.descriptor_derivatives(int(nn.sum()))
    d = oracle.bispectrum(pos, cell, types, 6.5, j_max, channel_weights=np.ones((1, 2)))
    assert _rel(dB, np.concatenate([d["dB"][i, :k] for i, k in enumerate(d["nn"])])) <= TOL[precision]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("j_max,channels,order,r_cut", [
    (0.5, 1, 1, 4.7), (4.0, 3, 1, 6.5), (4.5, 1, 1, 6.5), (2.0, 1, 2, 6.5), (2.5, 3, 2, 6.5), (4.0, 2, 2, 4.7)])
def test_evaluation_equals_the_rows(lib, precision, j_max, channels, order, r_cut):
    """Energies, forces and stress of mld_gpu_evaluate against the design rows of mld_gpu_predict (other
    kernels), with up to about 100 neighbours per atom."""
    from mld_gb300 import _lib
    structs = [_cell(n, n) for n in (2, 37, 70)]
    rng = np.random.default_rng(5)
    with _lib.Handle(_config(j_max, r_cut, channels, precision, order)) as h:
        h.set_structures([len(s[0]) for s in structs], np.concatenate([s[0] for s in structs]),
                         np.stack([s[1] for s in structs]), np.concatenate([s[2] for s in structs]))
        w = rng.normal(0.0, 1e-3, h.dim_design_line)
        w[1 + h.dim_desc:] *= 1e-3
        got, ref = h.evaluate(w), h.predict(w)
    for a, b in zip(got, ref):
        assert _rel(a, b) <= TOL[precision]

"""Energy and stress of structures whose atoms are summed in one part or in several (1024 atoms a part):
evaluation against the design rows times the weights, with structures on both sides of the edges in
one batch, and each one alone (bitwise: a structure's sums do not depend on its batch)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {0: 1e-10, 1: 2e-5}


@pytest.mark.parametrize("precision", [0, 1])
def test_structure_sums(lib, precision):
    from mld_gb300 import _lib, synth
    pos, cell = synth.bcc(10, 10, 11, synth.FE_A)
    rng = np.random.default_rng(7)
    structs = []
    for n in (2, 1023, 1024, 1025, 2049, 2200):
        keep = np.sort(rng.choice(len(pos), size=n, replace=False))
        structs.append(pos[keep] + rng.normal(0.0, 0.05, size=(n, 3)))
    c = _lib.default_config()
    c.j_max, c.r_cut, c.precision = 1.5, 4.0, precision
    nat = [len(p) for p in structs]
    cells = np.repeat(cell[None], len(structs), 0)
    with _lib.Handle(c) as h:
        h.set_structures(nat, np.concatenate(structs), cells, np.zeros(sum(nat), np.int32))
        w = rng.normal(0.0, 1e-2, h.dim_design_line)
        E, F, S = h.evaluate(w)
        Ep, Fp, Sp = h.predict(w)
        for a, b in ((E, Ep), (F, Fp), (S, Sp)):
            assert np.abs(a - b).max() <= TOL[precision] * np.abs(b).max()
        o = 0
        for i, p in enumerate(structs):
            h.set_structures([len(p)], p, cell[None], np.zeros(len(p), np.int32))
            e, f, s = h.evaluate(w)
            assert e[0] == E[i] and np.array_equal(np.ravel(s), np.ravel(S[i]))
            assert np.array_equal(np.ravel(f), np.ravel(F[o:o + len(p)]))
            o += len(p)

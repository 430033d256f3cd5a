"""The mixed evaluation takes the linear weights in more than 32 bits: the energy follows a change of all
weights by 2^-24, which 32-bit weights (here exactly representable ones) cannot hold.

8,192 Fe atoms, every term w_k B_k positive, no constant: E changes by the factor 1 + 2^-24.  The two
evaluations round at random within about 3 * 2^-24 of an atom's energy, 0.03 * 2^-24 of the sum of 8,192
atoms: a quarter of 2^-24 is eight times that.  The plain method holds it to rounding.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,order", [(0, 1), (1, 1), (1, 2)])
def test_energy_follows_the_last_bits_of_the_weights(lib, precision, order):
    from mld_gb300 import _lib, synth
    pos, cell = synth.bcc(16, 16, 16, synth.FE_A)
    pos = pos + np.random.default_rng(5).normal(0.0, 0.08, size=pos.shape)
    c = _lib.default_config()
    c.j_max, c.r_cut, c.precision, c.mld_order = 2.0, 4.7, precision, order
    with _lib.Handle(c) as h:
        h.set_structures([len(pos)], pos, cell[None], np.zeros(len(pos), np.int32))
        B, _ = h.descriptors()
        w = np.zeros(h.dim_design_line)
        w[1:1 + h.dim_desc] = np.sign(B.mean(0)) * 2.0 ** -10
        E1, E2 = h.evaluate(w)[0][0], h.evaluate(w * (1.0 + 2.0 ** -24))[0][0]
    assert E1 > 0.0
    assert abs((E2 - E1) / E1 * 2.0 ** 24 - 1.0) <= 0.25

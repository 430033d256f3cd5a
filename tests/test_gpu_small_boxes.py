"""Neighbour search of small boxes (periodic images) against the oracle's scan of every image: lists
equal in order, displacements within FP64 rounding.  Cases: one atom per cell, skewed cells,
unwrapped coordinates, one thin direction, and two thin directions (more images per atom than the
bit masks hold, the general scan)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RCUT = 4.7
CELLS = {
    "one_atom": (1, np.diag([2.9, 3.1, 3.0]), 0),
    "two_atoms_thin_first": (2, np.diag([1.3, 8.0, 9.0]), 0),
    "two_thin_directions": (2, np.diag([8.5, 1.2, 1.3]), 0),
    "skewed": (5, np.array([[6.0, 0.0, 0.0], [2.5, 5.5, 0.0], [-2.0, 1.5, 6.5]]), 0),
    "unwrapped": (33, np.diag([7.5, 8.1, 7.7]), 1),
    "many": (60, np.array([[9.0, 0.4, 0.0], [0.0, 9.2, 0.3], [0.2, 0.0, 9.1]]), 0),
}


@pytest.mark.parametrize("name", list(CELLS))
def test_small_box_lists_match_the_oracle(lib, name):
    import oracle
    from mld_gb300 import _lib
    n, cell, unwrap = CELLS[name]
    rng = np.random.default_rng(len(name))
    frac = rng.random((n, 3))
    if unwrap:
        frac = frac + rng.integers(-1, 2, size=(n, 3))
    pos = frac @ cell
    c = _lib.default_config()
    c.j_max, c.r_cut, c.precision = 1.0, RCUT, _lib.PLAIN_FP64
    with _lib.Handle(c) as h:
        h.set_structures([n], pos, cell[None], np.zeros(n, np.int32))
        _, nn = h.descriptors()
        nbr, u, _ = h.descriptor_derivatives(int(nn.sum()))
    o_nn, o_nbr, o_u, small = oracle.neighbours(pos, cell, RCUT)
    assert small and np.array_equal(nn, o_nn)
    assert np.array_equal(nbr, np.concatenate([o_nbr[i, :k] for i, k in enumerate(o_nn)]))
    assert np.abs(u - np.concatenate([o_u[i, :k] for i, k in enumerate(o_nn)])).max() <= 1e-12 * RCUT

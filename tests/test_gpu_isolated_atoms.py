"""Many atoms without neighbours behind ordinary ones in the work queue of the descriptor and evaluation
kernels: a CTA takes several of them one after the other, without a barrier of their own.

An atom without neighbours has B = 0, the constant as its energy, no force and no stress, exactly (the
energy of 2,197 equal terms in FP64: 1e-12).  The ordinary structures are bitwise what they are alone.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from test_gpu_j_range import _cell, _config  # noqa: E402


def _grid(n):
    """n^3 atoms at a distance of 12: about seven per persistent CTA."""
    g = 12.0 * np.arange(n)
    pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    return pos, np.eye(3) * 12.0 * n, (np.arange(n ** 3) % 2).astype(np.int32)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("channels,order", [(1, 1), (2, 1), (2, 2)])
def test_isolated_atoms_in_a_batch(lib, precision, channels, order):
    from mld_gb300 import _lib
    structs = [_cell(54, 1), _grid(13), _cell(70, 2)]
    rng = np.random.default_rng(9)
    with _lib.Handle(_config(2.0, 4.7, channels, precision, order)) as h:
        w = rng.normal(0.0, 1e-3, h.dim_design_line)
        w[1 + h.dim_desc:] *= 1e-3

        def run(s):
            h.set_structures([len(x[0]) for x in s], np.concatenate([x[0] for x in s]), np.stack([x[1] for x in s]),
                             np.concatenate([x[2] for x in s]))
            B, nn = h.descriptors()
            return (B, nn) + tuple(h.evaluate(w))

        alone = [run([structs[0]]), run([structs[2]])]
        for _ in range(5):
            B, nn, E, F, S = run(structs)
            lone = slice(54, 54 + 13 ** 3)
            assert not nn[lone].any() and not B[lone].any()
            assert abs(E[1] - 13 ** 3 * w[0]) <= 1e-12 * abs(13 ** 3 * w[0])
            assert not F[lone].any() and not S[1].any()
            for i, s, at in ((0, 0, slice(0, 54)), (1, 2, slice(54 + 13 ** 3, None))):
                assert np.array_equal(B[at], alone[i][0]) and np.array_equal(nn[at], alone[i][1])
                assert E[s] == alone[i][2][0] and np.array_equal(F[at], alone[i][3]) and np.array_equal(S[s], alone[i][4][0])

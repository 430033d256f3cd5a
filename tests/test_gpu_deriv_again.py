"""Derivatives asked for again: a second call returns what the first one formed, until the structures or
their lists are formed anew (another batch, other calls on the handle in between)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from test_gpu_j_range import _cell, _config  # noqa: E402


@pytest.mark.parametrize("precision", [0, 1])
def test_derivatives_again(lib, precision):
    from mld_gb300 import _lib
    one, two = [_cell(54, 1)], [_cell(n, n) for n in (70, 61, 66)]
    with _lib.Handle(_config(2.0, 4.7, 2, precision, 1)) as h:
        def stage(s):
            h.set_structures([len(x[0]) for x in s], np.concatenate([x[0] for x in s]), np.stack([x[1] for x in s]),
                             np.concatenate([x[2] for x in s]))
            return int(h.descriptors()[1].sum())

        w = np.random.default_rng(2).normal(0.0, 1e-2, h.dim_design_line)
        want = {}
        for name, s in (("one", one), ("two", two)):
            want[name] = h.descriptor_derivatives(stage(s))
        for name, s in (("one", one), ("two", two), ("one", one)):
            P = stage(s)
            for between in (lambda: None, lambda: h.predict(w), lambda: h.evaluate(w), h.descriptors, lambda: None):
                between()
                for a, b in zip(h.descriptor_derivatives(P), want[name]):
                    assert np.array_equal(a, b)

"""A batch's launch shapes are kept per kind of pass: what was tuned while the
members took two steps per pass is not the shape of single steps, nor the
other way round."""
import numpy as np
import pytest

from pfa_gb300 import ic

pytestmark = pytest.mark.gpu

GIB = 1 << 30
SMALL, LARGE = (202, 302), (1602, 1602)  # with LARGE the records exceed 96 MB: two steps per pass


def _fields(shape):
    return ic.grid2d(shape[1] - 2, shape[0] - 2, seed=shape[0], stripe_width=20, n_particles=2, radius=4.0)


def _shape_of(pfa, shapes):
    """The launch shape of an untuned batch of these members."""
    b = pfa.Batch(pfa.model_params(), GIB)
    for s in shapes:
        b.add(_fields(s))
    out = b.launch()
    b.close()
    return out


def test_tuned_shapes_stay_with_their_kind_of_pass(pfa):
    b = pfa.Batch(pfa.model_params(), GIB)
    b.add(_fields(SMALL))
    k = b.add(_fields(LARGE))
    b.tune(2)
    two = b.launch()
    assert two["rows"] >= 9
    b.remove(k)  # single steps from here
    assert b.launch() == _shape_of(pfa, [SMALL])
    b.tune(2)
    one = b.launch()
    k = b.add(_fields(LARGE))
    assert b.launch() == two
    b.remove(k)
    assert b.launch() == one
    b.set_launch(7, True)  # fixed for both
    assert (b.launch()["rows"], b.launch()["persistent"]) == (7, True)
    b.add(_fields(LARGE))
    assert (b.launch()["rows"], b.launch()["persistent"]) == (7, True)
    b.close()


def test_single_step_of_a_tuned_large_batch(pfa):
    """The odd step of a run whose double passes were tuned: the same bits as
    without tuning."""
    out = []
    for tuned in (False, True):
        b = pfa.Batch(pfa.model_params(), GIB)
        slots = [b.add(_fields(s)) for s in (SMALL, LARGE)]
        if tuned:
            b.tune(2)
        b.run(5)
        out.append([b.read(k) for k in slots])
        b.close()
    for f, g in zip(*out):
        for x, y in zip(f, g):
            assert np.array_equal(x[1:-1, 1:-1], y[1:-1, 1:-1])

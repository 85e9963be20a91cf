"""The quintic spline weights of a shift for every float64 that may come: the sum of the six truncated powers, term by term."""
import numpy as np
import pytest

from hcipy_gb300.atmosphere import quintic_weights


def term_by_term(shift):
    f, b = abs(shift), []
    for offset in (2.0 + f, 1.0 + f, f, 1.0 - f, 2.0 - f, 3.0 - f):
        acc, x = 0.0, offset + 3.0
        for c in (1.0, -6.0, 15.0, -20.0, 15.0, -6.0, 1.0):
            if x > 0.0:
                acc += c * x**5
            x -= 1.0
        b.append(acc / 120.0)
    return [0.0] + b if shift >= 0 else b[::-1] + [0.0]


@pytest.mark.parametrize('shift', [0.0, -0.0, 0.5, -0.5, 0.3, -1e-300, 1.0, -2.75, 7.5, float('nan'), float('inf'),
                                   float('-inf')])
def test_weights(shift):
    np.testing.assert_array_equal(quintic_weights(shift), np.array(term_by_term(shift)))

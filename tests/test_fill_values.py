"""Parameter vectors go into an engine's buffer as an array assignment takes
them: any sequence of numbers, what broadcasts to the buffer, and the same
exception for what does not."""
import numpy as np
import pytest

VALUES = [1.5, -2.0, 0.25]


@pytest.mark.parametrize("values", [
    VALUES, tuple(VALUES), np.array(VALUES), np.array(VALUES, np.float32), [1, 2, 3],
    np.array([VALUES]), np.array(VALUES)[::-1], [2.5], 4.0, np.array(7), [True, 2.0, np.float64(3)],
    ["1.5", "2", "3"], np.array(VALUES * 2)[::2]])
def test_accepted(values):
    from tf_pwa_b200.engine import _fill

    want, got = np.zeros(3), np.zeros(3)
    want[:] = values
    _fill(got, values)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("values", [[1.0, 2.0], [1.0] * 4, np.zeros((2, 3)), [], [1.0, "x", 2.0],
                                    [1.0, 1j, 2.0]])
def test_refused(values):
    from tf_pwa_b200.engine import _fill

    with pytest.raises(Exception) as want:
        np.zeros(3)[:] = values
    with pytest.raises(want.type):
        _fill(np.zeros(3), values)

"""The predicted time of a sweep follows the measured rates within a factor of three, wide and narrow."""
import pytest

from tropidist_gb300 import auto


# (peak bits, state-updates, measured seconds) of one uint8 sweep, 1000 x 2000 banded plans
@pytest.mark.parametrize("bits,work,seconds", [
    (31, 2.31e11, 19.6e-3), (30, 6.76e10, 6.51e-3), (28, 2.38e10, 2.92e-3), (26, 4.9e9, 1.74e-3), (24, 1.9e9, 1.72e-3),
    (22, 5.98e8, 2.12e-3), (21, 2.47e8, 2.71e-3), (19, 3.87e7, 2.33e-3), (16, 1.52e7, 1.41e-3)])
def test_prediction_is_near_the_measurement(bits, work, seconds):
    assert seconds / 3 <= auto.predicted_seconds(work, bits) <= 3 * seconds

"""The terrain's value noise at coordinates just below zero, whose remainder rounds to the period."""
import numpy as np

from aurora_b200 import scenes


def test_just_below_zero():
    x = np.array([[-1e-17, 0.0, 0.3]])
    h = scenes.value_noise_fbm(x, np.zeros_like(x), 5, 0.3, 4)
    assert h[0, 0] == h[0, 1]

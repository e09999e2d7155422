"""The autotuner's choice among shapes that are one launch: the same one in every run, whatever the timing's noise."""
import pytest

pytest.importorskip("torch")


def test_noise_does_not_choose_between_equal_shapes():
    from cemc_gb300 import autotune
    shapes = [(4, 1, 0), (8, 1, 0), (16, 1, 0), (8, 1, 6)]
    picks = {autotune._pick({s: 1e9 * (0.5 if s[0] == 4 else 1.0 + 0.002 * ((7 * i + 3 * k) % 5))
                             for k, s in enumerate(shapes)}) for i in range(10)}
    assert picks == {(8, 1, 0)}
    assert autotune._pick({(4, 1, 0): 1.0, (8, 1, 0): 1.03, (16, 1, 0): 1.035}) == (8, 1, 0)

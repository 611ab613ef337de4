"""Plans of sets whose indices span more than 2^31 along an axis: their tables' extents are formed in 64 bits, so that segments
too far apart for one table are never put into one."""
import numpy as np
import pytest

from test_plan_cpu import _run, plan_check  # noqa: F401  (the fixture)


@pytest.mark.parametrize("d", [1, 2, 3])
def test_indices_of_both_signs_near_the_limits(plan_check, d):  # noqa: F811
    rng = np.random.default_rng(d)
    top = 2 ** 31 - 1
    near = np.stack(np.meshgrid(*[np.arange(-5, 6)] * d, indexing="ij"), -1).reshape(-1, d)
    modes = np.concatenate([rng.integers(-top, top + 1, (150, d)), near, [[-top] * d, [top] * d]])
    _run(plan_check, [(rng.permutation(modes), np.ones(len(modes)))])

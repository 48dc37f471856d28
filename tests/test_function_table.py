"""What FunctionTable refuses before it reaches the GPU (no device needed)."""
from types import SimpleNamespace

import pytest

from pyquante_b200.engine import FunctionTable


def _bf(origin=(0.0, 0.0, 0.0), powers=(0, 0, 0), **kw):
    return SimpleNamespace(**dict(dict(origin=origin, powers=powers, pexps=[1.0], pcoefs=[1.0], pnorms=[1.0], norm=1.0),
                                  **kw))


@pytest.mark.parametrize("bfs", [
    [_bf(origin=(0.0, 0.0))],
    # two functions whose components add up to three each
    [_bf(origin=(0.0, 0.0)), _bf(origin=(0.0, 0.0, 0.0, 0.0))],
    [_bf(powers=(0, 0, 0, 1)), _bf(powers=(0, 0))],
    [_bf(pexps=[])],
    [_bf(pcoefs=[1.0, 2.0])],
    [_bf(pnorms=[])],
])
def test_inconsistent_functions_are_refused(bfs):
    with pytest.raises(ValueError):
        FunctionTable(bfs, 0)

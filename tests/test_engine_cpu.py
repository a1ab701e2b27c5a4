"""CPU tests of the engines' host side: what is handed to the kernels, and which plans are
taken, without a GPU."""

import pytest
import torch

from gravitation_gb300 import build as gbuild
from gravitation_gb300.adjoint import AdjointEngine


@pytest.fixture(scope='module', autouse=True)
def lib():
    gbuild.build()


@pytest.mark.parametrize('steps', [1, 2, 5])
def test_adjoint_steps_hands_over_the_stored_rows(steps):
    """Without a chained launch every backward step reads the caller's own accelerations, the
    last first, on the stream given."""
    eng = AdjointEngine.__new__(AdjointEngine)
    eng.chained, eng.sizes = False, [3]
    eng.device = torch.device('cpu')
    seen = []
    eng.step = lambda stream=None, a_in=None: seen.append((stream, a_in.data_ptr()))
    a = torch.arange(steps * 12, dtype=torch.float64).reshape(steps, 3, 4)
    eng.steps(a, stream='s')
    assert seen == [('s', a[k].data_ptr()) for k in reversed(range(steps))]

"""A call whose launch is refused (more threads than the kernel is built for) fails alone: the next call
of the same and of another engine works."""
import numpy as np
import pytest
import torch

from radtranbook_b200 import _lib
from radtranbook_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _engine(cuda):
    e = np.linspace(0.0, 1.0, 21)
    f = lambda v: torch.full((20,), v, dtype=torch.float64, device=cuda)  # noqa: E731
    return Engine("slab", e, np.array([0.0, 1.0]), np.diff(e)), (f(0.5), f(10.0), f(0.3))


def _step(eng, mat):
    eng.init_census(mat[0], 1000)
    return eng.transport(*mat, None, 1, 0.01, 1.0, 500, 0, 0, [None] * 4, (False,) * 4).report.n_transported


@pytest.mark.parametrize("other", [False, True])
def test_the_call_after_a_refused_launch(cuda, other):
    eng, mat = _engine(cuda)
    want = _step(eng, mat)
    eng.launch["block_size"] = 512
    with pytest.raises(_lib.ImcError, match="IMC_ERR_CUDA"):
        _step(eng, mat)
    eng.launch["block_size"] = 256
    assert _step(_engine(cuda)[0] if other else eng, mat) == want

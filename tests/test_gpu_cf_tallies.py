"""Carter-Forest with block tallies against the event-by-event form: w*s is added at every flight, the
lanes of one cell of a warp as one where there are several.  One cell (every lane), a few (some), many
(none), from one to many warps of histories, open and closed.

As the event form's own test: statistics exact, deposition and escapes relative 1e-12, intensity
relative L1 1e-12 (FP64 sums in another order)."""
import numpy as np
import pytest
import torch

from radtranbook_b200 import _lib
from radtranbook_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geometry", ["slab", "spherical", "xy"])
@pytest.mark.parametrize("nx,n", [(1, 3), (1, 33), (1, 40_000), (4, 5_000), (40, 40_000), (1200, 60_000)])
@pytest.mark.parametrize("closed", [False, True])
def test_intensity_matches_the_event_form(cuda, geometry, nx, n, closed):
    e1 = np.linspace(0.0, 0.5, nx + 1)
    e2 = np.linspace(0.0, 0.3, 2) if geometry == "xy" else np.array([0.0, 1.0])
    vol = {"slab": np.diff(e1), "spherical": 4 / 3 * np.pi * np.diff(e1 ** 3), "xy": np.diff(e1) * 0.3}[geometry]
    T = np.linspace(0.9, 0.4, nx)
    dev = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=cuda)  # noqa: E731
    runs = []
    for event in (0, 1):
        eng = Engine(geometry, e1, e2, vol, seed=0xCF7)
        eng.launch["event_based"] = event
        eng.init_census(dev(T), n)
        eng.transport(dev(T), dev(20.0 * T ** -1.0), dev(np.full(nx, 0.5)), None, 3, 2e-3, 1.0, n, 0 if closed else n, 0,
                      [None if closed else dev([1.0]), None, None, None], (closed,) * 4, max_events=1_000_000,
                      method=_lib.METHOD_CARTER_FOREST)
        runs.append((*eng.host_stats(), eng.dep.cpu().numpy(), eng.si.cpu().numpy()))
    (st, esc, dep, si), (st1, esc1, dep1, si1) = runs
    np.testing.assert_array_equal(st, st1)
    np.testing.assert_allclose(esc, esc1, rtol=1e-12, atol=0)
    np.testing.assert_allclose(dep, dep1, rtol=1e-12, atol=0)
    assert np.abs(si - si1).sum() <= 1e-12 * np.abs(si1).sum() and si1.sum() > 0

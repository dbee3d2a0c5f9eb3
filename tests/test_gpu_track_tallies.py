"""Where the tracking kernel sums its tallies: per block in shared memory (small meshes), one wide
block per SM with its main tally in shared memory (meshes up to about 26 thousand (group, cell)
entries), or global memory.  Each form against the event-by-event loop, which keeps its tallies in
global memory and stores every history as it ends: one transport step from the same census.

The histories are the same, so event statistics and the census agree exactly.  Deposition and
escaped energy are integer sums in units of a quantum that follows the FP64 sum of the tracked
weights (added in a run-dependent order, a few units of 2^-53 of it), so they agree to 1e-13; the
intensity of cells without absorption is an FP64 sum of at most 1e6 terms in another order: 1e-12.
Mesh sizes: both sides of the small-mesh limit (2048 entries) and of the wide block's.
"""
import numpy as np
import pytest
import torch

from radtranbook_b200 import _lib
from radtranbook_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _step(geometry, n1, n2, cuda, launch, ng=1, method=0):
    rng = np.random.default_rng(n1 * 1000 + n2)
    e1, e2 = np.linspace(0.0, 1.0, n1 + 1), np.linspace(0.0, 2.0, n2 + 1)
    vol = (np.pi * (e1[1:] ** 2 - e1[:-1] ** 2)[:, None] if geometry == "rz" else np.diff(e1)[:, None]) * np.diff(e2)
    nc = n1 * n2
    T = 0.1 + 0.4 * rng.random(nc)
    sig = 10.0 ** rng.uniform(-1.0, 2.5, (ng, nc))
    sig[:, : nc // 7] = 0.0  # cells without absorption
    d = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64).reshape(-1), device=cuda)  # noqa: E731
    eng = Engine(geometry, e1, e2, vol.T.reshape(-1), seed=0x7A11, n_groups=ng,
                 group_edges=np.logspace(-2, 1, ng + 1) if ng > 1 else None)
    eng.launch.update(launch)
    eng.init_census(d(T), 30_000)
    eng.transport(d(T), d(sig), d(np.full(nc, 0.05)), None, 3, 0.01, 1.0, 8000, 4000, 0,
                  [d(np.full(n2, 0.5)), None, d(np.full(n1, 0.4)), None], (False, True, False, False),
                  max_events=2000, rz_linear_source=geometry == "rz", method=method)
    stats, esc = eng.host_stats()
    w = eng.bank.view("weight").cpu().numpy()
    bank = [np.where(w > 0, eng.bank.view(k).cpu().numpy(), 0) for k in ("pos1", "pos2", "dir1", "dir2", "cell")]
    return stats, esc, eng.dep.cpu().numpy(), eng.si.cpu().numpy(), [w] + bank


@pytest.mark.parametrize("geometry,n1,n2,ng,method", [
    ("rz", 32, 64, 1, 0), ("rz", 41, 50, 1, 0), ("rz", 160, 165, 1, 0), ("rz", 165, 170, 1, 0),
    ("xy", 45, 46, 1, 0), ("xy", 7, 3, 1, 0), ("rz", 60, 70, 1, _lib.METHOD_CARTER_FOREST),
    ("xy", 50, 50, 1, _lib.METHOD_CARTER_FOREST), ("rz", 30, 41, 3, 0), ("xy", 60, 61, 9, 0)])
@pytest.mark.parametrize("shape", [(256, 4), (128, 1), (96, 3)])
def test_tally_forms_match_event_loop(cuda, geometry, n1, n2, ng, method, shape):
    a = _step(geometry, n1, n2, cuda, {"event_based": 1}, ng, method)
    b = _step(geometry, n1, n2, cuda, {"block_size": shape[0], "blocks_per_sm": shape[1]}, ng, method)
    np.testing.assert_array_equal(a[0], b[0])
    assert a[0][_lib.STAT_EVENTS] > 10_000
    np.testing.assert_allclose(a[1], b[1], rtol=1e-13)
    np.testing.assert_allclose(a[2], b[2], rtol=1e-13, atol=1e-13 * np.abs(a[2]).max())
    assert np.abs(a[3] - b[3]).sum() <= 1e-12 * np.abs(a[3]).sum()
    for x, y in zip(a[4], b[4]):
        np.testing.assert_array_equal(x, y)

"""A fixed source of zeros with a particle count: no source particles, and the step is the one without a
source, whatever the workspace held before (the plan writes no tables for such a source; the sum of the
tracked weights, which sets the weight floor and the tallies' unit, must not read them)."""
import numpy as np
import pytest
import torch

from radtranbook_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geometry,ng", [("slab", 1), ("spherical", 1), ("xy", 1), ("rz", 1), ("spherical", 3), ("xy", 3)])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_zero_source_is_no_source(cuda, geometry, ng, seed):
    e1 = np.linspace(0.1, 1.0, 11)
    e2 = np.linspace(0.0, 1.0, 6) if geometry in ("xy", "rz") else np.array([0.0, 1.0])
    nc = 10 * (len(e2) - 1)
    edges = np.geomspace(0.05, 10.0, ng + 1) if ng > 1 else None
    dev = lambda v, n: torch.full((n,), v, dtype=torch.float64, device=cuda)  # noqa: E731
    runs = []
    for source, n_source in ((None, 0), (dev(0.0, nc * ng), 5000)):
        eng = Engine(geometry, e1, e2, np.full(nc, 0.05), seed=0x50, n_groups=ng, group_edges=edges)
        eng.bank.ensure(40_000)
        eng._ws(eng.bank.capacity)
        eng.init_census(dev(0.5, nc), 3000)
        gen = torch.Generator(device=cuda).manual_seed(seed)
        eng.ws.copy_(torch.randint(0, 256, eng.ws.shape, dtype=torch.uint8, device=cuda, generator=gen))
        rep = eng.transport(dev(0.5, nc), dev(20.0, nc * ng), dev(0.1, nc), source, 2, 2e-3, 1.0, 4000, 2000, n_source,
                            [dev(0.8, len(e2) - 1 if len(e2) > 2 else 1), None, None, None], (False, True, True, True),
                            max_events=0 if geometry in ("slab", "spherical") else 1_000_000, rz_linear_source=ng == 1).report
        assert rep.n_source == 0
        runs.append((rep.n_transported, rep.weight_floor, *eng.host_stats(), eng.dep.cpu().numpy()))
    (n0, w0, st0, es0, d0), (n1, w1, st1, es1, d1) = runs
    assert n0 == n1 and st0[0] > 5000
    np.testing.assert_allclose(w1, w0, rtol=1e-12)
    np.testing.assert_array_equal(st0, st1)
    np.testing.assert_allclose(es1, es0, rtol=1e-11, atol=0)
    np.testing.assert_allclose(d1, d0, rtol=1e-11, atol=0)

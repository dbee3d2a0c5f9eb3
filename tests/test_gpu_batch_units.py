"""The batched tracking's work units against its entry queue (tables and tallies in global memory,
a lane refilled whenever its history ends): the same histories, so event counts and census sizes
agree exactly; depositions are integer sums in units of a quantum that follows each instance's FP64
weight sum (added in a run-dependent order), so temperatures agree to 1e-12 after three steps.
Sizes: one instance, instances of one cell and of two particles, instances without any particle
(no boundary source, cold), more instances than a block has threads, reflecting faces.
"""
import numpy as np
import pytest

from radtranbook_b200 import batch

pytestmark = pytest.mark.gpu


def _spec(K, cells, particles, reflect, cold):
    rng = np.random.default_rng(K * 7 + cells)
    n = np.maximum(rng.integers(1, cells + 1, K), 1)
    N = rng.integers(2, particles + 1, K)
    face = np.stack([np.where(rng.random(K) < cold, 0.0, rng.uniform(0.3, 1.0, K)), np.zeros(K)], 1)
    return batch.BatchSpec(n_cells=n, length=rng.uniform(0.05, 0.5, K), n_target=N - N // 2, n_boundary=N // 2,
                           n_max=4 * N, opacity_a=10.0 ** rng.uniform(0, 2.5, K), opacity_p=np.full(K, -3.0),
                           cv=rng.uniform(0.05, 1.0, K), face_T=face, reflect=np.full(K, reflect, np.int32),
                           seed=rng.integers(1, 2 ** 62, K, dtype=np.uint64))


@pytest.mark.parametrize("K,cells,particles,reflect,cold,shape", [
    (1, 1, 2, 0, 0.0, (256, 4)), (1, 800, 5000, 0, 0.0, (256, 4)), (300, 60, 400, 0, 0.3, (256, 4)),
    (40, 3, 9, 3, 0.0, (128, 1)), (70, 200, 3000, 2, 0.5, (96, 5))])
def test_units_match_entry_queue(cuda, K, cells, particles, reflect, cold, shape):
    spec = _spec(K, cells, particles, reflect, cold)
    out = []
    for form in (1, 2):
        eng = batch.BatchEngine(spec)
        eng.launch.update(form=form, block_size=shape[0], blocks_per_sm=shape[1])
        eng.init()
        eng.step(3, graph=False)
        eng.check()
        out.append((eng.s["stats"].cpu().numpy(), eng.census_sizes(), eng.s["T"].cpu().numpy(),
                    eng.s["tr"].cpu().numpy()))
    a, b = out
    np.testing.assert_array_equal(a[0], b[0])
    np.testing.assert_array_equal(a[1], b[1])
    np.testing.assert_allclose(a[2], b[2], rtol=1e-12)
    np.testing.assert_allclose(a[3], b[3], rtol=1e-12, atol=1e-15)

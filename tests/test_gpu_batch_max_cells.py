"""imc_batch.max_cells below the largest instance's cells (the caller's word; the entry-queue form does
not stage tables by it): the plan's shared-memory counts go by each instance's own cells, and the run is
the one with the right value."""
import numpy as np
import pytest

from radtranbook_b200 import batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("said", [0, 1, 39])
def test_queue_form_with_a_small_max_cells(cuda, said):
    K, cells = 6, np.array([40, 3, 700, 39, 1, 40])
    rng = np.random.default_rng(5)
    spec = batch.BatchSpec(n_cells=cells, length=rng.uniform(0.1, 0.4, K), n_target=np.full(K, 500),
                           n_boundary=np.full(K, 500), n_max=np.full(K, 800), opacity_a=10.0 ** rng.uniform(0, 2, K),
                           opacity_p=np.full(K, -3.0), cv=rng.uniform(0.05, 1.0, K),
                           face_T=np.stack([rng.uniform(0.5, 1.0, K), np.zeros(K)], 1),
                           reflect=np.zeros(K, np.int32), seed=rng.integers(1, 2 ** 62, K, dtype=np.uint64))
    runs = []
    for max_cells in (int(cells.max()), said):
        eng = batch.BatchEngine(spec)
        eng.launch["form"] = 2
        eng.cb.max_cells = max_cells
        eng.init()
        eng.step(3, graph=False)
        eng.check()
        runs.append(eng)
    # the batch's own tolerance: FP64 sums in another order, an FP32 near-tie that flips counts once
    for a, b in zip(runs[1].field("T"), runs[0].field("T")):
        assert np.abs(a - b).sum() <= 1e-4 * np.abs(b).sum()

"""The batched comb against the single-problem one, whose copies it must reproduce in order (a history's
draws follow its place in the bank, so a copy out of place shows in every later event): entries of many
thousand copies (several windows of a tile), instances of a few entries (many per tile), tiles that
straddle instances, instances that start off a multiple of four, combs that thin and that multiply.

Tolerances as for the batch's other parity tests: FP64 atomics add in a different order, and a history
whose event order flips on an FP32 near-tie counts once: median relative L1 of T 1e-9, largest 1e-4."""
import numpy as np
import pytest

from radtranbook_b200 import batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reflect", [0, 3])  # 3: thin and closed, every census lives to be combed
@pytest.mark.parametrize("K,cells,particles,n_max", [
    (2, 3, 5, 60_000), (45, 4, 9, 30), (5, 20, 1023, 1025), (3, 7, 4097, 500), (6, 50, 700, 20_000)])
def test_batched_comb_matches_single_problem(cuda, K, cells, particles, n_max, reflect):
    rng = np.random.default_rng(K * 31 + particles)
    N = particles + np.arange(K) % 3
    spec = batch.BatchSpec(n_cells=np.full(K, cells), length=rng.uniform(0.1, 0.4, K), n_target=N - N // 2,
                           n_boundary=N // 2, n_max=np.full(K, n_max), opacity_a=10.0 ** rng.uniform(0, 2, K) * (0.05 if reflect else 1.0),
                           opacity_p=np.full(K, 0.0 if reflect else -3.0), cv=rng.uniform(0.05, 1.0, K),
                           face_T=np.stack([rng.uniform(0.5, 1.0, K), np.zeros(K)], 1),
                           reflect=np.full(K, reflect, np.int32), seed=rng.integers(1, 2 ** 62, K, dtype=np.uint64))
    eng = batch.BatchEngine(spec)
    eng.init()
    eng.step(3, graph=False)
    eng.check()
    plain = batch.run_plain(spec, 3)
    errs = [np.abs(a - b).sum() / np.abs(b).sum() for a, b in zip(eng.field("T"), plain["T"])]
    assert max(errs) <= 1e-4 and np.median(errs) <= 1e-9, errs
    assert abs(eng.total_events() - plain["events"]) <= 1e-4 * plain["events"]
    if reflect:
        assert np.all(eng.census_sizes() > 0)

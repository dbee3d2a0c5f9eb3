"""The comb's and the plan's forms by size against the oracle on the same inputs.

Comb: weights are multiples of 2^-10, so every energy sum is exact in any order and the copies, cells,
groups and positions of the output agree exactly; copy weights to FP32 rounding (1e-7).  Sizes around a
tile of 1024 entries, tiles with more copies than the scatter's map, the counter-per-bin count (from 2^19
entries, bins that fit in shared memory) and the hash table on either side of it, the plan on one block
and on several (from 16,384 bins), combs that only drop dead entries, and a threshold.

Plan: source counts are integers from canonically ordered sums (particles tracked and issued energies,
exact to FP32 weights: 1e-7).  Sizes on both sides of the shared-memory counts (51,200 cells), with faces,
fixed source and emission; many energy groups (more edges than a block has threads)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from radtranbook_b200.engine import Engine

pytestmark = pytest.mark.gpu

SEED = 0x5EED0001


def _mesh(nx, ny):
    e1, e2 = np.linspace(0.0, 1.0, nx + 1), np.linspace(0.0, 2.0, ny + 1)
    return e1, e2, O.flat2d(np.diff(e1)[:, None] * np.diff(e2)[None, :])


@pytest.mark.parametrize("nx,ny,ng,n,n_max", [
    (8, 8, 1, 1, 1), (8, 8, 1, 3, 9000), (8, 8, 1, 1023, 700), (8, 8, 1, 1024, 5000), (8, 8, 1, 1025, 0),
    (8, 8, 1, 5000, -1000), (8, 8, 1, 600_001, 200_000), (60, 61, 1, 524_287, 300_000), (60, 61, 1, 524_288, 300_000),
    (160, 165, 1, 600_000, 400_000), (127, 129, 1, 40_000, 60_000), (128, 128, 1, 40_000, 60_000),
    (70, 71, 4, 50_000, 20_000), (20, 10, 4, 540_000, 100_000)])
def test_comb_forms_match_oracle(cuda, nx, ny, ng, n, n_max):
    e1, e2, vol = _mesh(nx, ny)
    edges = np.geomspace(0.01, 10.0, ng + 1) if ng > 1 else None
    eng = Engine("xy", e1, e2, vol, seed=SEED, n_groups=ng, group_edges=edges)
    orc = O.Oracle("xy", e1, e2, vol, SEED, n_groups=ng) if ng > 1 else O.Oracle("xy", e1, e2, vol, SEED)
    rng = np.random.default_rng(n + nx)
    w = rng.integers(100, 2000, n) / 1024.0
    if n > 100:
        w[rng.random(n) < 0.1] = 0.0  # dead entries
    cell = (rng.integers(0, nx * ny, n) if n_max % 200 else rng.integers(0, nx * ny, n) // 2).astype(np.int32)
    f = lambda: rng.uniform(0, 1, n).astype(np.float32).astype(np.float64)  # noqa: E731
    d1, d2, p1, p2 = f(), f(), f(), f()
    grp = (rng.integers(0, ng, n).astype(np.int32),) if ng > 1 else ()
    eng.bank.load(w, d1, d2, np.zeros(n), p1, p2, cell, *grp)
    orc.set_bank(w, d1, d2, np.zeros(n), p1, p2, cell, *grp)
    rep = eng.comb(n_max, 11, per_group=ng > 1)
    disc = orc.comb(n_max, 11, per_group=ng > 1)
    ob = orc.get_bank()
    assert rep.n_out == len(ob["weight"])
    for k in ("cell",) + (("group",) if ng > 1 else ()):
        np.testing.assert_array_equal(eng.bank.view(k).cpu().numpy(), ob[k])
    for k in ("pos1", "pos2", "dir1", "dir2"):
        np.testing.assert_array_equal(eng.bank.view(k).cpu().numpy(), ob[k].astype(np.float32))
    np.testing.assert_allclose(eng.bank.view("weight").cpu().numpy(), ob["weight"], rtol=1e-7)
    # the device's discrepancy is of its FP32 copies: 1e-7 of each bin's copies from the oracle's
    np.testing.assert_allclose(eng.disc.cpu().numpy()[: nx * ny * ng], disc, atol=1e-7 * 2.0 * w.sum())


@pytest.mark.parametrize("nx,ny", [(200, 255), (200, 256), (199, 260)])
@pytest.mark.parametrize("geometry", ["xy", "rz"])
def test_plan_counts_match_oracle(cuda, geometry, nx, ny):
    e1, e2, vol = _mesh(nx, ny)
    if geometry == "rz":
        vol = O.flat2d(np.pi * (e1[1:] ** 2 - e1[:-1] ** 2)[:, None] * np.diff(e2)[None, :])
    rng = np.random.default_rng(nx + ny)
    nc = nx * ny
    T = 0.05 + 0.5 * rng.random(nc)
    sig, cv = 10.0 ** rng.uniform(0, 2, nc), np.full(nc, 0.1)
    src = np.where(rng.random(nc) < 0.3, rng.random(nc), 0.0)
    face = [np.full(ny, 0.5), None, np.linspace(0.1, 0.6, nx), None]
    d = lambda a: None if a is None else torch.as_tensor(a, device=cuda)  # noqa: E731
    eng, orc = Engine(geometry, e1, e2, vol, seed=SEED), O.Oracle(geometry, e1, e2, vol, SEED)
    args = (3, 1e-3, 1.0, 70_000, 20_000, 30_000)
    res = eng.transport(d(T), d(sig), d(cv), d(src), *args, [d(f) for f in face], (False, True, False, True))
    ro = orc.transport(T, sig, cv, src, *args, face, (False, True, False, True))
    assert res.report.n_transported == ro["n_transported"]
    np.testing.assert_allclose(res.report.boundary_emission, ro["boundary_emission"], rtol=1e-7)
    np.testing.assert_allclose(res.report.source_emission, ro["source_emission"], rtol=1e-7)
    np.testing.assert_allclose(eng.emitted.cpu().numpy(), ro["emitted"], rtol=1e-7, atol=1e-300)


@pytest.mark.parametrize("ng", [255, 300])
def test_plan_of_many_groups_matches_oracle(cuda, ng):
    e1, e2, vol = _mesh(5, 7)
    edges = np.geomspace(0.01, 10.0, ng + 1)
    nc = 35
    T = np.linspace(0.2, 0.8, nc)
    sig = np.repeat(np.clip(5.0 * edges[1:] ** -1.0, 1e-2, 1e3)[:, None], nc, 1).reshape(-1)
    face = [np.full(7, 0.6), None, None, None]
    d = lambda a: None if a is None else torch.as_tensor(a, device=cuda)  # noqa: E731
    eng = Engine("xy", e1, e2, vol, seed=SEED, n_groups=ng, group_edges=edges)
    orc = O.Oracle("xy", e1, e2, vol, SEED, n_groups=ng)
    args = (2, 0.01, 1.0, 8000, 3000, 0)
    res = eng.transport(d(T), d(sig), d(np.full(nc, 0.2)), None, *args, [d(f) for f in face], (False,) * 4,
                        max_events=1_000_000, rz_linear_source=False)
    ro = orc.transport_mg(T, sig, np.full(nc, 0.2), None, *args, face, (False,) * 4, edges, max_events=1_000_000)
    assert res.report.n_transported == ro["n_transported"]
    np.testing.assert_allclose(res.report.boundary_emission, ro["boundary_emission"], rtol=1e-7)
    np.testing.assert_allclose(eng.emitted.cpu().numpy(), ro["emitted"], rtol=1e-7, atol=1e-300)

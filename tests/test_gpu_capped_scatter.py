"""Cells whose scatter distance is capped (sigma_s L > 1e4: the mean free path is L / 1e4), a slot of its
own in the tracking table, beside uncapped ones, against the oracle on the same sources and draws:
slab, sphere, xy, rz, Carter-Forest (the slot holds the absorption opacity), the multigroup sphere, and
the adjoint, where a capped cell samples independently of its opacity.

A step is some 30 capped mean free paths long, so histories hardly leave their cell and their events
follow from the draws: counts to 1e-3 (an FP32 near-tie that flips counts once), deposition relative L1
2e-4, the adjoint's gradient 2e-3, as the other parity tests."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from radtranbook_b200 import adjoint
from radtranbook_b200.engine import Engine
from radtranbook_b200 import _lib

pytestmark = pytest.mark.gpu

SEED, DT, L = 0xCA9, 1e-6, 0.01


def _mesh(geometry):
    e1 = L * np.arange(13) + (0.05 if geometry == "spherical" else 0.0)
    e2 = np.array([0.0, 1.0]) if geometry in ("slab", "spherical") else L * np.arange(11)
    if geometry == "slab":
        vol = np.diff(e1)
    elif geometry == "spherical":
        vol = 4 / 3 * np.pi * np.diff(e1 ** 3)
    elif geometry == "xy":
        vol = O.flat2d(np.diff(e1)[:, None] * np.diff(e2)[None, :])
    else:
        vol = O.flat2d(np.pi * (e1[1:] ** 2 - e1[:-1] ** 2)[:, None] * np.diff(e2)[None, :])
    nc = len(vol)
    # sigma L 2e4 (capped), 5e3, and 0.5 in turn; Fleck factors of 1/300 where it is thick
    sig = np.array([2e6, 5e5, 50.0])[np.arange(nc) % 3]
    return e1, e2, vol, np.full(nc, 1.0), sig, np.full(nc, 0.01)


def _check(dep, events, ro):
    assert ro["stats"][0] > 40_000
    assert abs(int(events) - int(ro["stats"][0])) <= 1e-3 * ro["stats"][0]
    assert np.abs(dep - ro["dep"]).sum() <= 2e-4 * np.abs(ro["dep"]).sum()


@pytest.mark.parametrize("method", ["fc", "cf"])
@pytest.mark.parametrize("geometry", ["slab", "spherical", "xy", "rz"])
def test_capped_cells(cuda, geometry, method):
    e1, e2, vol, T, sig, cv = _mesh(geometry)
    if method == "cf":
        cv = np.full_like(cv, 5.0)  # re-emission slower than the step: absorptions end histories too
    eng, orc = Engine(geometry, e1, e2, vol, seed=SEED), O.Oracle(geometry, e1, e2, vol, SEED)
    dev = lambda a: torch.as_tensor(a, device=cuda)  # noqa: E731
    eng.init_census(dev(T), 20000)
    b = eng.bank
    orc.set_bank(*(b.view(k).double().cpu().numpy() for k in ("weight", "dir1", "dir2", "time", "pos1", "pos2")),
                 b.view("cell").cpu().numpy())
    eng.transport(dev(T), dev(sig), dev(cv), None, 2, DT, 1.0, 20000, 0, 0, [None] * 4, (True,) * 4,
                  max_events=1_000_000, method=_lib.METHOD_CARTER_FOREST if method == "cf" else 0)
    ro = orc.transport(T, sig, cv, None, 2, DT, 1.0, 20000, 0, 0, [None] * 4, (True,) * 4, max_events=1_000_000,
                       method=method)
    _check(eng.dep.cpu().numpy(), eng.host_stats()[0][0], ro)


def test_capped_cells_multigroup_sphere(cuda):
    e1, e2, vol, T, sig, cv = _mesh("spherical")
    edges = np.geomspace(0.05, 20.0, 4)
    sg = np.stack([sig, np.roll(sig, 1), np.roll(sig, 2)]).reshape(-1)
    eng = Engine("spherical", e1, e2, vol, seed=SEED, n_groups=3, group_edges=edges)
    orc = O.Oracle("spherical", e1, e2, vol, SEED, n_groups=3)
    dev = lambda a: torch.as_tensor(a, device=cuda)  # noqa: E731
    eng.transport(dev(T), dev(sg), dev(cv), None, 2, DT, 1.0, 40000, 0, 0, [None] * 4, (True, True),
                  rz_linear_source=False)
    ro = orc.transport_mg1d(T, sg, cv, None, 2, DT, 1.0, 40000, 0, 0, [None] * 4, (True, True, False, False), edges)
    _check(eng.dep.cpu().numpy(), eng.host_stats()[0][0], ro)


def test_capped_cells_adjoint(cuda):
    e1, e2, vol, T, sig, cv = _mesh("xy")
    setup = adjoint.AdjointSetup("xy", e1, e2, T=1.0, cv=0.01, face_T=(1.0, 1.0, 1.0, 1.0),
                                 reflect=(False,) * 4, dt=DT, n_boundary=20000)
    cot = np.random.default_rng(4).standard_normal(len(vol))
    g = adjoint.AdjointProblem(setup).vjp(torch.as_tensor(sig, device=cuda), torch.as_tensor(cot, device=cuda)).cpu().numpy()
    o = O.Oracle("xy", e1, e2, vol, setup.seed)
    face = [np.full(10, 1.0), np.full(10, 1.0), np.full(12, 1.0), np.full(12, 1.0)]
    o.transport(T, sig, cv, None, 0, DT, 1.0, 0, setup.n_boundary, 0, face, setup.reflect, max_events=setup.max_events,
                sources_only=True)
    ref = o.adjoint_vjp(T, sig, cv, 0, DT, 1.0, setup.reflect, cot, max_events=setup.max_events)
    assert np.abs(g - ref).sum() <= 2e-3 * np.abs(ref).sum()

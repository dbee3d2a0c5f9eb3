"""Meshes long in one direction, whose edges would leave few blocks an SM or overfill a block's shared
memory: tracking, the event-by-event form and the adjoint read them through L1.  Sizes around the last
mesh that has a block tally (13,400 cells) and past what pairs (28,400) and single floats (57,000) of
edges would fit in; edges are multiples of 2^-12, exact in FP32.

Tracking against the event-by-event form (histories and tallies as in its own test: counts and census
entry by entry, deposition and escapes 1e-12) and against the oracle (FP32 against FP64 tracking, as
the other parity tests: events 1e-3, up to 40,000 cells deposition relative L1 2e-4); the adjoint against
the oracle's (relative L1 2e-3)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from radtranbook_b200.engine import Engine
from radtranbook_b200 import adjoint

from . import test_gpu_event_form as event_form

pytestmark = pytest.mark.gpu

SEED = 0x10E6


def _case(geometry, n):
    e1 = np.arange(n + 1) / 4096.0 + (1.0 if geometry == "spherical" else 0.0)
    e2 = np.array([0.0, 1.0])
    vol = 4 / 3 * np.pi * np.diff(e1 ** 3) if geometry == "spherical" else np.diff(e1)
    T = np.linspace(0.6, 0.3, n)
    face = [np.array([1.0]), None, None, None]
    return e1, e2, vol, T, 5.0 * T ** -1.0, np.full(n, 0.3), face


def _run(geometry, n, cuda, launch=None):
    e1, e2, vol, T, sig, cv, face = _case(geometry, n)
    eng = Engine(geometry, e1, e2, vol, seed=SEED)
    eng.launch.update(launch or {})
    dev = lambda a: None if a is None else torch.as_tensor(a, device=cuda)  # noqa: E731
    eng.init_census(dev(T), 20000)
    eng.transport(dev(T), dev(sig), dev(cv), None, 2, 1e-4, 1.0, 20000, 10000, 0, [dev(f) for f in face],
                  (False,) * 4, max_events=1_000_000)
    stats, esc = eng.host_stats()
    bank = {k: eng.bank.view(k).cpu().numpy() for k in ("weight", "pos1", "cell")}
    return stats, esc, eng.dep.cpu().numpy(), eng.si.cpu().numpy(), bank


@pytest.mark.parametrize("geometry", ["slab", "spherical"])
@pytest.mark.parametrize("n", [14_000, 28_000, 29_000, 40_000, 60_000])
def test_long_1d_mesh(cuda, geometry, n):
    gpu = _run(geometry, n, cuda)
    event_form._same(gpu, _run(geometry, n, cuda, {"event_based": 1}))
    e1, e2, vol, T, sig, cv, face = _case(geometry, n)
    orc = O.Oracle(geometry, e1, e2, vol, SEED)
    orc.init_ic(T, 20000)
    ro = orc.transport(T, sig, cv, None, 2, 1e-4, 1.0, 20000, 10000, 0, face, (False,) * 4, max_events=1_000_000)
    assert abs(int(gpu[0][0]) - int(ro["stats"][0])) <= 1e-3 * ro["stats"][0]
    if n <= 40_000:  # the bound is a coarse mesh's: a cell's deposition is off by FP32 ulps of its position over its width
        assert np.abs(gpu[2] - ro["dep"]).sum() <= 2e-4 * np.abs(ro["dep"]).sum()


# block tallies asked for (28 bytes a cell with one float per edge, so up to 8,100 cells) and the cell
# table alone (12 bytes: 19,000), where the tables fit but not beside a pair of floats per cell's edges
@pytest.mark.parametrize("n,launch", [(7_100, {"smem_cells": 1, "smem_tally": 1}),
                                      (8_000, {"smem_cells": 1, "smem_tally": 1}),
                                      (18_000, {"smem_cells": 1, "smem_tally": 0})])
def test_tables_asked_for_on_a_long_mesh(cuda, n, launch):
    event_form._same(_run("slab", n, cuda, launch), _run("slab", n, cuda, {"event_based": 1}))


@pytest.mark.parametrize("n", [29_000, 40_000])
def test_adjoint_on_a_long_mesh(cuda, n):
    e1, e2 = np.arange(n + 1) / 4096.0, np.array([0.0, 1.0])
    setup = adjoint.AdjointSetup("xy", e1, e2, T=0.3, cv=0.05, face_T=(1.0, 0.0, 0.0, 0.0),
                                 reflect=(False, False, True, True), dt=1e-3, n_boundary=20000)
    rng = np.random.default_rng(n)
    sigma = np.exp(np.log(8.0) + 0.6 * rng.standard_normal(n))
    cot = rng.standard_normal(n)
    cot /= np.linalg.norm(cot)
    g = adjoint.AdjointProblem(setup).vjp(torch.as_tensor(sigma, device=cuda),
                                          torch.as_tensor(cot, device=cuda)).cpu().numpy()
    o = O.Oracle("xy", e1, e2, np.diff(e1), setup.seed)
    Tc, cvc = np.full(n, 0.3), np.full(n, 0.05)
    o.transport(Tc, sigma, cvc, None, 0, setup.dt, 1.0, 0, setup.n_boundary, 0, [np.array([1.0]), None, None, None],
                setup.reflect, max_events=setup.max_events, sources_only=True)
    ref = o.adjoint_vjp(Tc, sigma, cvc, 0, setup.dt, 1.0, setup.reflect, cot, max_events=setup.max_events)
    assert np.abs(g - ref).sum() <= 2e-3 * np.abs(ref).sum()


def test_no_cliff_where_the_block_tally_ends(cuda):
    """14,000 cells against 13,000, the last thousand with a block tally: the step took 2.7 times as long
    with the edges in the shared memory of the one block that then fits an SM; 1.2 through L1."""
    def best(n):
        e1, e2, vol, T, sig, cv, face = _case("slab", n)
        eng = Engine("slab", e1, e2, vol, seed=SEED)
        dev = lambda a: None if a is None else torch.as_tensor(a, device=cuda)  # noqa: E731
        t = []
        for _ in range(4):  # the first one warms up
            eng.init_census(dev(T), 300_000)
            r = eng.transport(dev(T), dev(sig), dev(cv), None, 2, 1e-3, 1.0, 0, 0, 0, [None] * 4, (False,) * 4)
            t.append(r.report.ms_transport)
        return min(t)

    short, long = best(13_000), best(14_000)
    assert long <= 1.8 * short, (long, short)

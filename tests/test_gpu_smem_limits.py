"""Dynamic shared-memory limits of the kernels: a function's limit holds for every launch of it.

  - Launches just under 48 KB of dynamic shared memory, which a kernel's static bytes carry past it:
    tracking with block tallies (2-D and 1-D meshes of that size), the comb's counter per bin, the
    batched comb.  Against the event-by-event form (histories and tallies as in its own test), the
    oracle's comb, and the batch's queue form.
  - Engines on meshes of two sizes in four host threads, the larger ones' launches between the smaller
    ones': exactly the histories of the same runs one after the other.
  - A captured device loop on a mesh, replayed after an engine on a smaller one has stepped.
"""
import threading

import numpy as np
import pytest
import torch

from oracle import oracle as O
from radtranbook_b200 import batch, driver, imc2d, problems
from radtranbook_b200.engine import Engine

from . import test_gpu_comb_plan_forms as comb_forms
from . import test_gpu_event_form as event_form

pytestmark = pytest.mark.gpu


def test_block_tallies_just_under_the_limit_2d(cuda):
    e1, e2 = np.linspace(0.0, 1.0, 43), np.linspace(0.0, 1.0, 45)  # 42 x 44: 49,136 bytes
    vol = O.flat2d(np.diff(e1)[:, None] * np.diff(e2)[None, :])
    nc = 42 * 44
    T = np.linspace(0.9, 0.1, nc)
    args = ("xy", e1, e2, vol, T, 10 * T ** -3.0, np.full(nc, 0.3), [np.full(44, 1.0), None, None, None],
            (False, True, True, True), 20000, 20000)
    event_form._same(event_form._run(*args, False, cuda), event_form._run(*args, True, cuda))


@pytest.mark.parametrize("nx", [1405, 1406, 1407, 1408])  # 49,064 to 49,160 bytes
def test_block_tallies_just_under_the_limit_1d(cuda, nx):
    e1 = np.linspace(0.0, 0.2, nx + 1)
    T = np.linspace(0.9, 0.3, nx)
    args = ("slab", e1, np.array([0.0, 1.0]), np.diff(e1), T, 30 * T ** -3.0, np.full(nx, 0.3),
            [np.array([1.0]), None], (False, False), 10000, 10000)
    event_form._same(event_form._run(*args, False, cuda, max_events=0), event_form._run(*args, True, cuda, max_events=0))


@pytest.mark.parametrize("nx,ny", [(110, 111), (128, 96)])  # 48,840 and 49,152 bytes of counters
def test_counter_per_bin_just_under_the_limit(cuda, nx, ny):
    comb_forms.test_comb_forms_match_oracle(cuda, nx, ny, 1, 530_000, 300_000)


@pytest.mark.parametrize("K", [3570, 3580])
def test_batched_comb_just_under_the_limit(cuda, K):
    rng = np.random.default_rng(K)
    spec = batch.BatchSpec(n_cells=np.full(K, 2), length=rng.uniform(0.1, 0.4, K), n_target=np.full(K, 6),
                           n_boundary=np.full(K, 6), n_max=np.full(K, 10), opacity_a=10.0 ** rng.uniform(0, 2, K),
                           opacity_p=np.full(K, -3.0), cv=rng.uniform(0.05, 1.0, K),
                           face_T=np.stack([rng.uniform(0.5, 1.0, K), np.zeros(K)], 1),
                           reflect=np.zeros(K, np.int32), seed=rng.integers(1, 2 ** 62, K, dtype=np.uint64))
    runs = []
    for form in (0, 2):
        eng = batch.BatchEngine(spec)
        eng.launch["form"] = form
        eng.init()
        eng.step(3, graph=False)
        eng.check()
        runs.append(eng)
    # the batch's own tolerances: FP64 sums in another order, an FP32 near-tie that flips counts once
    errs = [np.abs(a - b).sum() / np.abs(b).sum() for a, b in zip(runs[0].field("T"), runs[1].field("T"))]
    assert max(errs) <= 1e-4 and np.median(errs) <= 1e-9, max(errs)
    assert abs(runs[0].total_events() - runs[1].total_events()) <= 1e-4 * runs[1].total_events()


def _problem(nr, nz, cuda):
    p = problems.crooked_pipe(scale=0.01, nr=nr, nz=nz)
    e1, e2 = p["edges1"], p["edges2"]
    vol = O.flat2d(np.pi * (e1[1:] ** 2 - e1[:-1] ** 2)[:, None] * np.diff(e2)[None, :])
    dev = lambda f: torch.as_tensor(O.flat2d(f), dtype=torch.float64, device=cuda)  # noqa: E731
    rc = 0.5 * (e1[:-1] + e1[1:])
    face = [None, None, torch.as_tensor(np.where(rc < 0.5, 0.5, 0.0), device=cuda), None]
    eng = Engine("rz", e1, e2, vol, seed=0x5A1E)
    T = dev(p["Tinit"])
    return eng, (T, dev(p["sigma_host"](p["Tinit"])), dev(p["cv_host"](p["Tinit"]))), face, p["reflect"]


def _steps(prob, n):
    """n transports of one small census, queued without waiting; event statistics, escapes and
    deposition of the last (the census loses weight from one to the next)."""
    eng, mat, face, reflect = prob
    eng.init_census(mat[0], 200)
    for k in range(n):
        eng.transport_async(*mat, None, 3, 0.01, 1.0, 0, 200, 0, face, reflect, max_events=1_000_000)
        if k % 500 == 499:
            torch.cuda.current_stream().synchronize()
    eng.comb_async(400, 3, None)
    sm = eng.fetch()
    return np.array(sm.stats[:]), np.array(sm.escaped[:]), eng.dep.cpu().numpy()


def test_threads_on_meshes_of_different_sizes(cuda):
    shapes = [(60, 210), (60, 150)]  # the same kernels: 12,600 and 9,000 cells of tally, and of plan counts
    n = 6000
    alone = [_steps(_problem(*s, cuda), n) for s in shapes]
    res, err = [None] * 4, []
    start = threading.Barrier(4, timeout=120)

    def body(q):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                prob = _problem(*shapes[q % 2], cuda)
                start.wait()
                res[q] = _steps(prob, n)
        except BaseException as ex:  # noqa: BLE001
            err.append(ex)

    th = [threading.Thread(target=body, args=(q,)) for q in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join(timeout=600)
    if err:
        raise err[0]
    for (st, esc, dep), (st1, esc1, dep1) in zip(res, alone * 2):
        np.testing.assert_array_equal(st, st1)
        np.testing.assert_allclose(esc, esc1, rtol=1e-12, atol=0)
        np.testing.assert_allclose(dep, dep1, rtol=1e-12, atol=0)


def _drop_in(nr, nz):
    p = problems.crooked_pipe(scale=0.01, nr=nr, nz=nz)
    st = imc2d.init_simulation(p["Ntarget"], p["Tinit"], p["Tr_init"], p["edges1"], p["edges2"], p["eos_dev"],
                               p["inv_eos_dev"], geometry="rz", seed=0xD159)
    return p, st


def _loop(p, st):
    return driver.DeviceLoop(st, Ntarget=p["Ntarget"], Nboundary=p["Nboundary"], Nsource=0, Nmax=p["Nmax"],
                             T_boundary=p["T_boundary"], sigma_a_func=p["sigma_dev"], inv_eos=p["inv_eos_dev"],
                             cv=p["cv_dev"], reflect=p["reflect"], geometry="rz",
                             boundary_source_func=p["boundary_source_func"])


def test_captured_loop_after_a_smaller_engine(cuda):
    runs = []
    for small_between in (False, True):
        p, st = _drop_in(60, 210)
        loop = _loop(p, st)
        loop.run([p["dt"]] * 2)
        if small_between:
            q, s2 = _drop_in(60, 150)
            for _ in range(2):
                s2, _ = imc2d.step(s2, q["Ntarget"], q["Nboundary"], 0, q["Nmax"], q["T_boundary"], q["dt"], q["edges1"],
                                   q["edges2"], q["sigma_dev"], q["inv_eos_dev"], q["cv_dev"], q["source"],
                                   reflect=q["reflect"], geometry="rz", boundary_source_func=q["boundary_source_func"])
        out = loop.run([p["dt"]] * 4)
        assert len(out["steps"]) == 4
        runs.append(st._T.cpu().numpy())
    # FP64 sums in another order; an FP32 near-tie that flips over the six steps counts once
    assert np.abs(runs[1] - runs[0]).sum() <= 1e-4 * np.abs(runs[0]).sum()

"""A step that raises between queueing its report and waiting for it leaves nothing in flight: the
report's kernels and copies write into pinned host buffers that torch's allocator may hand out again
once the state is gone, and it does not know of them.  A long device wait is queued before the report
and the comb (or what follows it) raises; on return the step's streams are idle."""
import numpy as np
import pytest
import torch

from radtranbook_b200 import imc1d, mg_imc1d, mg_imc2d, problems

pytestmark = pytest.mark.gpu


class Boom(RuntimeError):
    pass


def _raise_after_wait(monkeypatch, eng, update, call):
    """The engine's `update` queues a wait of some 0.1 s first, its `call` raises."""
    inner = getattr(eng, update)

    def slow(*a, **kw):
        torch.cuda._sleep(200_000_000)
        return inner(*a, **kw)

    def boom(*a, **kw):
        raise Boom

    monkeypatch.setattr(eng, update, slow)
    monkeypatch.setattr(eng, call, boom)


def _idle(eng):
    return torch.cuda.current_stream().query() and eng.side_stream().query()


def test_gray_step_that_raises_is_settled(cuda, monkeypatch):
    q = problems.marshak_slab(scale=0.2)
    st = imc1d.init_simulation(q["Ntarget"], q["Tinit"], q["Tr_init"], q["mesh"], q["eos_dev"], q["inv_eos_dev"])
    step = lambda: imc1d.step(st, q["Ntarget"], q["Nboundary"], 0, q["Nmax"], q["T_boundary"], q["dt"], q["mesh"],  # noqa: E731
                              q["sigma_dev"], q["inv_eos_dev"], q["cv_dev"], q["source"])
    step()
    with monkeypatch.context() as m:
        _raise_after_wait(m, st._engine, "material_update_law", "comb_async")
        with pytest.raises(Boom):
            step()
        assert _idle(st._engine)


def test_mg2d_step_that_raises_is_settled(cuda, monkeypatch):
    p = problems.mg_crooked_pipe(nr=30, nz=105, mode="quick")
    e1, e2, ge = p["edges1"], p["edges2"], p["energy_edges"]
    st = mg_imc2d.init_simulation(p["Ntarget"], p["Tinit"], p["Tr_init"], e1, e2, ge, p["eos_dev"],
                                  p["inv_eos_dev"], T_emit_floor=p["T_emit_floor"], geometry="rz", seed=0x4B1)
    step = lambda: mg_imc2d.step(st, p["Ntarget"], p["Nboundary"], 0, p["Nmax"], p["T_boundary"], p["dt_initial"],  # noqa: E731
                                 e1, e2, ge, p["sigma_dev"], p["inv_eos_dev"], p["cv_dev"], p["source"],
                                 reflect=p["reflect"], geometry="rz", boundary_source_func=p["boundary_source_func"],
                                 T_emit_floor=p["T_emit_floor"])
    step()
    with monkeypatch.context() as m:
        _raise_after_wait(m, st._engine, "material_update_law", "comb_async")
        with pytest.raises(Boom):
            step()
        assert _idle(st._engine)


def test_mg1d_step_that_raises_is_settled(cuda, monkeypatch):
    r, ge = np.linspace(0.0, 1.0, 21), np.geomspace(1e-3, 10.0, 5)
    mesh = np.stack([r[:-1], r[1:]], axis=1)
    fns = [lambda T, s=s: s * np.ones_like(T) for s in (20.0, 5.0, 1.0, 0.3)]
    T = np.full(20, 0.05)
    st = mg_imc1d.init_simulation(2000, T, T, mesh, ge, lambda T: 0.2 * T, lambda u: u / 0.2)
    step = lambda: mg_imc1d.step(st, 2000, 2000, 0, 6000, (0.0, 1.0), 0.01, mesh, ge, fns, lambda u: u / 0.2,  # noqa: E731
                                 lambda T: 0.2 * np.ones_like(T), np.zeros(20))
    step()
    with monkeypatch.context() as m:
        _raise_after_wait(m, st._engine, "fields_to_host", "queue_summary")
        with pytest.raises(Boom):
            step()
        assert _idle(st._engine)

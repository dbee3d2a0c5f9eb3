"""The adjoint's two gradient tallies (shared memory of one wide block per SM; global memory, on
meshes too large for that) against the FP64 oracle adjoint, on both sides of the size limit, with
hot material so that the scatter term counts, reflecting faces and an events-per-history cap.
Tolerance: the forward tests' of FP32 against FP64 tracking, relative L1 over cells <= 2e-3.
"""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from radtranbook_b200 import adjoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geometry,n1,n2,shape,cap", [
    ("xy", 168, 170, (256, 4), 1_000_000), ("xy", 170, 172, (256, 4), 1_000_000), ("rz", 9, 31, (96, 1), 1_000_000),
    ("xy", 1, 1, (256, 4), 1_000_000), ("xy", 20, 33, (128, 8), 12)])
def test_gradient_tallies_match_oracle(cuda, geometry, n1, n2, shape, cap):
    e1, e2 = np.linspace(0.0, 1.0, n1 + 1), np.linspace(0.0, 1.5, n2 + 1)
    setup = adjoint.AdjointSetup(geometry, e1, e2, T=0.8, cv=0.01, face_T=(0.0, 0.0, 1.0, 0.0),
                                 reflect=(True, False, False, True), dt=0.02, n_boundary=30_000, max_events=cap)
    rng = np.random.default_rng(n1)
    nc = n1 * n2
    sigma = np.exp(np.log(6.0) + 0.6 * rng.standard_normal(nc))
    cot = rng.standard_normal(nc)
    cot /= np.linalg.norm(cot)
    prob = adjoint.AdjointProblem(setup)
    prob.engine.launch.update(block_size=shape[0], blocks_per_sm=shape[1])
    g = prob.vjp(torch.as_tensor(sigma, device=cuda), torch.as_tensor(cot, device=cuda)).cpu().numpy()
    area = np.pi * (e1[1:] ** 2 - e1[:-1] ** 2) if geometry == "rz" else np.diff(e1)
    o = O.Oracle(geometry, e1, e2, O.flat2d(area[:, None] * np.diff(e2)[None, :]), setup.seed)
    T, cv = np.full(nc, setup.T), np.full(nc, setup.cv)
    o.transport(T, sigma, cv, None, 0, setup.dt, 1.0, 0, setup.n_boundary, 0, [None, None, np.full(n1, 1.0), None],
                setup.reflect, max_events=cap, sources_only=True)
    ref = o.adjoint_vjp(T, sigma, cv, 0, setup.dt, 1.0, setup.reflect, cot, max_events=cap)
    assert np.abs(g - ref).sum() <= 2e-3 * np.abs(ref).sum()

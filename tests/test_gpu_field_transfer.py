"""Cell fields between the flat device order c = i + nx j and the host's (nx, ny) order (an exact
permutation), and the per-(group, cell) moments of a 1-D bank against NumPy: FP64 sums of products
in a run-dependent order, so each bin agrees to n 2^-53 times its sum of magnitudes (n terms), plus
three roundings of the scaling.  Sizes: one cell, one row, one column, around a block of 256; banks
empty, of one entry, around a tile of 1024, with dead entries, and with entries past the count.
"""
import numpy as np
import pytest
import torch

from radtranbook_b200 import imc2d, problems
from radtranbook_b200.engine import C_LIGHT, Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 1), (5, 1), (1, 7), (16, 16), (15, 17), (257, 3), (60, 40)])
@pytest.mark.parametrize("n", [1, 3, 4])
def test_fields_both_ways(cuda, nx, ny, n):
    eng = Engine("xy", np.linspace(0, 1, nx + 1), np.linspace(0, 1, ny + 1), np.full(nx * ny, 1.0 / (nx * ny)))
    rng = np.random.default_rng(nx * 100 + ny)
    grid = rng.random((n, nx, ny))
    src = torch.empty(n * nx * ny, dtype=torch.float64, pin_memory=True)
    src.copy_(torch.from_numpy(grid.reshape(-1)))
    dst = [torch.zeros(nx * ny, dtype=torch.float64, device=eng.device) for _ in range(n)]
    eng.fields_from_host(src, dst)
    back = torch.zeros(n * nx * ny, dtype=torch.float64, pin_memory=True)
    done = eng.event("fields")
    eng.fields_to_host(dst, back, done)
    done.synchronize()
    for k in range(n):
        assert np.array_equal(dst[k].cpu().numpy(), grid[k].T.reshape(-1))  # c = i + nx j
    assert np.array_equal(back.numpy().reshape(n, nx, ny), grid)


@pytest.mark.parametrize("n,nc,G", [(0, 4, 2), (1, 1, 2), (1023, 7, 3), (1024, 1, 2), (1025, 50, 10), (30000, 100, 25)])
def test_bank_moments(cuda, n, nc, G):
    rng = np.random.default_rng(n + nc)
    vol = rng.uniform(0.5, 2.0, nc)
    eng = Engine("spherical", np.linspace(0, 1, nc + 1), np.array([0.0, 1.0]), vol, n_groups=G,
                 group_edges=np.geomspace(1e-3, 10.0, G + 1))
    extra = 37  # entries past the count, with cells of no mesh
    w = rng.uniform(0.0, 1.0, n + extra).astype(np.float32)
    w[:n][rng.random(n) < 0.2] = 0.0
    mu = rng.uniform(-1, 1, n + extra).astype(np.float32)
    cell, group = rng.integers(0, nc, n + extra), rng.integers(0, G, n + extra)
    cell[n:], group[n:] = nc + 1000, -5
    z = np.zeros(n + extra, np.float32)
    eng.bank.load(w, mu, z, z, z, z, cell, group)
    count = torch.tensor([n], dtype=torch.int64, device=eng.device)
    got = eng.moments(eng.bank, count.data_ptr()).cpu().numpy()
    b = (cell + nc * group)[:n]
    wd, wm = w[:n].astype(np.float64), w[:n].astype(np.float64) * mu[:n].astype(np.float64)
    for k, (v, scale) in enumerate([(wd, np.ones(nc)), (wm, C_LIGHT / vol)]):
        ref = np.bincount(b, v, nc * G).reshape(G, nc) * scale
        mag = np.bincount(b, np.abs(v), nc * G).reshape(G, nc) * scale
        assert np.all(np.abs(got[k] - ref) <= (n + 3) * 2.0 ** -53 * mag)


def test_host_callables_may_return_anything_array_like(cuda):
    """Object arrays, lists and scalars from host material callables give the float arrays' steps: the same
    histories, temperatures to the order of the FP64 weight sum (1e-12 after three steps)."""
    out = []
    for wrap in (lambda x: x, lambda x: x.astype(object), lambda x: x.tolist()):
        p = problems.crooked_pipe(nr=9, nz=20)
        st = imc2d.init_simulation(2000, p["Tinit"], p["Tr_init"], p["edges1"], p["edges2"], p["eos_host"],
                                   p["inv_eos_host"], geometry="rz")
        sig = lambda T: wrap(np.asarray(p["sigma_host"](T)))  # noqa: E731, B023
        inv = lambda e: wrap(np.asarray(p["inv_eos_host"](e)))  # noqa: E731, B023
        cv = lambda T: wrap(np.broadcast_to(p["cv_host"](T), T.shape).copy())  # noqa: E731, B023
        for _ in range(3):
            st, info = imc2d.step(st, 1500, 1500, 0, 6000, p["T_boundary"], p["dt"], p["edges1"], p["edges2"], sig, inv,
                                  cv, p["source"], reflect=p["reflect"], geometry="rz",
                                  boundary_source_func=p["boundary_source_func"])
        out.append((st.temperature.copy(), info["profiling"]["transport_events"]["total"]))
    for T, ev in out[1:]:
        assert ev == out[0][1]
        np.testing.assert_allclose(T, out[0][0], rtol=1e-12)

"""The wide block's open table of (group, cell) sums (meshes past its flat tally, with a few histories
per lane) against the event-by-event loop, which sums in global memory: meshes whose touched entries
fill the table many times over, and meshes whose histories sit in a few cells; with and without the
census sums the comb uses.

The histories are the same, so event statistics and the census agree exactly.  Deposition and escaped
energy are integer sums in units of a quantum that follows the FP64 sum of the tracked weights: 1e-13.
The census sums are FP64 sums of at most 1e6 positive terms in another order (relative error below
1e6 2^-53): 1e-9, against sums over the tracked bank."""
import numpy as np
import pytest
import torch

from radtranbook_b200 import _lib
from radtranbook_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _engine(geometry, n1, n2, ng, hot, launch, n, cuda):
    rng = np.random.default_rng(n1 + 7 * n2)
    e1, e2 = np.linspace(0.0, 1.0, n1 + 1), np.linspace(0.0, 2.0, n2 + 1)
    vol = (np.pi * (e1[1:] ** 2 - e1[:-1] ** 2)[:, None] if geometry == "rz" else np.diff(e1)[:, None]) * np.diff(e2)
    nc = n1 * n2
    T = np.full(nc, 1e-4) if hot else 0.2 + 0.2 * rng.random(nc)
    if hot:
        T[nc // 2:nc // 2 + 3] = 0.5
    sig = 10.0 ** rng.uniform(-1.0, 3.0, (ng, nc))
    sig[:, : nc // 9] = 0.0  # cells without absorption
    d = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64).reshape(-1), device=cuda)  # noqa: E731
    eng = Engine(geometry, e1, e2, vol.T.reshape(-1), seed=0x4A5F, n_groups=ng,
                 group_edges=np.logspace(-2, 1, ng + 1) if ng > 1 else None)
    eng.launch.update(launch)
    eng.init_census(d(T), n)
    eng.transport(d(T), d(sig), d(np.full(nc, 0.05)), None, 3, 0.002, 1.0, n // 4, n // 4, 0,
                  [d(np.full(n2, 0.5)), None, None, None], (False, True, False, False),
                  max_events=500, rz_linear_source=geometry == "rz")
    return eng, nc


@pytest.mark.parametrize("geometry,n1,n2,ng,hot,n,shape", [
    ("rz", 165, 170, 1, False, 30_000, (128, 1)), ("rz", 165, 170, 1, True, 30_000, (128, 1)),
    ("xy", 60, 61, 9, False, 300_000, (256, 4)), ("xy", 60, 61, 9, True, 300_000, (256, 4)),
    ("rz", 300, 400, 2, False, 120_000, (128, 2)), ("xy", 240, 240, 1, False, 400_000, (256, 4))])
def test_open_table_matches_event_loop(cuda, geometry, n1, n2, ng, hot, n, shape):
    a, nc = _engine(geometry, n1, n2, ng, hot, {"event_based": 1}, n, cuda)
    b, _ = _engine(geometry, n1, n2, ng, hot, {"block_size": shape[0], "blocks_per_sm": shape[1]}, n, cuda)
    assert b.bank.size >= 2 * 148 * shape[0] * shape[1]  # the table's side of the rule
    sa, ea = a.host_stats()
    sb, eb = b.host_stats()
    np.testing.assert_array_equal(sa, sb)
    np.testing.assert_allclose(ea, eb, rtol=1e-13)
    da, db = a.dep.cpu().numpy(), b.dep.cpu().numpy()
    np.testing.assert_allclose(da, db, rtol=1e-13, atol=1e-13 * np.abs(da).max())
    for k in ("weight", "pos1", "pos2", "dir1", "dir2", "cell"):
        w = a.bank.view("weight") > 0
        assert torch.equal(torch.where(w, a.bank.view(k), 0), torch.where(b.bank.view("weight") > 0, b.bank.view(k), 0))


@pytest.mark.parametrize("ng,hot", [(1, False), (1, True), (9, False), (9, True)])
def test_census_sums_reach_the_comb(cuda, ng, hot):
    n1, n2 = (165, 170) if ng == 1 else (60, 61)
    eng, nc = _engine("xy", n1, n2, ng, hot, {"block_size": 128, "blocks_per_sm": 1}, 60_000, cuda)
    T = torch.full((nc,), 0.3, dtype=torch.float64, device=cuda)
    sig = torch.full((ng * nc,), 5.0, dtype=torch.float64, device=cuda)
    cv = torch.full((nc,), 0.05, dtype=torch.float64, device=cuda)
    e = torch.zeros(nc, dtype=torch.float64, device=cuda)
    eng.transport_async(T, sig, cv, None, 4, 0.002, 1.0, 20_000, 0, 0, [None] * 4, (True,) * 4)
    eng.comb_async(40_000, 4, e, per_group=ng > 1, write_after=True)
    sm = eng.fetch()
    assert sm.flags & _lib.FLAG_COMB_OVERFLOW == 0
    w = eng.spare.view("weight").double()  # the tracked bank
    assert eng.spare.size >= 2 * 148 * 128
    total = float(w[w > 0].sum())
    assert sm.comb_before == pytest.approx(total, rel=1e-9)
    bins = eng.spare.view("cell").long() + (nc * eng.spare.view("group").long() if ng > 1 else 0)
    ref = torch.zeros(nc * ng, dtype=torch.float64, device=cuda).index_add_(0, bins[w > 0], w[w > 0])
    before = eng.disc + eng.comb_after
    assert torch.all((before - ref).abs() <= 1e-9 * ref.max())

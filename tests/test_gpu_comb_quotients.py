"""The comb's copies floor(w / ew + xi) where their FP32 quotient is at its weakest, exactly as the
oracle's FP64 ones: weights that are subnormal in FP32 or near its smallest and largest normal numbers,
and many copies an entry, where FP32 leaves a wide band around every integer open (at 2^17 copies,
half of an entry's fractions).  Weights are small integers times a power of two, so the energy sums
and the comb weights are the same in any order."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from radtranbook_b200.engine import Engine

pytestmark = pytest.mark.gpu

SEED = 0xC0B


# (power of two, integers below, entries, cells a side, target): copies an entry about target / entries
@pytest.mark.parametrize("p,top,n,side,n_max", [
    (-149, 40, 50_000, 4, 60_000), (-140, 40, 50_000, 4, 20_000), (-128, 40, 50_000, 4, 60_000),
    (-126, 400, 50_000, 4, 60_000), (121, 100, 50_000, 4, 50_000), (-20, 1 << 20, 50_000, 4, 60_000),
    (-20, 1 << 20, 3_000, 3, 600_000), (-20, 1 << 20, 40, 1, 5_000_000)])
def test_copies_match_fp64(cuda, p, top, n, side, n_max):
    e = np.linspace(0.0, 1.0, side + 1)
    vol = O.flat2d(np.diff(e)[:, None] * np.diff(e)[None, :])
    eng, orc = Engine("xy", e, e, vol, seed=SEED), O.Oracle("xy", e, e, vol, SEED)
    rng = np.random.default_rng(n + 1000 + p)
    w = np.ldexp(rng.integers(1, top, n).astype(np.float64), p)
    cell = rng.integers(0, side * side, n).astype(np.int32)
    d1, d2, p1, p2 = (rng.uniform(0, 1, n).astype(np.float32).astype(np.float64) for _ in range(4))
    assert np.array_equal(w, w.astype(np.float32).astype(np.float64))
    eng.bank.load(w, d1, d2, np.zeros(n), p1, p2, cell)
    orc.set_bank(w, d1, d2, np.zeros(n), p1, p2, cell)
    rep = eng.comb(n_max, 7)
    orc.comb(n_max, 7)
    ob = orc.get_bank()
    assert rep.n_out == len(ob["weight"])
    np.testing.assert_array_equal(eng.bank.view("cell").cpu().numpy(), ob["cell"])
    np.testing.assert_array_equal(eng.bank.view("pos1").cpu().numpy(), ob["pos1"].astype(np.float32))

"""Combs that make many copies of few entries: several blocks share a tile's copies, and past four times
the scatter's map every copy's entry is searched.  Against the oracle, exactly, as the comb's other forms:
one entry to a few tiles, targets on both sides of the split and of the map, by group, and a comb that
multiplies one bin's entries while most are dead."""
import pytest

from . import test_gpu_comb_plan_forms as comb_forms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,ng,n,n_max", [
    (1, 1, 1, 1, 70_000), (3, 3, 1, 7, 2_047), (3, 3, 1, 7, 2_051), (8, 8, 1, 100, 400_001), (8, 8, 1, 1_000, 8_193),
    (8, 8, 1, 1_000, 8_600), (8, 8, 1, 1_024, 1_000_001), (8, 8, 1, 1_025, 300_003), (8, 8, 1, 5_000, 1_000_001),
    (60, 61, 1, 3_000, 60_001), (8, 8, 4, 700, 200_001), (8, 8, 1, 200_000, 1_000_001)])
def test_many_copies_of_few_entries(cuda, nx, ny, ng, n, n_max):
    comb_forms.test_comb_forms_match_oracle(cuda, nx, ny, ng, n, n_max)

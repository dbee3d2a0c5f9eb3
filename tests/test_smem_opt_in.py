"""One place sets a kernel's dynamic shared-memory limit (smem_opt_in), and not to a launch's size: the
limit is the function's, so a second host thread's smaller launch would lower it under a larger one."""
import pathlib

CSRC = pathlib.Path(__file__).resolve().parent.parent / "radtranbook_b200" / "csrc"


def test_the_limit_is_set_in_one_place():
    uses = {p.name: p.read_text().count("cudaFuncSetAttribute(") for p in CSRC.iterdir() if p.suffix in (".cu", ".cuh", ".h")}
    assert {k: v for k, v in uses.items() if v} == {"imc_internal.h": 1}

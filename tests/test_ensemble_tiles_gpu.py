"""Ensembles of the performance build whose tiles cover fewer rows than the shape has,
and whose members run other tile shapes as single grids: the batched kernels of
every precision against single-grid runs and against the parity build, by the
ensemble tests' own measure (relative L2 of the variables in the plane, 1e-12 in
binary64, 1e-5 in binary32 and mixed) and psi in binary64 (it starts at zero:
1e-9; in the other precisions it is rounding noise for the first steps)."""
import pytest

from test_ensemble import _same

pytestmark = pytest.mark.gpu

# Members and the rows their list's tiles get on 148 SMs: 5, 13 and 19.
LISTS = {"five": [(64, 64), (100, 70), (37, 130)], "thirteen": [(160, 150), (96, 120), (200, 100)],
         "full": [(161, 97), (320, 300), (300, 320), (64, 64), (128, 256)]}


@pytest.mark.parametrize("order,solver", [("muscl", "hlld"), ("muscl", "hll"), ("first", "hlld")])
@pytest.mark.parametrize("precision", ["fp64", "fp32", "mixed"])
@pytest.mark.parametrize("sizes", sorted(LISTS))
def test_batched_tiles_match_single_grids_and_the_parity_build(pmhd_lib, sizes, precision, order, solver):
    common = dict(precision=precision, order=order, solver=solver)
    members = [pmhd_lib.member(nx, ny, pmhd_lib.PROBLEM_ORSZAG_TANG, (0.9 + 0.1 * k,), t_end=1e9)
               for k, (nx, ny) in enumerate(LISTS[sizes])]
    with pmhd_lib.Ensemble(members, **common) as e:
        e.advance(max_steps=4)
        for k, (nx, ny) in enumerate(LISTS[sizes]):
            got = e.get_state(k)
            for exact in (False, True):
                with pmhd_lib.Solver(nx=nx, ny=ny, exact=exact, **common) as s:
                    s.init_problem(pmhd_lib.PROBLEM_ORSZAG_TANG, [0.9 + 0.1 * k])
                    s.advance(max_steps=4)
                    ref = s.get_state()
                _same(got, ref, common, (nx, ny, exact))
                if precision == "fp64":
                    assert pmhd_lib.relative_l2(ref, got)[8] <= 1e-9

"""Which kernel variants the autotuner of a single grid may choose: the shapes every
handle has (32 x 19, of fewer rows here, and 32 x 8) and the grid's default one.
Split shapes, which round differently, are never a matter of timing: binary32
does not run them at all (grids and ensembles stay together), binary64 only where
they are the default."""
import pytest

pytestmark = pytest.mark.gpu


def _height(pmhd_lib, precision, n, autotune):
    with pmhd_lib.Solver(nx=n, ny=n, precision=precision, autotune=autotune) as s:
        s.init_problem(pmhd_lib.PROBLEM_ORSZAG_TANG)
        return s.advance(max_steps=64).tile_height


@pytest.mark.parametrize("n", [100, 110])
def test_tuned_choice_is_not_a_split_shape_unless_it_is_the_default(pmhd_lib, n):
    # Untuned on 148 SMs: tiles of 3 rows in binary32, split 32 x 4 tiles in binary64.
    assert _height(pmhd_lib, "fp32", n, False) == 3
    assert _height(pmhd_lib, "fp32", n, True) in (3, 8)
    assert _height(pmhd_lib, "fp64", n, False) == 4
    assert _height(pmhd_lib, "fp64", n, True) in (4, 3, 8)

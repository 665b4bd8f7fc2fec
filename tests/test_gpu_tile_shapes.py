"""Tile shapes and heights by grid size (kernels.cu default_shape, tile_rows), on
sizes that pick each of them, partial tiles included.  The performance build's
binary64, the only one with split shapes, stays within its parity bar of the
parity build, 1e-12 relative L2 per variable; the parity build, whose tiles have
between 2 and 19 rows here, equals the oracle in every precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [((4, 4), 2), ((95, 97), 2), ((129, 100), 4), ((131, 75), 4), ((193, 161), 8), ((255, 257), None),
         ((321, 320), None)]


@pytest.mark.parametrize("bc", [(0, 0, 0, 0), (0, 0, 1, 1)])
@pytest.mark.parametrize("size,height", SIZES)
def test_small_grid_shapes_match_the_parity_build(pmhd_lib, size, height, bc):
    nx, ny = size
    got = {}
    for exact in (True, False):
        with pmhd_lib.Solver(nx=nx, ny=ny, precision="fp64", exact=exact, bc=bc) as s:
            s.init_problem(pmhd_lib.PROBLEM_ORSZAG_TANG)
            st = s.advance(max_steps=6)
            assert st.steps == 6
            if height and not exact:
                assert st.tile_height == height
            got[exact] = s.get_state()
    rel = pmhd_lib.relative_l2(got[True], got[False])
    tol = np.array([1e-12] * 8 + [1e-9])  # psi starts at zero
    assert np.all(rel <= tol), rel


@pytest.mark.parametrize("size", [(64, 38), (200, 61), (161, 193), (96, 19 * 60)])
@pytest.mark.parametrize("prec,oprec", [("fp64", "f64"), ("fp32", "f32"), ("mixed", "mixed")])
def test_tile_rows_keep_the_parity_builds_bits(pmhd_lib, oracle, size, prec, oprec):
    import oracle_lib

    nx, ny = size
    cfg = oracle_lib.make_config(nx, ny, 1e9, max_steps=3)
    U = oracle_lib.init_ref_problem("f32" if prec == "fp32" else "f64", 0, nx, ny)
    oracle_lib.run(oprec, cfg, U)
    with pmhd_lib.Solver(nx=nx, ny=ny, precision=prec, exact=True) as s:
        s.init_problem(pmhd_lib.PROBLEM_ORSZAG_TANG)
        st = s.advance(max_steps=3)
        assert 2 <= st.tile_height <= 19
        np.testing.assert_array_equal(s.get_state(layout=pmhd_lib.LAYOUT_GHOSTED), U)


def test_autotuner_covers_every_shape(pmhd_lib):
    with pmhd_lib.Solver(nx=64, ny=64, precision="fp64", autotune=True) as s:
        s.init_problem(pmhd_lib.PROBLEM_ORSZAG_TANG)
        st = s.advance(max_steps=64)
        assert st.steps == 64 and st.tile_height in (2, 4, 8, 19)
        tuned = s.get_state()
    with pmhd_lib.Solver(nx=64, ny=64, precision="fp64") as s:
        s.init_problem(pmhd_lib.PROBLEM_ORSZAG_TANG)
        s.advance(max_steps=64)
        assert np.all(pmhd_lib.relative_l2(s.get_state(), tuned)[:8] <= 1e-11)

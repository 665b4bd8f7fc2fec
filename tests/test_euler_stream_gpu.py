"""The streaming 2D Euler step kernel (warps on strips of 28 columns) at the edges
of its strips and row blocks, both sweep orders: the parity build gives the
oracle's bits.  Binary32 streams at every size, binary64 past one wave of 32 x 12
tiles (296 of them), so its shapes here are long and thin."""
import numpy as np
import pytest

import euler_lib as EL

pytestmark = pytest.mark.gpu

SHAPES = [("fp32", s) for s in ((2, 2), (27, 5), (28, 6), (29, 7), (57, 3), (56, 40), (300, 131))]
SHAPES += [("fp64", s) for s in ((28, 3560), (57, 1790), (3000, 40), (29, 3553))]


@pytest.mark.parametrize("solver", ["hllc", "hll"])
@pytest.mark.parametrize("prec,shape", SHAPES)
def test_streaming_step_matches_the_oracle(oracle, pmhd_lib, prec, shape, solver):
    nx, ny = shape
    _, _, ref = EL.riemann2d(nx, 6, solver, prec, ny=ny, max_steps=5)
    with pmhd_lib.Euler2D(nx, ny, config=6, solver=solver, precision=prec, exact=True) as e:
        e.advance(max_steps=2)
        e.advance(max_steps=3)
        np.testing.assert_array_equal(e.prims(), ref)

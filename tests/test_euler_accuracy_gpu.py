"""How far the performance build's binary32 Euler runs are from binary64, against the
parity build's binary32 (the reference's expressions, correctly rounded).

A single run says little: the slip lines of configuration 3 amplify any rounding,
and two equally valid roundings differ by a quarter of their errors either way.  Over
eighteen runs that averages out to a quarter / sqrt(18) = 6 %, so the geometric mean
of the ratios stays below 1.15 unless the arithmetic itself has lost accuracy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _prims(pmhd_lib, n, config, solver, precision, exact):
    with pmhd_lib.Euler2D(n, n, config=config, solver=solver, precision=precision, exact=exact) as e:
        e.advance(1e9, 100)
        return e.prims().astype(np.float64)


def test_binary32_is_as_close_to_binary64_as_the_parity_build(pmhd_lib):
    ratios = []
    for config in (3, 6, 12):
        for solver in ("hllc", "hll"):
            for n in (200, 400, 1024):
                ref = _prims(pmhd_lib, n, config, solver, "fp64", True)
                err = [np.linalg.norm(_prims(pmhd_lib, n, config, solver, "fp32", exact) - ref)
                       for exact in (False, True)]
                ratios.append(err[0] / err[1])
    assert np.exp(np.mean(np.log(ratios))) < 1.15, ratios
